"""Parity of the fully fused gauge-attention layer (forward + backward) with
the oracle "reference fused Softmax (CPU) + reference eager transport /
segment-sum", on seeded inputs and on the golden fixtures the reference's
Python produced.

Tolerances: float64 1e-10; float32 1e-5 relative / 1e-6 absolute (absolute
part scaled by the tensor's magnitude for gradients); bf16 storage with fp32
accumulation 2e-2 relative to the tensor's magnitude, against the oracle run
in float32 on the bf16-rounded inputs."""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from oracle import oracle as O

from tests.helpers import assert_close, cuda, make_case, rel_err, seeded

pytestmark = pytest.mark.gpu

CASES = [
    (8, 16, 2 * math.pi / 8, {0: 3, 1: 2, 2: 1}, 2, "hard", 2),
    (8, 16, 2.5 * math.pi / 8, {0: 2, 1: 2}, 4, "quartic", 1),
    (6, 12, 2 * math.pi / 6, {1: 3, 3: 2}, 1, "hard", 3),
    (16, 32, 2 * math.pi / 16, {0: 4, 1: 4, 2: 4}, 2, "hard", 2),
    (12, 24, 3 * math.pi / 12, {0: 16, 1: 16, 2: 16}, 4, "hard", 1),  # the headline head type 16 x (m = 0, 1, 2), H = 4
    (8, 16, 2 * math.pi / 8, {0: 1, 1: 9}, 8, "quartic", 1),
]


def tables_for(c, dtype):
    from gm_attention_b200.attention import AttentionTables

    tdt = np.float64 if dtype == np.float64 else np.float32
    return AttentionTables(cuda(c.transport.astype(tdt)), cuda(c.bias.astype(tdt)), cuda(c.inside), cuda(c.row_ptr), cuda(c.source),
                           tuple(tuple(int(x) for x in row) for row in c.desc), c.heads, c.scale)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("case", CASES)
def test_fused_attention_matches_oracle(case, dtype):
    from gm_attention_b200.attention import attention_backward, attention_forward

    batch = case[6]
    c = make_case(*case[:5], dtype=dtype, window=case[5])
    q, k, v, g = seeded((batch * c.n_nodes, c.width), 31, dtype, 4)
    want = O.attention_forward(q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    dq_w, dk_w, dv_w = O.attention_backward(g, q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    t = tables_for(c, dtype)
    Q, K, V, G = cuda(q), cuda(k), cuda(v), cuda(g)
    out, lse = attention_forward(Q, K, V, t)
    rtol, atol = (1e-10, 1e-11) if dtype == np.float64 else (1e-5, 1e-6)
    assert_close(out.cpu().numpy(), want, rtol, atol * max(1.0, np.abs(want).max()), "out")
    dq, dk, dv = attention_backward(G, Q, K, V, out, lse, t)
    for name, got, ref in (("dq", dq, dq_w), ("dk", dk, dk_w), ("dv", dv, dv_w)):
        assert_close(got.cpu().numpy(), ref, rtol, 10 * atol * max(1.0, np.abs(ref).max()), name)


@pytest.mark.parametrize("case", CASES[:5])
def test_fused_attention_bf16_storage(case):
    from gm_attention_b200.attention import attention_backward, attention_forward

    batch = case[6]
    c = make_case(*case[:5], dtype=np.float32, window=case[5])
    rounded = [torch.from_numpy(x).bfloat16() for x in seeded((batch * c.n_nodes, c.width), 41, np.float32, 4)]
    q, k, v, g = (x.float().numpy() for x in rounded)
    want = O.attention_forward(q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    grads = O.attention_backward(g, q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    t = tables_for(c, np.float32)
    Q, K, V, G = (x.cuda() for x in rounded)
    out, lse = attention_forward(Q, K, V, t)
    assert rel_err(out.float().cpu().numpy(), want) < 2e-2
    got = attention_backward(G, Q, K, V, out, lse, t)
    for name, a, b in zip(("dq", "dk", "dv"), got, grads):
        assert rel_err(a.float().cpu().numpy(), b) < 2e-2, name


@pytest.mark.parametrize("name,rtol,atol", [("f64_hard", 1e-10, 1e-11), ("f32_quartic", 1e-5, 2e-6)])
def test_fused_attention_matches_reference_golden(golden_dir, name, rtol, atol):
    """Inputs and outputs produced by the reference's own Python (fused Softmax + eager value path + autograd)."""
    from gm_attention_b200.attention import AttentionTables, GaugeAttention

    g = np.load(golden_dir / f"attention_{name}.npz")
    t = AttentionTables(cuda(g["transport"]), cuda(g["bias"]), cuda(g["inside"]), cuda(g["row_ptr"]), cuda(g["source"]),
                        tuple(tuple(int(x) for x in row) for row in g["desc"]), int(g["heads"]), float(g["scale"]))
    q, k, v = (cuda(g[x]).requires_grad_(True) for x in ("q", "k", "v"))
    out = GaugeAttention.apply(q, k, v, t)
    assert_close(out.detach().cpu().numpy(), g["out"], rtol, atol, "out")
    (out * cuda(g["dout"])).sum().backward()
    for x, grad in (("dq", q.grad), ("dk", k.grad), ("dv", v.grad)):
        assert_close(grad.cpu().numpy(), g[x], rtol, 10 * atol * max(1.0, np.abs(g[x]).max()), x)


def test_unsupported_head_count_is_a_clear_error():
    from gm_attention_b200.attention import attention_forward

    c = make_case(6, 12, 2 * math.pi / 6, {0: 2}, 3, dtype=np.float32)
    q, = seeded((c.n_nodes, c.width), 1, np.float32)
    with pytest.raises(RuntimeError, match="heads must be 1, 2, 4 or 8"):
        attention_forward(cuda(q), cuda(q), cuda(q), tables_for(c, np.float32))


def test_one_infinite_value_reaches_its_neighbours_only():
    """The reference's edge loop (plain float arithmetic, ``nn/fused/attention.h:295-316`` + the eager value path) lets
    a non-finite value of a node reach exactly the targets that see the node, in that column.  The general (CSR)
    kernels do the same; the oracle on the same field is the witness.  (The lattice kernels, FMA and tensor-core, do
    not: owners that share staged neighbour rows multiply them by zero weights outside their own windows.)"""
    from gm_attention_b200.attention import attention_forward

    c = make_case(12, 24, 3 * math.pi / 12, {0: 4, 1: 4, 2: 4}, 2, dtype=np.float32)
    q, k, v = seeded((c.n_nodes, c.width), 77, np.float32, 3)
    node, column = 5 * c.nlon + 23, 6  # a scalar channel of the second head
    v[node, column] = np.inf
    want = O.attention_forward(q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, 1)
    seen_by = np.unique(c.target[c.source == node])
    assert np.array_equal(np.flatnonzero(~np.isfinite(want).all(1)), seen_by) and np.isfinite(np.delete(want, column, 1)).all()
    out, _ = attention_forward(cuda(q), cuda(k), cuda(v), tables_for(c, np.float32))
    out = out.cpu().numpy()
    assert np.array_equal(np.isfinite(out), np.isfinite(want))
    finite = np.isfinite(want)
    assert_close(out[finite], want[finite], 1e-5, 1e-6 * max(1.0, np.abs(want[finite]).max()), "finite entries")


# (heads, descriptor (n, copies, offset) in the descriptor's order, row length, degree).  Lane groups share a target's edges when
# a head's lanes are at least twice its copies; one scalar frequency with one to three others is the form with its own kernels.
GRAPHS = [
    (1, [(0, 4, 0), (1, 3, 4)], 10, 33),  # eight groups
    (1, [(0, 1, 0), (2, 1, 1)], 3, 40),  # 32 groups, odd rows: pairs of numbers
    (2, [(1, 5, 0), (0, 5, 20)], 30, 9),  # the scalar is not first
    (4, [(0, 8, 0), (1, 7, 32), (2, 8, 88)], 152, 21),  # one group, lanes without a copy
    (8, [(0, 2, 0), (1, 2, 16), (2, 1, 48), (3, 2, 64)], 96, 7),
    (2, [(1, 3, 0), (2, 3, 12), (3, 3, 24), (4, 3, 36), (5, 1, 48)], 52, 18),  # no scalar, five slots
    (1, [(0, 40, 0), (1, 33, 40)], 106, 5),  # two slots each
]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("graph", GRAPHS)
def test_lane_groups_share_edges(graph, dtype):
    """Against the oracle on graphs whose targets have none, one and many edges, some outside the window (with a source that
    no node has) and some of bias minus infinity (which count nothing, also as a target's first or as all that a group has).
    Tolerances as above."""
    from gm_attention_b200.attention import AttentionTables, attention_backward, attention_forward

    heads, rows, width, degree = graph
    n_nodes, batch = 37, 2
    rng = np.random.default_rng(5)
    counts = rng.integers(0, 2 * degree + 1, n_nodes)
    counts[:3] = 0, 1, 2
    row_ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    n_edges, orders = int(row_ptr[-1]), 1 + max(n for n, _, _ in rows)
    desc = np.array([(n, copies, offset, 0, 1 if n == 0 else 2) for n, copies, offset in rows], dtype=np.int64)
    source = rng.integers(0, n_nodes, n_edges)
    angle = rng.uniform(-np.pi, np.pi, (n_edges, 1)) * np.arange(orders)
    transport = np.stack([np.cos(angle), np.sin(angle)], -1).astype(dtype)
    bias = rng.standard_normal(n_edges).astype(dtype)
    silent, inside = rng.random(n_edges) < 0.3, (rng.random(n_edges) < 0.8).astype(np.uint8)
    silent[row_ptr[:-1][counts > 0]] = True  # each target's first
    last = row_ptr[1:][counts > 0] - 1  # (one edge of each counts)
    silent[last], inside[last] = False, 1
    q, k, v, g = seeded((batch * n_nodes, width), 13, dtype, 4)
    keep = (inside & ~silent).astype(np.uint8)  # what the oracle sees
    args = (transport, bias, keep, desc, row_ptr, source, heads, 0.3, batch)
    want = O.attention_forward(q, k, v, *args)
    grads = O.attention_backward(g, q, k, v, *args)
    elsewhere = np.where(inside != 0, source, -(1 << 40))
    bias = np.where(silent, dtype(-np.inf), bias)
    t = AttentionTables(cuda(transport), cuda(bias), cuda(inside), cuda(row_ptr), cuda(elsewhere), tuple(map(tuple, desc.tolist())), heads, 0.3)
    Q, K, V, G = map(cuda, (q, k, v, g))
    out, lse = attention_forward(Q, K, V, t)
    rtol, atol = (1e-10, 1e-11) if dtype == np.float64 else (1e-5, 1e-6)
    assert_close(out.cpu().numpy(), want, rtol, atol * max(1.0, np.abs(want).max()), "out")
    for name, got, ref in zip(("dq", "dk", "dv"), attention_backward(G, Q, K, V, out, lse, t), grads):
        assert_close(got.cpu().numpy(), ref, rtol, 10 * atol * max(1.0, np.abs(ref).max()), name)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("graph", GRAPHS)
def test_targets_whose_edges_all_count_nothing(graph, dtype):
    """A target all of whose edges in the window have bias minus infinity is one without edges: zeros forward, zeros backward, and
    its neighbours' gradients are those of the other targets.  Tolerances as above."""
    from gm_attention_b200.attention import AttentionTables, attention_backward, attention_forward

    heads, rows, width, degree = graph
    n_nodes, batch = 29, 2
    rng = np.random.default_rng(6)
    counts = rng.integers(1, 2 * degree + 1, n_nodes)
    row_ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    n_edges, orders = int(row_ptr[-1]), 1 + max(n for n, _, _ in rows)
    desc = np.array([(n, copies, offset, 0, 1 if n == 0 else 2) for n, copies, offset in rows], dtype=np.int64)
    source = rng.integers(0, n_nodes, n_edges)
    angle = rng.uniform(-np.pi, np.pi, (n_edges, 1)) * np.arange(orders)
    transport = np.stack([np.cos(angle), np.sin(angle)], -1).astype(dtype)
    bias = rng.standard_normal(n_edges).astype(dtype)
    inside = (rng.random(n_edges) < 0.8).astype(np.uint8)
    inside[row_ptr[:-1]] = 1
    silent = np.repeat(np.arange(n_nodes) % 3 == 0, counts)
    q, k, v, g = seeded((batch * n_nodes, width), 17, dtype, 4)
    # what the oracle sees: the other targets' edges
    ptr = np.concatenate([[0], np.cumsum(np.where(np.arange(n_nodes) % 3 == 0, 0, counts))]).astype(np.int64)
    args = (transport[~silent], bias[~silent], inside[~silent], desc, ptr, source[~silent], heads, 0.3, batch)
    want = O.attention_forward(q, k, v, *args)
    grads = O.attention_backward(g, q, k, v, *args)
    bias = np.where(silent, dtype(-np.inf), bias)
    t = AttentionTables(cuda(transport), cuda(bias), cuda(inside), cuda(row_ptr), cuda(source), tuple(map(tuple, desc.tolist())), heads, 0.3)
    Q, K, V, G = map(cuda, (q, k, v, g))
    out, lse = attention_forward(Q, K, V, t)
    dq, dk, dv = attention_backward(G, Q, K, V, out, lse, t)
    nothing = torch.arange(batch * n_nodes, device="cuda") % n_nodes % 3 == 0
    assert not out[nothing].any() and not dq[nothing].any() and bool((lse[nothing] == -np.inf).all())
    rtol, atol = (1e-10, 1e-11) if dtype == np.float64 else (1e-5, 1e-6)
    assert_close(out.cpu().numpy(), want, rtol, atol * max(1.0, np.abs(want).max()), "out")
    for name, got, ref in zip(("dq", "dk", "dv"), (dq, dk, dv), grads):
        assert_close(got.cpu().numpy(), ref, rtol, 10 * atol * max(1.0, np.abs(ref).max()), name)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("graph", GRAPHS)
def test_what_is_not_a_number_reaches_the_neighbours_gradients(graph, dtype):
    """A NaN in a target's q and an infinity in a source's k make their targets' outputs NaN, in their head; the gradients are not
    finite where the oracle's are not: of those targets, and of all that they see."""
    from gm_attention_b200.attention import AttentionTables, attention_backward, attention_forward

    heads, rows, width, degree = graph
    n_nodes, batch = 211, 2
    rng = np.random.default_rng(8)
    counts = rng.integers(1, 6, n_nodes)
    counts[7], counts[60] = 2 * degree, degree
    row_ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    n_edges, orders = int(row_ptr[-1]), 1 + max(n for n, _, _ in rows)
    desc = np.array([(n, copies, offset, 0, 1 if n == 0 else 2) for n, copies, offset in rows], dtype=np.int64)
    source = rng.integers(0, n_nodes, n_edges)
    angle = rng.uniform(-np.pi, np.pi, (n_edges, 1)) * np.arange(orders)
    transport = np.stack([np.cos(angle), np.sin(angle)], -1).astype(dtype)
    bias, inside = rng.standard_normal(n_edges).astype(dtype), np.ones(n_edges, np.uint8)
    q, k, v, g = seeded((batch * n_nodes, width), 19, dtype, 4)
    q[7, rows[0][2]] = np.nan
    k[n_nodes + source[row_ptr[60]], rows[-1][2]] = np.inf
    args = (transport, bias, inside, desc, row_ptr, source, heads, 0.3, batch)
    want = O.attention_forward(q, k, v, *args)
    grads = O.attention_backward(g, q, k, v, *args)
    t = AttentionTables(cuda(transport), cuda(bias), cuda(inside), cuda(row_ptr), cuda(source), tuple(map(tuple, desc.tolist())), heads, 0.3)
    Q, K, V, G = map(cuda, (q, k, v, g))
    out, lse = attention_forward(Q, K, V, t)
    seen = np.arange(n_edges)[row_ptr[7]:row_ptr[8]]
    assert not np.isfinite(grads[2][source[seen]]).all(1).any()
    for name, got, ref in zip(("out", "dq", "dk", "dv"), (out, *attention_backward(G, Q, K, V, out, lse, t)), (want, *grads)):
        assert np.array_equal(np.isfinite(got.cpu().numpy()), np.isfinite(ref)), name
