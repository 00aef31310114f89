"""Parity of the op-level CUDA kernels (scores + softmax, depthwise convolution;
forward and backward) with the reference's own compiled CPU drivers, through
the extension-shim -> C ABI -> kernel path.

Tolerances: float64 1e-11 relative (summation order only); float32 1e-5
relative / 1e-6 absolute, scaled by the magnitude of the compared tensor for
gradients that sum hundreds of terms."""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from oracle import oracle as O

from tests.helpers import assert_close, cuda, make_case, seeded

pytestmark = pytest.mark.gpu

CASES = [
    (8, 16, 2 * math.pi / 8, {0: 3, 1: 2, 2: 1}, 2, "hard"),
    (8, 16, 2.5 * math.pi / 8, {0: 2, 1: 2}, 4, "quartic"),
    (6, 12, 2 * math.pi / 6, {1: 3, 3: 2}, 1, "hard"),
    (16, 32, 2 * math.pi / 16, {0: 4, 1: 4, 2: 4}, 2, "hard"),  # 4 x (m = 0, 1, 2) per head, 2 heads, on a half-size grid
    (12, 24, 3 * math.pi / 12, {0: 5, 1: 3}, 3, "quartic"),  # odd offsets, H = 3
]


def magnitude(a) -> float:
    return max(float(np.abs(a).max()), 1.0) if a.size else 1.0


def tolerances(dtype):
    return (1e-11, 1e-12) if dtype == np.float64 else (1e-5, 1e-6)


@pytest.fixture(scope="module")
def ext():
    from gm_attention_b200.nn import fused_attention as fa

    return fa.extension(True)


def reference_or_oracle_softmax(reference_modules, c, q, k, da):
    t = torch.from_numpy
    ref = reference_modules["gm_fused_attention_cpu"]
    alpha = ref.softmax_forward(t(q), t(k), t(c.transport), t(c.bias), t(c.inside), t(c.desc), t(c.row_ptr), t(c.source), c.heads,
                                c.scale, c.max_degree)
    dq, dk = ref.softmax_backward(t(da), t(q), t(k), t(c.transport), t(c.bias), t(c.inside), t(c.desc), t(c.row_ptr), t(c.source),
                                  alpha, c.heads, c.scale, c.max_degree)
    return alpha.numpy(), dq.numpy(), dk.numpy()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("case", CASES)
def test_softmax_forward_backward(ext, reference_modules, case, dtype):
    c = make_case(*case[:5], dtype=dtype, window=case[5])
    q, k = seeded((c.n_nodes, c.width), 11, dtype, 2)
    da, = seeded((c.source.shape[0], c.heads), 12, dtype)
    alpha_ref, dq_ref, dk_ref = reference_or_oracle_softmax(reference_modules, c, q, k, da)
    tables = [cuda(x) for x in (c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source)]
    alpha = ext.softmax_forward(cuda(q), cuda(k), *tables, c.heads, c.scale, c.max_degree)
    rtol, atol = tolerances(dtype)
    assert_close(alpha.cpu().numpy(), alpha_ref, rtol, atol, "alpha")
    dq, dk = ext.softmax_backward(cuda(da), cuda(q), cuda(k), *tables, cuda(alpha_ref), c.heads, c.scale, c.max_degree)
    scale = magnitude(dk_ref)
    assert_close(dq.cpu().numpy(), dq_ref, rtol, atol * scale * 10, "dq")
    assert_close(dk.cpu().numpy(), dk_ref, rtol, atol * scale * 10, "dk")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("case", CASES)
def test_conv_forward_backward(ext, reference_modules, case, dtype):
    nlat, nlon, radius, types, _, window = case
    c = make_case(nlat, nlon, radius, types, 1, dtype=dtype, window=window)
    a0 = types.get(0, 0)
    w = sum(4 * a for n, a in types.items() if n)
    e = c.source.shape[0]
    v, g = seeded((c.n_nodes, c.width), 13, dtype, 2)
    rc, = seeded((e, a0), 14, dtype)
    cc, = seeded((e, w), 15, dtype)
    t = torch.from_numpy
    ref = reference_modules["gm_fused_attention_cpu"]
    args = (t(rc), t(cc), t(c.transport), t(c.angular), t(c.rho), t(c.weights), t(c.desc), t(c.row_ptr), t(c.source), a0, w)
    out_ref = ref.conv_forward(t(v), *args).numpy()
    dv_ref, drc_ref, dcc_ref = (x.numpy() for x in ref.conv_backward(t(g), t(v), *args))
    dev = [cuda(x) for x in (rc, cc, c.transport, c.angular, c.rho, c.weights, c.desc, c.row_ptr, c.source)]
    out = ext.conv_forward(cuda(v), *dev, a0, w)
    rtol, atol = tolerances(dtype)
    assert_close(out.cpu().numpy(), out_ref, rtol, atol * magnitude(out_ref), "conv out")
    dv, drc, dcc = ext.conv_backward(cuda(g), cuda(v), *dev, a0, w)
    assert_close(dv.cpu().numpy(), dv_ref, rtol, atol * magnitude(dv_ref), "dv")
    assert_close(drc.cpu().numpy(), drc_ref, rtol, atol * magnitude(drc_ref), "drc")
    assert_close(dcc.cpu().numpy(), dcc_ref, rtol, atol * magnitude(dcc_ref), "dcc")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("types, heads", [
    ({0: 4, 1: 4}, 1),         # four items a pass: eight groups of lanes take a node's edges in turn
    ({0: 8, 1: 5, 2: 3}, 1),   # eight scalar items, eight complex ones, aligned pairs
    ({0: 3, 1: 9}, 1),         # pairs at odd offsets: read number by number
    ({1: 17, 3: 16}, 1),       # 33 complex items: a pass of 32 and one of one; the third frequency's power
    ({0: 4, 1: 4, 2: 4}, 2),   # scores: two heads of four lanes, four groups
    ({0: 5, 1: 5, 2: 5}, 4),   # five copies in groups of eight lanes
    ({0: 2, 1: 2, 2: 2, 3: 2}, 8),
    ({0: 8, 1: 8}, 4),         # as many copies as lanes
    ({0: 5, 1: 6, 2: 5}, 8),   # a second round of copies, pairs at even offsets
    ({0: 16, 1: 15, 2: 16, 3: 13}, 8),  # four rounds
    ({1: 17, 2: 3}, 2),        # no scalars
    ({1: 3, 0: 5}, 2),         # the scalars behind others (scores)
    ({2: 17, 0: 9, 1: 20}, 2),  # ... and between others: 34 and 40 complex items, 18 scalar ones
    ({3: 2, 2: 1, 0: 3, 1: 4, 4: 1}, 4),  # five rows
])
def test_ops_with_lanes_that_share_edges(ext, types, heads, dtype):
    """Neighbourhoods of 0 to 130 edges -- fewer than the groups, one more than they take at a time, many turns -- against the oracle
    in float64: float64 1e-12 of the largest value, float32 2e-6 (sums of at most 130 terms of O(1) and of 2 x 51 products)."""
    orders = 2 * max(types) + 1
    degrees = np.array([0, 1, 3, 4, 5, 17, 130, 33, 2, 64, 0, 12])
    n, e = len(degrees), int(degrees.sum())
    rng = np.random.default_rng(3)
    row_ptr = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int64)
    source = rng.integers(0, n, e).astype(np.int64)
    phases = np.exp(1j * rng.uniform(0, 6.28, (2, e, 1)) * np.arange(orders))
    transport, angular = (np.stack([x.real, x.imag], -1) for x in phases)
    rho, weights, bias = rng.uniform(0.1, 1.0, e), rng.standard_normal(e), rng.standard_normal(e)
    inside = (rng.random(e) > 0.2).astype(np.uint8)
    inside[row_ptr[:-1][degrees > 0]] = 1
    desc, flat, coef = [], 0, 0
    for f, a in types.items():
        dim = 1 if f == 0 else 2
        desc.append([f, a, flat, coef if f else 0, dim])
        flat += heads * a * dim
        coef += 4 * a if f else 0
    desc = np.array(desc, np.int64)
    cast = lambda *xs: [x.astype(dtype) for x in xs]
    tolerance = 1e-12 if dtype == np.float64 else 2e-6

    def compare(got, want, names):
        for name, a, b in zip(names, got, want):
            assert_close(a.cpu().numpy(), b.astype(dtype), 0.0, tolerance * magnitude(b), name)

    q, k, da = cast(rng.standard_normal((n, flat)), rng.standard_normal((n, flat)), rng.standard_normal((e, heads)))
    transport, angular, rho, weights, bias = cast(transport, angular, rho, weights, bias)
    wide = lambda *xs: [x.astype(np.float64) for x in xs]
    alpha = O.softmax_forward(*wide(q, k, transport, bias), inside, desc, row_ptr, source, heads, 0.3)
    tables = [cuda(x) for x in (transport, bias, inside, desc, row_ptr, source)]
    compare([ext.softmax_forward(cuda(q), cuda(k), *tables, heads, 0.3, 130)], [alpha], ["alpha"])
    want = O.softmax_backward(*wide(da, q, k, transport), desc, row_ptr, source, alpha, heads, 0.3)
    for largest in (130, 1):  # uneven neighbourhoods, and as if all were alike
        compare(ext.softmax_backward(cuda(da), cuda(q), cuda(k), *tables, cuda(alpha.astype(dtype)), heads, 0.3, largest), want, ["dq", "dk"])
    if heads == 1:
        a0 = types.get(0, 0)
        rc, cc = cast(rng.standard_normal((e, a0)), rng.standard_normal((e, coef)))
        edge = [rc, cc, transport, angular, rho, weights]
        dev = [cuda(x) for x in (*edge, desc, row_ptr, source)]
        compare([ext.conv_forward(cuda(q), *dev, a0, coef)], [O.conv_forward(*wide(q, *edge), desc, row_ptr, source, a0, coef)], ["out"])
        want = O.conv_backward(*wide(k, q, *edge), desc, row_ptr, source, a0, coef)
        compare(ext.conv_backward(cuda(k), cuda(q), *dev, a0, coef), want, ["dv", "drc", "dcc"])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n, degree, longest", [
    (12400, 24, 24),   # pairs of dk at once, sources not read ahead
    (12400, 5, 5),     # by numbers, not ahead; forward: no groups of lanes
    (12400, 12, 600),  # uneven: pairs, ahead
    (700, 8, 8),       # few targets: by numbers, ahead (float64: not)
    (700, 24, 24),     # pairs, ahead
])
def test_scores_by_every_kernel(ext, n, degree, longest, dtype):
    """Scores and their gradients where each of the kernels' variants is chosen, against the oracle in float64: to 1e-12 of the
    largest value, in float32 to 2e-6 (a gradient of dk sums about as many terms as a target has edges, up to 600 of dq)."""
    rng = np.random.default_rng(7)
    degrees = np.full(n, degree)
    degrees[:1] = longest
    row_ptr = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int64)
    e, heads = int(row_ptr[-1]), 2
    source = rng.integers(0, n, e).astype(np.int64)
    desc = np.array([[0, 3, 0, 0, 1], [1, 4, 6, 0, 2]], np.int64)
    phase = np.exp(1j * rng.uniform(0, 6.28, (e, 1)) * np.arange(2))
    q, k, da, transport, bias = (x.astype(dtype) for x in (rng.standard_normal((n, 22)), rng.standard_normal((n, 22)), rng.standard_normal((e, heads)),
                                                           np.stack([phase.real, phase.imag], -1), rng.standard_normal(e)))
    inside = np.ones(e, np.uint8)
    wide = lambda *xs: [x.astype(np.float64) for x in xs]
    alpha = O.softmax_forward(*wide(q, k, transport, bias), inside, desc, row_ptr, source, heads, 0.3)
    want = O.softmax_backward(*wide(da, q, k, transport), desc, row_ptr, source, alpha, heads, 0.3)
    tables = [cuda(x) for x in (transport, bias, inside, desc, row_ptr, source)]
    got = [ext.softmax_forward(cuda(q), cuda(k), *tables, heads, 0.3, longest),
           *ext.softmax_backward(cuda(da), cuda(q), cuda(k), *tables, cuda(alpha.astype(dtype)), heads, 0.3, longest)]
    for name, a, b in zip(("alpha", "dq", "dk"), got, (alpha, *want)):
        assert_close(a.cpu().numpy(), b.astype(dtype), 0.0, (1e-12 if dtype == np.float64 else 2e-6) * magnitude(b), name)


def test_softmax_large_neighbourhood_spills_to_global(ext):
    """A row whose logits exceed the shared-memory budget keeps them in alpha."""
    n, deg, heads, d = 3, 30000, 2, 4
    rng = np.random.default_rng(0)
    q = rng.standard_normal((n, d)).astype(np.float32)
    k = rng.standard_normal((n, d)).astype(np.float32)
    source = np.concatenate([rng.integers(0, n, deg), [1], [0, 2]]).astype(np.int64)
    row_ptr = np.array([0, deg, deg + 1, deg + 3], np.int64)
    e = source.shape[0]
    transport = np.tile(np.array([[[1.0, 0.0], [0.6, 0.8]]], np.float32), (e, 1, 1))
    bias = rng.standard_normal(e).astype(np.float32)
    inside = (rng.random(e) > 0.2).astype(np.uint8)
    inside[[0, deg, deg + 1]] = 1
    desc = np.array([[1, 1, 0, 0, 2]], np.int64)
    want = O.softmax_forward(q, k, transport, bias, inside, desc, row_ptr, source, heads, 0.5)
    got = ext.softmax_forward(cuda(q), cuda(k), cuda(transport), cuda(bias), cuda(inside), cuda(desc), cuda(row_ptr), cuda(source),
                              heads, 0.5, deg)
    assert_close(got.cpu().numpy(), want, 2e-5, 1e-7, "alpha (spilled logits)")


def test_float32_masked_edge_never_sets_the_shift(ext):
    """The reference's float32 boundary case (tests/nn/test_fused_attention.py:376-404)."""
    desc = np.array([[0, 1, 0, 0, 1]], np.int64)
    q = np.array([[1.0], [1.0]], np.float32)
    k = np.array([[1.0], [1e4]], np.float32)
    row_ptr = np.array([0, 2, 3], np.int64)
    source = np.array([0, 1, 1], np.int64)
    transport = np.tile(np.array([[[1.0, 0.0]]], np.float32), (3, 1, 1))
    bias = np.array([0.0, np.log(np.finfo(np.float32).tiny), 0.0], np.float32)
    inside = np.array([1, 0, 1], np.uint8)
    alpha = ext.softmax_forward(cuda(q), cuda(k), cuda(transport), cuda(bias), cuda(inside), cuda(desc), cuda(row_ptr), cuda(source),
                                1, 1.0, 2)
    assert alpha.cpu().numpy().reshape(-1).tolist() == [1.0, 0.0, 1.0]


def test_empty_problems_and_isolated_nodes(ext):
    dev = torch.device("cuda")
    desc = torch.tensor([[0, 2, 0, 0, 1]], device=dev)
    z = lambda *s, dt=torch.float32: torch.zeros(*s, dtype=dt, device=dev)
    # no nodes at all
    alpha = ext.softmax_forward(z(0, 2), z(0, 2), z(0, 1, 2), z(0), z(0, dt=torch.uint8), desc, z(1, dt=torch.int64), z(0, dt=torch.int64), 1, 1.0, 1)
    assert alpha.shape == (0, 1)
    # nodes without any edge: conv output is zero, softmax backward gives zero dq
    out = ext.conv_forward(torch.ones(3, 2, device=dev), z(0), z(0), z(0, 1, 2), z(0, 1, 2), z(0), z(0), desc, z(4, dt=torch.int64),
                           z(0, dt=torch.int64), 2, 0)
    assert torch.equal(out, z(3, 2))
    dq, dk = ext.softmax_backward(z(0, 1), torch.ones(3, 2, device=dev), torch.ones(3, 2, device=dev), z(0, 1, 2), z(0),
                                  z(0, dt=torch.uint8), desc, z(4, dt=torch.int64), z(0, dt=torch.int64), z(0, 1), 1, 1.0, 1)
    assert torch.equal(dq, z(3, 2)) and torch.equal(dk, z(3, 2))


def test_contract_errors_match_the_reference_wording(ext):
    dev = torch.device("cuda")
    q = torch.zeros(2, 2, device=dev)
    with pytest.raises(RuntimeError, match="contiguous"):
        ext.softmax_forward(q.t(), q, torch.zeros(1, 1, 2, device=dev), torch.zeros(1, device=dev),
                            torch.zeros(1, dtype=torch.uint8, device=dev), torch.tensor([[0, 2, 0, 0, 1]], device=dev),
                            torch.tensor([0, 1, 1], device=dev), torch.tensor([0], device=dev), 1, 1.0, 1)
    with pytest.raises(RuntimeError, match="at most 8 heads"):
        ext.softmax_forward(q, q, torch.zeros(1, 1, 2, device=dev), torch.zeros(1, device=dev),
                            torch.zeros(1, dtype=torch.uint8, device=dev), torch.tensor([[0, 2, 0, 0, 1]], device=dev),
                            torch.tensor([0, 1, 1], device=dev), torch.tensor([0], device=dev), 9, 1.0, 1)


def test_autograd_functions_run_end_to_end(ext):
    """Softmax.apply / Depthwise.apply with the reference's argument orders."""
    from gm_attention_b200.nn import fused_attention as fa

    c = make_case(8, 16, 2 * math.pi / 8, {0: 3, 1: 2, 2: 1}, 2, dtype=np.float64)
    q, k = (cuda(x).requires_grad_(True) for x in seeded((c.n_nodes, c.width), 21, np.float64, 2))
    tables = [cuda(x) for x in (c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source)]
    alpha = fa.Softmax.apply(q, k, *tables, c.heads, c.scale, c.max_degree)
    weight = cuda(seeded(tuple(alpha.shape), 22, np.float64)[0])
    (alpha * weight).sum().backward()
    dq_ref, dk_ref = O.softmax_backward(weight.cpu().numpy(), q.detach().cpu().numpy(), k.detach().cpu().numpy(), c.transport, c.desc,
                                        c.row_ptr, c.source, alpha.detach().cpu().numpy(), c.heads, c.scale)
    assert_close(q.grad.cpu().numpy(), dq_ref, 1e-10, 1e-11, "dq through autograd")
    assert_close(k.grad.cpu().numpy(), dk_ref, 1e-10, 1e-11, "dk through autograd")


@pytest.mark.parametrize("heads, head", [(1, {0: 5}), (2, {0: 4, 1: 4, 2: 4}), (4, {0: 8, 1: 8, 2: 8, 3: 8}), (8, {0: 4, 1: 4, 2: 4, 3: 4}), (4, {0: 20, 1: 16})])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_one_or_two_warps_per_target(ext, heads, head, dtype):
    """The number of warps that share a target's scores follows the edges per edge of the longest target (a hint to these
    kernels): both give the same bits, so that chunks equal the whole whatever each is given.  The backward's additions to dk,
    by numbers or by pairs, agree to the rounding of sums in another order."""
    c = make_case(24, 40, 3 * math.pi / 24, head, heads, dtype=dtype)
    q, k = (cuda(x) for x in seeded((c.n_nodes, c.width), 23, dtype, 2))
    da = cuda(seeded((c.source.shape[0], heads), 24, dtype)[0])
    tables = [cuda(x) for x in (c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source)]
    n_edges = c.source.shape[0]
    assert 4096 < n_edges <= 4096 * c.max_degree
    two = ext.softmax_forward(q, k, *tables, heads, c.scale, c.max_degree)
    one = ext.softmax_forward(q, k, *tables, heads, c.scale, 1)
    assert torch.equal(one, two) and bool(torch.isfinite(one).all())
    # a third of the nodes' worth of edges more than 24 a node: by pairs; the same edges as those of many more nodes: by numbers
    more = torch.cat([tables[4], tables[4][-1:].expand(n_edges)])
    wide = [torch.cat([x, torch.zeros(n_edges, c.width, dtype=x.dtype, device="cuda")]) for x in (q, k)]
    pairs = ext.softmax_backward(da, q, k, *tables, two, heads, c.scale, c.max_degree)
    numbers = ext.softmax_backward(da, *wide, *tables[:4], more, tables[5], two, heads, c.scale, 1)
    for a, b in zip(pairs, numbers):
        assert float((a - b[:c.n_nodes]).abs().max()) <= (1e-5 if dtype == np.float32 else 1e-13) * float(a.abs().max())


@pytest.mark.parametrize("heads, head", [(1, {0: 5, 1: 3}), (2, {0: 4, 1: 4, 2: 4}), (4, {0: 4, 1: 2, 2: 3, 3: 4}), (8, {0: 2, 1: 2})])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_lane_groups_give_the_same_bits(ext, heads, head, dtype):
    """Groups of lanes that share a target's edges come with seven edges per target and more: the same edges as those of
    targets enough for none give the same scores bit for bit, as a chunk of few edges per target must."""
    c = make_case(12, 24, 3 * math.pi / 12, head, heads, dtype=dtype)
    q, k = (cuda(x) for x in seeded((c.n_nodes, c.width), 29, dtype, 2))
    tables = [cuda(x) for x in (c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source)]
    n_edges = c.source.shape[0]
    assert n_edges >= 7 * c.n_nodes
    more = torch.cat([tables[4], tables[4][-1:].expand(n_edges)])
    wide = [torch.cat([x, torch.zeros(n_edges, c.width, dtype=x.dtype, device="cuda")]) for x in (q, k)]
    shared = ext.softmax_forward(q, k, *tables, heads, c.scale, c.max_degree)
    assert torch.equal(ext.softmax_forward(*wide, *tables[:4], more, tables[5], heads, c.scale, c.max_degree), shared)


def test_chunked_scores_equal_the_whole_edge_set(ext):
    """Exact chunking over contiguous target ranges (reference ``nn/attention.py:344-402``): every chunk holds whole
    neighbourhoods, its constants are views of the parent's, and the softmax stays a partition of unity inside it --
    the op over the chunks, concatenated, equals the op over the whole edge set bit for bit."""
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_attention as fa

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(12, 24, dev)
    cutoff = 2 * math.pi / 12
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=2, dtype=torch.float32)
    heads, attn = 2, FieldType({0: 4, 1: 4, 2: 4})
    owner = type("Layer", (), {})()
    p = fa._plan(owner, attn, attn.scaled(heads), heads)
    desc = fa.descriptors(owner, p, dev)
    q, k = (cuda(x) for x in seeded((lattice.n_nodes, p.width), 21, np.float32, 2))
    scale = 1.0 / math.sqrt(attn.dimension)
    whole = fa.geometry(edges, cutoff, "quartic", torch.float32)
    alpha = ext.softmax_forward(q, k, whole.transport, whole.bias, whole.inside, desc, whole.row_ptr, whole.source, heads, scale, whole.max_degree)
    pieces = []
    for first in range(0, lattice.n_nodes, 37):
        last = min(lattice.n_nodes, first + 37)
        chunk, e_first, e_last = edges.target_range(first, last)
        fa.register_chunk(chunk, edges, e_first, e_last)
        g = fa.geometry(chunk, cutoff, "quartic", torch.float32)
        assert g.base is whole and g.transport.data_ptr() == whole.transport[e_first:e_last].data_ptr()
        part = ext.softmax_forward(q, k, g.transport, g.bias, g.inside, desc, g.row_ptr, g.source, heads, scale, max(g.max_degree, 1))
        sums = torch.zeros(lattice.n_nodes, heads, device=dev).index_add_(0, chunk.target_index, part)
        assert torch.allclose(sums[first:last], torch.ones_like(sums[first:last]), atol=1e-5)
        pieces.append(part)
    assert torch.equal(torch.cat(pieces), alpha)
