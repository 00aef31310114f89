"""Factored steerable kernel (forward, aggregate, backward, aggregated backward)
and pair-term kernels against the reference's own compiled CPU drivers, through
the extension shim and the C ABI.  float64 to 1e-10; float32 rtol 1e-4 / atol
1e-5 scaled by magnitude (the reference's own test tolerances,
tests/nn/test_fused_factored.py:126-158, 272-334)."""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from tests.helpers import assert_close, cuda, make_case, rel_err, seeded

pytestmark = pytest.mark.gpu


def blocks_for(type_in: dict[int, int], type_out: dict[int, int]):
    """Readout order of the reference kernel: real (0, 0) first, then for every (n, m) pair linear, then antilinear."""
    blocks, powers = [], {}
    if 0 in type_in and 0 in type_out:
        blocks.append((0, 0, "real"))
    for n in sorted(type_in):
        for m in sorted(type_out):
            if n == 0 and m == 0:
                continue
            blocks.append((n, m, "linear"))
            powers[(n, m, "linear")] = abs(m - n)
            if n >= 1 and m >= 1:
                blocks.append((n, m, "antilinear"))
                powers[(n, m, "antilinear")] = m + n
    return blocks, powers


FACTORED_CASES = [
    ({0: 2, 1: 2}, {0: 2, 1: 3}, 5),
    ({0: 8, 1: 8, 2: 8}, {0: 4, 1: 4, 2: 4}, 17),  # value kernel of the 32 x 64 configuration: 13 blocks, wc 48, wr 4
    ({1: 3}, {0: 2, 2: 2}, 4),                       # no real block
    ({0: 32, 1: 32, 2: 32, 3: 32}, {0: 8, 1: 8, 2: 8, 3: 8}, 17),  # the 128 x 256 layer (32 x (m <= 3) -> 8 x (m <= 3)): packed width 392 > the reference's 320
]


def factored_problem(type_in, type_out, k, dtype, seed):
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.nn import fused_factored as ff

    c = make_case(8, 16, 2 * math.pi / 8, {0: 1}, 1, dtype=dtype, max_frequency=6)
    blocks, powers = blocks_for(type_in, type_out)
    p = ff.plan_blocks(blocks, FieldType(type_out), powers)
    e, n = c.source.shape[0], c.n_nodes
    h, = seeded((e, k - 1), seed, dtype)
    zc, = seeded((n, k, p.wc, 2), seed + 1, dtype)
    zr, = seeded((n, k, p.wr), seed + 2, dtype)
    desc = np.array([b.row() for b in p.blocks], np.int32).reshape(-1, 8)
    return c, p, h, zc, zr, desc


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("case", FACTORED_CASES)
def test_factored_against_reference_driver(reference_modules, case, dtype):
    from gm_attention_b200.nn import fused_factored as ff

    type_in, type_out, k = case
    c, p, h, zc, zr, desc = factored_problem(type_in, type_out, k, dtype, 61)
    too_wide_for_reference = 2 * p.wc + p.wr > 320
    ext = ff.extension(True)
    t = torch.from_numpy
    order, group_ptr, group_source = ff.source_groups(t(c.source))
    dev = [cuda(x) for x in (h, zc, zr, c.angular, c.transport, c.rho, desc, c.source)]
    groups = [x.cuda() for x in (order, group_ptr, group_source)]
    rows = ext.forward(*dev, *groups, p.d_out, p.max_bm)
    weights, = seeded((c.source.shape[0],), 64, dtype)
    out = ext.aggregate(rows, cuda(weights), cuda(c.row_ptr))
    g_rows, = seeded((c.source.shape[0], p.d_out), 65, dtype)
    g_nodes, = seeded((c.n_nodes, p.d_out), 66, dtype)
    dh, dzc, dzr = ext.backward(cuda(g_rows), *dev, *groups)
    agg = ext.backward_aggregated(cuda(g_nodes), cuda(c.target), cuda(weights), rows, *dev, *groups)
    rtol, atol = (1e-10, 1e-11) if dtype == np.float64 else (1e-4, 1e-5)
    if too_wide_for_reference:
        # the reference refuses this width; check the linear-algebra identities instead:
        # aggregate = weighted segment sum of the rows, and <g, rows> = <dh, h> + <dZ, Z> (the map is bilinear in (h~, Z))
        rows_np = rows.cpu().numpy().astype(np.float64)
        want = np.add.reduceat(rows_np * weights[:, None], c.row_ptr[:-1], axis=0)
        assert_close(out.cpu().numpy(), want, 10 * rtol, 10 * atol * max(1.0, np.abs(want).max()), "aggregate")
        lhs = float((g_rows.astype(np.float64) * rows_np).sum())
        zsum = float((dzc.cpu().numpy().astype(np.float64) * zc).sum() + (dzr.cpu().numpy().astype(np.float64) * zr).sum())
        assert abs(zsum - lhs) <= 1e-3 * abs(lhs) + 1e-6  # rows are linear in Z
        # ... and the numpy restatement of the reference arithmetic, which has no width limit
        from oracle import ops_np

        mag = lambda x: max(1.0, float(np.abs(x).max())) if x.size else 1.0
        rows_np2 = ops_np.factored_forward(h, zc, zr, c.angular, c.transport, c.rho, desc, c.source, p.d_out)
        assert_close(rows.cpu().numpy(), rows_np2, 10 * rtol, 10 * atol * mag(rows_np2), "rows vs restatement")
        for name, got, ref_np in zip(("dh", "dzc", "dzr"), (dh, dzc, dzr),
                                     ops_np.factored_backward(g_rows, h, zc, zr, c.angular, c.transport, c.rho, desc, c.source)):
            assert_close(got.cpu().numpy(), ref_np, 10 * rtol, 100 * atol * mag(ref_np), name + " vs restatement")
        return
    ref = reference_modules["gm_factored_cpu"]
    cpu = [t(x) for x in (h, zc, zr, c.angular, c.transport, c.rho, desc, c.source)]
    rows_ref = ref.forward(*cpu, order, group_ptr, group_source, p.d_out, p.max_bm)
    mag = lambda x: max(1.0, float(np.abs(x).max())) if x.size else 1.0
    assert_close(rows.cpu().numpy(), rows_ref.numpy(), rtol, atol * mag(rows_ref.numpy()), "rows")
    out_ref = ref.aggregate(rows_ref, t(weights), t(c.row_ptr))
    assert_close(out.cpu().numpy(), out_ref.numpy(), rtol, 10 * atol * mag(out_ref.numpy()), "aggregate")
    for name, got, want in zip(("dh", "dzc", "dzr"), (dh, dzc, dzr), ref.backward(t(g_rows), *cpu, order, group_ptr, group_source)):
        assert_close(got.cpu().numpy(), want.numpy(), rtol, 10 * atol * mag(want.numpy()), name)
    agg_ref = ref.backward_aggregated(t(g_nodes), t(c.target), t(weights), rows_ref, *cpu, order, group_ptr, group_source)
    for name, got, want in zip(("dh", "dzc", "dzr", "dweights"), agg, agg_ref):
        assert_close(got.cpu().numpy(), want.numpy(), rtol, 100 * atol * mag(want.numpy()), "aggregated " + name)


def test_source_groups_known_answer():
    """The grouping of the reference's tests/nn/test_fused_factored.py:105-123."""
    from gm_attention_b200.nn import fused_factored as ff

    order, ptr, sources = ff.source_groups(torch.tensor([2, 1, 2, 0, 1, 2]))
    assert order.tolist() == [3, 1, 4, 0, 2, 5] and ptr.tolist() == [0, 1, 3, 6] and sources.tolist() == [0, 1, 2]


def test_factored_autograd_functions():
    from gm_attention_b200.nn import fused_factored as ff

    c, p, h, zc, zr, desc = factored_problem({0: 2, 1: 2}, {0: 2, 1: 3}, 5, np.float64, 71)
    order, group_ptr, group_source = (x.cuda() for x in ff.source_groups(torch.from_numpy(c.source)))
    H, ZC, ZR = (cuda(x).requires_grad_(True) for x in (h, zc, zr))
    W = cuda(seeded((c.source.shape[0],), 72, np.float64)[0]).requires_grad_(True)
    tables = [cuda(x) for x in (c.angular, c.transport, c.rho, desc, c.source)]
    out = ff.FactoredAggregate.apply(H, ZC, ZR, W, *tables, cuda(c.target), cuda(c.row_ptr), order, group_ptr, group_source, p.d_out, p.max_bm)
    rows = ff.Factored.apply(H, ZC, ZR, *tables, order, group_ptr, group_source, p.d_out, p.max_bm)
    want = torch.segment_reduce(rows * W[:, None], "sum", offsets=cuda(c.row_ptr))
    assert torch.allclose(out, want, rtol=1e-10, atol=1e-11)
    g = cuda(seeded(tuple(out.shape), 73, np.float64)[0])
    grads_a = torch.autograd.grad((out * g).sum(), (H, ZC, ZR, W), retain_graph=True)
    grads_b = torch.autograd.grad((want * g).sum(), (H, ZC, ZR, W))
    for a, b in zip(grads_a, grads_b):
        assert torch.allclose(a, b, rtol=1e-9, atol=1e-10)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("type_in, type_out, k, degrees", [
    ({0: 1}, {0: 3}, 1, [1, 2]),                                        # no trunk, no complex block
    ({0: 2, 1: 2}, {0: 2, 1: 3}, 2, [64, 65, 0, 63]),                   # tile of 64 edges: exact, one more, one less; a source without edges
    ({1: 3}, {0: 5, 2: 5}, 6, [3, 130]),                                # no scalar block; k - 1 = 5 is no multiple of 4
    ({0: 8, 1: 8, 2: 8}, {0: 4, 1: 4, 2: 4}, 17, [92, 7, 129]),
    ({0: 2, 1: 2, 2: 2}, {0: 8, 1: 8, 2: 8}, 20, [66, 31]),             # 200 packed columns: two dZ patches per thread
    ({0: 2, 1: 2, 2: 2, 3: 2}, {0: 9, 1: 9, 2: 9, 3: 9}, 17, [70, 5]),  # 441 packed columns: smaller tiles in float64
    ({0: 2, 1: 2, 2: 2}, {0: 25, 1: 25, 2: 25}, 11, [33]),              # 625 packed columns: several passes over the edges
])
def test_factored_against_plain_sums(type_in, type_out, k, degrees, dtype):
    """Rows and all gradients against the op's definition written with torch in float64: float64 to 1e-10, float32 to
    2e-6 of each tensor's magnitude (sums of at most 130 edges x 441 columns of O(1) terms)."""
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.nn import fused_factored as ff

    blocks, powers = blocks_for(type_in, type_out)
    p = ff.plan_blocks(blocks, FieldType(type_out), powers)
    n_f, n = 8, len(degrees)
    rng = np.random.default_rng(5)
    source = rng.permutation(np.repeat(np.arange(n), degrees))
    e = source.shape[0]
    h, zc, zr, g = (rng.standard_normal(shape).astype(dtype) for shape in ((e, k - 1), (n, k, p.wc, 2), (n, k, p.wr), (e, p.d_out)))
    phase = np.exp(1j * rng.uniform(0, 6.28, (2, e, 1)) * np.arange(n_f))
    angular, transport = (np.stack([x.real, x.imag], -1).astype(dtype) for x in phase)
    rho = rng.uniform(0.1, 1.0, e).astype(dtype)
    # the definition
    H, ZC, ZR = (torch.from_numpy(x.astype(np.float64)).requires_grad_(True) for x in (h, zc, zr))
    src = torch.from_numpy(source)
    A, T = (torch.view_as_complex(torch.from_numpy(x.astype(np.float64))) for x in (angular, transport))
    hh = torch.cat([torch.ones(e, 1, dtype=torch.float64), H], 1)
    uc, ur = torch.einsum("et,etcx->ecx", hh, ZC[src]), torch.einsum("et,etc->ec", hh, ZR[src])
    order = lambda table, o: table[:, o] if o >= 0 else table[:, -o].conj()
    want = torch.zeros(e, p.d_out, dtype=torch.float64)
    for b in p.blocks:
        if b.kind == 0:
            part = ur[:, b.z_offset:b.z_offset + b.b_m]
        else:
            factor = order(A, b.angular) * order(T, b.transport) * torch.from_numpy(rho.astype(np.float64)) ** b.power
            z = factor[:, None] * torch.view_as_complex(uc[:, b.z_offset:b.z_offset + b.b_m].contiguous())
            part = z.real if b.take_real else torch.view_as_real(z).reshape(e, -1)
        want = want + torch.nn.functional.pad(part, (b.out_offset, p.d_out - b.out_offset - part.shape[1]))
    grads = torch.autograd.grad((want * torch.from_numpy(g.astype(np.float64))).sum(), (H, ZC, ZR), allow_unused=True)
    # the op
    desc = np.array([b.row() for b in p.blocks], np.int32).reshape(-1, 8)
    groups = [x.cuda() for x in ff.source_groups(src)]
    leaves = [cuda(x).requires_grad_(True) for x in (h, zc, zr)]
    rows = ff.Factored.apply(*leaves, *(cuda(x) for x in (angular, transport, rho, desc, source)), *groups, p.d_out, p.max_bm)
    got = torch.autograd.grad(rows, leaves, cuda(g))
    tolerance = 1e-10 if dtype == np.float64 else 2e-6
    for name, a, b in zip(("rows", "dh", "dzc", "dzr"), (rows.detach(), *got), (want.detach(), *grads)):
        if b is None or b.numel() == 0:
            continue
        assert rel_err(a.cpu().numpy(), b.numpy()) < tolerance, name


@pytest.mark.parametrize("scales", [0, 3])
@pytest.mark.parametrize("type_in, type_out, k, degrees", [
    ({0: 8, 1: 8, 2: 8}, {0: 4, 1: 4, 2: 4}, 17, [92, 16, 0, 129, 17, 47]),  # full trunk; steps of 16 edges: exact, one more, one less
    ({0: 2, 1: 2}, {0: 4, 1: 4}, 2, [64, 100]),                            # one trunk output
    ({0: 2, 1: 2}, {0: 3, 1: 9}, 16, [64, 65, 63, 300]),                   # uneven blocks: a round more than their mean asks for; an odd trunk
    ({1: 3}, {0: 5, 2: 5}, 6, [130, 200]),                                 # no scalar block; gradient rows of an odd width
    ({0: 2, 1: 2, 2: 2}, {0: 25, 1: 25, 2: 25}, 11, [90, 33]),             # 91 tiles: three rounds of 32 backward
])
def test_factored_tensor_cores_against_float64(type_in, type_out, k, degrees, scales):
    """Rows, weighted sums' gradients and all others of the float32 kernels, against the float64 kernels (which the tests above pin)
    on the same numbers (rows by the tensor cores from k 10 on, the last graph's gradients too; ``both_factored_kernels`` below has
    edges enough for the others'): sums of at most 300 edges x 19 trunk outputs or 575 columns of O(1)
    terms whose rounding errors of 2^-24 add up like their square root, 2e-6 of each tensor's norm."""
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.nn import fused_factored as ff

    blocks, powers = blocks_for(type_in, type_out)
    p = ff.plan_blocks(blocks, FieldType(type_out), powers)
    n_f, n = 8, len(degrees)
    rng = np.random.default_rng(15)
    source = rng.permutation(np.repeat(np.arange(n), degrees))
    e = source.shape[0]
    phase = np.exp(1j * rng.uniform(0, 6.28, (2, e, n_f)))
    angular, transport = (np.stack([x.real, x.imag], -1) for x in phase)
    rho = rng.uniform(0.1, 1.0, (e, scales) if scales else e)
    desc = np.array([b.row() for b in p.blocks], np.int32).reshape(-1, 8)
    if scales:
        desc[:, 5] %= scales
    values = [x.astype(np.float32) for x in (rng.standard_normal((e, k - 1)), rng.standard_normal((n, k, p.wc, 2)), rng.standard_normal((n, k, p.wr)),
                                             angular, transport, rho)]
    targets = np.sort(rng.integers(0, 5, e))
    g, weights = rng.standard_normal((5, p.d_out)).astype(np.float32), rng.standard_normal(e).astype(np.float32)
    groups = [x.cuda() for x in ff.source_groups(torch.from_numpy(source))]
    ext, results = ff.extension(True), []
    for dtype in (np.float32, np.float64):
        args = (*(cuda(x.astype(dtype)) for x in values), cuda(desc), cuda(source))
        rows = ext.forward(*args, *groups, p.d_out, p.max_bm, bool(scales))
        plain = ext.backward(rows, *args, *groups, bool(scales))
        summed = [] if scales else ext.backward_aggregated(cuda(g.astype(dtype)), cuda(targets), cuda(weights.astype(dtype)), rows, *args, *groups)
        results.append((rows, *plain, *summed))
    for x, (a, b) in enumerate(zip(*results)):
        assert a.shape == b.shape and (b.numel() == 0 or float((a.double() - b).norm() / b.norm()) < 2e-6), x


def both_factored_kernels(type_in, type_out, k, degrees, scales, spoil=lambda **fields: None, dtypes=(np.float32,)):
    """Rows, plain gradients and (no ``scales``) aggregated ones by the kernels that sources of many edges take in float32 and by
    the others, which a grouping with as many empty runs of further nodes as make the mean run short sends the same edges to.
    ``spoil`` may change the numbers before.  Per dtype a pair of dicts of tensors, rows of edges or of the nodes with edges first."""
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.nn import fused_factored as ff

    blocks, powers = blocks_for(type_in, type_out)
    p = ff.plan_blocks(blocks, FieldType(type_out), powers)
    n_f, n, e = 8, len(degrees), sum(degrees)
    more = e // 24 + 1
    rng = np.random.default_rng(15)
    source = rng.permutation(np.repeat(np.arange(n), degrees))
    phase = np.exp(1j * rng.uniform(0, 6.28, (2, e, n_f)))
    desc = np.array([b.row() for b in p.blocks], np.int32).reshape(-1, 8)
    if scales:
        desc[:, 5] %= scales
    fields = dict(h=rng.standard_normal((e, k - 1)), zc=rng.standard_normal((n + more, k, p.wc, 2)), zr=rng.standard_normal((n + more, k, p.wr)),
                  angular=np.stack([phase[0].real, phase[0].imag], -1), transport=np.stack([phase[1].real, phase[1].imag], -1),
                  rho=rng.uniform(0.1, 1.0, (e, scales) if scales else e))
    upstream = dict(g=rng.standard_normal((e, p.d_out)), gt=rng.standard_normal((5, p.d_out)), weights=rng.uniform(0.1, 0.5, e))
    fields, upstream = ({name: x.astype(np.float32) for name, x in d.items()} for d in (fields, upstream))
    targets = np.sort(rng.integers(0, 5, e))
    spoil(source=source, targets=targets, **fields, **upstream)
    order, ptr, nodes = [x.cuda() for x in ff.source_groups(torch.from_numpy(source))]
    long = (order, torch.cat([ptr, ptr[-1:].expand(more)]), torch.cat([nodes, torch.arange(n, n + more, device="cuda")]))
    ext, results = ff.extension(True), []
    for dtype in dtypes:
        args = (*(cuda(x.astype(dtype)) for x in fields.values()), cuda(desc), cuda(source))
        g, gt, weights = (cuda(x.astype(dtype)) for x in upstream.values())
        pair = []
        for groups in ((order, ptr, nodes), long):
            rows = ext.forward(*args, *groups, p.d_out, p.max_bm, bool(scales))
            got = dict(rows=rows, **dict(zip(("dh", "dzc", "dzr"), ext.backward(g, *args, *groups, bool(scales)))))
            if not scales:
                # (the same forward rows for both)
                shared = pair[0]["rows"] if pair else rows
                got |= dict(zip(("dh_t", "dzc_t", "dzr_t", "dw_t"), ext.backward_aggregated(gt, cuda(targets), weights, shared, *args, *groups)))
            pair.append({name: x[: n if "z" in name else e] for name, x in got.items() if x.numel()})
        results.append(pair)
    return results


# (edges enough for the tensor-core kernels of both directions; k 2: the backward's only)
FACTORED_TENSOR_CORES = [
    ({0: 8, 1: 8, 2: 8}, {0: 4, 1: 4, 2: 4}, 17, 70 * [92, 16, 0, 129, 17, 47]),
    ({0: 2, 1: 2}, {0: 4, 1: 4}, 2, 800 * [64, 100]),
    ({0: 2, 1: 2}, {0: 3, 1: 9}, 16, 100 * [64, 65, 63, 300]),  # two rounds of tiles forward
    ({1: 3}, {0: 5, 2: 5}, 12, 200 * [130, 200]),
    ({0: 2, 1: 2, 2: 2}, {0: 25, 1: 25, 2: 25}, 11, [90, 33]),  # three rounds backward
]


@pytest.mark.parametrize("case", FACTORED_TENSOR_CORES)
def test_factored_weights_gradients_are_the_same_sums(case):
    """An edge's ``<g, row>`` has no matrix product in it: the tensor-core kernel adds it up as the other does."""
    (tensor_cores, others), = both_factored_kernels(*case, 0)
    assert torch.equal(tensor_cores["dw_t"], others["dw_t"])


@pytest.mark.parametrize("scales", [0, 3])
@pytest.mark.parametrize("case", FACTORED_TENSOR_CORES)
def test_factored_kernels_agree_on_values_no_bfloat16_holds(case, scales):
    """Infinities, NaN and finite numbers that round to infinity in bfloat16, in every operand: the tensor-core kernels give
    infinities, NaN and finite values where the others give them, and the latter to the rounding of sums in another order: rows
    with values above 1e30 to 1e-5 of the largest (up to 575 terms, of which one is 1e35 times the others), the rest to 2e-6 of their
    norm, as above, those of the sources of 1e24 for themselves.  Products that overflow are among them."""
    big = np.float32(3.4e38)  # (the largest bfloat16 is 3.39e38)

    def spoil(source, targets, h, zc, zr, angular, transport, rho, g, gt, weights):
        # hundredths, so that a product with `big` stays finite
        for x in (h, zc, zr, g, gt):
            x *= np.float32(0.01)
        of = [np.flatnonzero(source == j) for j in range(int(source.max()) + 1)]
        t = h.shape[1] - 1
        h[of[0][3], t], h[of[0][40], 0] = np.inf, big
        zc[1, t + 1, 0, 1], zc[1, 1, -1, 0] = -big, np.inf
        if zr.shape[-1]:
            zr[1, 1, 0] = big
        h[of[1][5], 0], h[of[1][-1], t] = -big, np.nan
        g[of[0][17], -1], g[of[0][18], 0] = -np.inf, big
        gt[1, 0], gt[3, -1], weights[of[0][50]] = -np.inf, np.inf, big  # (no two of `big` in a product: whether that overflows hangs on the order)
        if len(of) > 3:
            zc[3, 0, 0, 0], zc[3, 1, 1, 0] = np.inf, big  # (the constant feature's)
            h[of[3][-1], 0] = -np.inf
        if len(of) > 5:
            # overflowing sums, in the order of the trunk's outputs (rows) and of a source's edges (dZ)
            h[of[4]] *= np.float32(1e26)
            g[of[4]] *= np.float32(1e26)
            h[of[5]] *= np.float32(1e26)
            zc[5] *= np.float32(1e26)
            zr[5] *= np.float32(1e26)

    (tensor_cores, others), = both_factored_kernels(*case, scales, spoil)
    for name, want in others.items():
        got = tensor_cores[name]
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()), name
        assert torch.equal(got[got.isinf()], want[got.isinf()]), name
        a, b = (torch.where(x.isfinite(), x, 0.0).double().reshape(len(x), -1) for x in (got, want))
        largest = b.abs().amax(1, keepdim=True)
        huge = largest > 1e30
        assert bool(((a - b).abs() <= 1e-5 * largest)[huge[:, 0]].all()), name
        for rows in ((largest < 1e10)[:, 0], ((largest >= 1e10) & ~huge)[:, 0]):
            assert float((a - b)[rows].norm()) <= 2e-6 * float(b[rows].norm()), name


@pytest.mark.parametrize("scales", [0, 3])
@pytest.mark.parametrize("k", [2, 9, 10, 11, 17])
def test_factored_tensor_cores_round_no_worse(k, scales):
    """The 2-norms of the errors against the float64 kernels, over 30 000 edges: none larger than the CUDA-core kernels' (rows of a
    short trunk are theirs)."""
    (tensor_cores, others), (want, _) = both_factored_kernels({0: 4, 1: 4}, {0: 8, 1: 8}, k, [150] * 200, scales, dtypes=(np.float32, np.float64))
    for name, x in want.items():
        here, there = (float((y[name].double() - x).norm()) for y in (tensor_cores, others))
        assert here <= there, (name, here / there)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_factored_sources_without_edges(dtype):
    """A grouping that lists every node, most of them with an empty run between two full ones (more runs than the forward
    has CTAs, so that a CTA meets both), gives the rows and gradients of the grouping without them, bit for bit: an empty
    run leaves no copy behind that the next source's could race with, and its node's gradient is zero."""
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.nn import fused_factored as ff

    blocks, powers = blocks_for({0: 2, 1: 2}, {0: 2, 1: 3})
    p = ff.plan_blocks(blocks, FieldType({0: 2, 1: 3}), powers)
    n, k, n_f = 9000, 6, 4
    degrees = np.where(np.arange(n) % 3 == 1, 1 + np.arange(n) % 5, 0)
    rng = np.random.default_rng(9)
    source = rng.permutation(np.repeat(np.arange(n), degrees))
    e = source.shape[0]
    draw = lambda *shape: cuda(rng.standard_normal(shape).astype(dtype))
    h, zc, zr, angular, transport, rho = draw(e, k - 1), draw(n, k, p.wc, 2), draw(n, k, p.wr), draw(e, n_f, 2), draw(e, n_f, 2), draw(e)
    desc, src = cuda(np.array([b.row() for b in p.blocks], np.int32)), cuda(source)
    args = (h, zc, zr, angular, transport, rho, desc, src)
    order, group_ptr, group_source = ff.source_groups(src)
    every_ptr = torch.zeros(n + 1, dtype=torch.long, device=src.device)
    every_ptr[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    every = (order, every_ptr, torch.arange(n, device=src.device))
    assert group_source.shape[0] < n
    ext, g = ff.extension(True), draw(e, p.d_out)
    rows = ext.forward(*args, order, group_ptr, group_source, p.d_out, p.max_bm)
    grads = ext.backward(g, *args, order, group_ptr, group_source)
    assert torch.equal(ext.forward(*args, *every, p.d_out, p.max_bm), rows)
    for got, want in zip(ext.backward(g, *args, *every), grads):
        assert torch.equal(got, want)
    empty = torch.from_numpy(degrees == 0).to(src.device)
    assert bool((grads[1][empty] == 0).all()) and bool((grads[2][empty] == 0).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_factored_backward_without_columns(dtype):
    """Blocks of no columns: dh is zero and dweights = <g, row>, whatever the memory held."""
    from gm_attention_b200.nn import fused_factored as ff

    dev = torch.device("cuda", 0)
    draw = lambda *shape: torch.randn(*shape, dtype=dtype, device=dev)
    n, e, k, d_out = 5, 37, 4, 3
    source, target = torch.arange(e, device=dev) % n, torch.arange(e, device=dev) // 8
    desc = torch.tensor([[1, 0, 0, 1, 1, 1, 0, 0]], dtype=torch.int32, device=dev)
    args = (draw(e, k - 1), draw(n, k, 0, 2), draw(n, k, 0), draw(e, 2, 2), draw(e, 2, 2), draw(e), desc, source)
    g, weights, rows = draw(e, d_out), draw(e), draw(e, d_out)
    del draw
    for _ in range(2):  # the second call's outputs come from memory the first one left non-zero
        scrap = [torch.full((e, k - 1), 7.0, dtype=dtype, device=dev), torch.full((e,), 7.0, dtype=dtype, device=dev)]
        del scrap
        dh, _, _, dweights = ff.extension(True).backward_aggregated(g, target, weights, rows, *args, *ff.source_groups(source))
        assert bool((dh == 0).all())
        torch.testing.assert_close(dweights, (g[target] * rows).sum(1), rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("k, blocks, n_f, backward", [
    (1, 127, 4, False),   # 8 128 packed columns without a trunk
    (2, 63, 4, False),    # 4 032 over a trunk of one
    (4, 32, 4, False),    # 2 048 over a trunk of three: the tiled form holds the float32 one only
    (5, 2, 2000, True),   # phase tables of 2 000 orders, most of them unused
])
def test_factored_sizes_beyond_the_tiled_kernels(k, blocks, n_f, backward, dtype):
    """Rows (and gradients, where the backward's own buffers fit) of sizes whose tiles outgrow shared memory, against the
    numpy restatement: float64 1e-10, float32 1e-5 of each tensor's magnitude (sums of up to 127 blocks x 4 terms)."""
    from gm_attention_b200.nn import fused_factored as ff
    from oracle import ops_np

    rng = np.random.default_rng(11)
    width, n, e = 32, 3, 150
    desc = np.array([[1, width * i, width, (i % 3) + n_f - 4, -(i % 2), i % 4, 0, 0] for i in range(blocks)], np.int32)
    draw = lambda *shape: rng.standard_normal(shape).astype(dtype)
    h, zc, zr, rho, g = draw(e, k - 1), draw(n, k, width * blocks, 2), draw(n, k, 0), rng.uniform(0.1, 1.0, e).astype(dtype), draw(e, 2 * width)
    phase = np.exp(1j * rng.uniform(0, 6.28, (2, e, 1)) * np.arange(n_f))
    angular, transport = (np.stack([x.real, x.imag], -1).astype(dtype) for x in phase)
    source = rng.integers(0, n, e)
    args = (h, zc, zr, angular, transport, rho, desc, source)
    groups = ff.source_groups(cuda(source))
    ext = ff.extension(True)
    bound = 1e-10 if dtype == np.float64 else 1e-5
    wide = [x.astype(np.float64) if x.dtype == np.float32 else x for x in args]
    rows = ext.forward(*map(cuda, args), *groups, 2 * width, width)
    assert rel_err(rows.cpu().numpy(), ops_np.factored_forward(*wide, 2 * width)) < bound
    if backward:
        for got, want in zip(ext.backward(cuda(g), *map(cuda, args), *groups), ops_np.factored_backward(g.astype(np.float64), *wide)):
            assert got.numel() == 0 or rel_err(got.cpu().numpy(), want) < bound


PAIR_CASES = [
    (3, 2, 5, 2 | 8),          # real block: U_REAL | OUT_REAL
    (4, 8, 16, 1 | 2),         # 0 -> m: MATRIX_COMPLEX | U_REAL
    (8, 4, 16, 1 | 4 | 8),     # n -> 0: MATRIX_COMPLEX | CONJ_U | OUT_REAL
    (16, 16, 16, 1),           # linear
    (2, 3, 7, 1 | 4),          # antilinear
]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("case", PAIR_CASES)
def test_pairs_against_reference_driver(reference_modules, case, dtype):
    from gm_attention_b200.nn import fused_pairs as fp

    a, b, trunk, flags = case
    ref = reference_modules["gm_fused_pairs_cpu"]
    ext = fp.extension()
    e = 301
    width = (2 if flags & 1 else 1) * a * b
    cdt = torch.complex64 if dtype == np.float32 else torch.complex128
    rnd = lambda shape, seed: torch.from_numpy(seeded(shape, seed, dtype)[0])
    cx = lambda shape, seed: torch.view_as_complex(rnd((*shape, 2), seed))
    hidden, weight, bias = rnd((e, trunk), 81), rnd((width, trunk), 82), rnd((width,), 83)
    u = rnd((e, a), 84) if flags & 2 else cx((e, a), 84)
    pre = torch.polar(torch.ones(e, dtype=torch.from_numpy(np.zeros(1, dtype)).dtype), rnd((e,), 85))
    post = torch.polar(torch.ones(e, dtype=pre.real.dtype), rnd((e,), 86))
    scale = rnd((e,), 87).abs()
    out0 = rnd((e, b), 88) if flags & 8 else cx((e, b), 88)
    grad_out = rnd((e, b), 89) if flags & 8 else cx((e, b), 89)
    assert pre.dtype == cdt
    out_ref = out0.clone()
    ref.forward(hidden, weight, bias, u, pre, post, scale, out_ref, a, b, flags)
    out = out0.clone().cuda()
    dev = [x.cuda() for x in (hidden, weight, bias, u, pre, post, scale)]
    ext.forward(*dev, out, a, b, flags)
    rtol, atol = (1e-10, 1e-11) if dtype == np.float64 else (1e-4, 1e-5)
    as_np = lambda x: torch.view_as_real(x).cpu().numpy() if x.is_complex() else x.cpu().numpy()
    mag = lambda x: max(1.0, float(np.abs(x).max()))
    assert_close(as_np(out), as_np(out_ref), rtol, atol * mag(as_np(out_ref)), "out")
    gu_ref, gh_ref, gk_ref = torch.ones_like(u), torch.ones_like(hidden), torch.zeros(width, e, dtype=hidden.dtype)
    ref.backward(hidden, weight, bias, u, pre, post, scale, grad_out, gu_ref, gh_ref, gk_ref, a, b, flags)
    gu, gh, gk = torch.ones_like(u).cuda(), torch.ones_like(hidden).cuda(), torch.zeros(width, e, dtype=hidden.dtype).cuda()
    ext.backward(*dev, grad_out.cuda(), gu, gh, gk, a, b, flags)
    for name, got, want in (("grad_u", gu, gu_ref), ("grad_hidden", gh, gh_ref), ("grad_k", gk, gk_ref)):
        assert_close(as_np(got), as_np(want), rtol, 10 * atol * mag(as_np(want)), name)


def test_pairs_plan_order():
    """Term order of the reference planner (tests/nn/test_fused_pairs.py:136-147): m outer, n inner; linear before antilinear."""
    from types import SimpleNamespace

    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.nn import fused_pairs as fp

    tin, tout = FieldType({0: 2, 1: 3}), FieldType({0: 1, 1: 2})
    ranges, powers = {}, {}
    offset = 0
    for n, m in [(0, 1), (1, 0), (1, 1)]:
        width = 2 * tout.multiplicity(m) * tin.multiplicity(n)
        ranges[(n, m, "linear")], powers[(n, m, "linear")] = slice(offset, offset + width), abs(m - n)
        offset += width
        if n and m:
            ranges[(n, m, "antilinear")], powers[(n, m, "antilinear")] = slice(offset, offset + width), m + n
            offset += width
    kernel = SimpleNamespace(field_type_in=tin, field_type_out=tout, _pair_ranges=ranges, _pair_powers=powers)
    terms = fp.plan(kernel)
    assert [(t.n, t.m, t.role) for t in terms] == [(0, 0, "real"), (1, 0, "linear"), (0, 1, "linear"), (1, 1, "linear"), (1, 1, "antilinear")]
    assert [t.flags for t in terms] == [2 | 8, 1 | 4 | 8, 1 | 2, 1, 1 | 4]
    assert [(t.pre_order, t.post_order) for t in terms] == [(None, None), (1, None), (None, 1), (0, None), (2, None)]


# ----------------------------------------------------------------------------- the pair-term driver (_FusedPairs, forward_general)

DRIVER_CASES = [
    ({0: 2, 1: 2, 2: 1}, {0: 1, 1: 2, 2: 2}, True),
    ({0: 2, 1: 2, 2: 1}, {0: 1, 1: 2, 2: 2}, False),
    ({0: 3}, {0: 2}, True),
    ({1: 2, 2: 1}, {1: 1, 2: 2}, True),
    ({0: 2, 1: 1}, {1: 2}, True),
    ({1: 2}, {0: 2}, True),
    ({1: 16}, {1: 16}, True),
    ({0: 5, 1: 7}, {0: 6, 2: 5}, True),  # block sides outside the reference's CPU size list
]


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("field_in, field_out, bias", DRIVER_CASES)
@pytest.mark.parametrize("level", ["node", "edge"])
def test_pairs_driver_matches_the_pair_loop(monkeypatch, level, field_in, field_out, bias, dtype):
    """``forward_general`` against the plain-PyTorch pair loop on the same device, on a node field (the factored form) and
    on the field gathered onto the edges (one launch per term, blocked readout gradient): values and every gradient (input
    field, trunk, both heads), the logic of the reference's ``tests/nn/test_fused_pairs.py:73-93``.  float64 1e-11 / 1e-10;
    float32 1e-5 relative to the tensor's magnitude."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp

    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(6, 12, dev)
    cutoff = 1.4 * math.pi / 6
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=dtype)
    kernel = StandInKernel(field_in, field_out, cutoff, trunk=16, bias=bias, dtype=dtype).to(dev)
    flat0 = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, generator=torch.Generator().manual_seed(5), dtype=dtype).to(dev)

    taken = []
    recognise = fp._factored_inputs
    monkeypatch.setattr(fp, "_factored_inputs", lambda *a: taken.append(recognise(*a)) or taken[-1])

    def run(fused: bool):
        flat = flat0.clone().requires_grad_(True)
        x = FeatureField.from_flat(kernel.field_type_in, flat if level == "node" else flat.index_select(0, edges.source_index))
        out = fp.forward_general(kernel, x, edges).coefficients if fused else kernel.pair_loop(x, edges)
        loss = sum((out[m] * torch.linspace(0.1, 1.0, out[m].numel(), dtype=dtype, device=dev).reshape(out[m].shape)).sum() for m in out)
        return {m: v.detach() for m, v in out.items()}, [g.detach() for g in torch.autograd.grad(loss, [flat, *kernel.parameters()])]

    y_plain, g_plain = run(False)
    y_fused, g_fused = run(True)
    assert [found is not None for found in taken] == [level == "node"]
    tol_y, tol_g = (1e-11, 1e-10) if dtype == torch.float64 else (1e-5, 1e-5)
    for m in y_plain:
        scale = max(1.0, float(y_plain[m].abs().max()))
        assert float((y_fused[m] - y_plain[m]).abs().max()) <= tol_y * scale, m
    for a, b in zip(g_fused, g_plain):
        assert float((a - b).abs().max()) <= tol_g * max(1.0, float(b.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("field_in, field_out, trunk, bias", [
    ({0: 3, 1: 5}, {0: 3, 1: 2, 2: 1}, 5, True),       # odd scalar block before complex ones, a trunk that is no multiple of 4
    ({0: 8, 1: 8, 2: 8}, {0: 4, 1: 4, 2: 4}, 16, True),
    ({0: 16, 1: 16}, {0: 8, 1: 8}, 16, False),
    ({1: 2}, {0: 2}, 1, True),                          # complex readout only
    ({0: 3}, {0: 2}, 16, True),                         # real readout only
])
def test_node_level_field_equals_the_pair_terms(monkeypatch, field_in, field_out, trunk, bias, dtype):
    """The factored form of ``forward_general`` against the pair terms on the same call: outputs (contiguous, as before) and
    every gradient; a node field that is a strided view takes it too, the same field gathered onto the edges takes the pair
    terms.  float64 1e-11; float32 4e-6 of each tensor's magnitude (sums over ~2 000 edges in another order)."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=dtype)
    kernel = StandInKernel(field_in, field_out, cutoff, trunk=trunk, bias=bias, dtype=dtype).to(dev)
    generator = torch.Generator().manual_seed(7)
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, generator=generator, dtype=dtype).to(dev).requires_grad_(True)
    taken = []
    recognise = fp._factored_inputs
    monkeypatch.setattr(fp, "_factored_inputs", lambda *a: taken.append(recognise(*a)) or taken[-1])

    def run(values):
        out = fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, values), edges).coefficients
        assert all(v.is_contiguous() for v in out.values())
        g = torch.Generator().manual_seed(8)
        loss = sum((v * torch.randn(*v.shape, generator=g, dtype=dtype).to(dev)).sum() for v in out.values())
        return [*(v.detach() for v in out.values()), *torch.autograd.grad(loss, [flat, *kernel.parameters()])]

    node = run(flat)
    assert taken[-1] is not None
    strided = run(torch.cat([flat, flat], 1)[:, :flat.shape[1]])
    assert taken[-1] is not None
    edge = run(flat.index_select(0, edges.source_index))
    assert taken[-1] is None
    monkeypatch.setattr(fp, "_factored_inputs", lambda *a: None)
    terms = run(flat)
    bound = 1e-11 if dtype == torch.float64 else 4e-6
    for got in (node, strided, edge):
        for a, b in zip(got, terms):
            assert a.shape == b.shape and rel_err(a.cpu().numpy(), b.cpu().numpy()) < bound


@pytest.mark.parametrize("warm", [False, True])
def test_pair_driver_under_capture(monkeypatch, warm):
    """A graph captures ``forward_general`` on an edge set it has never seen (pair terms: grouping the edges would
    synchronise) and on one an eager call has grouped (factored form); replayed, both give the eager result."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(8, 18, dev)
    cutoff = 1.9 * math.pi / 8
    make = lambda: compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float32)
    seen, fresh = make(), make()
    kernel = StandInKernel({0: 3, 1: 2}, {0: 2, 1: 2}, cutoff, trunk=8, dtype=torch.float32).to(dev)
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev)
    taken = []
    recognise = fp._factored_inputs
    monkeypatch.setattr(fp, "_factored_inputs", lambda *a: taken.append(recognise(*a)) or taken[-1])
    run = lambda edges: fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, flat), edges).coefficients
    with torch.no_grad():
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            want = run(seen)
            run(seen)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = run(seen if warm else fresh)
        assert (taken[-1] is not None) == warm
        graph.replay()
        torch.cuda.synchronize()
    for m in want:
        assert rel_err(out[m].cpu().numpy(), want[m].cpu().numpy()) < 4e-6


def test_node_field_with_too_few_rows_is_refused():
    """A field shorter than the edges' largest source + 1 is an error on the host, from the pair driver and from the
    factored drivers; one row per source is enough, and rows beyond the sources are read by nobody."""
    from types import SimpleNamespace

    from gm_attention_b200.fields import FeatureField, FieldType
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_factored as ff
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float32)
    kernel = StandInKernel({0: 2, 1: 2}, {0: 2, 1: 2}, cutoff, dtype=torch.float32).to(dev)
    flat = torch.randn(lattice.n_nodes + 5, kernel.field_type_in.dimension, device=dev)
    general = lambda n: fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, flat[:n]), edges).coefficients
    want = general(lattice.n_nodes)
    for m, values in general(lattice.n_nodes + 5).items():
        assert torch.equal(values, want[m])
    with pytest.raises(RuntimeError, match="the node field has"):
        general(lattice.n_nodes - 1)
    blocks, powers = blocks_for({0: 2, 1: 2}, {0: 2, 1: 2})
    factored = SimpleNamespace(field_type_out=FieldType({0: 2, 1: 2}), _pair_powers=powers, _blocks=lambda: blocks, radial_basis=SimpleNamespace(cutoff=cutoff),
                               _trunk_hidden=lambda e: torch.ones(e.n_edges, 3, device=dev))
    products = lambda n: {b: torch.ones(n, 4, 2, device=dev, dtype=torch.float32 if b[2] == "real" else torch.complex64) for b in blocks}
    weights = torch.ones(edges.n_edges, device=dev)
    for call in (lambda n: ff.forward(factored, None, edges, products(n)), lambda n: ff.forward_aggregated(factored, None, edges, weights, products(n))):
        assert call(lattice.n_nodes).isfinite().all()
        with pytest.raises(RuntimeError, match="the node field has"):
            call(lattice.n_nodes - 1)


def test_node_level_field_after_the_edges_were_overwritten(monkeypatch):
    """``forward_general`` reads the indices as they are at the call: an ``edge_index`` overwritten in place, and a
    ``source_index`` kept apart from it and replaced, give what the pair terms give for the new sources."""
    from types import SimpleNamespace

    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float64)
    kernel = StandInKernel({0: 2, 1: 2}, {0: 2, 1: 2}, cutoff).to(dev)
    x = FeatureField.from_flat(kernel.field_type_in, torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev, dtype=torch.float64))
    apart = SimpleNamespace(**{name: getattr(edges, name) for name in ("edge_index", "n_edges", "row_ptr", "distances", "angular_phases", "transport_phases",
                                                                       "max_frequency", "angular_harmonic", "transport_harmonic")})
    apart.source_index = edges.source_index.clone()
    for _ in range(2):
        for e in (edges, apart):
            got = fp.forward_general(kernel, x, e).coefficients
            with monkeypatch.context() as patch:
                patch.setattr(fp, "_factored_inputs", lambda *a: None)
                want = fp.forward_general(kernel, x, e).coefficients
            for m in want:
                assert rel_err(got[m].detach().cpu().numpy(), want[m].detach().cpu().numpy()) < 1e-11
        edges.edge_index[1] = edges.edge_index[1].flip(0)
        apart.source_index = apart.source_index.roll(11)


def test_pair_driver_under_capture_beside_a_dead_edge_set(monkeypatch):
    """An entry left by a freed edge set under the key of a new one does not count as that set's grouping: under capture
    the call takes the pair terms, as on any edge set it has not seen, instead of building groups inside the graph."""
    import weakref

    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_factored as ff
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(8, 18, dev)
    cutoff = 1.9 * math.pi / 8
    seen, fresh = (compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float32) for _ in range(2))
    kernel = StandInKernel({0: 3, 1: 2}, {0: 2, 1: 2}, cutoff, trunk=8, dtype=torch.float32).to(dev)
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev)
    run = lambda edges: fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, flat), edges).coefficients
    taken = []
    recognise = fp._factored_inputs
    monkeypatch.setattr(fp, "_factored_inputs", lambda *a: taken.append(recognise(*a)) or taken[-1])
    with torch.no_grad():
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            want = run(seen)
            with monkeypatch.context() as patch:  # the pair terms once, so that the library behind torch's products is set up
                patch.setattr(fp, "_factored_inputs", lambda *a: None)
                run(seen)
        torch.cuda.current_stream().wait_stream(side)
        gone = torch.zeros(3)
        ff._GROUPS[ff._slot(fresh)[0]] = ff._Kept(weakref.ref(gone), ff.grouping_for(seen, seen.source_index), torch.cuda.current_stream())
        del gone
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = run(fresh)
        assert taken[-1] is None
        graph.replay()
        torch.cuda.synchronize()
    for m in want:
        assert rel_err(out[m].cpu().numpy(), want[m].cpu().numpy()) < 4e-6


def test_captured_pair_driver_outlives_the_grouping_cache(monkeypatch):
    """A graph that captured the factored form replays the eager result after other edge sets have filled the cache of
    groupings several times over: the groups it reads by address stay while the edge set lives."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_factored as ff
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(8, 18, dev)
    cutoff = 1.9 * math.pi / 8
    make = lambda: compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float32)
    seen = make()
    kernel = StandInKernel({0: 3, 1: 2}, {0: 2, 1: 2}, cutoff, trunk=8, dtype=torch.float32).to(dev)
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev)
    run = lambda edges: fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, flat), edges).coefficients
    monkeypatch.setattr(ff, "GROUP_CACHE_SIZE", 2)
    with torch.no_grad():
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            want = {m: v.clone() for m, v in run(seen).items()}
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = run(seen)
        entry = ff._GROUPS[ff._slot(seen)[0]]
        assert entry.captured
        others = [make() for _ in range(8)]
        for e in others:
            ff.grouping_for(e, e.source_index)
        assert ff._GROUPS[ff._slot(seen)[0]] is entry and len(ff._GROUPS) <= 3 + sum(kept.captured for kept in ff._GROUPS.values())
        graph.replay()
        torch.cuda.synchronize()
    for m in want:
        assert torch.equal(out[m], want[m])


def test_grouping_shared_between_streams(monkeypatch):
    """Groups built at the end of one stream's queue are complete for a call on another stream, without an order between
    the two; and groups that are dropped while that stream still waits to read them are not handed out again."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_factored as ff
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(16, 40, dev)
    cutoff = 1.9 * math.pi / 16
    edges, same = (compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float32) for _ in range(2))
    kernel = StandInKernel({0: 3, 1: 2}, {0: 2, 1: 2}, cutoff, trunk=8, dtype=torch.float32).to(dev)
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev)
    run = lambda e: fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, flat), e).coefficients
    with torch.no_grad():
        want = run(same)
        torch.cuda.synchronize()
        first, second = torch.cuda.Stream(), torch.cuda.Stream()
        with torch.cuda.stream(first):
            torch.cuda._sleep(100_000_000)
            found = ff.grouping_for(edges, edges.source_index)
        with torch.cuda.stream(second):
            out = run(edges)
            torch.cuda._sleep(100_000_000)
            late = run(edges)
        shapes = [t.shape for t in found.groups]
        del found
        del ff._GROUPS[ff._slot(edges)[0]]
        with torch.cuda.stream(first):  # zeros are harmless groups, and not these
            again = [torch.zeros(s, dtype=torch.long, device=dev) for s in shapes for _ in range(3)]
        torch.cuda.synchronize()
    assert again
    for m in want:
        assert torch.equal(out[m], want[m]) and torch.equal(late[m], want[m])


class _Field:
    """A field of any coefficients, complex ones among them."""

    def __init__(self, field_type, coefficients):
        self.field_type, self.coefficients = field_type, coefficients

    def __getitem__(self, frequency):
        return self.coefficients[frequency]


def test_node_level_field_with_lazy_conjugates(monkeypatch):
    """Complex coefficients and phase tables that are conjugate views, and real ones with a pending sign, give the factored
    form the values the pair terms see.  float64, 1e-11."""
    import dataclasses

    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    plain = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float64)
    lazy = dataclasses.replace(plain, angular_phases=plain.angular_phases.conj(), transport_phases=plain.transport_phases.conj())
    kernel = StandInKernel({0: 2, 1: 3, 2: 1}, {0: 2, 1: 2}, cutoff).to(dev)
    draw = lambda a: torch.randn(lattice.n_nodes, a, dtype=torch.complex128, device=dev, requires_grad=True)
    z0, z1, z2 = draw(2), draw(3), draw(1)
    for edges in (plain, lazy):
        results = []
        for factored in (True, False):
            values = {0: z0.conj().imag, 1: z1.conj(), 2: torch.view_as_real(z2)}
            assert values[0].is_neg() and values[1].is_conj()
            with monkeypatch.context() as patch:
                if not factored:
                    patch.setattr(fp, "_factored_inputs", lambda *a: None)
                out = fp.forward_general(kernel, _Field(kernel.field_type_in, values), edges).coefficients
            loss = sum((v * torch.linspace(-1.0, 1.0, v.numel(), dtype=v.dtype, device=dev).reshape(v.shape)).sum() for v in out.values())
            results.append([*out.values(), *(torch.view_as_real(g.resolve_conj()) for g in torch.autograd.grad(loss, [z0, z1, z2]))])
        for a, b in zip(*results):
            assert rel_err(a.detach().cpu().numpy(), b.detach().cpu().numpy()) < 1e-11


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_node_level_field_uses_the_kernels_radial_table(monkeypatch, dtype):
    """A kernel whose table of radial factors is not the powers of one ratio (column 0 is not 1 either) gets its own
    columns from the factored form, forward and backward, as from the pair terms.  float64 1e-11; float32 4e-6."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=dtype)
    kernel = StandInKernel({0: 2, 1: 3, 2: 1}, {0: 2, 1: 2, 2: 2}, cutoff, dtype=dtype).to(dev)
    columns = torch.randn(edges.n_edges, 5, dtype=dtype, device=dev)
    kernel._radial_powers = lambda distances: columns
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, dtype=dtype, device=dev, requires_grad=True)
    taken, results = [], []
    recognise = fp._factored_inputs
    for factored in (True, False):
        monkeypatch.setattr(fp, "_factored_inputs", lambda *a: taken.append(recognise(*a) if factored else None) or taken[-1])
        out = fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, flat), edges).coefficients
        loss = sum((v * torch.linspace(-1.0, 1.0, v.numel(), dtype=dtype, device=dev).reshape(v.shape)).sum() for v in out.values())
        results.append([*out.values(), *torch.autograd.grad(loss, [flat, *kernel.parameters()])])
    assert taken[0] is not None
    for a, b in zip(*results):
        assert rel_err(a.detach().cpu().numpy(), b.detach().cpu().numpy()) < (1e-11 if dtype == torch.float64 else 4e-6)


def test_node_level_field_on_a_callers_own_types(monkeypatch):
    """An edge set without ``row_ptr`` takes the pair terms; field types that know their frequencies and multiplicities
    only, in any order, take the factored form.  float64, 1e-11 against the pair terms."""
    from types import SimpleNamespace

    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float64)
    names = ("edge_index", "source_index", "n_edges", "distances", "angular_phases", "transport_phases", "max_frequency", "angular_harmonic",
             "transport_harmonic")
    bare = SimpleNamespace(**{name: getattr(edges, name) for name in names})
    kernel = StandInKernel({0: 2, 1: 3}, {0: 2, 1: 1, 2: 2}, cutoff).to(dev)
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev, dtype=torch.float64)
    coefficients = FeatureField.from_flat(kernel.field_type_in, flat).coefficients
    multiplicity = {2: 2, 0: 2, 1: 1}
    kernel.field_type_out = SimpleNamespace(frequencies=tuple(multiplicity), multiplicity=multiplicity.__getitem__)
    taken = []
    recognise = fp._factored_inputs
    monkeypatch.setattr(fp, "_factored_inputs", lambda *a: taken.append(recognise(*a)) or taken[-1])
    with torch.no_grad():
        results = [fp.forward_general(kernel, _Field(kernel.field_type_in, coefficients), e).coefficients for e in (edges, bare)]
    assert [found is not None for found in taken] == [True, False]
    assert list(results[0]) == list(results[1]) == [2, 0, 1]
    for m in multiplicity:
        assert rel_err(results[0][m].cpu().numpy(), results[1][m].cpu().numpy()) < 1e-11


@pytest.mark.parametrize("field_in, field_out, trunk", [({0: 2, 1: 2}, {0: 2, 1: 2}, 17), ({0: 17}, {0: 2}, 8), ({0: 2, 1: 2}, {1: 17}, 8)])
def test_pair_driver_bounds_do_not_depend_on_the_graph(field_in, field_out, trunk):
    """Trunks above 16 and multiplicities above 16 are refused for a node-level field as for the same field on the edges."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float32)
    kernel = StandInKernel(field_in, field_out, cutoff, trunk=trunk, dtype=torch.float32).to(dev)
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev)
    for values in (flat, flat[edges.source_index]):
        with pytest.raises(RuntimeError, match="must be in 1..16"):
            fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, values), edges)


def test_wide_node_field_takes_the_pair_terms():
    """A packed input beyond what the node products stage (2048 columns) is served by the pair terms, bit for bit the
    result on the gathered field."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(6, 14, dev)
    cutoff = 1.9 * math.pi / 6
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=70, dtype=torch.float32)
    kernel = StandInKernel({n: 16 for n in range(67)}, {0: 1}, cutoff, trunk=2, dtype=torch.float32).to(dev)
    assert kernel.field_type_in.dimension > fp.MAX_NODE_WIDTH and edges.n_edges >= 4 * lattice.n_nodes
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev)
    with torch.no_grad():
        node, edge = (fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, v), edges)[0] for v in (flat, flat[edges.source_index]))
    assert torch.equal(node, edge)


def test_node_level_route_only_for_tensors_its_kernels_can_read(monkeypatch):
    """What the route's kernels would read out of range or as other numbers does not take it: readouts with missing rows
    or columns, of another dtype or place, a field of another shape than the input type's, tables of another length,
    32-bit sources.  (Judged on the tensors alone: nothing is launched.)"""
    import dataclasses
    from types import SimpleNamespace

    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float32)
    x = FeatureField.from_flat(StandInKernel({0: 2, 1: 3}, {0: 2, 1: 1}, cutoff).field_type_in, torch.randn(lattice.n_nodes, 8, device=dev)).coefficients

    def takes(values=x, over=edges, spoil=None):
        kernel = StandInKernel({0: 2, 1: 3}, {0: 2, 1: 1}, cutoff, dtype=torch.float32).to(dev)
        if spoil is not None:
            spoil(kernel)
        hidden = fp._trunk_output(kernel, edges.distances)
        return fp._factored_inputs(kernel, values, over, hidden, fp.plan(kernel), kernel._radial_powers(edges.distances)) is not None

    def replace(head, **parts):
        def spoil(kernel):
            old = getattr(kernel, head)
            del kernel._modules[head]
            setattr(kernel, head, SimpleNamespace(weight=parts.get("weight", lambda w: w)(old.weight), bias=parts.get("bias", lambda b: b)(old.bias)))
        return spoil

    assert takes() and takes(spoil=replace("real_head")) and takes(spoil=replace("complex_head", bias=lambda b: None))
    for head in ("real_head", "complex_head"):
        for parts in ({"weight": lambda w: w[:-1]}, {"weight": lambda w: w[:, :-1]}, {"weight": lambda w: w.double()}, {"weight": lambda w: w.cpu()},
                      {"bias": lambda b: b[:-1]}, {"bias": lambda b: b.double()}, {"bias": lambda b: b.cpu()}):
            assert not takes(spoil=replace(head, **parts)), (head, parts)
    for values in ({0: x[0][:, :1], 1: x[1]}, {0: x[0], 1: x[1][:, :2]}, {0: x[0], 1: x[1].flatten(1)}, {0: x[0][:-1], 1: x[1]},
                   {0: torch.complex(x[0], x[0]), 1: x[1]}, {0: x[0].double(), 1: x[1].double()}):
        assert not takes(values=values)
    short = {name: getattr(edges, name)[:-1] for name in ("angular_phases", "transport_phases")}
    assert not takes(over=dataclasses.replace(edges, **short))
    assert not takes(over=dataclasses.replace(edges, edge_index=edges.edge_index.int()))


def test_kernel_saved_after_a_call_and_loaded_elsewhere():
    """A kernel saved after a call, loaded with its tensors on the host and moved back, gives what it gave before, from the
    pair driver and from the factored one: the descriptors it kept are uploaded again."""
    import io

    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_factored as ff
    from gm_attention_b200.nn import fused_pairs as fp
    from tests.helpers import StandInKernel

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(9, 22, dev)
    cutoff = 1.9 * math.pi / 9
    edges = compute_edge_geometry(lattice, lattice.frames, cutoff, max_frequency=4, dtype=torch.float32)
    kernel = StandInKernel({0: 2, 1: 2}, {0: 2, 1: 2}, cutoff, dtype=torch.float32).to(dev)
    flat = torch.randn(lattice.n_nodes, kernel.field_type_in.dimension, device=dev)
    kernel.plan_of_blocks = blocks_for({0: 2, 1: 2}, {0: 2, 1: 2})[0]
    products = {b: torch.randn(lattice.n_nodes, 9, 2, device=dev, dtype=torch.float32 if b[2] == "real" else torch.complex64) for b in kernel.plan_of_blocks}

    def results(kernel):
        kernel._blocks = lambda: kernel.plan_of_blocks
        kernel._trunk_hidden = lambda e: kernel.radial_trunk(kernel.radial_basis(e.distances))
        with torch.no_grad():
            out = fp.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, flat), edges).coefficients
            out = [*out.values(), ff.forward(kernel, None, edges, dict(products))]
        del kernel._blocks, kernel._trunk_hidden
        return out

    want = results(kernel)
    file = io.BytesIO()
    torch.save(kernel, file)
    file.seek(0)
    loaded = torch.load(file, map_location="cpu", weights_only=False).to(dev)
    assert loaded.__dict__["_fused_node_descriptors"][str(dev)][0].device.type == "cpu"
    for a, b in zip(results(loaded), want, strict=True):
        assert torch.equal(a, b)


# (nodes, copies of the input frequencies, of the output ones, k): copies about what a thread holds (16) or sums (8), columns
# about what is staged together (128), nodes about a tile (32)
NODE_PRODUCTS = [
    (1, (1, 1), (1, 2), 2),
    (33, (8, 9), (4, 3), 17),
    (31, (16, 17), (2, 5), 5),
    (70, (33, 3), (40, 31), 6),
    (300, (7, 8, 4), (3, 4, 2), 17),
    (40, (2, 5), (150, 1), 3),
]


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("case", NODE_PRODUCTS)
def test_node_products_against_float64(case, dtype, aligned):
    """``Z_t = M_t x~`` and its gradients against the sums in float64.  A sum of ``n`` products of complex numbers errs by at most
    ``(2 n + 2)`` roundings of the sum of the terms' magnitudes (a float64 result: of twice that, the oracle's own)."""
    from gm_attention_b200.nn.fused_pairs import NodeProducts

    n_nodes, ins, outs, k = case
    offsets = np.concatenate([[0], np.cumsum([a if n == 0 else 2 * a for n, a in enumerate(ins)])])
    rows, counts, widths = [], [0, 0], [0, 0]
    for n, a in enumerate(ins):
        for m, b in enumerate(outs):
            for mode in (0,) if n == 0 else (1, 2) if m else (2,):
                c = int(n > 0 or m > 0)
                rows.append((c, widths[c], b, a, int(offsets[n]), mode, counts[c], 0))
                widths[c] += b
                counts[c] += (2 if c else 1) * a * b
    wr, wc = (w + 3 for w in widths)  # (columns of no block)
    gen = torch.Generator().manual_seed(3)

    def normal(*shape):
        return torch.randn(*shape, generator=gen, dtype=torch.float64).to(dtype).cuda()

    x, cw, cb, rw, rb = normal(n_nodes, int(offsets[-1])), normal(counts[1], k - 1), normal(counts[1]), normal(counts[0], k - 1), normal(counts[0])
    gc, gr = normal(n_nodes, k, wc, 2), normal(n_nodes, k, wr)
    if not aligned:  # the same numbers one element on
        gc = torch.cat([gc.new_zeros(1), gc.reshape(-1)])[1:].view(gc.shape)
    leaves = [t.requires_grad_() for t in (x, cw, cb, rw, rb)]
    zc, zr = NodeProducts.apply(*leaves, torch.tensor(rows, dtype=torch.int32).cuda(), k, wc, wr)
    grads = torch.autograd.grad((zc, zr), leaves, (gc, gr))

    def oracle(sign, x, cw, cb, rw, rb, gc, gr):
        """zc, zr (columns of no block zero) and the gradients, from real parts so that magnitudes can be put through too
        (they add: ``sign`` 1 in place of -1)."""
        cm, rm = torch.cat([cb[:, None], cw], 1), torch.cat([rb[:, None], rw], 1)
        zc, zr = torch.zeros_like(gc), torch.zeros_like(gr)
        dx, dcm, drm = torch.zeros_like(x), torch.zeros_like(cm), torch.zeros_like(rm)
        for c, z0, b, a, x0, mode, row0, _ in rows:
            if mode == 0:
                xr, xi = x[:, x0 : x0 + a], torch.zeros_like(x[:, x0 : x0 + a])
            else:
                xr, xi = x[:, x0 : x0 + 2 * a].view(-1, a, 2).unbind(-1)
                xi = sign * xi if mode == 2 else xi
            if c:
                mr, mi = cm[row0 : row0 + 2 * a * b].view(b, a, 2, k).unbind(2)
                g_r, g_i = gc[:, :, z0 : z0 + b].unbind(-1)
            else:
                mr = rm[row0 : row0 + a * b].view(b, a, k)
                mi, g_r = torch.zeros_like(mr), gr[:, :, z0 : z0 + b]
                g_i = torch.zeros_like(g_r)
            product = lambda m, y: torch.einsum("bak,na->nkb", m, y)
            z_r, z_i = product(mr, xr) + sign * product(mi, xi), product(mr, xi) + product(mi, xr)
            back = lambda m, g: torch.einsum("bak,nkb->na", m, g)
            d_r, d_i = back(mr, g_r) + back(mi, g_i), back(mr, g_i) + sign * back(mi, g_r)
            outer = lambda g, y: torch.einsum("nkb,na->bak", g, y)
            w_r, w_i = outer(g_r, xr) + outer(g_i, xi), outer(g_i, xr) + sign * outer(g_r, xi)
            if c:
                zc[:, :, z0 : z0 + b] = torch.stack([z_r, z_i], -1)
                dcm[row0 : row0 + 2 * a * b] = torch.stack([w_r, w_i], 2).reshape(2 * a * b, k)
            else:
                zr[:, :, z0 : z0 + b] = z_r
                drm[row0 : row0 + a * b] = w_r.reshape(a * b, k)
            if mode == 0:
                dx[:, x0 : x0 + a] += d_r
            else:
                dx[:, x0 : x0 + 2 * a] += torch.stack([d_r, sign * d_i if mode == 2 else d_i], -1).reshape(n_nodes, 2 * a)
        return zc, zr, dx, dcm[:, 1:], dcm[:, 0], drm[:, 1:], drm[:, 0]

    inputs = [t.detach().double().cpu() for t in (*leaves, gc, gr)]
    want, size = oracle(-1.0, *inputs), oracle(1.0, *(t.abs() for t in inputs))
    columns = [torch.zeros(w, dtype=torch.bool) for w in (wr, wc)]
    for c, z0, b, *_ in rows:
        columns[c][z0 : z0 + b] = True
    zc, zr = torch.where(columns[1][:, None], zc.detach().cpu(), 0.0), torch.where(columns[0], zr.detach().cpu(), 0.0)
    terms = (max(ins), max(ins), k * sum(outs) * 2, n_nodes, n_nodes, n_nodes, n_nodes)
    unit = torch.finfo(dtype).eps / 2 * (2 if dtype == torch.float64 else 1)
    for name, got, ref, scale, n in zip(("zc", "zr", "dx", "dcw", "dcb", "drw", "drb"), (zc, zr, *grads), want, size, terms):
        excess = (got.cpu().double() - ref).abs() - (2 * n + 2) * unit * scale
        assert got.shape == ref.shape and excess.max() <= 0, (name, float(excess.max()))


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("d_out", [1, 2, 5, 20, 33, 64, 127, 128])
def test_aggregate_widths(d_out, dtype, offset):
    """A target's weighted sum of its rows (0 to 300 of them) against float64: a sum of ``n`` products errs by at most ``n + 1``
    roundings of the sum of their magnitudes.  ``offset`` 1: rows that do not start on a 16-byte boundary."""
    from gm_attention_b200.nn import fused_factored as ff

    degrees = torch.tensor([0, 1, 300, 2, 7, 33, 0, 64, 15, 128])
    row_ptr = torch.cat([torch.zeros(1, dtype=torch.int64), degrees.cumsum(0)])
    n_edges = int(row_ptr[-1])
    gen = torch.Generator().manual_seed(d_out)
    rows = torch.randn(n_edges * d_out + offset, generator=gen, dtype=torch.float64).to(dtype).cuda()[offset:].view(n_edges, d_out)
    weights = torch.randn(n_edges, generator=gen, dtype=torch.float64).to(dtype).cuda()
    got = ff.extension(True).aggregate(rows, weights, row_ptr.cuda()).cpu().double()
    terms = weights.cpu().double()[:, None] * rows.cpu().double()
    target = torch.repeat_interleave(torch.arange(len(degrees)), degrees)
    want = torch.zeros(len(degrees), d_out, dtype=torch.float64).index_add(0, target, terms)
    size = torch.zeros_like(want).index_add(0, target, terms.abs())
    assert ((got - want).abs() <= (degrees[:, None] + 1) * torch.finfo(dtype).eps * size).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("d_out", [1, 8, 20, 33, 50])
def test_aggregate_many_targets_of_few_edges(d_out, dtype):
    """12 300 targets of 0 to 12 edges, by columns where vectors would cost more; the bound of ``test_aggregate_widths``."""
    from gm_attention_b200.nn import fused_factored as ff

    gen = torch.Generator().manual_seed(d_out)
    degrees = torch.randint(0, 13, (12300,), generator=gen)
    row_ptr = torch.cat([torch.zeros(1, dtype=torch.int64), degrees.cumsum(0)])
    n_edges = int(row_ptr[-1])
    rows, weights = (torch.randn(*shape, generator=gen, dtype=torch.float64).to(dtype) for shape in ((n_edges, d_out), (n_edges,)))
    got = ff.extension(True).aggregate(rows.cuda(), weights.cuda(), row_ptr.cuda()).cpu().double()
    terms = weights.double()[:, None] * rows.double()
    target = torch.repeat_interleave(torch.arange(len(degrees)), degrees)
    want = torch.zeros(len(degrees), d_out, dtype=torch.float64).index_add(0, target, terms)
    size = torch.zeros_like(want).index_add(0, target, terms.abs())
    assert ((got - want).abs() <= (degrees[:, None] + 1) * torch.finfo(dtype).eps * size).all()
