"""The lattice depthwise convolution (coefficient table per (row pair, offset) instead of a per-edge stream) against the
reference's depthwise op (``nn/fused/attention.h:174-232, 265-287``, restated in ``oracle/gm_oracle.c`` and pinned to the
reference's compiled driver) fed with the SAME coefficients expanded to every edge.

* whole problem on small lattices, float32 and bf16 storage, batches 1 / 3 / 4 (every samples-per-CTA variant), plain and
  normalised aggregation weights: output, field gradient, and the coefficient gradient summed over the edges of an entry;
* 256 x 512, radius 4 pi / 256, batch 4, 64 x (m = 0, 1, 2) (a_0 = 64, W = 512, 22 999 040 edges per sample): sampled
  targets and sources (complete rows, exact), the coefficient gradient of one complete lattice row, and -- on the whole
  problem -- the adjoint identities  <g, y> = <table, dtable> = <dv, v>  that hold because y is bilinear in (table, v).

Tolerances: float32 1e-5 relative with an absolute part of 1e-5 of the tensor's largest magnitude for sums of hundreds
to thousands of terms; bf16 storage 2e-2 of the largest magnitude against the oracle in float32 on the rounded inputs.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from oracle import geometry_np as G
from oracle import oracle as O
from oracle import sampled as S

from tests.helpers import assert_close, cuda, descriptor_rows, make_case, rel_err, seeded

pytestmark = pytest.mark.gpu


def magnitude(a) -> float:
    return max(float(np.abs(a).max()), 1.0)


def entry_of(tables, target: np.ndarray, source: np.ndarray) -> np.ndarray:
    """Table entry of every edge (target <- source), from the windows alone."""
    lat = tables.lattice
    span = 2 * lat.halo + 1
    cnt, lo, off = (x.cpu().numpy().reshape(-1) for x in (lat.win_cnt, lat.win_lo, lat.win_off))
    ri, li, rj, lj = target // lat.nlon, target % lat.nlon, source // lat.nlon, source % lat.nlon
    w = ri * span + (rj - ri + lat.halo)
    d = (lj - li - lo[w]) % lat.nlon
    assert (d < cnt[w]).all()
    return off[w] + d


def package_tables(c, head_type, normalize: bool):
    from gm_attention_b200.nn.lattice_depthwise import conv_tables

    weights = c.weights
    if normalize:
        mass = np.add.reduceat(c.weights, c.row_ptr[:-1])
        weights = (c.weights / np.repeat(np.maximum(mass, 1e-12), np.diff(c.row_ptr))).astype(c.weights.dtype)
    geometry = SimpleNamespace(transport=cuda(c.transport.astype(np.float32)), angular=cuda(c.angular.astype(np.float32)),
                               rho=cuda(c.rho.astype(np.float32)), bias=cuda(c.bias.astype(np.float32)), inside=cuda(c.inside),
                               row_ptr=cuda(c.row_ptr), source=cuda(c.source))
    rows = descriptor_rows(c.head_type, 1)
    return conv_tables(geometry, cuda((c.rho * c.radius).astype(np.float32)), cuda(weights.astype(np.float32)), rows, c.nlat, c.nlon), weights


@pytest.mark.parametrize("batch,storage,normalize", [(1, "f32", False), (3, "f32", True), (4, "f32", False), (3, "bf16", False), (4, "bf16", True)])
def test_whole_problem(batch, storage, normalize):
    from gm_attention_b200.nn.lattice_depthwise import lattice_depthwise

    head = {0: 4, 1: 3, 2: 2}
    c = make_case(16, 32, 3 * math.pi / 16, head, 1, dtype=np.float32)
    a0, w = 4, 4 * 3 + 4 * 2
    tables, weights = package_tables(c, head, normalize)
    n_entries = tables.n_entries
    rc_t, = seeded((n_entries, a0), 31, np.float32)
    cc_t, = seeded((n_entries, w), 32, np.float32)
    fields = seeded((batch * c.n_nodes, c.width), 33, np.float32, 2)
    bf16 = storage == "bf16"
    if bf16:
        dev = [torch.from_numpy(x).bfloat16().cuda() for x in fields]
        fields = [x.float().cpu().numpy() for x in dev]
    else:
        dev = [cuda(x) for x in fields]
    v, g = fields
    entry = entry_of(tables, c.target, c.source)
    rc, cc = rc_t[entry], cc_t[entry]
    args = (rc[None], cc[None], c.transport, c.angular, c.rho, weights, c.desc, c.row_ptr, c.source, a0, w)
    want_out, want_dv = np.zeros_like(v), np.zeros_like(v)
    want_drc, want_dcc = np.zeros_like(rc_t), np.zeros_like(cc_t)
    for b in range(batch):
        rows = slice(b * c.n_nodes, (b + 1) * c.n_nodes)
        want_out[rows] = O.conv_forward(v[rows], *args)
        dv, drc, dcc = O.conv_backward(g[rows], v[rows], *args)
        want_dv[rows] = dv
        np.add.at(want_drc, entry, drc.reshape(-1, a0))
        np.add.at(want_dcc, entry, dcc.reshape(-1, w))
    V = dev[0].requires_grad_(True)
    RC, CC = cuda(rc_t).requires_grad_(True), cuda(cc_t).requires_grad_(True)
    out = lattice_depthwise(V, RC, CC, tables)
    out.backward(dev[1])
    got = {"out": out.detach(), "dv": V.grad, "drc": RC.grad, "dcc": CC.grad}
    want = {"out": want_out, "dv": want_dv, "drc": want_drc, "dcc": want_dcc}
    for name in want:
        a = got[name].float().cpu().numpy()
        if bf16:
            assert rel_err(a, want[name]) < 2e-2, name
        else:
            assert_close(a, want[name], 1e-5, 1e-5 * magnitude(want[name]), name)


def test_only_true_neighbours_are_touched():
    """One Inf in the field reaches exactly the targets that see that node, as in the reference's edge loop."""
    from gm_attention_b200.nn.lattice_depthwise import fold, _apply

    head = {0: 4, 1: 3, 2: 2}
    c = make_case(16, 32, 3 * math.pi / 16, head, 1, dtype=np.float32)
    tables, _ = package_tables(c, head, False)
    rc_t, = seeded((tables.n_entries, 4), 41, np.float32)
    cc_t, = seeded((tables.n_entries, 20), 42, np.float32)
    v, = seeded((c.n_nodes, c.width), 43, np.float32)
    node = 5 * c.nlon + 31
    v[node, 5] = np.inf  # the imaginary part of the first m = 1 copy
    out = _apply(cuda(v), fold(cuda(rc_t), cuda(cc_t), tables), tables, False).cpu().numpy()
    seen_by = np.unique(c.target[c.source == node])
    bad = np.flatnonzero(~np.isfinite(out).all(1))
    assert np.array_equal(bad, seen_by)
    assert np.isfinite(out[:, :4]).all() and np.isfinite(out[:, 10:]).all()  # other channels stay finite everywhere


# ----------------------------------------------------------------------------- 256 x 512, radius 4 pi / 256, batch 4

@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("nlat, nlon, reach, head, batch", [
    (6, 8, 1.5, {0: 2, 1: 1}, 1),                    # one tile; windows of whole rows; stages longer than the row
    (6, 24, 2.0, {0: 10, 1: 10}, 3),                 # node rows of 60 / 120 bytes: 4-byte copies; an odd batch
    (5, 144, 1.6, {0: 6, 1: 5, 2: 5}, 2),            # tiles beyond the last longitude, windows of several stages
    (4, 32, 1.2, {0: 64, 1: 64, 2: 64}, 2),          # 160 items: two tiles fill 320 threads
    (4, 16, 1.2, {0: 130, 1: 130, 2: 130}, 1),       # 325 items: more than a CTA has threads, the kernel without stages
])
def test_apply_against_the_host_loops(nlat, nlon, reach, head, batch, storage):
    """Both forms of the apply kernel, forward and transposed, against numpy loops in float64 on the same (rounded) field:
    at most ~300 products per output, 1e-5 of the largest in float32; one rounding to bf16 (2^-9) on top in bf16."""
    from types import SimpleNamespace

    from gm_attention_b200.nn.lattice_depthwise import _apply, conv_tables
    from tests.test_lattice_depthwise_cpu import _apply_on_the_host

    c = make_case(nlat, nlon, reach * math.pi / nlat, head, 1, dtype=np.float32)
    geometry = SimpleNamespace(transport=cuda(c.transport), angular=cuda(c.angular), rho=cuda(c.rho), bias=cuda(c.bias), inside=cuda(c.inside),
                               row_ptr=cuda(c.row_ptr), source=cuda(c.source))
    t = conv_tables(geometry, cuda(c.rho * np.float32(c.radius)), cuda(c.weights), descriptor_rows(c.head_type, 1), nlat, nlon)
    lat = t.lattice
    table, = seeded((t.n_entries, t.table_width), 61, np.float32)
    x = torch.from_numpy(seeded((batch * c.n_nodes, c.width), 62, np.float32)[0]).to(torch.bfloat16 if storage == "bf16" else torch.float32)
    items = t.items.cpu().numpy().tolist()
    sample = slice((batch - 1) * c.n_nodes, batch * c.n_nodes)
    for transposed in (False, True):
        windows = (lat.t_win_cnt, lat.t_win_lo, lat.t_win_off) if transposed else (lat.win_cnt, lat.win_lo, lat.win_off)
        used = table[lat.t_entry.cpu().numpy()] if transposed else table
        want = _apply_on_the_host(x[sample].double().numpy(), used.astype(np.float64), *(w.cpu().numpy() for w in windows), items, nlat, nlon, lat.halo,
                                  transposed)
        got = _apply(x.cuda(), cuda(used), t, transposed)[sample].float().cpu().numpy()
        atol = 1e-5 * np.abs(want).max()
        assert_close(got, want, 2.0 ** -8 if storage == "bf16" else 1e-5, atol, "transposed" if transposed else "forward")


# bfloat16 rows of a multiple of 16 bytes: tensor cores.  One tile of 8 longitudes; column blocks of 32 partly filled; more
# than 64 tiles (two CTAs along a row, chunks of 32 tiles with a remainder); windows of one to several stages
TENSOR_CORE_CASES = [
    (5, 8, 1.5, {0: 2, 1: 1, 2: 2}, 1),
    (6, 24, 2.0, {0: 8, 1: 8}, 3),
    (4, 560, 1.3, {0: 8, 1: 8, 2: 8}, 2),
    (12, 136, 3.0, {0: 4, 1: 14}, 1),
    (4, 24, 1.4, {0: 8}, 15),                        # 14 samples of 3 tiles share a CTA, one is left; one half of a block of 16 columns
    (3, 256, 1.2, {0: 8, 1: 8, 2: 8}, 3),            # two samples of 32 tiles fill a CTA, one is left
    (2, 512, 1.1, {0: 2, 1: 3}, 1),                  # 64 tiles; a window of 519 positions: four groups of 24 offsets and fewer
    (3, 520, 1.1, {1: 20}, 2),                       # 65 tiles: blocks of 33 and 32
]


def tensor_core_case(nlat, nlon, reach, head):
    from types import SimpleNamespace

    from gm_attention_b200.nn.lattice_depthwise import conv_tables

    c = make_case(nlat, nlon, reach * math.pi / nlat, head, 1, dtype=np.float32)
    geometry = SimpleNamespace(transport=cuda(c.transport), angular=cuda(c.angular), rho=cuda(c.rho), bias=cuda(c.bias), inside=cuda(c.inside),
                               row_ptr=cuda(c.row_ptr), source=cuda(c.source))
    return c, conv_tables(geometry, cuda(c.rho * np.float32(c.radius)), cuda(c.weights), descriptor_rows(c.head_type, 1), nlat, nlon)


@pytest.mark.parametrize("nlat, nlon, reach, head, batch", TENSOR_CORE_CASES)
def test_tensor_core_kernels_against_the_host_loops(nlat, nlon, reach, head, batch):
    """apply (one rounding to bf16, 2^-9, and 1e-5 of the largest for the float32 sums), transposed and not, and the table
    gradient (float32 sums over nlon x batch products of bf16 values: 1e-5 of the largest) against float64, whatever order
    the blocks come in."""
    import dataclasses

    from gm_attention_b200.nn.lattice_depthwise import _apply, _table_gradient
    from tests.test_lattice_depthwise_cpu import _apply_on_the_host

    c, t = tensor_core_case(nlat, nlon, reach, head)
    lat = t.lattice
    assert c.width % 8 == 0
    table, = seeded((t.n_entries, t.table_width), 71, np.float32)
    x, g = (torch.from_numpy(v).bfloat16() for v in seeded((batch * c.n_nodes, c.width), 72, np.float32, 2))
    items = t.items.cpu().numpy().tolist()
    sample = slice((batch - 1) * c.n_nodes, batch * c.n_nodes)
    for transposed in (False, True):
        windows = (lat.t_win_cnt, lat.t_win_lo, lat.t_win_off) if transposed else (lat.win_cnt, lat.win_lo, lat.win_off)
        used = table[lat.t_entry.cpu().numpy()] if transposed else table
        want = _apply_on_the_host(x[sample].double().numpy(), used.astype(np.float64), *(w.cpu().numpy() for w in windows), items, nlat, nlon, lat.halo,
                                  transposed)
        got = _apply(x.cuda(), cuda(used), t, transposed, tensor_cores=True)[sample].float().cpu().numpy()
        assert_close(got, want, 2.0 ** -8, 1e-5 * np.abs(want).max(), "transposed" if transposed else "forward")
    cnt, lo, off = (w.cpu().numpy() for w in (lat.win_cnt, lat.win_lo, lat.win_off))
    X, G = (v.double().numpy().reshape(batch, nlat, nlon, c.width) for v in (x, g))
    want = np.zeros((t.n_entries, t.table_width))
    for i in range(nlat):
        for w in range(2 * lat.halo + 1):
            for d in range(int(cnt[i, w])):
                xs = np.roll(X[:, i + w - lat.halo], -(int(lo[i, w]) + d), axis=1)
                for kind, col, fcol in items:
                    m = np.einsum("bla,blc->ac", G[:, i, :, col:col + 2], xs[:, :, col:col + 2])
                    want[off[i, w] + d, fcol:fcol + (4 if kind == 0 else 2)] = m.reshape(-1) if kind == 0 else (m[0, 0], m[1, 1])
    order = torch.randperm(t.blocks.shape[0], generator=torch.Generator().manual_seed(5))
    for blocks in (t.blocks, t.blocks[order.to(t.blocks.device)].contiguous()):
        got = _table_gradient(g.cuda(), x.cuda(), dataclasses.replace(t, blocks=blocks), tensor_cores=True)
        assert_close(got.cpu().numpy(), want, 1e-5, 1e-5 * np.abs(want).max(), "table gradient")


@pytest.mark.parametrize("head", [{0: 8, 1: 12, 2: 8}, {0: 16, 1: 40, 2: 40}])
def test_tensor_core_kernels_with_several_blocks_of_columns_per_cta(head):
    """Launches of so many CTAs that apply gives one CTA up to 2 of 3 or 5 of 11 blocks of 16 columns, table_grad 5 of 6 blocks of 32,
    the last of each fewer, against the FMA kernels (which take a field on an 8-byte boundary): apply to two roundings to bf16 (2^-8 each)
    and 1e-5 of the largest, the table gradient to 1e-5 of the largest.  Infinities and NaN in the first, a middle and the last block of
    several samples and rows reach the same outputs as there."""
    from gm_attention_b200.nn.lattice_depthwise import _apply, _table_gradient

    batch = 32
    c, t = tensor_core_case(24, 520, 1.1, head)
    gen = torch.Generator(device="cuda").manual_seed(75)
    x, g = (torch.randn(batch * c.n_nodes, c.width, generator=gen, device="cuda").bfloat16() for _ in range(2))
    table = torch.randn(t.n_entries, t.table_width, generator=gen, device="cuda")
    shifted = torch.empty(x.numel() + 4, dtype=x.dtype, device="cuda")[4:].view(x.shape)
    for node, col, value in [(0, 0, None)] + [(b * c.n_nodes + row * 520 + lon, col, value) for b, row, lon in ((0, 12, 519), (17, 5, 8), (31, 23, 260))
                                             for col, value in ((3, np.inf), (17, np.nan), (c.width - 1, -np.inf), (c.width // 2, np.nan))]:
        if value is None:
            shifted.copy_(x)
            want, got = _table_gradient(g, shifted, t), _table_gradient(g, x, t, tensor_cores=True)
            assert_close(got.cpu().numpy(), want.cpu().numpy(), 0.0, 1e-5 * float(want.abs().max()), "table gradient")
            for transposed in (False, True):
                want, got = (_apply(v, table, t, transposed, tensor_cores=v is x).float() for v in (shifted, x))
                assert bool(((got - want).abs() <= 2.0 ** -7 * want.abs() + 1e-5 * float(want.abs().max())).all())
        else:
            x[node, col] = value
    shifted.copy_(x)
    for transposed in (False, True):
        want, got = (_apply(v, table, t, transposed, tensor_cores=v is x).float() for v in (shifted, x))
        finite = want.isfinite()
        assert not bool(finite.all()) and torch.equal(got.isfinite(), finite) and torch.equal(got.isnan(), want.isnan())
        assert torch.equal(got[want.isinf()], want[want.isinf()])
        assert bool(((got - want).abs() <= 2.0 ** -7 * want.abs() + 1e-5 * float(want[finite].abs().max()))[finite].all())


def test_tensor_core_apply_touches_only_true_neighbours():
    """An Inf, a NaN and a value whose products overflow reach exactly the targets that see their nodes, in their own channel."""
    from gm_attention_b200.nn.lattice_depthwise import _apply

    c, t = tensor_core_case(16, 64, 3.0, {0: 4, 1: 6})
    table, = seeded((t.n_entries, t.table_width), 73, np.float32)
    v, = seeded((c.n_nodes, c.width), 74, np.float32)
    clean = torch.from_numpy(v).bfloat16().cuda()
    want = _apply(clean, cuda(table), t, False, tensor_cores=True)
    dirty = clean.clone()
    nodes = [(5 * c.nlon + 63, 5, float("inf")), (9 * c.nlon + 20, 2, float("nan")), (0, 9, 3e38)]
    for node, col, value in nodes:
        dirty[node, col] = value
    got = _apply(dirty, cuda(table), t, False, tensor_cores=True)
    touched = torch.zeros_like(got, dtype=torch.bool)
    for node, col, value in nodes:
        seen_by = torch.from_numpy(np.unique(c.target[c.source == node])).cuda()
        first = col if col < 4 else col - col % 2  # scalar channels stand alone, (re, im) go together
        for x in range(first, first + (1 if col < 4 else 2)):
            touched[seen_by, x] = True
            if value != 3e38:
                assert not torch.isfinite(got[seen_by, x].float()).any()
    assert torch.equal(got[~touched], want[~touched])


@pytest.mark.parametrize("order", ["random", "sorted"])
@pytest.mark.parametrize("nlat, nlon, reach", [(6, 512, 2), (32, 256, 4), (24, 48, 2.5)])
def test_tensor_core_apply_rounds_no_worse_than_the_fma_kernel(nlat, nlon, reach, order):
    """Sums that cancel show the rounding of the accumulation, which the bf16 result hides otherwise: along a longitude the
    field is constant and the last entry of every window takes away the sum of the others.  In float64 what is left is
    about 2^-24 of a term, so the result is the error.  Bound: the FMA kernel's (which takes a field on an 8-byte boundary)."""
    from gm_attention_b200.nn.lattice_depthwise import _apply

    c = make_case(nlat, nlon, reach * math.pi / nlat, {0: 8, 1: 8}, 1, dtype=np.float32)
    t, _ = package_tables(c, None, False)
    lat, D = t.lattice, 24
    gen = np.random.default_rng(7)
    table = gen.standard_normal((t.n_entries, t.table_width)).astype(np.float32)
    cnt, off = (x.cpu().numpy().reshape(-1) for x in (lat.win_cnt, lat.win_off))
    sums = np.zeros((cnt.size, t.table_width))
    for w in np.flatnonzero(cnt > 0):
        rows = slice(off[w], off[w] + cnt[w])
        if order == "sorted":  # partial sums of the size of the window, and back
            table[rows] = -np.sort(-table[rows], axis=0)
        last = off[w] + cnt[w] - 1
        table[last] = -table[rows][:-1].astype(np.float64).sum(0)
        sums[w] = table[rows].astype(np.float64).sum(0)
    ring = torch.from_numpy(gen.standard_normal((nlat, D)).astype(np.float32)).bfloat16()
    x = ring.float().double().numpy()
    want = np.zeros((nlat, D))
    items, span = t.items.cpu().numpy(), 2 * lat.halo + 1
    for i in range(nlat):
        for w in range(span):
            j = i + w - lat.halo
            if 0 <= j < nlat and cnt[i * span + w]:
                for kind, col, fcol in items:
                    m = sums[i * span + w, fcol:fcol + 4]
                    m = m.reshape(2, 2) if kind == 0 else np.diag(m[:2])
                    want[i, col:col + 2] += m @ x[j, col:col + 2]
    field = ring[:, None, :].expand(nlat, nlon, D).reshape(nlat * nlon, D).contiguous().cuda()
    shifted = torch.empty(field.numel() + 4, dtype=field.dtype, device="cuda")[4:].view(field.shape)
    shifted.copy_(field)
    table = cuda(table)
    error = []
    for tensor_cores in (True, False):
        got = _apply(field if tensor_cores else shifted, table, t, False, tensor_cores=tensor_cores).float().double().cpu().numpy().reshape(nlat, nlon, D)
        error.append((float(np.sqrt(((got - want[:, None]) ** 2).mean())), float(np.abs(got - want[:, None]).max())))
    assert error[0][0] <= error[1][0] and error[0][1] <= error[1][1], error


@pytest.mark.parametrize("share", [3e-4, 1e-2, 1.0])
@pytest.mark.parametrize("head, nlon", [({0: 8, 1: 8}, 88), ({0: 4, 1: 10, 2: 12}, 552)])
def test_tensor_core_apply_of_non_finite_fields(head, nlon, share):
    """Infinities and NaNs everywhere or here and there, with zeros in the table: the same outputs are NaN, infinite and finite
    as by the FMA kernel (which takes a field on an 8-byte boundary); finite ones to the bf16 storage's 2^-7."""
    from gm_attention_b200.nn.lattice_depthwise import _apply

    c = make_case(7, nlon, 2 * math.pi / 7, head, 1, dtype=np.float32)
    t, _ = package_tables(c, None, False)
    gen = torch.Generator(device="cuda").manual_seed(8)
    table = torch.randn(t.n_entries, t.table_width, generator=gen, device="cuda")
    table[torch.rand(table.shape, generator=gen, device="cuda") < 0.2] = 0.0
    x = torch.randn(2 * c.n_nodes, c.width, generator=gen, device="cuda")
    odd = torch.rand(x.shape, generator=gen, device="cuda") < share
    values = torch.tensor([math.nan, math.inf, -math.inf], device="cuda")[torch.randint(3, x.shape, generator=gen, device="cuda")]
    field = torch.where(odd, values, x).bfloat16()
    shifted = torch.empty(field.numel() + 4, dtype=field.dtype, device="cuda")[4:].view(field.shape)
    shifted.copy_(field)
    assert c.width % 8 == 0 and field.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 == 8
    got, want = _apply(field, table, t, False, tensor_cores=True).float(), _apply(shifted, table, t, False).float()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
    assert bool(want.isnan().any()) and (share == 1.0 or bool(want.isfinite().any()))
    finite = want.isfinite()
    if bool(finite.any()):
        assert float((got - want)[finite].abs().max()) <= 2.0 ** -7 * float(want[finite].abs().max())


@pytest.mark.parametrize("head", [{0: 2, 1: 1}, {0: 6, 1: 5, 2: 7}, {1: 3}, {0: 130, 1: 130}, {0: 4}])
def test_fold_kernel_equals_the_tensor_algebra(head):
    """One launch each way against :func:`fold` and its autograd gradients: a handful of float32 products per value, 2e-6 of
    the largest; float64 coefficients are rounded first, as :func:`fold` does."""
    from types import SimpleNamespace

    from gm_attention_b200.nn.lattice_depthwise import _fold, conv_tables, fold

    c = make_case(6, 16, 1.7 * math.pi / 6, head, 1, dtype=np.float32)
    geometry = SimpleNamespace(transport=cuda(c.transport), angular=cuda(c.angular), rho=cuda(c.rho), bias=cuda(c.bias), inside=cuda(c.inside),
                               row_ptr=cuda(c.row_ptr), source=cuda(c.source))
    t = conv_tables(geometry, cuda(c.rho * np.float32(c.radius)), cuda(c.weights), descriptor_rows(c.head_type, 1), 6, 16)
    for dtype in (np.float32, np.float64):
        coefficients = [cuda(seeded((t.n_entries, w), 63 + w, dtype)[0]).requires_grad_(True) if w else None for w in (t.a_0, t.complex_width)]
        leaves = [x for x in coefficients if x is not None]
        got, want = _fold(*coefficients, t), fold(*coefficients, t)
        assert "FoldTable" in type(got.grad_fn).__name__ and got.shape == want.shape and got.is_contiguous()
        g = cuda(seeded(tuple(got.shape), 64, np.float32)[0])
        for name, a, b in zip(("table", "first", "second"), (got, *torch.autograd.grad(got, leaves, g)), (want, *torch.autograd.grad(want, leaves, g))):
            assert a.dtype == b.dtype and rel_err(a.detach().cpu().numpy(), b.detach().cpu().numpy()) < 2e-6, name


NLAT, NLON, BATCH, COPIES = 256, 512, 4, 64
HEAD = {0: COPIES, 1: COPIES, 2: COPIES}
RADIUS = 4 * math.pi / NLAT


@pytest.fixture(scope="module")
def big():
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_attention as fa
    from gm_attention_b200.nn.lattice_depthwise import conv_tables

    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(NLAT, NLON, dev)
    edges = compute_edge_geometry(lattice, lattice.frames, RADIUS, max_frequency=4, dtype=torch.float32)
    assert edges.n_edges == 22_999_040
    geo = fa.geometry(edges, RADIUS, "hard", torch.float32)
    rows = descriptor_rows(FieldType(HEAD), 1)
    tables = conv_tables(geo, edges.distances.float(), geo.weights, rows, NLAT, NLON)
    assert tables.n_entries == 22_999_040 // NLON
    gen = torch.Generator(device="cuda").manual_seed(5)
    a0, w = COPIES, 8 * COPIES
    rc_t = torch.randn(tables.n_entries, a0, generator=gen, device=dev) / 4
    cc_t = torch.randn(tables.n_entries, w, generator=gen, device=dev) / 4
    return tables, rows, rc_t, cc_t


@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_sampled_targets_256x512(big, storage):
    from gm_attention_b200.nn.lattice_depthwise import lattice_depthwise

    tables, rows, rc_t, cc_t = big
    n1, D = NLAT * NLON, 5 * COPIES
    a0, w = COPIES, 8 * COPIES
    dtype = torch.bfloat16 if storage == "bf16" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(6)
    V, Gd = (torch.randn(BATCH * n1, D, generator=gen, device="cuda").to(dtype) for _ in range(2))
    V.requires_grad_(True)
    RC, CC = rc_t.clone().requires_grad_(True), cc_t.clone().requires_grad_(True)
    out = lattice_depthwise(V, RC, CC, tables)
    out.backward(Gd)
    # adjoint identities on the whole problem (float64 sums of the kernels' own results)
    from gm_attention_b200.nn.lattice_depthwise import fold, _table_gradient

    table = fold(rc_t, cc_t, tables)
    dtable = _table_gradient(Gd, V.detach(), tables)
    lhs = float((Gd.double() * out.detach().double()).sum())
    assert abs(float((table.double() * dtable.double()).sum()) - lhs) < (2e-2 if storage == "bf16" else 1e-4) * abs(lhs)
    assert abs(float((V.grad.double() * V.detach().double()).sum()) - lhs) < (2e-2 if storage == "bf16" else 1e-4) * abs(lhs)
    # sampled targets / sources of the LAST sample against the oracle
    lat = G.midpoint_lattice(NLAT, NLON)
    t_rows = [0, 1, 4, 9, NLAT // 2, NLAT - 1]
    targets = np.array([r * NLON + col for r in t_rows for col in (0, NLON - 1, NLON // 2 + 1)], np.int64)
    sources = np.array([9 * NLON, (NLAT // 2) * NLON + NLON - 1, 40 * NLON + 7], np.int64)
    sample = S.sample_problem(lat, RADIUS, targets, sources, 4, np.float32)
    b = BATCH - 1
    pick = lambda x, nodes: x[torch.from_numpy(b * n1 + nodes).cuda()].float().cpu().numpy()
    tgt = np.repeat(sample.nodes, np.diff(sample.row_ptr))
    entry = entry_of(tables, tgt, sample.nodes[sample.source_index])
    rc, cc = rc_t[torch.from_numpy(entry).cuda()].cpu().numpy(), cc_t[torch.from_numpy(entry).cuda()].cpu().numpy()
    want = S.run_conv(sample, pick(V.detach(), sample.nodes), pick(Gd, sample.nodes), rc, cc, rows, RADIUS, a0, w)
    got = {"out": pick(out.detach(), sample.targets), "dv": pick(V.grad, sample.sources)}
    for name in got:
        if storage == "bf16":
            assert rel_err(got[name], want[name]) < 2e-2, name
        else:
            assert_close(got[name], want[name], 1e-5, 1e-5 * magnitude(want[name]), name)
    # the coefficient gradient of every entry of ONE complete lattice row (row 9: 421 neighbours per node): all 512
    # targets of the row, all samples, per-edge gradients of the oracle summed per entry
    row = 9
    row_targets = row * NLON + np.arange(NLON, dtype=np.int64)
    whole = S.sample_problem(lat, RADIUS, row_targets, np.zeros(0, np.int64), 4, np.float32)
    tgt = np.repeat(whole.nodes, np.diff(whole.row_ptr))
    entry = entry_of(tables, tgt, whole.nodes[whole.source_index])
    index = torch.from_numpy(entry).cuda()
    rc, cc = rc_t[index].cpu().numpy(), cc_t[index].cpu().numpy()
    first, count = int(entry.min()), int(entry.max()) - int(entry.min()) + 1
    want_rc, want_cc = np.zeros((count, a0), np.float64), np.zeros((count, w), np.float64)
    for s in range(BATCH):
        rows_of = lambda x: x[torch.from_numpy(s * n1 + whole.nodes).cuda()].float().cpu().numpy()
        r = S.run_conv(whole, rows_of(V.detach()), rows_of(Gd), rc, cc, rows, RADIUS, a0, w)
        np.add.at(want_rc, entry - first, r["drc"])
        np.add.at(want_cc, entry - first, r["dcc"])
    got_rc, got_cc = RC.grad[first:first + count].cpu().numpy(), CC.grad[first:first + count].cpu().numpy()
    covered = np.unique(entry - first)
    for name, a, ref in (("drc", got_rc, want_rc), ("dcc", got_cc, want_cc)):
        if storage == "bf16":
            assert rel_err(a[covered], ref[covered]) < 2e-2, name
        else:
            assert_close(a[covered], ref[covered].astype(np.float32), 1e-4, 1e-5 * magnitude(ref), name)


# ----------------------------------------------------------------------------- the reference's own convolution layer

@pytest.mark.parametrize("name", ["plain", "normalized"])
def test_reference_convolution_layer(name):
    """A depthwise ``SO2Convolution`` with its radial network, as the reference's Python evaluates it through its eager
    path (fixtures of ``tests/golden/make_golden.py: depthwise_case``, float64), against the package's chain in float32:
    geometry on the device, radial network on the table entries, fold, apply; gradients of the field and of every
    parameter of the network."""
    from pathlib import Path

    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
    from gm_attention_b200.nn import fused_attention as fa
    from gm_attention_b200.nn.lattice_depthwise import conv_tables, lattice_depthwise
    from tests.test_lattice_depthwise_cpu import load_network

    z = np.load(Path(__file__).resolve().parent / "golden" / f"depthwise_{name}.npz")
    nlat, nlon, radius = int(z["nlat"]), int(z["nlon"]), float(z["radius"])
    head = FieldType({int(n): int(a) for n, a in z["types"]})
    dev = torch.device("cuda", 0)
    lattice = midpoint_lattice(nlat, nlon, dev)
    edges = compute_edge_geometry(lattice, lattice.frames, radius, max_frequency=4, dtype=torch.float32)
    geo = fa.geometry(edges, radius, "hard", torch.float32)
    weights = geo.aggregation_weights(bool(int(z["normalize"])), 1e-12)
    tables = conv_tables(geo, edges.distances.float(), weights, descriptor_rows(head, 1), nlat, nlon)
    net = load_network(z, torch.float32, dev)
    v = cuda(z["v"].astype(np.float32)).requires_grad_(True)
    out = lattice_depthwise(v, *net(tables.distances), tables)
    out.backward(cuda(z["dout"].astype(np.float32)))
    assert_close(out.detach().cpu().numpy(), z["out"].astype(np.float32), 2e-5, 2e-5 * magnitude(z["out"]), "out")
    assert_close(v.grad.cpu().numpy(), z["dv"].astype(np.float32), 2e-5, 2e-5 * magnitude(z["dv"]), "dv")
    for key, parameter in net.named_parameters():
        want = z["grad__" + key.replace(".", "__")].astype(np.float32)
        assert_close(parameter.grad.cpu().numpy(), want, 1e-4, 1e-4 * magnitude(want), key)
