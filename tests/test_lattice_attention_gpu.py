"""The equiangular-lattice fast path of the fused layer against the oracle and
against the general CSR kernels: forward and the deterministic two-pass
backward, float32 (1e-5 relative / 1e-6 absolute, absolute part scaled by the
tensor's magnitude) and bf16 storage (2e-2 relative to the magnitude)."""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from oracle import oracle as O

from tests.helpers import assert_close, cuda, make_case, rel_err, seeded

pytestmark = pytest.mark.gpu

CASES = [
    # nlat, nlon, radius, head type, heads, window, batch
    (16, 32, 2 * math.pi / 16, {0: 4, 1: 4, 2: 4}, 2, "hard", 2),         # 2 heads of 4 x (m = 0, 1, 2)
    (12, 24, 3 * math.pi / 12, {0: 16, 1: 16, 2: 16}, 4, "hard", 1),      # headline layout; polar windows are whole rows
    (8, 16, 2.5 * math.pi / 8, {0: 2, 1: 2}, 4, "quartic", 2),             # pairs outside the quartic window's support
    (10, 20, 2 * math.pi / 10, {0: 8, 1: 8, 2: 8, 3: 8}, 4, "hard", 1),   # 4 heads of 8 x (m = 0..3)
    (8, 256, 1.2 * math.pi / 8, {0: 4, 1: 4, 2: 4}, 2, "hard", 1),        # wide windows: several staged chunks per row
    (8, 16, 2 * math.pi / 8, {1: 6, 2: 6}, 1, "hard", 2),                 # no scalar block, runs of 2 with idle slots
    (8, 16, 2 * math.pi / 8, {0: 3, 2: 5}, 2, "hard", 1),                 # odd multiplicities: unaligned runs
]


def tables_for(c):
    from gm_attention_b200.attention import AttentionTables, build_lattice_tables

    rows = tuple(tuple(int(x) for x in row) for row in c.desc)
    general = AttentionTables(cuda(c.transport), cuda(c.bias), cuda(c.inside), cuda(c.row_ptr), cuda(c.source), rows, c.heads, c.scale)
    return general, build_lattice_tables(general, c.nlat, c.nlon, rows, c.heads, c.scale)


@pytest.mark.parametrize("case", CASES)
def test_lattice_matches_oracle_float32(case):
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    batch = case[6]
    c = make_case(*case[:5], dtype=np.float32, window=case[5])
    q, k, v, g = seeded((batch * c.n_nodes, c.width), 51, np.float32, 4)
    want = O.attention_forward(q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    grads = O.attention_backward(g, q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    _, lat = tables_for(c)
    assert lat.n_edges == c.source.shape[0]
    Q, K, V, G = cuda(q), cuda(k), cuda(v), cuda(g)
    out, lse = lattice_attention_forward(Q, K, V, lat)
    assert_close(out.cpu().numpy(), want, 1e-5, 1e-6 * max(1.0, np.abs(want).max()), "out")
    got = lattice_attention_backward(G, Q, K, V, out, lse, lat)
    for name, a, b in zip(("dq", "dk", "dv"), got, grads):
        assert_close(a.cpu().numpy(), b, 1e-5, 1e-5 * max(1.0, np.abs(b).max()), name)


# one head layout or more per tile: (copies per lane, lanes per owner) follow the larger multiplicity, then the number of frequencies
LAYOUTS = [
    {0: 1}, {0: 4, 1: 3, 2: 3}, {0: 2, 1: 4, 2: 4, 3: 4}, {1: 3, 2: 3, 3: 3, 4: 3},               # 4 x 1
    {0: 6, 1: 5}, {0: 5, 1: 5, 2: 5}, {1: 6, 2: 6, 3: 6}, {0: 5, 1: 6, 2: 6, 3: 6, 4: 6},          # 3 x 2
    {0: 7, 1: 7}, {0: 8, 1: 7, 2: 7}, {0: 7, 1: 8, 2: 8, 3: 8}, {1: 7, 2: 7, 3: 7, 4: 7},          # 4 x 2
    {0: 12, 1: 11}, {0: 9, 1: 9, 2: 9}, {0: 10, 1: 9, 2: 9, 3: 9}, {1: 12, 2: 12, 3: 12, 4: 12},   # 3 x 4
    {0: 16, 1: 2}, {0: 13, 1: 13}, {0: 15, 1: 14, 2: 14}, {0: 16, 1: 13, 2: 13, 3: 13}, {0: 16, 1: 16, 2: 16, 3: 16, 4: 16},  # 4 x 4
]


@pytest.mark.parametrize("head", LAYOUTS)
@pytest.mark.parametrize("shape", [(6, 14, 2.0, 1, 1), (4, 320, 1.6, 2, 4), (4, 320, 1.6, 2, 32)])
def test_lattice_float32_layouts(head, shape):
    """Every (copies per lane, lanes per owner, frequencies) tile, ragged runs padded with zeros, on three shapes: one whose
    neighbours are split over eight lanes and whose tile outgrows the lattice row; one of 10 240 owners (several stages per
    window, a tile remainder), split over 8 / 4 / 2 lanes in the forward and 4 / 2 / 1 in the backward at 1 / 2 / 4 lanes per owner;
    and one of 81 920, where nothing is split (148 SMs x 256 threads of owners' lanes are, with two owners a lane, 75 776 owners).
    Float32 against the oracle on the float32 tables for the last sample, tolerances as above."""
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    nlat, nlon, reach, heads, batch = shape
    c = make_case(nlat, nlon, reach * math.pi / nlat, head, heads, dtype=np.float32)
    q, k, v, g = seeded((c.n_nodes, c.width), 56, np.float32, 4)
    _, lat = tables_for(c)
    sample = slice((batch - 1) * c.n_nodes, batch * c.n_nodes)
    generator = torch.Generator(device="cuda").manual_seed(57)
    others = [torch.randn(batch * c.n_nodes, c.width, device="cuda", generator=generator) for _ in range(4)]
    for field, values in zip(others, (q, k, v, g)):
        field[sample] = cuda(values)
    Q, K, V, G = others
    out, lse = lattice_attention_forward(Q, K, V, lat)
    got = lattice_attention_backward(G, Q, K, V, out, lse, lat)
    args = (c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, 1)
    want = O.attention_forward(q, k, v, *args)
    grads = O.attention_backward(g, q, k, v, *args)
    assert_close(out[sample].cpu().numpy(), want, 1e-5, 1e-6 * max(1.0, np.abs(want).max()), "out")
    for name, a, b in zip(("dq", "dk", "dv"), got, grads):
        assert_close(a[sample].cpu().numpy(), b, 1e-5, 1e-5 * max(1.0, np.abs(b).max()), name)


@pytest.mark.parametrize("case", CASES[:4])
def test_lattice_bf16_storage(case):
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    batch = case[6]
    c = make_case(*case[:5], dtype=np.float32, window=case[5])
    rounded = [torch.from_numpy(x).bfloat16() for x in seeded((batch * c.n_nodes, c.width), 52, np.float32, 4)]
    q, k, v, g = (x.float().numpy() for x in rounded)
    want = O.attention_forward(q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    grads = O.attention_backward(g, q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    _, lat = tables_for(c)
    Q, K, V, G = (x.cuda() for x in rounded)
    out, lse = lattice_attention_forward(Q, K, V, lat)
    assert rel_err(out.float().cpu().numpy(), want) < 2e-2
    got = lattice_attention_backward(G, Q, K, V, out, lse, lat)
    for name, a, b in zip(("dq", "dk", "dv"), got, grads):
        assert rel_err(a.float().cpu().numpy(), b) < 2e-2, name


def test_lattice_agrees_with_the_general_kernels_and_is_deterministic():
    from gm_attention_b200.attention import (attention_backward, attention_forward, lattice_attention_backward,
                                             lattice_attention_forward)

    c = make_case(16, 32, 3 * math.pi / 16, {0: 16, 1: 16, 2: 16}, 4, dtype=np.float32)
    general, lat = tables_for(c)
    Q, K, V, G = (cuda(x) for x in seeded((2 * c.n_nodes, c.width), 53, np.float32, 4))
    out_a, lse_a = attention_forward(Q, K, V, general)
    out_b, lse_b = lattice_attention_forward(Q, K, V, lat)
    assert_close(out_b.cpu().numpy(), out_a.cpu().numpy(), 1e-5, 2e-6, "out")
    assert_close(lse_b.cpu().numpy(), lse_a.cpu().numpy(), 1e-5, 1e-5, "lse")
    first = lattice_attention_backward(G, Q, K, V, out_b, lse_b, lat)
    again = lattice_attention_backward(G, Q, K, V, out_b, lse_b, lat)
    for a, b in zip(first, again):
        assert torch.equal(a, b)  # no atomics: bit-identical reruns
    for name, a, b in zip(("dq", "dk", "dv"), first, attention_backward(G, Q, K, V, out_a, lse_a, general)):
        assert_close(a.cpu().numpy(), b.cpu().numpy(), 1e-5, 1e-5 * max(1.0, float(b.abs().max())), name)


def test_lattice_through_autograd_and_unsupported_layout():
    from gm_attention_b200.attention import GaugeAttention, build_lattice_tables, lattice_layout_supported

    c = make_case(8, 16, 2 * math.pi / 8, {0: 4, 1: 4, 2: 4}, 2, dtype=np.float32)
    _, lat = tables_for(c)
    q, k, v = (cuda(x).requires_grad_(True) for x in seeded((c.n_nodes, c.width), 54, np.float32, 3))
    g, = seeded((c.n_nodes, c.width), 55, np.float32)
    out = GaugeAttention.apply(q, k, v, lat)
    (out * cuda(g)).sum().backward()
    grads = O.attention_backward(g, q.detach().cpu().numpy(), k.detach().cpu().numpy(), v.detach().cpu().numpy(), c.transport, c.bias,
                                 c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, 1)
    for name, a, b in zip(("dq", "dk", "dv"), (q.grad, k.grad, v.grad), grads):
        assert_close(a.cpu().numpy(), b, 1e-5, 1e-5 * max(1.0, np.abs(b).max()), name)
    odd = make_case(6, 12, 2 * math.pi / 6, {1: 3, 3: 2}, 1, dtype=np.float32)
    rows = tuple(tuple(int(x) for x in row) for row in odd.desc)
    assert not lattice_layout_supported(rows)
    assert lattice_layout_supported(lat.desc_rows)


#: headline head layout on a wide lattice: every unit of staging, tiles that wrap the longitude seam and
#: tiles that do not, windows from a few positions (one staged chunk) to whole rows (several chunks)
STAGING_CASE = (6, 256, 1.2 * math.pi / 6, {0: 16, 1: 16, 2: 16}, 2, "hard", 2)
TC_CASES = [CASES[0], CASES[1], CASES[2], CASES[3], CASES[4], (8, 16, 2 * math.pi / 8, {1: 6, 2: 6}, 1, "hard", 2), STAGING_CASE]


@pytest.fixture(params=["one-head", "four-heads"])
def kernel_family(request, monkeypatch):
    """The two tensor-core kernel families: one head per CTA (default) and all four heads of a tile per CTA (opt-in;
    layouts it does not serve fall through to the first)."""
    from gm_attention_b200 import attention

    monkeypatch.setattr(attention, "FOUR_HEADS", "1" if request.param == "four-heads" else "0")
    return request.param


FOUR_HEAD_CASES = [
    (12, 48, 3 * math.pi / 12, {0: 16, 1: 16, 2: 16}, 4, "hard", 2),      # headline layout: whole-row polar windows, tiles across the seam
    (6, 256, 1.2 * math.pi / 6, {0: 16, 1: 16, 2: 16}, 4, "hard", 2),     # wide windows: several chunks per row pair, tensor copies and seam chunks
    (10, 64, 2 * math.pi / 10, {0: 16, 1: 16}, 4, "quartic", 1),          # one complex frequency, masked pairs inside the windows
    (8, 40, 2 * math.pi / 8, {0: 16, 1: 16, 2: 16, 3: 16}, 4, "hard", 1), # three complex frequencies (20-word entries), the smallest row length served
]


@pytest.mark.parametrize("case", FOUR_HEAD_CASES)
def test_four_head_kernels_match_the_oracle_and_the_one_head_kernels(case, monkeypatch):
    """The persistent four-heads-per-CTA kernels (128-byte rows, producer / consumer warps): forward and both backward
    passes against the oracle (2e-2 of each tensor's magnitude) and against the one-head kernels on the same inputs;
    bit-identical reruns; no wait on a barrier ran out."""
    import ctypes

    from gm_attention_b200 import _lib, attention
    from gm_attention_b200.attention import four_head_layout_supported, lattice_attention_backward, lattice_attention_forward

    batch = case[6]
    c = make_case(*case[:5], dtype=np.float32, window=case[5])
    rounded = [torch.from_numpy(x).bfloat16() for x in seeded((batch * c.n_nodes, c.width), 62, np.float32, 4)]
    q, k, v, g = (x.float().numpy() for x in rounded)
    want = O.attention_forward(q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    grads = O.attention_backward(g, q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    _, lat = tables_for(c)
    assert four_head_layout_supported(lat, c.width)
    Q, K, V, G = (x.cuda() for x in rounded)
    results = {}
    # the other family: the one-head tensor-core kernels, or the FMA lattice kernels where those have no instantiation
    # (16 copies of three complex frequencies)
    other_tc = attention.tensor_core_layout_supported(lat.desc_rows)
    for family in ("1", "0"):
        monkeypatch.setattr(attention, "FOUR_HEADS", family)
        tc = True if family == "1" else other_tc
        out, lse = lattice_attention_forward(Q, K, V, lat, tensor_cores=tc)
        results[family] = (out, lse, *lattice_attention_backward(G, Q, K, V, out, lse, lat, tensor_cores=tc))
    monkeypatch.setattr(attention, "FOUR_HEADS", "1")
    out, lse = lattice_attention_forward(Q, K, V, lat, tensor_cores=True)
    again = (out, lse, *lattice_attention_backward(G, Q, K, V, out, lse, lat, tensor_cores=True))
    for a, b in zip(results["1"], again):
        assert torch.equal(a, b)
    for name, a, b in zip(("out", "dq", "dk", "dv"), (results["1"][0], *results["1"][2:]), (want, *grads)):
        assert rel_err(a.float().cpu().numpy(), b) < 2e-2, name
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), results["1"], results["0"]):
        assert rel_err(a.float().cpu().numpy(), b.float().cpu().numpy()) < 2e-2, name
    expired = ctypes.c_int(-1)
    _lib.call("gm_lattice_attention_tc4_wait_expired", ctypes.byref(expired))
    assert expired.value == 0


@pytest.mark.parametrize("case", TC_CASES)
def test_tensor_core_forward_bf16(case):
    """mma.sync Gram / value tiles against the oracle (2e-2 of the output's magnitude) and against the FMA
    lattice kernel on the same bf16 inputs (they differ only by the bf16 rounding of the attention weights)."""
    from gm_attention_b200.attention import lattice_attention_forward, tensor_core_layout_supported

    batch = case[6]
    c = make_case(*case[:5], dtype=np.float32, window=case[5])
    rounded = [torch.from_numpy(x).bfloat16() for x in seeded((batch * c.n_nodes, c.width), 57, np.float32, 3)]
    q, k, v = (x.float().numpy() for x in rounded)
    want = O.attention_forward(q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    _, lat = tables_for(c)
    assert tensor_core_layout_supported(lat.desc_rows)
    Q, K, V = (x.cuda() for x in rounded)
    out_tc, lse_tc = lattice_attention_forward(Q, K, V, lat, tensor_cores=True)
    out_fma, lse_fma = lattice_attention_forward(Q, K, V, lat, tensor_cores=False)
    assert rel_err(out_tc.float().cpu().numpy(), want) < 2e-2
    assert rel_err(out_tc.float().cpu().numpy(), out_fma.float().cpu().numpy()) < 2e-2
    assert_close(lse_tc.cpu().numpy(), lse_fma.cpu().numpy(), 1e-4, 1e-4, "lse")


@pytest.mark.parametrize("case", TC_CASES)
def test_tensor_core_backward_bf16(case):
    """Both backward passes on tensor cores against the oracle (fp32 on the bf16-rounded inputs, 2e-2 of each
    gradient's magnitude); reruns are bit-identical (no atomics)."""
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    batch = case[6]
    c = make_case(*case[:5], dtype=np.float32, window=case[5])
    rounded = [torch.from_numpy(x).bfloat16() for x in seeded((batch * c.n_nodes, c.width), 58, np.float32, 4)]
    q, k, v, g = (x.float().numpy() for x in rounded)
    grads = O.attention_backward(g, q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    _, lat = tables_for(c)
    Q, K, V, G = (x.cuda() for x in rounded)
    out, lse = lattice_attention_forward(Q, K, V, lat, tensor_cores=True)
    got = lattice_attention_backward(G, Q, K, V, out, lse, lat, tensor_cores=True)
    again = lattice_attention_backward(G, Q, K, V, out, lse, lat, tensor_cores=True)
    for name, a, b, a2 in zip(("dq", "dk", "dv"), got, grads, again):
        assert rel_err(a.float().cpu().numpy(), b) < 2e-2, name
        assert torch.equal(a, a2), name


def test_tensor_core_backward_ignores_stale_shared_memory():
    """A step of 16 staged positions may start inside a window and end beyond it: the rows beyond carry weight zero, and
    whatever an earlier kernel left in shared memory (here NaN, on every SM) must not reach the sums."""
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    batch = STAGING_CASE[6]
    c = make_case(*STAGING_CASE[:5], dtype=np.float32, window=STAGING_CASE[5])
    _, lat = tables_for(c)
    Q, K, V, G = (torch.from_numpy(x).bfloat16().cuda() for x in seeded((batch * c.n_nodes, c.width), 58, np.float32, 4))
    out, lse = lattice_attention_forward(Q, K, V, lat, tensor_cores=True)
    poison = torch.full_like(Q, float("nan"))
    for _ in range(4):  # the fp32-arithmetic and the tensor-core kernel stage these rows over most of an SM's shared memory
        for tensor_cores in (False, True):
            lattice_attention_forward(poison, poison, poison, lat, tensor_cores=tensor_cores)
        lattice_attention_backward(poison, poison, poison, poison, poison, torch.full_like(lse, float("nan")), lat, tensor_cores=True)
        for name, got in zip(("dq", "dk", "dv"), lattice_attention_backward(G, Q, K, V, out, lse, lat, tensor_cores=True)):
            assert bool(torch.isfinite(got.float()).all()), name


@pytest.mark.parametrize("offset", [4, 2, 1])
def test_staging_in_units_of_every_size(offset):
    """Neighbour rows are staged in copies of 16, 8, 4 or 2 bytes, as the fields' addresses allow (here views at an element
    offset of 0, 4, 2, 1): the same arithmetic on the same values, bit for bit."""
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    batch = STAGING_CASE[6]
    c = make_case(*STAGING_CASE[:5], dtype=np.float32, window=STAGING_CASE[5])
    _, lat = tables_for(c)
    fields = [torch.from_numpy(x).bfloat16().cuda() for x in seeded((batch * c.n_nodes, c.width), 60, np.float32, 4)]
    moved = [torch.empty(x.numel() + offset, dtype=x.dtype, device="cuda")[offset:].view(x.shape).copy_(x) for x in fields]
    assert all(x.data_ptr() % 16 == 0 for x in fields) and all(x.data_ptr() % 16 == 2 * offset for x in moved)
    results = []
    for Q, K, V, G in (fields, moved):
        out, lse = lattice_attention_forward(Q, K, V, lat, tensor_cores=True)
        results.append((out, lse, *lattice_attention_backward(G, Q, K, V, out, lse, lat, tensor_cores=True)))
    for x, y in zip(*results):
        assert torch.equal(x, y)
    assert torch.isfinite(results[0][0].float()).all()


def test_host_pipeline_equals_the_device_path():
    """Host-resident fields, sample chunks pipelined over three streams: same numbers as one device-resident call."""
    from gm_attention_b200.attention import HostPipeline, lattice_attention_backward, lattice_attention_forward

    batch = 5
    c = make_case(8, 16, 2 * math.pi / 8, {0: 4, 1: 4, 2: 4}, 2, dtype=np.float32)
    _, lat = tables_for(c)
    host = [torch.from_numpy(x).pin_memory() for x in seeded((batch * c.n_nodes, c.width), 59, np.float32, 4)]
    outs = [torch.empty_like(host[0]).pin_memory() for _ in range(4)]
    pipe = HostPipeline(lat, batch, c.width, torch.float32, torch.device("cuda", 0), chunk=1)
    for _ in range(2):  # the second run reuses the staging buffers
        pipe.run(*host, *outs)
        torch.cuda.synchronize()
    for x in outs:
        x.zero_()
    for _ in range(3):  # enqueue-only calls overlap one another; join before reading
        pipe.run(*host, *outs, wait=False)
    pipe.join()
    torch.cuda.synchronize()
    Q, K, V, G = (x.cuda() for x in host)
    out, lse = lattice_attention_forward(Q, K, V, lat)
    want = (out, *lattice_attention_backward(G, Q, K, V, out, lse, lat))
    for got, ref in zip(outs, want):
        assert torch.equal(got, ref.cpu())


def test_layer_split_around_a_halo_exchange_equals_one_call():
    """The row subsets used to overlap the halo exchange (interior / boundary target rows; halo / owned source rows)
    reproduce the unsplit forward and backward of a rank's band bit for bit (one GPU, no exchange: the band of rank 1
    of 3 with its halo rows filled from the full fields)."""
    import dataclasses

    from gm_attention_b200.attention import AttentionTables, build_lattice_tables, lattice_attention_backward, lattice_attention_forward
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.geometry import midpoint_lattice
    from gm_attention_b200.nn import fused_attention as fa
    from gm_attention_b200.parallel import BandPlan, band_geometry, overlap_tables

    dev = torch.device("cuda", 0)
    nlat, nlon, heads, batch = 24, 64, 2, 2
    radius = 2.5 * math.pi / nlat
    attn = FieldType({0: 16, 1: 16, 2: 16})
    full = attn.scaled(heads)
    lattice = midpoint_lattice(nlat, nlon, dev)
    plan = BandPlan(nlat, nlon, lattice.band(radius), (0, 7, 16, 24))
    rank = 1
    elo, ehi = plan.extended(rank)
    edges = band_geometry(lattice, plan, rank, radius, max_frequency=2, dtype=torch.float32)
    geo = fa.geometry(edges, radius, "hard", torch.float32)
    p = fa._plan(type("Layer", (), {})(), attn, full, heads)
    gen = AttentionTables(geo.transport, geo.bias, geo.inside, geo.row_ptr, geo.source, p.rows, heads, 1 / math.sqrt(attn.dimension))
    t = build_lattice_tables(gen, ehi - elo, nlon, p.rows, heads, gen.scale)
    split = overlap_tables(t, plan, rank)
    assert split.interior.row_order.numel() > 0 and split.boundary.row_order.numel() > 0
    assert split.interior.row_order.numel() + split.boundary.row_order.numel() == t.row_order.numel()
    assert split.halo_sources.t_row_order.numel() + split.owned_sources.t_row_order.numel() == t.t_row_order.numel()
    n = batch * (ehi - elo) * nlon
    Q, K, V, G = (torch.from_numpy(x).bfloat16().to(dev) for x in seeded((n, full.dimension), 61, np.float32, 4))
    out, lse = lattice_attention_forward(Q, K, V, t)
    want = (out, lse, *lattice_attention_backward(G, Q, K, V, out, lse, t))
    out2, lse2 = lattice_attention_forward(Q, K, V, split.interior)
    lattice_attention_forward(Q, K, V, split.boundary, out=out2, lse=lse2)
    ws = (torch.zeros_like(Q), torch.zeros_like(Q), torch.zeros_like(Q), torch.empty((n, heads), dtype=torch.float32, device=dev))
    lattice_attention_backward(G, Q, K, V, out2, lse2, split.full, passes=3, workspace=ws)
    lattice_attention_backward(G, Q, K, V, out2, lse2, split.halo_sources, passes=4, workspace=ws)
    lattice_attention_backward(G, Q, K, V, out2, lse2, split.owned_sources, passes=4, workspace=ws)
    for a, b in zip(want, (out2, lse2, *ws[:3])):
        assert torch.equal(a, b)


# tiles of 4 rows x 8 or 16 longitudes with remainders both ways, copies of 2 / 8 / 16 bytes at a time, windows cut into
# chunks, more neighbour rows than a warp has lanes, a lattice narrower than a tile
PACKED_CASES = [
    (5, 8, 2 * math.pi / 5, {0: 5, 1: 5}, 3, "hard", 2),
    (7, 30, 2.5 * math.pi / 7, {0: 4, 1: 4, 2: 4}, 2, "quartic", 1),
    (33, 40, 3 * math.pi / 33, {0: 8, 1: 8, 2: 8, 3: 8}, 1, "hard", 2),
    (4, 320, 1.6 * math.pi / 4, {0: 16, 1: 16, 2: 16}, 1, "hard", 1),
    (40, 12, 15.5 * math.pi / 40, {1: 6, 2: 6}, 1, "hard", 1),
]


@pytest.mark.parametrize("case", PACKED_CASES)
def test_packed_tensor_core_kernels(case, monkeypatch):
    """The tensor-core kernels with a plan, without one (every CTA packs its own lists) and after the tables were written in
    place (the entries are read in every launch; windows that are not the plan's are packed anew), against the oracle on the rounded inputs; bf16 storage: 2e-2 of the magnitude."""
    import dataclasses

    from gm_attention_b200 import attention
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    monkeypatch.setattr(attention, "PLANNED_FROM", 0)
    batch = case[6]
    c = make_case(*case[:5], dtype=np.float32, window=case[5])
    rounded = [torch.from_numpy(x).bfloat16() for x in seeded((batch * c.n_nodes, c.width), 63, np.float32, 4)]
    q, k, v, g = (x.float().numpy() for x in rounded)
    Q, K, V, G = (x.cuda() for x in rounded)
    _, lat = tables_for(c)
    assert all(plan is not None for plan in lat.tc_plans)

    def run(t):
        out, lse = lattice_attention_forward(Q, K, V, t, tensor_cores=True)
        return out, lse, *lattice_attention_backward(G, Q, K, V, out, lse, t, tensor_cores=True)

    planned = run(lat)
    for a, b in zip(planned, run(dataclasses.replace(lat, tc_plans=(None, None, None)))):
        assert torch.equal(a, b)
    want = O.attention_forward(q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    grads = O.attention_backward(g, q, k, v, c.transport, c.bias, c.inside, c.desc, c.row_ptr, c.source, c.heads, c.scale, batch)
    for name, a, b in zip(("out", "dq", "dk", "dv"), (planned[0], *planned[2:]), (want, *grads)):
        assert float(np.abs(a.float().cpu().numpy() - b).max()) < 2e-2 * max(1.0, np.abs(b).max()), name
    lat.entries[:, :2 * lat.orders].mul_(-1.0)
    turned = run(lat)
    assert torch.equal(turned[0], run(dataclasses.replace(lat, tc_plans=(None, None, None)))[0]) and not torch.equal(turned[0], planned[0])


def test_tables_without_a_plan():
    """Head layouts the tensor-core kernels do not take (orders out of turn) still make tables for the others."""
    from gm_attention_b200.attention import AttentionTables, build_lattice_tables, lattice_attention_forward

    c = make_case(6, 16, 2 * math.pi / 6, {0: 2, 1: 2, 2: 2}, 1, dtype=np.float32)
    rows = [tuple(int(x) for x in row) for row in c.desc]
    general = AttentionTables(cuda(c.transport), cuda(c.bias), cuda(c.inside), cuda(c.row_ptr), cuda(c.source), tuple(rows), c.heads, c.scale)
    q, k, v = (cuda(x) for x in seeded((c.n_nodes, c.width), 64, np.float32, 3))
    want, _ = lattice_attention_forward(q, k, v, build_lattice_tables(general, c.nlat, c.nlon, tuple(rows), c.heads, c.scale))
    turned = build_lattice_tables(general, c.nlat, c.nlon, (rows[0], rows[2], rows[1]), c.heads, c.scale)
    assert turned.tc_plans == (None, None, None)
    got, _ = lattice_attention_forward(q, k, v, turned)
    assert float((got - want).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))


def test_kernels_read_the_tables_in_every_launch(monkeypatch):
    """Writes into the tables show at once: by a captured graph's replay, past the tensors' write counters, and where they
    change the windows that the plans were made from (some row tiles, then all); bit for bit as without plans.  Copies keep
    their plans."""
    import copy
    import dataclasses

    from gm_attention_b200 import attention
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    monkeypatch.setattr(attention, "PLANNED_FROM", 0)

    c = make_case(13, 40, 2.5 * math.pi / 13, {0: 8, 1: 8}, 2, dtype=np.float32)
    Q, K, V, G = (torch.from_numpy(x).bfloat16().cuda() for x in seeded((c.n_nodes, c.width), 65, np.float32, 4))
    _, lat = tables_for(c)
    bare = dataclasses.replace(lat, tc_plans=(None, None, None))
    out, lse = torch.empty_like(Q), torch.empty((c.n_nodes, c.heads), device="cuda")
    grads = [torch.empty_like(Q) for _ in range(3)] + [torch.empty_like(lse)]

    def run(t, out, lse, grads):
        lattice_attention_forward(Q, K, V, t, tensor_cores=True, out=out, lse=lse)
        lattice_attention_backward(G, Q, K, V, out, lse, t, tensor_cores=True, workspace=tuple(grads))

    run(lat, out, lse, grads)  # loads the kernels before the capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(lat, out, lse, grads)
    results = []

    def compare():
        for x in (out, lse, *grads):
            x.fill_(float("nan"))
        graph.replay()
        other = [torch.empty_like(x) for x in (out, lse, *grads)]
        run(bare, other[0], other[1], other[2:])
        eager = [torch.empty_like(x) for x in (out, lse, *grads)]
        run(copy.deepcopy(lat), eager[0], eager[1], eager[2:])
        for a, b, x in zip((out, lse, *grads), other, eager):
            assert torch.equal(a, b) and torch.equal(x, b)
        results.append([x.clone() for x in (out, *grads[:3])])
        for earlier in results[:-1]:
            assert not torch.equal(earlier[0], out)

    assert all(plan.layout == lat.plan_layout() for plan in copy.deepcopy(lat).tc_plans)
    compare()
    lat.entries[:, :2].mul_(-1.0)
    compare()
    lat.entries.data[:, 2].add_(torch.linspace(0.0, 1.0, lat.entries.shape[0], device="cuda"))
    lat.t_entries.data[:, :2].mul_(-1.0)
    compare()
    assert not torch.equal(results[2][2], results[1][2])  # dk: the transposed entries
    lat.win_cnt.data[6].clamp_(max=3)  # one row of one tile
    compare()
    lat.win_lo.data.add_(1)
    lat.t_win_cnt.data.clamp_(max=4)
    compare()


@pytest.mark.parametrize("head", [{0: 8, 1: 8}, {0: 5, 1: 6, 2: 6}])
def test_fields_on_odd_addresses(head):
    """bf16 fields that start on a 2-byte boundary only (contiguous views at an odd element offset), each alone and all
    together: bit for bit the aligned call's results."""
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    c = make_case(6, 24, 2 * math.pi / 6, head, 2, dtype=np.float32)
    _, lat = tables_for(c)
    aligned = [torch.from_numpy(x).bfloat16().cuda() for x in seeded((c.n_nodes, c.width), 66, np.float32, 4)]
    results = [torch.empty_like(aligned[0]) for _ in range(4)]

    def odd(x):
        view = torch.empty(x.numel() + 1, dtype=x.dtype, device="cuda")[1:].view(x.shape)
        view.copy_(x)
        assert view.data_ptr() % 4 == 2 and view.is_contiguous()
        return view

    def run(fields, results):
        q, k, v, g = fields
        out, dq, dk, dv = results
        _, lse = lattice_attention_forward(q, k, v, lat, tensor_cores=True, out=out)
        delta = torch.empty_like(lse)
        lattice_attention_backward(g, q, k, v, out, lse, lat, tensor_cores=True, workspace=(dq, dk, dv, delta))
        return [x.clone() for x in (*results, lse, delta)]

    want = run(aligned, results)
    for moved in [{x} for x in range(8)] + [set(range(8))]:
        fields = [odd(x) if i in moved else x for i, x in enumerate(aligned)]
        places = [odd(x) if i + 4 in moved else x for i, x in enumerate(results)]
        for a, b in zip(run(fields, places), want):
            assert torch.equal(a, b), moved


@pytest.mark.parametrize("planned_from", [0, 1 << 40])
def test_short_row_lists(planned_from, monkeypatch):
    """Lists with fewer rows than the lattice has row tiles (whose grid is made for the tiles they can touch): rows of one tile
    and of several, out of order, at both poles and in the last, partial tile give the bits of the whole call; other rows
    keep what they held."""
    import dataclasses

    from gm_attention_b200 import attention
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    monkeypatch.setattr(attention, "PLANNED_FROM", planned_from)
    rows, nlon, batch = 37, 24, 2
    c = make_case(rows, nlon, 2 * math.pi / rows, {0: 8, 1: 8}, 2, dtype=np.float32)
    Q, K, V, G = (torch.from_numpy(x).bfloat16().cuda() for x in seeded((batch * c.n_nodes, c.width), 67, np.float32, 4))
    _, lat = tables_for(c)
    out, lse = lattice_attention_forward(Q, K, V, lat, tensor_cores=True)
    whole = lattice_attention_backward(G, Q, K, V, out, lse, lat, tensor_cores=True)
    banded = lambda x: x.view(batch, rows, nlon, -1)
    for listed in ([36], [0], [17], [36, 0], [9, 8, 11], [20, 5, 6, 33, 2], [0, 1, 2, 3, 4, 35, 36, 18, 19]):
        order = torch.tensor(listed, dtype=torch.int32, device="cuda")
        part = dataclasses.replace(lat, row_order=order, t_row_order=order)
        got = lattice_attention_forward(Q, K, V, part, tensor_cores=True, out=torch.full_like(out, 7.0), lse=torch.full_like(lse, 7.0))
        places = tuple(torch.full_like(Q, 7.0) for _ in range(3)) + (torch.full_like(lse, 7.0),)
        lattice_attention_backward(G, Q, K, V, out, lse, part, tensor_cores=True, passes=3, workspace=places)
        delta = places[3].clone()
        full_delta = torch.empty_like(lse)
        lattice_attention_backward(G, Q, K, V, out, lse, lat, tensor_cores=True, passes=1, workspace=places[:3] + (full_delta,))
        lattice_attention_backward(G, Q, K, V, out, lse, part, tensor_cores=True, passes=4, workspace=places[:3] + (full_delta,))
        other = [r for r in range(rows) if r not in listed]
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), (*got, *places[:3]), (out, lse, *whole)):
            assert torch.equal(banded(a)[:, listed], banded(b)[:, listed]), (name, listed)
            assert bool((banded(a)[:, other] == 7.0).all()), (name, listed)
        assert bool((banded(delta)[:, other] == 7.0).all())


def test_plans_of_another_format_or_layout_are_not_used(monkeypatch):
    """Plans that were saved with another record format, or for another head count, lattice or halo, are left alone (their
    records, here of no use to anyone, are never read): the kernels pack their own lists."""
    import dataclasses

    from gm_attention_b200 import _lib, attention
    from gm_attention_b200.attention import lattice_attention_backward, lattice_attention_forward

    monkeypatch.setattr(attention, "PLANNED_FROM", 0)
    c = make_case(9, 24, 2 * math.pi / 9, {0: 8, 1: 8}, 2, dtype=np.float32)
    Q, K, V, G = (torch.from_numpy(x).bfloat16().cuda() for x in seeded((c.n_nodes, c.width), 68, np.float32, 4))
    _, lat = tables_for(c)

    def run(t):
        before = _lib.CALLS["gm_lattice_plan_refresh"]
        out, lse = lattice_attention_forward(Q, K, V, t, tensor_cores=True)
        return (out, lse, *lattice_attention_backward(G, Q, K, V, out, lse, t, tensor_cores=True)), _lib.CALLS["gm_lattice_plan_refresh"] - before

    want, refreshed = run(lat)
    assert refreshed == 3
    tag, desc, heads, rows, nlon, halo, orders = lat.plan_layout()
    for layout in ((tag - 1, desc, heads, rows, nlon, halo, orders), (desc, heads, rows, nlon, halo, orders), (tag, desc, heads + 1, rows, nlon, halo, orders),
                   (tag, desc, heads, rows, nlon, halo + 1, orders)):
        other = tuple(dataclasses.replace(p, layout=layout, records=torch.full_like(p.records, 255)) for p in lat.tc_plans)
        got, refreshed = run(dataclasses.replace(lat, tc_plans=other))
        assert refreshed == 0
        for a, b in zip(got, want):
            assert torch.equal(a, b)
