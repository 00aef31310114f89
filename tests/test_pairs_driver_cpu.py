"""The pair-term driver (``_FusedPairs`` and ``forward_general``) against a plain-PyTorch pair loop, on CPU:
the Python logic of the driver -- term loop, table indexing, in-place accumulation, the blocked readout gradient --
runs here over the REFERENCE's compiled CPU pair driver (oracle/_ref) standing in for the CUDA extension, which
has the same functions and signatures.  float64: values 1e-12, gradients 1e-11 (the bounds of the reference's own
``tests/nn/test_fused_pairs.py:73-93``); the field-type cases are the ones that test uses."""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from oracle import geometry_np as G

from tests.helpers import StandInKernel

CASES = [
    ({0: 2, 1: 2, 2: 1}, {0: 1, 1: 2, 2: 2}, True),   # (0,0), (0,m), (n,0), (n,m) with m - n of both signs
    ({0: 2, 1: 2, 2: 1}, {0: 1, 1: 2, 2: 2}, False),  # no bias
    ({0: 3}, {0: 2}, True),                            # real head only
    ({1: 2, 2: 1}, {1: 1, 2: 2}, True),                # complex head only
    ({0: 2, 1: 1}, {1: 2}, True),                      # real input into complex output only
    ({1: 2}, {0: 2}, True),                            # complex input into the real output only
    ({1: 16}, {1: 16}, True),                          # the largest block the kernels take
]


def cpu_edges(dtype=np.float64):
    from gm_attention_b200.geometry import EdgeGeometry

    lat = G.midpoint_lattice(5, 8)
    e = G.lattice_edges(lat, 1.3 * math.pi / 5, 4, dtype)
    t = torch.from_numpy
    return EdgeGeometry(t(e.edge_index), t(e.row_ptr), t(e.log_coordinates), t(e.distances), t(e.polar_angles), t(e.transport_angles),
                        t(e.tangent_quadrature_weights), t(e.angular_phases), t(e.transport_phases)), 1.3 * math.pi / 5


def run(kernel, flat, edges, fused: bool):
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.nn import fused_pairs as fp

    flat = flat.detach().clone().requires_grad_(True)
    x = FeatureField.from_flat(kernel.field_type_in, flat)
    if fused:
        out = fp.forward_general(kernel, x, edges).coefficients
    else:
        out = kernel.pair_loop(x, edges)
    loss = sum((out[m] * torch.arange(1, out[m].numel() + 1, dtype=flat.dtype).reshape(out[m].shape) / out[m].numel()).sum() for m in out)
    grads = torch.autograd.grad(loss, [flat, *kernel.parameters()])
    return {m: v.detach() for m, v in out.items()}, [g.detach() for g in grads]


@pytest.mark.parametrize("field_in, field_out, bias", CASES)
def test_driver_matches_the_pair_loop(reference_modules, monkeypatch, field_in, field_out, bias):
    from gm_attention_b200.nn import fused_pairs as fp

    monkeypatch.setattr(fp, "extension", lambda *sizes: reference_modules["gm_fused_pairs_cpu"])
    edges, cutoff = cpu_edges()
    kernel = StandInKernel(field_in, field_out, cutoff, trunk=5, bias=bias)
    gen = torch.Generator().manual_seed(3)
    flat = torch.randn(edges.n_edges, kernel.field_type_in.dimension, generator=gen, dtype=torch.float64)  # an edge-level field
    y_plain, g_plain = run(kernel, flat, edges, False)
    y_fused, g_fused = run(kernel, flat, edges, True)
    for m in y_plain:
        torch.testing.assert_close(y_fused[m], y_plain[m], atol=1e-12, rtol=0.0)
    assert len(g_fused) == len(g_plain)
    for a, b in zip(g_fused, g_plain):
        torch.testing.assert_close(a, b, atol=1e-11, rtol=0.0)


def test_plan_order_and_node_level_fields(reference_modules, monkeypatch):
    """Term order = for every output frequency, for every input frequency (reference ``tests/nn/test_fused_pairs.py:136-147``);
    a node-level field is gathered by the driver itself; the blocked readout gradient equals the plain product."""
    from gm_attention_b200.fields import FeatureField
    from gm_attention_b200.nn import fused_pairs as fp

    monkeypatch.setattr(fp, "extension", lambda *sizes: reference_modules["gm_fused_pairs_cpu"])
    edges, cutoff = cpu_edges()
    kernel = StandInKernel({0: 1, 1: 2}, {0: 2, 1: 1}, cutoff)
    assert [(t.n, t.m, t.role) for t in fp.plan(kernel)] == [(0, 0, "real"), (1, 0, "linear"), (0, 1, "linear"), (1, 1, "linear"), (1, 1, "antilinear")]
    nodes = torch.randn(40, kernel.field_type_in.dimension, dtype=torch.float64, generator=torch.Generator().manual_seed(4))
    x = FeatureField.from_flat(kernel.field_type_in, nodes)
    gathered = FeatureField.from_flat(kernel.field_type_in, nodes[edges.source_index])
    a, b = fp.forward_general(kernel, x, edges), fp.forward_general(kernel, gathered, edges)
    for m in a.field_type.frequencies:
        assert torch.equal(a[m], b[m])
    monkeypatch.setattr(fp, "GRADIENT_BLOCK_ROWS", 7)
    gk, op = torch.randn(6, 40, dtype=torch.float64), torch.randn(40, 5, dtype=torch.float64)
    torch.testing.assert_close(fp._coefficient_product(gk, op), gk @ op, atol=1e-12, rtol=0)


def test_sources_beyond_the_node_field_are_refused():
    """The grouping knows the range of its sources; what reads a node field through it refuses one with too few rows."""
    from gm_attention_b200.nn import fused_factored as ff

    edges, _ = cpu_edges()
    found = ff.grouping_for(edges, edges.source_index)
    assert (found.lowest, found.highest) == (int(edges.source_index.min()), int(edges.source_index.max()))
    assert found.require_nodes(found.highest + 1) is found.groups
    with pytest.raises(RuntimeError, match="the node field has"):
        found.require_nodes(found.highest)
    with pytest.raises(RuntimeError, match="the node field has"):
        ff.grouping(torch.tensor([3, -1, 2])).require_nodes(4)
    empty = ff.grouping(torch.zeros(0, dtype=torch.long))
    assert [t.shape[0] for t in empty.require_nodes(0)] == [0, 1, 0]


def test_grouping_follows_indices_written_in_place():
    """An edge set whose indices are overwritten in place is grouped anew, whether it is written through ``edge_index`` or
    through a view of it, and so is a registered chunk; unchanged indices keep their grouping."""
    from gm_attention_b200.nn import fused_attention
    from gm_attention_b200.nn import fused_factored as ff

    edges, _ = cpu_edges()
    order_of = lambda e: ff.groups_for(e, e.source_index)[0]
    first = order_of(edges)
    assert order_of(edges) is first
    edges.edge_index[1] = edges.edge_index[1].flip(0)
    assert torch.equal(order_of(edges), torch.argsort(edges.source_index, stable=True)) and not torch.equal(order_of(edges), first)
    edges.source_index.copy_(edges.source_index.roll(7))
    assert torch.equal(order_of(edges), torch.argsort(edges.source_index, stable=True))
    chunk, lo, hi = edges.target_range(3, 9)
    fused_attention.register_chunk(chunk, edges, lo, hi)
    assert order_of(chunk) is order_of(chunk)
    chunk.edge_index[1] = chunk.edge_index[1].flip(0)
    assert torch.equal(order_of(chunk), torch.argsort(chunk.source_index, stable=True))


def test_a_dead_edge_sets_grouping_is_nobodys():
    """An entry whose edge set is gone is not found under the key of the set that took its id and address, neither by the
    query nor by the builder, and is dropped."""
    import weakref

    from gm_attention_b200.nn import fused_factored as ff

    edges, _ = cpu_edges()
    device = edges.source_index.device
    assert ff.cached_grouping(edges, device) is None
    gone = torch.zeros(3)
    reference = weakref.ref(gone)
    del gone
    key, _ = ff._slot(edges)
    stale = ff.Grouping(ff.source_groups(edges.source_index.flip(0)), 0, 39)
    ff._GROUPS[key] = ff._Kept(reference, stale, None)
    assert ff.cached_grouping(edges, device) is None and key not in ff._GROUPS
    ff._GROUPS[key] = ff._Kept(reference, stale, None)
    found = ff.grouping_for(edges, edges.source_index)
    assert found is not stale and torch.equal(found.groups[0], torch.argsort(edges.source_index, stable=True))
    assert ff.cached_grouping(edges, device) is found
    assert ff._cached(key, None, device) is None and ff._cached(key, edges.row_ptr, device) is None and key in ff._GROUPS


def test_groupings_read_by_a_graph_outlive_the_cache(monkeypatch):
    """A grouping handed out during a capture is kept until its edge set goes, past any number of others; the rest are
    bounded, least recently used first, and dead edge sets' entries go when one is added."""
    from gm_attention_b200.nn import fused_factored as ff

    monkeypatch.setattr(ff, "_GROUPS", type(ff._GROUPS)())
    monkeypatch.setattr(ff, "GROUP_CACHE_SIZE", 3)
    sets = [cpu_edges()[0] for _ in range(6)]
    find = lambda e: ff.grouping_for(e, e.source_index)
    captured = find(sets[0])
    ff._GROUPS[ff._slot(sets[0])[0]].captured = True
    built = [find(e) for e in sets[1:]]
    assert len(ff._GROUPS) == 4 and find(sets[0]) is captured
    assert [find(e) is b for e, b in zip(sets[3:], built[2:])] == [True] * 3
    assert ff.cached_grouping(sets[1], sets[1].source_index.device) is None
    del sets[0]
    find(sets[0])
    assert len(ff._GROUPS) == 3 and not any(kept.captured for kept in ff._GROUPS.values())


@pytest.mark.parametrize("n_nodes, n_edges, repaid", [(100, 399, False), (100, 400, True), (8192, 4 * 8192, True), (8193, 4 * 8193, False),
                                                      (30000, 299_999, False), (30000, 300_000, True)])
def test_where_the_node_products_are_repaid(n_nodes, n_edges, repaid):
    from gm_attention_b200.nn import fused_pairs as fp

    assert fp._products_repaid(n_nodes, n_edges) is repaid
