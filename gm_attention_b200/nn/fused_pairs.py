"""Host driver of the fused pair terms of the general steerable kernel.

Mirror of the reference's ``gm_attention/nn/fused_pairs.py``: ``MODE``,
``SUPPORTED``, ``Term``, ``plan``, ``enabled``, ``extension``, the flags, the
autograd function ``_FusedPairs`` (``fused_pairs.py:156-238``) and the driver
entry ``forward_general`` (``:247-295``).  The reference compiles one CUDA
extension per ``(a, b, trunk)``; here a single kernel serves every
``a, b, trunk <= 16`` (runtime sizes, bounds unrolled), so ``extension()``
takes the sizes only for signature compatibility.

``_FusedPairs.apply(hidden, complex_weight, complex_bias, real_weight, real_bias,
meta, phases, scales, *vectors)`` keeps the reference's argument order and
``meta`` keys (``terms``, ``tables``, ``in_index``, ``out_index``,
``out_frequencies``, ``out_multiplicity``): one launch per term forward, one per
term backward (input and trunk gradients accumulated in place, the term's
coefficient-major slab of the coefficient gradient written), then the readout
weight / bias gradients as ONE product of the coefficient gradient with
``[hidden | 1]``, summed over blocks of 16 384 edges like the reference's
``_blocked_weight_gradient`` (``nn/kernels.py:49-64``).

``forward_general`` on a NODE-level field takes the factored form instead: an edge's phases commute with the sum over the
input copies, so ``M(e) (pre u~)`` is a phase times ``sum_t h~_t(e) Z_t(source(e))`` with ``Z_t = W_t x`` formed once per node
(:class:`NodeProducts`) -- ``a`` times fewer multiply-adds per edge, no per-edge coefficient gradients, and the readout's
gradient a sum over nodes.  Edge-level fields, and anything :func:`_factored_inputs` does not recognise, take the pair terms.
"""

from __future__ import annotations

import functools
import os
from dataclasses import dataclass
from typing import Any

import torch
from torch import Tensor

MAX_MULT, MAX_TRUNK = 16, 16
#: every block size up to MAX_MULT is served (the reference's CPU build lists a fixed set)
SUPPORTED = tuple(range(1, MAX_MULT + 1))
MATRIX_COMPLEX, U_REAL, CONJ_U, OUT_REAL = 1, 2, 4, 8
MODE = os.environ.get("GM_FUSED_PAIRS", "0")


@functools.cache
def extension(a: int | None = None, b: int | None = None, trunk: int | None = None) -> Any:
    from gm_attention_b200 import _lib
    from gm_attention_b200.nn.ext import PairsExtension

    _lib.lib()
    return PairsExtension()


@dataclass(frozen=True)
class Term:
    """One (n, m, role) pair term: block shape, flags, rows of the readout, phase orders, radial power."""

    n: int
    m: int
    role: str
    flags: int
    a: int
    b: int
    real_head: bool
    rows: slice
    pre_order: int | None
    post_order: int | None
    power: int | None


def plan(kernel: Any) -> list[Term]:
    """The terms in the order of the general kernel's pair loop (reference ``fused_pairs.py:98-123``):
    for every output frequency m, for every input frequency n."""
    cached = kernel.__dict__.get("_fused_plan")
    if cached is not None:
        return cached  # type: ignore[no-any-return]
    terms: list[Term] = []
    for m in kernel.field_type_out.frequencies:
        b = kernel.field_type_out.multiplicity(m)
        for n in kernel.field_type_in.frequencies:
            a = kernel.field_type_in.multiplicity(n)
            if n == 0 and m == 0:
                terms.append(Term(n, m, "real", U_REAL | OUT_REAL, a, b, True, slice(0, a * b), None, None, None))
                continue
            rows, power = kernel._pair_ranges[(n, m, "linear")], kernel._pair_powers[(n, m, "linear")]
            if n == 0:
                terms.append(Term(n, m, "linear", MATRIX_COMPLEX | U_REAL, a, b, False, rows, None, m, power))
            elif m == 0:
                terms.append(Term(n, m, "linear", MATRIX_COMPLEX | CONJ_U | OUT_REAL, a, b, False, rows, n, None, power))
            else:
                terms.append(Term(n, m, "linear", MATRIX_COMPLEX, a, b, False, rows, m - n, None, power))
                terms.append(Term(n, m, "antilinear", MATRIX_COMPLEX | CONJ_U, a, b, False, kernel._pair_ranges[(n, m, "antilinear")],
                                  m + n, None, kernel._pair_powers[(n, m, "antilinear")]))
    kernel.__dict__["_fused_plan"] = terms
    return terms


def enabled(kernel: Any, x: Any, edges: Any) -> bool:
    if MODE == "0":
        return False
    if MODE == "cpu":
        raise RuntimeError("GM_FUSED_PAIRS=cpu is not provided by gm_attention_b200 (no CPU path)")
    if x.device.type != "cuda" or x.dtype not in (torch.float32, torch.float64):
        return False
    head = kernel.complex_head if kernel.complex_head is not None else kernel.real_head
    if not 1 <= head.in_features <= MAX_TRUNK:
        return False
    for term in plan(kernel):
        if not (1 <= term.a <= MAX_MULT and 1 <= term.b <= MAX_MULT):
            return False
        if any(o is not None and abs(o) > edges.max_frequency for o in (term.pre_order, term.post_order)):
            return False
    return True


# ----------------------------------------------------------------------------- the autograd function

#: edges per block of the readout-gradient product (the reference's SPLIT_K_ROWS, ``nn/kernels.py:33``)
GRADIENT_BLOCK_ROWS = 16384


def _complex_of(real_dtype: torch.dtype) -> torch.dtype:
    return torch.complex128 if real_dtype == torch.float64 else torch.complex64


def _none(like: Tensor) -> Tensor:
    return like.new_empty(0)


def _head_rows(term: Term, cw: Tensor | None, cb: Tensor | None, rw: Tensor | None, rb: Tensor | None) -> tuple[Tensor, Tensor]:
    """The readout rows (and bias entries, or an empty tensor) that produce the term's block."""
    weight, bias = (rw, rb) if term.real_head else (cw, cb)
    if weight is None:
        raise RuntimeError(f"term ({term.n}, {term.m}, {term.role}) needs the {'real' if term.real_head else 'complex'} head")
    return weight[term.rows].contiguous(), (_none(weight) if bias is None else bias[term.rows].contiguous())


def _coefficient_product(grad_k: Tensor, operand: Tensor) -> Tensor:
    """``grad_k (width, E) @ operand (E, K) -> (width, K)``, summed over blocks of GRADIENT_BLOCK_ROWS edges (a batched
    product over the whole blocks, one more for the remainder): partial sums of bounded length, as the reference forms them."""
    width, e = grad_k.shape
    blocks = e // GRADIENT_BLOCK_ROWS
    if blocks < 2:
        return grad_k @ operand
    whole = blocks * GRADIENT_BLOCK_ROWS
    left = grad_k[:, :whole].reshape(width, blocks, GRADIENT_BLOCK_ROWS).permute(1, 0, 2)  # (blocks, width, rows): a view
    right = operand[:whole].reshape(blocks, GRADIENT_BLOCK_ROWS, operand.shape[1])
    total = torch.bmm(left, right).sum(0)
    if whole < e:
        total = total + grad_k[:, whole:] @ operand[whole:]
    return total


class _FusedPairs(torch.autograd.Function):
    """Every pair term of one general-kernel call (reference ``fused_pairs.py:156-238``)."""

    @staticmethod
    def forward(ctx: Any, hidden: Tensor, complex_weight: Tensor | None, complex_bias: Tensor | None, real_weight: Tensor | None,  # type: ignore[override]
                real_bias: Tensor | None, meta: dict[str, Any], phases: tuple[Tensor, ...], scales: tuple[Tensor, ...],
                *vectors: Tensor) -> tuple[Tensor, ...]:
        ext = extension()
        e = hidden.shape[0]
        outputs = [torch.zeros(e, meta["out_multiplicity"][m], dtype=hidden.dtype if m == 0 else _complex_of(hidden.dtype), device=hidden.device)
                   for m in meta["out_frequencies"]]
        for term, (pre, post, power) in zip(meta["terms"], meta["tables"], strict=True):
            weight, bias = _head_rows(term, complex_weight, complex_bias, real_weight, real_bias)
            ext.forward(hidden, weight, bias, vectors[meta["in_index"][term.n]],
                        _none(hidden) if pre is None else phases[pre], _none(hidden) if post is None else phases[post],
                        _none(hidden) if power is None else scales[power], outputs[meta["out_index"][term.m]], term.a, term.b, term.flags)
        ctx.save_for_backward(hidden, complex_weight, complex_bias, real_weight, real_bias, *phases, *scales, *vectors)
        ctx.meta, ctx.sizes = meta, (len(phases), len(scales))
        return tuple(outputs)

    @staticmethod
    def backward(ctx: Any, *grad_outputs: Tensor | None) -> tuple[Any, ...]:  # type: ignore[override]
        meta = ctx.meta
        n_phases, n_scales = ctx.sizes
        hidden, cw, cb, rw, rb, *rest = ctx.saved_tensors
        phases, scales, vectors = rest[:n_phases], rest[n_phases:n_phases + n_scales], rest[n_phases + n_scales:]
        ext = extension()
        e = hidden.shape[0]
        upstream = []
        for g, m in zip(grad_outputs, meta["out_frequencies"], strict=True):
            if g is None:
                g = torch.zeros(e, meta["out_multiplicity"][m], dtype=hidden.dtype if m == 0 else _complex_of(hidden.dtype), device=hidden.device)
            upstream.append(g.contiguous())
        grad_hidden = torch.zeros_like(hidden)
        grad_vectors = [torch.zeros_like(v) for v in vectors]
        # coefficient gradients, coefficient-major (width, E): a term's rows are one contiguous slab
        slabs = {True: None if rw is None else hidden.new_empty(rw.shape[0], e), False: None if cw is None else hidden.new_empty(cw.shape[0], e)}
        for term, (pre, post, power) in zip(meta["terms"], meta["tables"], strict=True):
            weight, bias = _head_rows(term, cw, cb, rw, rb)
            slot = meta["in_index"][term.n]
            ext.backward(hidden, weight, bias, vectors[slot], _none(hidden) if pre is None else phases[pre],
                         _none(hidden) if post is None else phases[post], _none(hidden) if power is None else scales[power],
                         upstream[meta["out_index"][term.m]], grad_vectors[slot], grad_hidden, slabs[term.real_head][term.rows],
                         term.a, term.b, term.flags)
        # d weight = grad_k hidden, d bias = grad_k 1: one product against [hidden | 1]
        any_bias = cb is not None or rb is not None
        operand = torch.cat((hidden, hidden.new_ones(e, 1)), 1) if any_bias else hidden

        def readout_gradients(grad_k: Tensor | None, bias: Tensor | None) -> tuple[Tensor | None, Tensor | None]:
            if grad_k is None:
                return None, None
            product = _coefficient_product(grad_k, operand)
            if not any_bias:
                return product, None
            return product[:, :-1], (product[:, -1] if bias is not None else None)

        grad_cw, grad_cb = readout_gradients(slabs[False], cb)
        grad_rw, grad_rb = readout_gradients(slabs[True], rb)
        return (grad_hidden, grad_cw, grad_cb, grad_rw, grad_rb, None, None, None, *grad_vectors)


# ----------------------------------------------------------------------------- node-level fields: the factored form

#: nodes per partial sum of the readout's gradient
NODE_CHUNK = 128
#: widest packed node field gm_node_products_* take (its rows are staged in shared memory)
MAX_NODE_WIDTH = 2048


class NodeProducts(torch.autograd.Function):
    """``(x (N, D), complex / real readout) -> zc (N, k, wc, 2), zr (N, k, wr)``: every block's ``Z_t = M_t x~``."""

    @staticmethod
    def forward(ctx: Any, x: Tensor, cw: Tensor | None, cb: Tensor | None, rw: Tensor | None, rb: Tensor | None,  # type: ignore[override]
                desc: Tensor, k: int, wc: int, wr: int) -> tuple[Tensor, Tensor]:
        from gm_attention_b200 import _lib

        x, cw, cb, rw, rb = (None if t is None else t.contiguous() for t in (x, cw, cb, rw, rb))
        zc, zr = x.new_empty(x.shape[0], k, wc, 2), x.new_empty(x.shape[0], k, wr)
        with torch.cuda.device(x.device):
            _lib.call("gm_node_products_forward", *(_lib.ptr(t) for t in (x, cw, cb, rw, rb, desc)), x.shape[0], desc.shape[0], x.shape[1], k, wc, wr,
                      _lib.dtype_code(x.dtype), _lib.ptr(zc), _lib.ptr(zr), _lib.stream(x.device))
        ctx.save_for_backward(x, cw, cb, rw, rb, desc)
        return zc, zr

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx: Any, dzc: Tensor, dzr: Tensor) -> tuple[Any, ...]:  # type: ignore[override]
        from gm_attention_b200 import _lib

        x, cw, cb, rw, rb, desc = ctx.saved_tensors
        dzc, dzr = dzc.contiguous(), dzr.contiguous()
        k, wc, wr = dzc.shape[1], dzc.shape[2], dzr.shape[2]
        chunks = -(-x.shape[0] // NODE_CHUNK)
        rows = [0 if w is None else w.shape[0] for w in (cw, rw)]
        dx = torch.empty_like(x)
        parts = [x.new_zeros(chunks, r, k) for r in rows]
        with torch.cuda.device(x.device):
            _lib.call("gm_node_products_backward", *(_lib.ptr(t) for t in (x, cw, cb, rw, rb, desc, dzc, dzr)), x.shape[0], desc.shape[0], x.shape[1],
                      k, wc, wr, *rows, NODE_CHUNK, _lib.dtype_code(x.dtype), _lib.ptr(dx), _lib.ptr(parts[0]), _lib.ptr(parts[1]),
                      _lib.stream(x.device))
        grads: list[Tensor | None] = []
        for part, w, b in ((parts[0], cw, cb), (parts[1], rw, rb)):
            total = None if w is None else part.sum(0)
            grads += [None if total is None else total[:, 1:], None if b is None else total[:, 0]]  # type: ignore[index]
        return (dx, *grads, None, None, None, None)


@dataclass(frozen=True)
class NodePlan:
    """What the node-level route knows of a kernel from its terms alone."""

    served: bool  # the terms are within the bounds of the pair terms and of the route's kernels, their readout rows plain runs
    factored: Any = None  # the factored plan of the terms
    rows: tuple = ()  # descriptor rows of the node products
    inputs: tuple = ()  # (frequency, multiplicity) of the input type, in its order
    needed: tuple = ()  # (real head?, readout rows its terms read)
    width: int = 0  # packed columns of the products, padded to whole 16-byte vectors
    order: int = 0  # highest order of the phase tables
    power: int = 0  # highest column of the radial table


def _node_plan(kernel: Any, terms: list[Term]) -> NodePlan:
    """The kernel's :class:`NodePlan`, kept on it like the terms."""
    cached = kernel.__dict__.get("_fused_node_plan")
    if cached is None:
        cached = kernel.__dict__["_fused_node_plan"] = _built_node_plan(kernel, terms)
    return cached  # type: ignore[no-any-return]


def _built_node_plan(kernel: Any, terms: list[Term]) -> NodePlan:
    from gm_attention_b200.fields import FieldType
    from gm_attention_b200.nn import fused_factored as ff

    # the pair terms' own bounds first: what they refuse is refused on any graph
    if not terms or any(not (1 <= t.a <= MAX_MULT and 1 <= t.b <= MAX_MULT) for t in terms):
        return NodePlan(False)
    # the rows' layout is this route's own: what the kernel's field type is asked is what the pair terms ask
    p = ff.plan_blocks([(t.n, t.m, t.role) for t in terms], FieldType({t.m: t.b for t in terms}),
                       {(t.n, t.m, t.role): t.power for t in terms if t.power is not None})
    inputs = tuple((n, kernel.field_type_in.multiplicity(n)) for n in kernel.field_type_in.frequencies)
    offsets, at = {}, 0
    for n, copies in inputs:
        offsets[n] = at
        at += copies * (1 if n == 0 else 2)
    by_block = {(t.n, t.m, t.role): t for t in terms}
    rows = []
    for b in p.blocks:
        t = by_block[b.block]
        operand = 0 if t.flags & U_REAL else (2 if t.flags & CONJ_U else 1)
        rows.append((b.kind, b.z_offset, t.b, t.a, offsets[t.n], operand, t.rows.start or 0, 0))
    needed: dict[bool, int] = {}
    plain = True
    for t in terms:
        start, width = t.rows.start or 0, t.a * t.b * (2 if t.flags & MATRIX_COMPLEX else 1)
        plain = plain and start >= 0 and t.rows.stop == start + width and t.rows.step in (None, 1)
        needed[t.real_head] = max(needed.get(t.real_head, 0), start + width)
    powers = [b.power for b in p.blocks]
    served = plain and at <= MAX_NODE_WIDTH and p.d_out <= ff.MAX_OUT and p.max_bm <= ff.MAX_BM and min(powers) >= 0
    return NodePlan(served, p, tuple(rows), inputs, tuple(needed.items()), -(-(2 * p.wc + p.wr) // 4) * 4,
                    max(max(abs(b.angular), abs(b.transport)) for b in p.blocks), max(powers))


def _readouts_fit(kernel: Any, needed: tuple, hidden: Tensor) -> bool:
    """Whether both heads hold, in the trunk's dtype and place, the rows their terms read."""
    for real, rows in needed:
        head = kernel.real_head if real else kernel.complex_head
        weight, bias = getattr(head, "weight", None), getattr(head, "bias", None)
        if weight is None or weight.dim() != 2 or weight.shape[0] < rows or weight.shape[1] != hidden.shape[1]:
            return False
        if weight.dtype != hidden.dtype or weight.device != hidden.device:
            return False
        if bias is not None and (bias.shape != weight.shape[:1] or bias.dtype != hidden.dtype or bias.device != hidden.device):
            return False
    return True


def _products_repaid(n_nodes: int, n_edges: int) -> bool:
    """Whether a node's products serve enough edges, so that no kernel measured loses by the factored form, a first pass
    on an edge set (0.25 to 0.5 ms for its grouping) included.  Forward and backward, float32, trunk 16, ms as factored form /
    pair terms.  Beyond 8 192 nodes the narrow kernels on many nodes decide: {2, 2} -> {8, 8} on 80 000 nodes 2.91 / 2.24 at
    4.9 edges per node, 3.16 / 2.90 at 8.8, 3.26 / 3.34 at 10.9; others would gain earlier ({16, 16} -> {8, 8} there 4.03 / 4.88 at
    4.9, on 30 000 nodes 1.72 / 2.70; {8, 8, 8} -> {4, 4, 4} 1.71 / 2.72).  Up to 8 192 nodes both wait for their launches, of which the
    factored form has fewer: {2, 2} -> {8, 8} 1.16 / 1.37 from 1 to 8 edges per node, three frequencies 1.24 / 2.05."""
    return n_edges >= (4 if n_nodes <= 8192 else 10) * n_nodes


def _field_fits(inputs: tuple, values: list[Tensor], n_nodes: int, like: Tensor) -> bool:
    """Whether the coefficients are ``(N, a_0)`` reals and ``(N, a_n)`` complex numbers or ``(N, a_n, 2)`` pairs, in ``like``'s
    real dtype and place."""
    for (n, copies), v in zip(inputs, values, strict=True):
        as_complex = v.is_complex()
        if v.device != like.device or v.dtype != (_complex_of(like.dtype) if as_complex else like.dtype):
            return False
        if (n == 0 and as_complex) or v.shape != ((n_nodes, copies) if n == 0 or as_complex else (n_nodes, copies, 2)):
            return False
    return True


def _uploaded(kernel: Any, device: torch.device) -> tuple[Tensor, Tensor] | None:
    """The kernel's descriptors on ``device``, if they are there: a kernel loaded from a file may bring others' under its name."""
    from gm_attention_b200.nn import fused_factored as ff

    found = kernel.__dict__.get("_fused_node_descriptors", {}).get(str(device))
    return found if found is not None and all(ff.is_on(t, device) for t in found) else None


def _prepared(kernel: Any, edges: Any, device: torch.device) -> bool:
    """Whether an earlier call left the kernel's descriptors on the device and grouped these edges by source."""
    from gm_attention_b200.nn import fused_factored as ff

    return _uploaded(kernel, device) is not None and ff.cached_grouping(edges, device) is not None


def _factored_inputs(kernel: Any, x: Any, edges: Any, hidden: Tensor, terms: list[Term], table: Tensor | None) -> tuple | None:
    """What the factored form needs of this call, or ``None`` where the pair terms serve it: an edge-level or mixed field,
    too few edges per node (:func:`_products_repaid`), phase tables that are not plain per-edge
    ``angular_phases`` / ``transport_phases`` of one width or that want gradients, sizes beyond the factored kernels, and any
    tensor that does not have the shape, dtype or place the kernels read it with."""
    from gm_attention_b200.nn import fused_factored as ff

    device, dtype = hidden.device, hidden.dtype
    if device.type != "cuda" or dtype not in (torch.float32, torch.float64) or hidden.dim() != 2 or not 1 <= hidden.shape[1] <= MAX_TRUNK:
        return None
    node = _node_plan(kernel, terms)
    k = hidden.shape[1] + 1
    if not node.served or k > ff.MAX_K or k * node.width > ff.MAX_KC:
        return None
    values = [x[n] for n, _ in node.inputs]
    n_nodes, n_edges = int(values[0].shape[0]), int(edges.n_edges)
    if n_nodes == n_edges or n_nodes == 0 or not _products_repaid(n_nodes, n_edges) or not _field_fits(node.inputs, values, n_nodes, hidden):
        return None
    angular, transport = getattr(edges, "angular_phases", None), getattr(edges, "transport_phases", None)
    if angular is None or transport is None or not hasattr(edges, "edge_index") or not hasattr(edges, "row_ptr"):
        return None
    for phases in (angular, transport):
        if phases.dim() != 2 or phases.shape != angular.shape or phases.dtype != _complex_of(dtype) or phases.device != device or phases.requires_grad:
            return None
    source, index = edges.source_index, edges.edge_index
    if source.shape != (n_edges,) or source.dtype != torch.int64 or source.device != device:
        return None
    if index is not edges.edge_index or ff.version(source) < 0 or source.untyped_storage().data_ptr() != index.untyped_storage().data_ptr():
        return None  # no grouping to keep, or one whose key could not tell other indices: an edge_index formed on every access,
        # inference tensors, sources kept apart from edge_index
    if hidden.shape[0] != n_edges or angular.shape[0] != n_edges or node.order >= angular.shape[1] or not _readouts_fit(kernel, node.needed, hidden):
        return None
    scales = hidden.new_ones(n_edges, 1) if table is None else table.detach()  # table None: no block has a scale
    if scales.dim() != 2 or scales.shape[0] != n_edges or scales.shape[1] <= node.power or scales.dtype != dtype or scales.device != device:
        return None
    if torch.cuda.is_current_stream_capturing() and not _prepared(kernel, edges, device):
        return None  # grouping the edges by source and uploading the descriptors synchronise: not while a graph is captured
    return node, values, angular, transport, scales, source, n_nodes


def _forward_factored(kernel: Any, x: Any, edges: Any, hidden: Tensor, found: tuple) -> Any:
    from gm_attention_b200.nn import fused_factored as ff

    node, values, angular, transport, scales, source, n_nodes = found
    p = node.factored
    device = hidden.device
    # the kernels read memory: conjugations and signs that torch has put off are carried out first
    flat = [(torch.view_as_real(v.resolve_conj()) if v.is_complex() else v.resolve_neg()).reshape(n_nodes, -1) for v in values]
    packed = flat[0] if len(flat) == 1 else torch.cat(flat, 1)
    uploaded = _uploaded(kernel, device)
    if uploaded is None:
        uploaded = (torch.tensor(node.rows, dtype=torch.int32, device=device).reshape(-1, 8),
                    torch.tensor([b.row() for b in p.blocks], dtype=torch.int32, device=device).reshape(-1, 8))
        kernel.__dict__.setdefault("_fused_node_descriptors", {})[str(device)] = uploaded
    node_desc, desc = uploaded
    params = [q for head in (kernel.complex_head, kernel.real_head) for q in ((None, None) if head is None else (head.weight, head.bias))]
    zc, zr = NodeProducts.apply(packed, *params, node_desc, hidden.shape[1] + 1, p.wc, p.wr)
    source = source.contiguous()
    order, group_ptr, group_source = ff.grouping_for(edges, source).require_nodes(n_nodes)
    out = ff.Factored.apply(hidden, zc, zr, *(torch.view_as_real(t.resolve_conj().contiguous()) for t in (angular, transport)), scales.resolve_neg().contiguous(),
                            desc, source, order, group_ptr, group_source, p.d_out, p.max_bm, True)
    widths = {m: kernel.field_type_out.multiplicity(m) * (2 if m else 1) for m in sorted(kernel.field_type_out.frequencies)}
    parts = dict(zip(widths, out.split(list(widths.values()), 1), strict=True))
    return {m: parts[m].contiguous() if m == 0 else parts[m].contiguous().reshape(hidden.shape[0], -1, 2) for m in kernel.field_type_out.frequencies}


# ----------------------------------------------------------------------------- driver entry

def _trunk_output(kernel: Any, distances: Tensor) -> Tensor:
    """Radial basis then the Linear / SiLU trunk, ``(E, trunk width)`` (reference ``nn/kernels.py:108-117, 605-607``)."""
    hidden = kernel.radial_basis(distances)
    for layer in kernel.radial_trunk:
        hidden = layer(hidden)
    return hidden.contiguous()


def _transported_vectors(x: Any, edges: Any, frequencies: list[int]) -> tuple[Tensor, ...]:
    """Per input frequency the source node's coefficients in the TARGET gauge, per edge: ``e^{i n gamma} x_n[source]``
    as ``(E, a_n)`` complex, ``x_0[source]`` as ``(E, a_0)`` real (reference ``nn/kernels.py:156-189``).  ``x`` is an
    edge-level field when its leading size is the edge count, a node-level field otherwise."""
    out = []
    for n in frequencies:
        values = x[n]
        if values.shape[0] != edges.n_edges:
            values = values.index_select(0, edges.source_index)
        if n == 0:
            out.append(values.contiguous())
        else:
            z = torch.view_as_complex(values.contiguous()) if not values.is_complex() else values
            out.append((edges.transport_harmonic(n).unsqueeze(-1) * z).contiguous())
    return tuple(out)


def forward_general(kernel: Any, x: Any, edges: Any) -> Any:
    """``kernel._forward_general(x, edges)`` through the fused terms (reference ``fused_pairs.py:247-295``).

    ``kernel`` is the reference's ``SO2SteerableKernel`` or any object with its attributes (``field_type_in / _out``,
    ``radial_basis``, ``radial_trunk``, ``complex_head`` / ``real_head``, ``_pair_ranges``, ``_pair_powers``,
    ``_radial_powers``); ``x`` maps a frequency to ``(E or N, a_n[, 2])`` coefficients and carries ``field_type``; the
    result is built with ``type(x)(field_type_out, {m: coefficients})``."""
    terms = plan(kernel)
    with torch.profiler.record_function("gm::kernel/radial"):
        hidden = _trunk_output(kernel, edges.distances)
    powers = sorted({t.power for t in terms if t.power is not None})
    table = kernel._radial_powers(edges.distances) if powers else None
    found = _factored_inputs(kernel, x, edges, hidden, terms, table)
    if found is not None:
        with torch.profiler.record_function("gm::kernel/pairs"):
            return type(x)(kernel.field_type_out, _forward_factored(kernel, x, edges, hidden, found))
    in_frequencies, out_frequencies = list(kernel.field_type_in.frequencies), list(kernel.field_type_out.frequencies)
    with torch.profiler.record_function("gm::transport"):
        vectors = _transported_vectors(x, edges, in_frequencies)
    orders = sorted({o for t in terms for o in (t.pre_order, t.post_order) if o is not None})
    phases = tuple(edges.angular_harmonic(o).contiguous() for o in orders)
    scales = tuple(table[:, p].contiguous() for p in powers)
    where_order, where_power = {o: i for i, o in enumerate(orders)}, {p: i for i, p in enumerate(powers)}
    meta = {
        "terms": terms,
        "tables": [(where_order.get(t.pre_order), where_order.get(t.post_order), where_power.get(t.power)) for t in terms],
        "in_index": {n: i for i, n in enumerate(in_frequencies)},
        "out_index": {m: i for i, m in enumerate(out_frequencies)},
        "out_frequencies": out_frequencies,
        "out_multiplicity": {m: kernel.field_type_out.multiplicity(m) for m in out_frequencies},
    }
    heads = (kernel.complex_head, kernel.real_head)
    params = [p for head in heads for p in ((None, None) if head is None else (head.weight, head.bias))]
    with torch.profiler.record_function("gm::kernel/pairs"):
        outputs = _FusedPairs.apply(hidden, *params, meta, phases, scales, *vectors)
    return type(x)(kernel.field_type_out, {m: (out if m == 0 else torch.view_as_real(out)) for m, out in zip(out_frequencies, outputs, strict=True)})


__all__ = ["MODE", "SUPPORTED", "Term", "enabled", "extension", "forward_general", "plan"]
