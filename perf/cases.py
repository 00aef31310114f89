"""Performance cases: what a user of this package has it do, one pass each through the public entry points.

A case is a dict of plain values; ``op`` says which part of the package it drives:

``attention``          the fused layer on an equiangular lattice (``GaugeAttention`` over ``LatticeTables``)
``graph_attention``    the same layer on a point set without longitude symmetry (``GaugeAttention`` over ``AttentionTables``)
``scores``             scores + neighbourhood softmax, the drop-in op (``fused_attention.softmax``)
``depthwise``          depthwise steerable convolution under per-edge coefficients, the drop-in op (``forward_depthwise``)
``lattice_depthwise``  depthwise convolution with its radial network on a lattice (``RadialCoefficients`` + ``lattice_depthwise``)
``factored``           factored steerable kernel with the weighted sum per target (``fused_factored.forward_aggregated``)
``pairs``              pair terms of the general steerable kernel (``fused_pairs.forward_general``)

``train`` passes run forward and backward and return the output and every gradient; the others run forward only.
"""

from __future__ import annotations

import math
from types import SimpleNamespace
from typing import Any

import numpy as np
import torch
from torch import nn

from gm_attention_b200.attention import AttentionTables, GaugeAttention, build_lattice_tables
from gm_attention_b200.fields import FeatureField, FieldType
from gm_attention_b200.geometry import compute_edge_geometry, midpoint_lattice
from gm_attention_b200.nn import fused_attention, fused_factored, fused_pairs
from gm_attention_b200.nn.lattice_depthwise import RadialCoefficients, conv_tables, lattice_depthwise

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
TRUNK = 16  # width of the radial networks' hidden layer
BASIS = 4  # Gaussian rings of the radial networks


def listed() -> list[dict[str, Any]]:
    return [
        # the smallest layer of the benchmark family (32 x 64, batch 2, 2 heads): a training pass that is all launches and latency
        _attention("attention_f32_32x64", 32, 64, 2, batch=2, heads=2, copies=4, top=2, dtype="f32"),
        # the middle configuration, four frequencies (m <= 3), in both storage types
        _attention("attention_f32_128x256", 128, 256, 3, batch=4, heads=4, copies=8, top=3, dtype="f32"),
        _attention("attention_bf16_128x256", 128, 256, 3, batch=4, heads=4, copies=8, top=3, dtype="bf16"),
        # the headline configuration: the largest training pass
        _attention("attention_bf16_256x512", 256, 512, 3, batch=8, heads=4, copies=16, top=2, dtype="bf16"),
        # inference (no gradients) on a lattice no tile divides, odd number of rows, smooth window, odd batch
        _attention("infer_bf16_91x180", 91, 180, 2.5, batch=3, heads=4, copies=16, top=2, dtype="bf16", window="quartic", train=False),
        # training on a point set without longitude symmetry (a spiral lattice of as many points as a subdivided icosahedron)
        dict(name="graph_f32_10242", op="graph_attention", points=10242, radius=0.12, batch=2, heads=4, copies=8, top=2, dtype="f32",
             window="hard", train=True),
        # the drop-in operators at the size their table in the benchmark uses
        dict(name="scores_f32_128x256", op="scores", rows=128, columns=256, radius=3.0, heads=4, copies=8, top=3, dtype="f32", train=True),
        dict(name="depthwise_f32_128x256", op="depthwise", rows=128, columns=256, radius=3.0, copies=16, top=2, dtype="f32", train=True),
        # the depthwise layer with its radial network: the large configuration in bf16, and a small odd one in float32
        dict(name="convolution_bf16_256x512", op="lattice_depthwise", rows=256, columns=512, radius=4.0, batch=4, copies=64, top=2,
             dtype="bf16", train=True),
        dict(name="convolution_f32_45x88", op="lattice_depthwise", rows=45, columns=88, radius=4.0, batch=3, copies=32, top=2,
             dtype="f32", train=True),
        # the value kernel {8, 8, 8} -> {4, 4, 4} with a trunk of 16: factored form at the benchmark's size, pair form on a coarser level
        dict(name="factored_f32_128x256", op="factored", rows=128, columns=256, radius=3.0, copies_in=8, copies_out=4, top=2, dtype="f32",
             train=True),
        dict(name="pairs_f32_64x128", op="pairs", rows=64, columns=128, radius=3.0, copies_in=8, copies_out=4, top=2, dtype="f32",
             train=True),
    ]


def _attention(name: str, rows: int, columns: int, radius: float, *, batch: int, heads: int, copies: int, top: int, dtype: str,
               window: str = "hard", train: bool = True) -> dict[str, Any]:
    return dict(name=name, op="attention", rows=rows, columns=columns, radius=float(radius), batch=batch, heads=heads, copies=copies,
                top=top, dtype=dtype, window=window, train=train)


def draw(rng: Any) -> dict[str, Any]:
    """One more case of the same ranges; sizes are drawn over their logarithm, and a draw that would cost more than the
    largest listed case of its kind is drawn again."""
    op = rng.choice(["attention"] * 5 + ["graph_attention", "scores", "depthwise", "lattice_depthwise", "lattice_depthwise", "factored", "pairs"])
    dtype = rng.choice(["f32", "bf16", "bf16"]) if op in ("attention", "lattice_depthwise") else "f32"
    # multiply-adds (attention, factored kernel, pair terms) and coefficients (depthwise) a draw may hold: below its kind's largest listed case
    most = {("attention", "f32"): 8e9, ("attention", "bf16"): 1.2e11, ("lattice_depthwise", "f32"): 6e9, ("lattice_depthwise", "bf16"): 5e10,
            ("graph_attention", "f32"): 5e8, ("scores", "f32"): 3e9, ("depthwise", "f32"): 4.2e8, ("factored", "f32"): 4.8e9,
            ("pairs", "f32"): 1.0e10}[op, dtype]
    while True:
        rows = _spread(rng, 24, 256 if op in ("attention", "lattice_depthwise") else 128)
        columns = 2 * rows if rng.random() < 0.5 else 2 * _spread(rng, max(24, rows // 2), 2 * rows)
        lattice = dict(rows=rows, columns=columns, radius=rng.choice([2.0, 2.5, 3.0, 3.0, 4.0]))
        if op == "attention":
            case = dict(op=op, **lattice, batch=rng.randint(1, 8), heads=rng.choice([1, 2, 4, 4, 8]), copies=rng.choice([4, 5, 8, 8, 12, 16, 16]),
                        top=rng.choice([1, 2, 2, 3]), dtype=dtype, window=rng.choice(["hard", "hard", "quartic"]), train=rng.random() < 0.75)
            case["columns"] = max(columns, 48)
            if case["top"] == 3:  # four frequencies come with the narrower heads
                case["copies"] = min(case["copies"], 8)
        elif op == "graph_attention":
            points = _spread(rng, 640, 12000)
            degree = rng.uniform(12.0, 48.0)
            case = dict(op=op, points=points, radius=math.acos(1.0 - 2.0 * degree / points), batch=rng.randint(1, 4), heads=rng.choice([1, 2, 4, 8]),
                        copies=rng.choice([4, 5, 8]), top=rng.choice([1, 2, 3]), dtype=dtype, window=rng.choice(["hard", "quartic"]), train=True)
        elif op == "scores":
            case = dict(op=op, **lattice, heads=rng.choice([1, 2, 4, 8]), copies=rng.choice([4, 5, 8, 16]), top=rng.choice([1, 2, 3]), dtype=dtype, train=True)
            if _width(case) > fused_attention.MAX_D:
                continue
        elif op == "depthwise":
            case = dict(op=op, **lattice, copies=rng.choice([4, 7, 8, 16, 32]), top=rng.choice([1, 2]), dtype=dtype, train=True)
        elif op == "lattice_depthwise":
            case = dict(op=op, **lattice, batch=rng.randint(1, 4), copies=rng.choice([8, 10, 16, 32, 64]), top=rng.choice([1, 2]), dtype=dtype, train=True)
            case["columns"] = max(24, columns // 8 * 8)
        else:
            case = dict(op=op, **lattice, copies_in=rng.choice([4, 6, 8, 16]), copies_out=rng.choice([2, 3, 4, 8]), top=rng.choice([1, 2]), dtype=dtype,
                        train=True)
        if _size(case) <= most:
            return case


def _spread(rng: Any, low: int, high: int) -> int:
    return round(math.exp(rng.uniform(math.log(low), math.log(high))))


# --------------------------------------------------------------------------- shapes

def _field_type(copies: int, top: int) -> FieldType:
    return FieldType.uniform(copies, top)


def _width(case: dict[str, Any]) -> int:
    return case["copies"] * (1 + 2 * case["top"]) * case.get("heads", 1)


def _edges(case: dict[str, Any]) -> int:
    """Edges of one sample: counted row pair by row pair on a lattice, expected on the spiral point set."""
    if case["op"] == "graph_attention":
        return round(case["points"] ** 2 * (1.0 - math.cos(case["radius"])) / 2.0)
    return _lattice_entries(case) * case["columns"]


def _lattice_entries(case: dict[str, Any]) -> int:
    """Neighbours summed over one target per lattice row."""
    rows, columns, radius = case["rows"], case["columns"], case["radius"] * math.pi / case["rows"] + 1e-10
    theta = (np.arange(rows) + 0.5) * math.pi / rows
    cosine = (math.cos(radius) - np.outer(np.cos(theta), np.cos(theta))) / np.outer(np.sin(theta), np.sin(theta))
    reach = np.arccos(np.clip(cosine, -1.0, 1.0)) * columns / (2.0 * math.pi)
    counts = np.where(cosine > 1.0, 0, np.minimum(2 * np.floor(reach) + 1, columns))
    return int(counts.sum())


def _blocks(case: dict[str, Any]) -> tuple[list[tuple[int, int, str]], dict[tuple[int, int, str], int]]:
    """Coefficient blocks of the steerable kernel in readout order, with their radial powers."""
    blocks: list[tuple[int, int, str]] = [(0, 0, "real")]
    powers = {}
    for n in range(case["top"] + 1):
        for m in range(case["top"] + 1):
            if n == 0 and m == 0:
                continue
            for role, power in [("linear", abs(m - n))] + ([("antilinear", m + n)] if n and m else []):
                blocks.append((n, m, role))
                powers[(n, m, role)] = power
    return blocks, powers


def _size(case: dict[str, Any]) -> float:
    op, edges = case["op"], _edges(case) * case.get("batch", 1)
    if op in ("attention", "graph_attention", "scores"):
        return edges * _width(case) * (3 if case["train"] else 1)
    if op == "depthwise":
        return edges * case["copies"] * (1 + 4 * case["top"])
    if op == "lattice_depthwise":
        return edges * case["copies"] * (1 + 4 * case["top"])
    blocks = len(_blocks(case)[0])
    if op == "factored":
        return edges * (TRUNK + 1) * (2 * blocks - 1) * case["copies_out"]
    return edges * (TRUNK + 1) * (2 * blocks - 1) * case["copies_in"] * case["copies_out"]


# --------------------------------------------------------------------------- what a user's program holds before the call

class _SteerableKernel(nn.Module):
    """What the steerable-kernel drivers read of a kernel: field types, the readout's block layout, the radial network."""

    def __init__(self, case: dict[str, Any], cutoff: float) -> None:
        super().__init__()
        self.field_type_in, self.field_type_out = _field_type(case["copies_in"], case["top"]), _field_type(case["copies_out"], case["top"])
        block_list, self._pair_powers = _blocks(case)
        self._block_list, self.cutoff = block_list, cutoff
        self.radial_basis = _RadialBasis(cutoff)
        self.radial_trunk = nn.Sequential(nn.Linear(BASIS, TRUNK), nn.SiLU())
        entries = case["copies_in"] * case["copies_out"]
        self._pair_ranges = {b: slice(2 * entries * i, 2 * entries * (i + 1)) for i, b in enumerate(b for b in block_list if b[2] != "real")}
        self.complex_head = nn.Linear(TRUNK, 2 * entries * len(self._pair_ranges))
        self.real_head = nn.Linear(TRUNK, entries)

    def _blocks(self) -> list[tuple[int, int, str]]:
        return self._block_list

    def _radial_powers(self, distances: torch.Tensor) -> torch.Tensor:
        rho = distances / self.cutoff
        return torch.stack([rho**p for p in range(max(self._pair_powers.values()) + 1)], -1)

    def _trunk_hidden(self, edges: Any) -> torch.Tensor:
        return self.radial_trunk(self.radial_basis(edges.distances))


class _RadialBasis(nn.Module):
    """Gaussian rings in the squared relative distance."""

    def __init__(self, cutoff: float) -> None:
        super().__init__()
        self.cutoff = cutoff
        self.register_buffer("centers", torch.linspace(0.0, 1.0, BASIS))

    def forward(self, distances: torch.Tensor) -> torch.Tensor:
        offset = (distances / self.cutoff).square().unsqueeze(-1) - self.centers
        return torch.exp(-0.5 * (offset * (BASIS - 1)).square())


def _spiral(points: int) -> SimpleNamespace:
    """Points of a golden-angle spiral with equal quadrature weights and (east, north) frames."""
    device = torch.device("cuda")
    index = torch.arange(points, dtype=torch.float64, device=device)
    z = 1.0 - (2.0 * index + 1.0) / points
    phi = index * (math.pi * (3.0 - math.sqrt(5.0)))
    s = torch.sqrt(1.0 - z * z)
    nodes = torch.stack([s * phi.cos(), s * phi.sin(), z], -1)
    east = torch.stack([-phi.sin(), phi.cos(), torch.zeros_like(phi)], -1)
    north = torch.stack([-z * phi.cos(), -z * phi.sin(), s], -1)
    weights = torch.full((points,), 4.0 * math.pi / points, dtype=torch.float64, device=device)
    return SimpleNamespace(nodes=nodes, exact_nodes=nodes, quadrature_weights=weights, frames=torch.stack([east, north], -1))


def prepare(case: dict[str, Any], seed: int) -> dict[str, Any]:
    device = torch.device("cuda")
    generator = torch.Generator(device=device).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    op, top, train = case["op"], case["top"], case["train"]

    def normal(*shape: int, grad: bool = False, scale: float = 1.0, kind: torch.dtype = dtype) -> torch.Tensor:
        values = torch.randn(*shape, generator=generator, device=device, dtype=torch.float32)
        return (values if scale == 1.0 else values * scale).to(kind).requires_grad_(grad)

    if op == "graph_attention":
        grid, radius = _spiral(case["points"]), case["radius"]
        nodes = case["points"]
    else:
        grid, radius = midpoint_lattice(case["rows"], case["columns"], device), case["radius"] * math.pi / case["rows"]
        nodes = case["rows"] * case["columns"]
    orders = top if op in ("attention", "graph_attention", "scores") else 2 * top
    edges = compute_edge_geometry(grid, grid.frames, radius, max_frequency=orders, dtype=torch.float32)
    state: dict[str, Any] = {"op": op, "train": train}

    if op in ("attention", "graph_attention", "scores"):
        head, heads = _field_type(case["copies"], top), case["heads"]
        window = case.get("window", "hard")
        scale = 1.0 / math.sqrt(head.dimension)
        # the layer's module as the drivers read it
        layer = SimpleNamespace(field_type_attn=head, field_type_in=head.scaled(heads), num_heads=heads, cutoff=radius,
                                heads=[SimpleNamespace(window=window, _score_scale=scale)])
        plan = fused_attention.plan(layer)
        constants = fused_attention.geometry(edges, radius, window, torch.float32)
        batch = case.get("batch", 1)
        if op == "scores":
            state |= {"layer": layer, "edges": edges, "q": normal(nodes, plan.width, grad=True), "k": normal(nodes, plan.width, grad=True),
                      "upstream": normal(edges.n_edges, heads)}
            return state
        tables = AttentionTables(constants.transport, constants.bias, constants.inside, constants.row_ptr, constants.source, plan.rows, heads, scale)
        if op == "attention":
            tables = build_lattice_tables(tables, case["rows"], case["columns"], plan.rows, heads, scale)
        state |= {"tables": tables} | {name: normal(batch * nodes, plan.width, grad=train) for name in ("q", "k", "v")}
        if train:
            state["upstream"] = normal(batch * nodes, plan.width)
        return state

    if op in ("depthwise", "lattice_depthwise"):
        field = _field_type(case["copies"], top)
        layer = SimpleNamespace(kernel=SimpleNamespace(field_type=field), cutoff=radius, window="hard", normalize=False, eps=1e-6)
        plan = fused_attention.plan_depthwise(layer)
        constants = fused_attention.geometry(edges, radius, "hard", torch.float32)
        if op == "depthwise":
            state |= {"layer": layer, "edges": edges, "v": normal(nodes, plan.width, grad=True), "upstream": normal(nodes, plan.width),
                      "rc": normal(1, edges.n_edges, plan.a_0, grad=True), "cc": normal(1, edges.n_edges, plan.complex_width, grad=True)}
            return state
        batch = case["batch"]
        state["tables"] = conv_tables(constants, edges.distances, constants.weights, plan.rows, case["rows"], case["columns"])
        network = RadialCoefficients(plan.a_0, plan.complex_width, radius, n_radial_basis=BASIS, radial_hidden_features=(TRUNK,), device=device)
        _fill(network, normal)
        state |= {"network": network, "v": normal(batch * nodes, plan.width, grad=True), "upstream": normal(batch * nodes, plan.width)}
        return state

    kernel = _SteerableKernel(case, radius).to(device)
    _fill(kernel, normal)
    state |= {"kernel": kernel, "edges": edges}
    out_width = kernel.field_type_out.dimension
    if op == "factored":
        # the node-side products of the kernel's readout with the field: one (nodes, 1 + trunk, b) mix per block
        b = case["copies_out"]
        products = {block: (normal(nodes, TRUNK + 1, b, grad=True) if block[2] == "real" else
                            torch.view_as_complex(normal(nodes, TRUNK + 1, b, 2)).requires_grad_(True)) for block in kernel._blocks()}
        weights = fused_attention.geometry(edges, radius, "hard", torch.float32).weights
        state |= {"products": products, "weights": weights.clone().requires_grad_(True), "upstream": normal(nodes, out_width)}
        return state
    state["x"] = normal(nodes, kernel.field_type_in.dimension, grad=True)
    state["upstream"] = {m: normal(edges.n_edges, b, *([2] if m else [])) for m, b in kernel.field_type_out.items()}
    return state


def _fill(module: nn.Module, normal: Any) -> None:
    """Parameters ~ N(0, 1 / fan_in) from the case's seed."""
    for parameter in module.parameters():
        fan_in = parameter.shape[1] if parameter.dim() == 2 else parameter.shape[0]
        parameter.data.copy_(normal(*parameter.shape, scale=1.0 / math.sqrt(fan_in), kind=torch.float32))


# --------------------------------------------------------------------------- one pass

def run(state: dict[str, Any]) -> Any:
    op = state["op"]
    if op in ("attention", "graph_attention"):
        q, k, v = state["q"], state["k"], state["v"]
        if not state["train"]:
            with torch.no_grad():
                return GaugeAttention.apply(q, k, v, state["tables"])
        out = GaugeAttention.apply(q, k, v, state["tables"])
        return out.detach(), *torch.autograd.grad(out, (q, k, v), state["upstream"])
    if op == "scores":
        q, k = state["q"], state["k"]
        alpha = fused_attention.softmax(state["layer"], q, k, state["edges"])
        return alpha.detach(), *torch.autograd.grad(alpha, (q, k), state["upstream"])
    if op == "depthwise":
        v, rc, cc = state["v"], state["rc"], state["cc"]
        out = fused_attention.forward_depthwise(state["layer"], v, rc, cc, state["edges"])
        return out.detach(), *torch.autograd.grad(out, (v, rc, cc), state["upstream"])
    if op == "lattice_depthwise":
        v, network, tables = state["v"], state["network"], state["tables"]
        out = lattice_depthwise(v, *network(tables.distances), tables)
        return out.detach(), *torch.autograd.grad(out, (v, *network.parameters()), state["upstream"])
    kernel, edges = state["kernel"], state["edges"]
    if op == "factored":
        products, weights = state["products"], state["weights"]
        out = fused_factored.forward_aggregated(kernel, None, edges, weights, dict(products))
        trained = [*kernel.radial_trunk.parameters(), *products.values(), weights]
        return out.detach(), *torch.autograd.grad(out, trained, state["upstream"])
    x = state["x"]
    out = fused_pairs.forward_general(kernel, FeatureField.from_flat(kernel.field_type_in, x), edges).coefficients
    orders = sorted(out)
    gradients = torch.autograd.grad([out[m] for m in orders], [x, *kernel.parameters()], [state["upstream"][m] for m in orders])
    return *(out[m].detach() for m in orders), *gradients


# --------------------------------------------------------------------------- bounds

def work(case: dict[str, Any]) -> dict[str, float]:
    """Compulsory traffic (every input once, every output once) and arithmetic of one pass.

    A contraction over a head's columns is two operations per scalar copy and eight per complex copy (the transport is
    part of it).  Attention has two of them forward and four backward (d alpha, dq, dk, dv); the lattice layers read
    their tables per (row pair, offset), the other operators read theirs per edge."""
    op, train, top = case["op"], case["train"], case["top"]
    elem = 2 if case["dtype"] == "bf16" else 4
    edges, batch = _edges(case), case.get("batch", 1)
    nodes = case["points"] if op == "graph_attention" else case["rows"] * case["columns"]
    edge_constants = edges * (4 * 2 * (top + 1) + 4 + 1 + 8)  # transport, bias, window flag, source index
    if op in ("attention", "graph_attention", "scores"):
        fields = nodes * batch * _width(case) * elem
        contraction = edges * batch * case["heads"] * case["copies"] * (2 + 8 * top)
        if op == "scores":  # forward: q, k -> alpha; backward: d alpha -> dq, dk
            return {"bytes": 4 * fields + 2 * edges * case["heads"] * 4 + edge_constants, "flops": 3.0 * contraction}
        constants = edge_constants if op == "graph_attention" else _lattice_entries(case) * (8 * top + 4)
        return {"bytes": (8 if train else 4) * fields + constants, "flops": (6.0 if train else 2.0) * contraction}
    if op in ("depthwise", "lattice_depthwise"):
        fields = nodes * batch * case["copies"] * (1 + 2 * top) * elem
        coefficients = case["copies"] * (1 + 4 * top)
        flops = 3.0 * edges * batch * case["copies"] * (2 + 8 * top)  # forward, field gradient, coefficient gradient
        if op == "depthwise":
            tables = edges * (2 * 8 * (2 * top + 1) + 4 + 4 + 8)
            return {"bytes": 4 * fields + 2 * edges * coefficients * 4 + tables, "flops": flops}
        return {"bytes": 4 * fields + _lattice_entries(case) * (4 + 16 * top), "flops": flops}
    blocks = len(_blocks(case)[0])
    out_width = case["copies_out"] * (1 + 2 * top)
    tables = edges * (2 * 8 * (2 * top + 1) + 4 + 8 + 4)
    if op == "factored":  # rows = h~ Z(source), then weighted sums; backward dh, dZ, dweights
        packed = (TRUNK + 1) * (2 * blocks - 1) * case["copies_out"]
        return {"bytes": 2 * nodes * packed * 4 + 2 * nodes * out_width * 4 + 2 * edges * 4 + tables, "flops": 3.0 * 2.0 * edges * packed}
    matrix = (2 * blocks - 1) * case["copies_in"] * case["copies_out"]
    in_width = case["copies_in"] * (1 + 2 * top)
    return {"bytes": 2 * nodes * in_width * 4 + 2 * edges * out_width * 4 + tables, "flops": 3.0 * 2.0 * edges * matrix * (TRUNK + 2)}


def tolerance(case: dict[str, Any]) -> dict[str, float]:
    """About four times the 2-norm error measured against the same operator in float64: 2.5e-3 for bf16 storage, 2e-7 to
    3.4e-7 for float32 attention, up to 2.7e-6 where a gradient is summed over every edge into a few parameters."""
    if case["dtype"] == "bf16":
        return {"rel": 1e-2}
    return {"rel": 2e-6 if case["op"] in ("attention", "graph_attention", "scores") else 1e-5}
