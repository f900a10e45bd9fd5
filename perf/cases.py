"""What this framework is timed on: the calls its users make, over the sizes they make them with.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (inputs from the seed, layers,
edge lists), ``run`` is one pass through the public entry points, ``work`` is what a pass cannot do without and
``tolerance`` what two correct float32 / bfloat16 implementations may differ by.  Eight kinds of call:

graph       spherical harmonics -> ``SO3LinearGraph`` on an edge list: the message-passing step of an equivariant
            network, as a training step (all gradients) or as inference
edge        ``SO3Linear`` on per-edge features, the drop-in form of the same layer
molecular   per-edge radial weights in bfloat16: ``gather_rows`` -> ``SO3Linear`` 'uu' -> ``segment_sum``
so2         ``WignerD`` -> rotate -> ``SO2Linear`` -> rotate back, the high-order path
product     ``TensorProduct`` of two channelled operands with full channel mixing
mix         ``IrrepsLinear``, the channel mixing between layers
epilogue    ``Gate`` -> ``BatchRMSNorm`` -> ``LayerRMSNorm``, what follows a tensor product
features    ``EdgeFeaturizer``: positions to radius graph, harmonics, radial basis and cutoff
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

from equitorch_b200 import nn as enn
from equitorch_b200.graph import EdgeGraph
from equitorch_b200.irreps import Irreps
from equitorch_b200.ops.graph_ops import gather_rows, segment_sum
from equitorch_b200.transforms import EdgeFeaturizer, RadiusGraph

DEV = "cuda:0"
IRREPS = {1: "0e+1o", 2: "0e+1o+2e", 3: "0e+1o+2e+3o"}
MOLECULAR = "4x0e+2x1o+2e"            # 128x0e + 64x1o + 32x2e with 32 channels


def listed():
    return [
        # One layer of a large training step: random geometric graph, about 2M edges, the scaling configuration.
        dict(name="graph_train_100k_nodes", kind="graph", nodes=100_000, edges=2_000_000, geometric=True, l_max=3,
             channels=64, mode="uv", train=True),
        # 200k edges with sources anywhere in a node table of 10k rows (the microbenchmark configuration).
        dict(name="graph_train_random_200k", kind="graph", nodes=10_000, edges=200_000, geometric=False, l_max=3,
             channels=64, mode="uv", train=True),
        # A mid-size batch with ragged counts, channel-wise weights and lower degree, edges in no order.
        dict(name="graph_train_uu_ragged", kind="graph", nodes=7_013, edges=110_003, geometric=False, l_max=2,
             channels=128, mode="uu", train=True),
        # A molecular-dynamics sized forward pass: few nodes, latency counts.
        dict(name="graph_infer_960_nodes", kind="graph", nodes=960, edges=20_500, geometric=True, l_max=2,
             channels=32, mode="uv", train=False),
        # The smallest call: 1024 samples, 16 channels, channel-wise shared weights.
        dict(name="edge_uu_1024", kind="edge", samples=1_024, l_max=2, channels=16, mode="uu"),
        # The per-edge layer with full channel mixing on an odd number of edges.
        dict(name="edge_uv_20011", kind="edge", samples=20_011, l_max=3, channels=64, mode="uv"),
        # Molecular batch (32 graphs of 30 atoms): bfloat16 operands, weights produced per edge by a radial network.
        dict(name="molecular_bf16", kind="molecular", nodes=960, edges=20_480, channels=32),
        # High-order rotated path, 49 components.
        dict(name="so2_l6_100k_edges", kind="so2", edges=100_000, l_max=6, channels=32),
        # Self-interaction of node features.
        dict(name="product_uvw_2000", kind="product", samples=2_000, l_max=2, channels=32),
        # Channel mixing between two layers.
        dict(name="mix_50021_nodes", kind="mix", nodes=50_021, l_max=3, channels=64, channels_out=128),
        # Gate and normalisations of the large training step.
        dict(name="epilogue_100k_nodes", kind="epilogue", nodes=100_000, l_max=3, channels=64),
        # Edge featurisation of a point cloud as large as the large training step's.
        dict(name="features_100k_points", kind="features", nodes=100_000, shell=18, l_max=3, basis=8),
    ]


def _log(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["graph", "graph", "graph", "edge", "edge", "molecular", "so2", "product", "mix", "epilogue", "features"])
    if kind == "graph":
        l_max, channels = rng.choice([1, 2, 3, 3]), rng.choice([16, 32, 64, 64, 128])
        nodes = _log(rng, 300, {16: 15_000, 128: 20_000}.get(channels, 40_000))
        edges = int(nodes * rng.uniform(3, 10 if channels == 16 else 30))
        return dict(kind=kind, nodes=nodes, edges=edges, geometric=rng.random() < 0.5, l_max=l_max, channels=channels,
                    mode=rng.choice(["uv", "uv", "uu"]), train=rng.random() < 0.7)
    if kind == "edge":
        return dict(kind=kind, samples=_log(rng, 200, 20_000), l_max=rng.choice([1, 2, 3]), channels=rng.choice([16, 32, 64]),
                    mode=rng.choice(["uv", "uu"]))
    if kind == "molecular":
        nodes = _log(rng, 100, 3_000)
        return dict(kind=kind, nodes=nodes, edges=int(nodes * rng.uniform(8, 25)), channels=rng.choice([16, 32, 64]))
    if kind == "so2":
        return dict(kind=kind, edges=_log(rng, 1_000, 80_000), l_max=rng.randint(2, 6), channels=rng.choice([32, 32, 64]) if
                    rng.random() < 0.7 else 16)
    if kind == "product":
        return dict(kind=kind, samples=_log(rng, 100, 2_000), l_max=rng.choice([1, 2]), channels=rng.choice([16, 32]))
    if kind == "mix":
        return dict(kind=kind, nodes=_log(rng, 500, 50_000), l_max=rng.choice([1, 2, 3]), channels=rng.choice([32, 64]),
                    channels_out=rng.choice([32, 64, 128]))
    if kind == "epilogue":
        return dict(kind=kind, nodes=_log(rng, 500, 100_000), l_max=rng.choice([1, 2, 3]), channels=rng.choice([32, 64]))
    return dict(kind=kind, nodes=_log(rng, 1_000, 100_000), shell=rng.choice([6, 18, 26]), l_max=rng.choice([1, 2, 3]), basis=8)


# ---- inputs ------------------------------------------------------------------------------------------------------------
class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, scale=1.0, dtype=torch.float32):
        return (torch.randn(*shape, generator=self.g, device=DEV) * scale).to(dtype)

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device=DEV)

    def integers(self, high, *shape):
        return torch.randint(0, high, shape, generator=self.g, device=DEV)


def _leaf(t, grad=True):
    return t.contiguous().requires_grad_(grad)


def _morton(cell):
    code = torch.zeros(cell.shape[0], dtype=torch.long, device=DEV)
    for bit in range(10):
        for axis in range(3):
            code |= ((cell[:, axis] >> bit) & 1) << (3 * bit + axis)
    return torch.argsort(code, stable=True)


def _edges(rnd, case):
    """(src, dst, edge vectors) with exactly ``case["edges"]`` edges."""
    nodes, edges = case["nodes"], case["edges"]
    if not case["geometric"]:
        src, dst = rnd.integers(nodes, edges), rnd.integers(nodes, edges)
        return src, (torch.sort(dst).values if edges % 2 == 0 else dst), rnd.normal(edges, 3)
    # points uniform in a cube in Morton order, each joined to its neighbours: the shortest pairs, ordered by destination
    box = (nodes * nodes * 4.0 / 3.0 * math.pi / edges) ** (1.0 / 3.0)
    pos, r = rnd.uniform(nodes, 3) * box, 1.05
    pos = pos[_morton(pos.long())].contiguous()
    while True:
        data = RadiusGraph(r, max_num_neighbors=128)(SimpleNamespace(pos=pos))
        if data.edge_index.shape[1] >= edges:
            break
        r *= 1.05
    keep = torch.sort(torch.topk(data.edge_vec.norm(dim=-1), edges, largest=False).indices).values
    return data.edge_index[0][keep], data.edge_index[1][keep], data.edge_vec[keep]


# cutoff between two shells of neighbours of a cubic lattice
_SHELL_CUTOFF = {6: 1.20, 18: 1.57, 26: 1.86}


def _lattice(rnd, nodes):
    """Atoms displaced about the sites of a cubic lattice (the edge count does not depend on the displacements)."""
    side = math.ceil(nodes ** (1.0 / 3.0))
    i = torch.arange(nodes, device=DEV)
    site = torch.stack([i % side, i // side % side, i // (side * side)], dim=-1)
    site = site[_morton(site)]
    return (site + (rnd.uniform(nodes, 3) - 0.5) * 0.06).contiguous()


def prepare(case, seed):
    rnd, kind = _Random(seed), case["kind"]
    s = SimpleNamespace(kind=kind, case=case)
    c = case.get("channels")
    if kind == "graph":
        ir, dim, train = IRREPS[case["l_max"]], (case["l_max"] + 1) ** 2, case["train"]
        src, dst, vec = _edges(rnd, case)
        s.graph = EdgeGraph(src, dst, case["nodes"])
        s.sh = enn.SphericalHarmonics(case["l_max"])
        s.layer = enn.SO3LinearGraph(ir, ir, ir, c, c, internal_weights=False, feature_mode=case["mode"]).to(DEV)
        s.x, s.vec = _leaf(rnd.normal(case["nodes"], dim, c), train), _leaf(vec, train)
        s.w = _leaf(rnd.normal(*s.layer.weight_shape, scale=c ** -0.5 if case["mode"] == "uv" else 1.0), train)
        s.cot = rnd.normal(case["nodes"], dim, c) if train else None
    elif kind == "edge":
        ir, n, dim = IRREPS[case["l_max"]], case["samples"], (case["l_max"] + 1) ** 2
        s.sh = enn.SphericalHarmonics(case["l_max"])
        s.layer = enn.SO3Linear(ir, ir, ir, c, c, internal_weights=False, feature_mode=case["mode"]).to(DEV)
        s.x, s.vec, s.cot = _leaf(rnd.normal(n, dim, c)), _leaf(rnd.normal(n, 3)), rnd.normal(n, dim, c)
        s.w = _leaf(rnd.normal(*s.layer.weight_shape, scale=c ** -0.5))
    elif kind == "molecular":
        nodes, edges = case["nodes"], case["edges"]
        src, dst = rnd.integers(nodes, edges), torch.sort(rnd.integers(nodes, edges)).values
        s.layer = enn.SO3Linear(MOLECULAR, IRREPS[2], MOLECULAR, c, c, internal_weights=False, feature_mode="uu").to(DEV)
        s.sh, s.src, s.vec = enn.SphericalHarmonics(2), src, rnd.normal(edges, 3)
        s.ptr = torch.zeros(nodes + 1, dtype=torch.long, device=DEV)
        s.ptr[1:] = torch.cumsum(torch.bincount(dst, minlength=nodes), 0)
        s.x = _leaf(rnd.normal(nodes, 15, c, dtype=torch.bfloat16))
        s.w = _leaf(rnd.normal(edges, *s.layer.weight_shape, dtype=torch.bfloat16))
        s.cot = rnd.normal(nodes, 15, c)
    elif kind == "so2":
        ir, n, dim = Irreps((0, case["l_max"])), case["edges"], (case["l_max"] + 1) ** 2
        s.wigner, s.rotate = enn.WignerD(ir).to(DEV), enn.DenseWignerRotation(ir)
        s.layer = enn.SO2Linear(ir, ir, c, c, internal_weights=False, feature_mode="uv").to(DEV)
        s.x, s.cot = _leaf(rnd.normal(n, dim, c)), rnd.normal(n, dim, c)
        u = rnd.uniform(n, 3) * 2 - 1                           # Haar rotations as ZYZ angles
        s.angles = _leaf(torch.stack([math.pi * u[:, 0], torch.acos(u[:, 1].clamp(-1, 1)), math.pi * u[:, 2]], dim=-1))
        s.w = _leaf(rnd.normal(*s.layer.weight_shape, scale=c ** -0.5))
    elif kind == "product":
        ir, n, dim = IRREPS[case["l_max"]], case["samples"], (case["l_max"] + 1) ** 2
        s.layer = enn.TensorProduct(ir, ir, ir, c, c, c, internal_weights=False, feature_mode="uvw").to(DEV)
        s.x, s.y, s.cot = _leaf(rnd.normal(n, dim, c)), _leaf(rnd.normal(n, dim, c)), rnd.normal(n, dim, c)
        s.w = _leaf(rnd.normal(*s.layer.weight_shape, scale=1.0 / c))
    elif kind == "mix":
        ir, n, dim, co = IRREPS[case["l_max"]], case["nodes"], (case["l_max"] + 1) ** 2, case["channels_out"]
        s.layer = enn.IrrepsLinear(ir, ir, c, co, internal_weights=False).to(DEV)
        s.x, s.cot = _leaf(rnd.normal(n, dim, c)), rnd.normal(n, dim, co)
        s.w = _leaf(rnd.normal(*s.layer.weight_shape, scale=c ** -0.5))
    elif kind == "epilogue":
        ir, n, dim = IRREPS[case["l_max"]], case["nodes"], (case["l_max"] + 1) ** 2
        s.gate = enn.Gate(ir, activation=torch.nn.Sigmoid()).to(DEV)
        # momentum 1: the running statistics are those of the pass, so that a repeated pass gives the same buffer
        s.bn, s.ln = enn.BatchRMSNorm(ir, c, momentum=1.0).to(DEV).train(), enn.LayerRMSNorm(ir, c).to(DEV)
        s.x, s.gates, s.cot = _leaf(rnd.normal(n, dim, c)), _leaf(rnd.normal(n, case["l_max"] + 1, c)), rnd.normal(n, dim, c)
    else:
        r = _SHELL_CUTOFF[case["shell"]]
        s.pos = _lattice(rnd, case["nodes"])
        s.featurizer = EdgeFeaturizer(r, case["l_max"], enn.BesselBasis(r, case["basis"]).to(DEV), enn.PolynomialCutoff(r),
                                      max_num_neighbors=64)
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------------
def run(s):
    if s.kind == "graph":
        if not s.case["train"]:
            with torch.no_grad():
                return s.layer(s.x, s.sh(s.vec), s.graph, s.w)
        out = s.layer(s.x, s.sh(s.vec), s.graph, s.w)
        return [out, *torch.autograd.grad(out, [s.x, s.vec, s.w], s.cot)]
    if s.kind == "edge":
        out = s.layer(s.x, s.sh(s.vec), s.w)
        return [out, *torch.autograd.grad(out, [s.x, s.vec, s.w], s.cot)]
    if s.kind == "molecular":
        message = s.layer(gather_rows(s.x, s.src), s.sh(s.vec).bfloat16(), s.w)
        out = segment_sum(message.float(), s.ptr)
        return [out, *torch.autograd.grad(out, [s.x, s.w], s.cot)]
    if s.kind == "so2":
        d = s.wigner(s.angles[:, 0], s.angles[:, 1], s.angles[:, 2])
        out = s.rotate(s.layer(s.rotate(s.x, d), s.w), d.transpose(-1, -2))
        return [out, *torch.autograd.grad(out, [s.x, s.w, s.angles], s.cot)]
    if s.kind == "product":
        out = s.layer(s.x, s.y, s.w)
        return [out, *torch.autograd.grad(out, [s.x, s.y, s.w], s.cot)]
    if s.kind == "mix":
        out = s.layer(s.x, s.w)
        return [out, *torch.autograd.grad(out, [s.x, s.w], s.cot)]
    if s.kind == "epilogue":
        out = s.ln(s.bn(s.gate(s.x, s.gates)))
        return [out, *torch.autograd.grad(out, [s.x, s.gates, s.bn.weight, s.ln.weight], s.cot), s.bn.running_squared_norm]
    f = s.featurizer.features(s.pos)
    return [f.src, f.dst, f.ptr, f.vec, f.length, f.sh, f.bessel, f.cutoff]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------
def _paths(ls1, ls2, ls_out):
    """(paths, intermediate rows, (m_1, m_2) cells in use) of a product over (l, parity) lists."""
    paths = rows = 0
    cells = set()
    for i, (a, pa) in enumerate(ls1):
        for j, (b, pb) in enumerate(ls2):
            for o, po in ls_out:
                if abs(a - b) <= o <= a + b and pa * pb == po:
                    paths += 1
                    rows += 2 * o + 1
                    cells.add((i, j))
    return paths, rows, sum((2 * ls1[i][0] + 1) * (2 * ls2[j][0] + 1) for i, j in cells)


def _natural(l_max):
    return [(l, (-1) ** l) for l in range(l_max + 1)]


def work(case):
    kind, c = case["kind"], case.get("channels")
    if kind == "features":
        e = case["nodes"] * case["shell"]
        width = 16 + 12 + 4 + 4 * (case["l_max"] + 1) ** 2 + 4 * case["basis"] + 4
        return dict(bytes=case["nodes"] * (12 + 8) + e * width, flops=e * 150)
    if kind == "molecular":
        ls = [(0, 1)] * 4 + [(1, -1)] * 2 + [(2, 1)]
        paths, rows, cells = _paths(ls, _natural(2), ls)
        n, e = case["nodes"], case["edges"]
        return dict(bytes=n * 15 * c * (2 + 4 + 4 + 2) + e * (12 + 16 + 2 * paths * c * 2), flops=e * c * 2 * (3 * cells + 3 * rows))
    dim = (case["l_max"] + 1) ** 2
    if kind == "so2":
        n, l = case["edges"], case["l_max"]
        block = sum((2 * k + 1) ** 2 for k in range(l + 1))
        terms = sum((1 if m == 0 else 4) * (l + 1 - m) ** 2 for m in range(l + 1))
        w = sum((1 if m == 0 else 2) * (l + 1 - m) ** 2 for m in range(l + 1)) * c * c * 4
        return dict(bytes=n * (4 * dim * c * 4 + 24) + 2 * w, flops=n * (6 * 2 * block * c + 3 * 2 * terms * c * c))
    if kind == "epilogue":
        n, k = case["nodes"], case["l_max"] + 1
        return dict(bytes=n * c * 4 * (4 * dim + 2 * k), flops=n * c * dim * 24)
    if kind == "mix":
        n, co, k = case["nodes"], case["channels_out"], case["l_max"] + 1
        return dict(bytes=n * dim * 8 * (c + co) + 2 * k * c * co * 4, flops=3 * 2 * n * dim * c * co)
    paths, rows, cells = _paths(*[_natural(case["l_max"])] * 3)
    if kind == "product":
        n, w = case["samples"], paths * c ** 3 * 4
        return dict(bytes=n * dim * c * 4 * 6 + 2 * w, flops=n * (4 * 2 * rows * c ** 3))
    mixing = 2 * c if case["mode"] == "uv" else 2
    w = paths * c * (c if case["mode"] == "uv" else 1) * 4
    if kind == "edge":
        n = case["samples"]
        return dict(bytes=n * (4 * dim * c * 4 + 24) + 2 * w, flops=n * c * (3 * 2 * cells + 4 * rows * mixing))
    n, e = case["nodes"], case["edges"]
    if not case["train"]:
        return dict(bytes=n * 2 * dim * c * 4 + e * (12 + 16) + w, flops=e * c * 2 * cells + n * c * rows * mixing)
    return dict(bytes=n * 4 * dim * c * 4 + e * (24 + 16) + 2 * w, flops=e * c * 3 * 2 * cells + n * c * 4 * rows * mixing)


def tolerance(case):
    # Measured against the same path in float64: float32 up to 3.7e-6 (three-product TF32 sums in 'uvw'), two such results
    # differ by twice that at most; bfloat16 6.5e-3 (gradients summed over a node's edges), 5e-3 between two passes.
    return {"rel": 1.5e-2} if case["kind"] == "molecular" else {"rel": 1e-5}
