"""Generate ``generated/walk_specs.inc``: straight-line Clebsch-Gordan code for the kernels in which one warp walks the
edges of its nodes on its own (``tp_walk.cu``).

For the index structures of the registry of :mod:`gen_tp_specs`.  A lane holds a channel (or a few) of *all* cells
``Q[m_y, m_feat]`` of the per-node outer product, so a warp needs nothing from other warps; where that is more than a lane's
registers hold (l_max 3: 234 cells), the components of the channelled operand are dealt to two halves, each a warp's, such
that every intermediate row belongs to one half.

The rows are emitted by output component ``K``, and inside one by path ``P``: what the weight step of a layer with
channel-wise weights needs to finish a component in registers, ``out[K] = sum_P w[P] row(K, P)``.

    python -m equitorch_b200.csrc.gen_walk_specs        # rewrites generated/walk_specs.inc
"""
from __future__ import annotations

import hashlib
import os
from typing import List, NamedTuple, Optional

import numpy as np

from .gen_tp_specs import HERE, REGISTRY, Structure, structure_from_info, structure_key, tc_plan

OUT = os.path.join(HERE, "generated", "walk_specs.inc")
MOST_CELLS = 96        # of one lane; more are split over two warps


class RowMap(NamedTuple):
    """Weight step of a layer: intermediate row r goes to output component ``comp[r]`` with the weight ``path[r]``."""
    comp: np.ndarray
    path: np.ndarray


def row_map(info) -> Optional[RowMap]:
    """From the ``info_M_fwd`` table of a TensorProductInfo; None where it has scales or a row order of its own."""
    if info.index1 is not None or info.scale is not None or info.gather_index is not None or info.index_out is not None:
        return None
    seg = np.arange(info.out_size + 1) if info.seg_out is None else info.seg_out.cpu().numpy()
    path = np.arange(seg[-1]) if info.index2 is None else info.index2.cpu().numpy()
    if len(path) != seg[-1]:
        return None
    return RowMap(np.repeat(np.arange(len(seg) - 1), np.diff(seg)).astype(np.int64), path.astype(np.int64))


def mix_key(s: Structure, m: Optional[RowMap]) -> int:
    """Identifies a structure together with its weight step; 0: none."""
    if m is None or len(m.comp) != s.num_rows:
        return 0
    h = hashlib.sha256(structure_key(s).to_bytes(8, "little"))
    for col in (m.comp, m.path):
        h.update(np.ascontiguousarray(col, dtype=np.int64).tobytes())
    return int.from_bytes(h.digest()[:7], "little")


class Half(NamedTuple):
    comps: List[int]       # components of the channelled operand, in the order of a ring slot
    cells: List[tuple]     # (m_y, position in comps): the accumulators
    pairs: int             # the first 2 pairs of them are neighbours (2 n, 2 n + 1) in m_y for packed multiply-adds
    rows: List[int]        # rows it produces, by output component, then path
    entries: List[int]     # entry ids in the order of use
    paths: List[int]       # paths of its rows


def halves(s: Structure, m: RowMap) -> Optional[List[Half]]:
    cells = sorted(set(zip(s.mf.tolist(), s.my.tolist())))
    if len(cells) <= MOST_CELLS:
        parts = [list(range(s.d_feat))]
    else:
        plan = tc_plan(s)                    # a split in which no row needs both parts
        if plan is None:
            return None
        parts = plan.mlist
    out = []
    for n, comps in enumerate(parts):
        at = {c: i for i, c in enumerate(comps)}
        mine = {(k, at[c]) for c, k in cells if c in at}
        paired = sorted((t for t in mine if (t[0] ^ 1, t[1]) in mine), key=lambda t: (t[1], t[0]))
        mine = paired + sorted(mine - set(paired), key=lambda t: (t[1], t[0]))
        rows = sorted({int(r) for r, c in zip(s.row, s.mf) if int(c) in at} |
                      (set(range(s.num_rows)) - set(s.row.tolist()) if n == 0 else set()),     # rows without entries are zeros
                      key=lambda r: (int(m.comp[r]), int(m.path[r]), r))
        entries = [t for r in rows for t in np.nonzero(s.row == r)[0].tolist()]
        out.append(Half(list(comps), mine, len(paired) // 2, rows, entries, sorted({int(m.path[r]) for r in rows})))
    return out


def _emit_half(s: Structure, m: RowMap, h: int, half: Half, num_out: int) -> List[str]:
    index = {(k, half.comps[i]): n for n, (k, i) in enumerate(half.cells)}
    by_row = {r: [t for t in half.entries if s.row[t] == r] for r in half.rows}
    place = {t: n for n, t in enumerate(half.entries)}
    local = {p: n for n, p in enumerate(half.paths)}
    out = []
    # per edge: q[cell] += x[m_feat] y[m_y]; component i of the slot is CW floats behind component i - 1
    out.append(f"  template <int V, int CW> __device__ __forceinline__ static void outer{h}(float (&q)[NC][V], const float* xs, "
               "const float (&y)[YF]) {")
    out.append("    float x[V];")
    for i in range(len(half.comps)):
        out.append(f"    EQT_LDX(x, xs + {i} * CW);")
        for n, (k, j) in enumerate(half.cells):
            if j == i and n >= 2 * half.pairs:
                out.append(f"    EQT_FMA(q[{n}], x, y[{k}]);")
            elif j == i and n % 2 == 0:
                out.append(f"    EQT_FMA2(q[{n}], q[{n + 1}], x, y[{k}], y[{k + 1}]);")
    out.append("  }")
    # adjoint, per edge: a[m_y] = sum of x[m_feat] h[cell] over the lane's channels
    out.append(f"  template <int V, int CW> __device__ __forceinline__ static void dot{h}(float (&a)[DY], const float* xs, "
               "const float (&q)[NC][V]) {")
    out.append("    float x[V];")
    out += [f"    a[{k}] = 0.f;" for k in range(s.d_y)]
    for i in range(len(half.comps)):
        out.append(f"    EQT_LDX(x, xs + {i} * CW);")
        for n, (k, j) in enumerate(half.cells):
            if j == i and n >= 2 * half.pairs:
                out.append(f"    EQT_DOT(a[{k}], x, q[{n}]);")
            elif j == i and n % 2 == 0:
                out.append(f"    EQT_DOT2(a[{k}], a[{k + 1}], x, q[{n}], q[{n + 1}]);")
    out.append("  }")

    def scale(t, loaded):
        text = [f"    c = sc[{place[t] // 4}];"] if place[t] // 4 != loaded else []
        return text, f"c.{'xyzw'[place[t] % 4]}", place[t] // 4

    # per node: rows from the accumulators, handed to the sink by output component
    out.append(f"  template <int V, class Sink> __device__ __forceinline__ static void rows{h}(const float (&q)[NC][V], const float4* sc, "
               "Sink& sink) {")
    out.append("    float4 c; float v[V];")
    loaded = -1
    for k in range(num_out):
        out.append(f"    sink.template open<{k}>();")
        for r in [r for r in half.rows if m.comp[r] == k]:
            if not by_row[r]:
                out.append("    EQT_ZERO(v);")
            for n, t in enumerate(by_row[r]):
                text, term, loaded = scale(t, loaded)
                out += text
                out.append(f"    {'EQT_FMA' if n else 'EQT_MUL'}(v, q[{index[int(s.my[t]), int(s.mf[t])]}], {term});")
            out.append(f"    sink.template row<{r}, {k}, {int(m.path[r])}, {local[int(m.path[r])]}>(v);")
        out.append(f"    sink.template close<{k}>();")
    out.append("  }")
    # adjoint, per node: h[cell] = sum_t scale[t] g[row[t]]
    out.append(f"  template <int V, class Source> __device__ __forceinline__ static void cells{h}(float (&q)[NC][V], const float4* sc, "
               "Source& source) {")
    out.append("    float4 c; float g[V];")
    loaded, touched = -1, set()
    for k in range(num_out):
        mine = [r for r in half.rows if m.comp[r] == k and by_row[r]]
        if mine:
            out.append(f"    source.template open<{k}>();")
        for r in mine:
            out.append(f"    source.template row<{r}, {k}, {int(m.path[r])}>(g);")
            for t in by_row[r]:
                text, term, loaded = scale(t, loaded)
                out += text
                cell = index[int(s.my[t]), int(s.mf[t])]
                out.append(f"    {'EQT_FMA' if cell in touched else 'EQT_MUL'}(q[{cell}], g, {term});")
                touched.add(cell)
    out.append("  }")
    return out


def emit(idx: int, s: Structure, m: RowMap, note: str) -> Optional[str]:
    parts = halves(s, m)
    if parts is None:
        return None
    num_out, num_paths = int(m.comp.max()) + 1, int(m.path.max()) + 1
    longest = max((len(p.entries) + 3) // 4 * 4 for p in parts)
    both = parts if len(parts) == 2 else parts * 2
    order = [t for p in parts for t in p.entries + [-1] * (longest - len(p.entries))]
    out = [f"// {note}",
           f"static __device__ const short walk_order{idx}[{len(order)}] = {{{', '.join(str(t) for t in order)}}};",
           f"struct Walk{idx} {{",
           f"  static constexpr uint64_t KEY = {structure_key(s)}ull, MIX_KEY = {mix_key(s, m)}ull;",
           f"  static constexpr int T = {len(s.row)}, R = {s.num_rows}, DF = {s.d_feat}, DY = {s.d_y}, YF = {(s.d_y + 3) // 4 * 4};",
           f"  static constexpr int K = {num_out}, P = {num_paths}, HALVES = {len(parts)};",
           f"  static constexpr int NC = {max(len(p.cells) for p in parts)}, NX = {max(len(p.comps) for p in parts)}, "
           f"NP = {max(len(p.paths) for p in parts)}, TH = {longest};",
           "  // scales of half h in the order of use: entry order(TH h + i) of the table, or -1 (padding)",
           f"  __device__ static int order(int i) {{ return walk_order{idx}[i]; }}",
           "  // component of the channelled operand at place i of half h, and path of the half's place i",
           "  __device__ static int comp(int h, int i) {",
           "    switch (i) {"]
    for i in range(max(len(p.comps) for p in parts)):
        a, b = (p.comps[i] if i < len(p.comps) else 0 for p in both)
        out.append(f"      case {i}: return h ? {b} : {a};")
    out += ["      default: return 0;", "    }", "  }", "  __device__ static int path(int h, int i) {", "    switch (i) {"]
    for i in range(max(len(p.paths) for p in parts)):
        a, b = (p.paths[i] if i < len(p.paths) else -1 for p in both)
        out.append(f"      case {i}: return h ? {b} : {a};")
    out += ["      default: return -1;", "    }", "  }"]
    for h, part in enumerate(parts):
        out += _emit_half(s, m, h, part, num_out)
    if len(parts) == 1:
        out += ["  template <int V, int CW> __device__ __forceinline__ static void outer1(float (&)[NC][V], const float*, const float (&)[YF]) {}",
                "  template <int V, int CW> __device__ __forceinline__ static void dot1(float (&)[DY], const float*, const float (&)[NC][V]) {}",
                "  template <int V, class Sink> __device__ __forceinline__ static void rows1(const float (&)[NC][V], const float4*, Sink&) {}",
                "  template <int V, class Source> __device__ __forceinline__ static void cells1(float (&)[NC][V], const float4*, Source&) {}"]
    out.append("};")
    return "\n".join(out)


def collect() -> List[tuple]:
    from ..irreps import Irreps
    from ..tables import tp_infos
    seen, specs = set(), []
    for o, a, b in REGISTRY:
        io, i1, i2 = Irreps(o), Irreps(a), Irreps(b)
        fwd, bwd1, _, _ = tp_infos(io, i1, i2)
        for s, info, note in ((structure_from_info(fwd.info_Mij_fwd, True, i1.dim, i2.dim), fwd.info_M_fwd, "forward"),
                              (structure_from_info(bwd1.info_Mij_fwd, False, io.dim, i2.dim), bwd1.info_M_fwd, "grad of input1")):
            m = row_map(info)
            if m is not None and mix_key(s, m) not in seen:
                seen.add(mix_key(s, m))
                specs.append((s, m, f"{a} (x) {b} -> {o}: {note}"))
    return specs


def generate(path: str = OUT) -> str:
    body = ["// AUTO-GENERATED by equitorch_b200/csrc/gen_walk_specs.py - do not edit.", "#pragma once", ""]
    names = []
    for n, (s, m, note) in enumerate(collect()):
        text = emit(n, s, m, note)
        if text:
            body += [text, ""]
            names.append(f"Walk{n}")
    body.append("#define EQT_FOR_EACH_WALK(X) " + " ".join(f"X({n})" for n in names))
    text = "\n".join(body) + "\n"
    os.makedirs(os.path.dirname(path), exist_ok=True)
    if not os.path.exists(path) or open(path).read() != text:
        with open(path, "w") as fh:
            fh.write(text)
    return path


if __name__ == "__main__":
    print(generate())
