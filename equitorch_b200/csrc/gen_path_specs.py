"""Generate ``generated/path_specs.inc``: one Clebsch-Gordan block per (l_out, l_1, l_2) as straight-line code.

A layer's table is a list of paths (k, i, j) between irreps; what a path does depends on its three degrees only.  For
degrees up to ``MAX_L`` the block's multiply-adds are emitted with the CG values as immediates, on register blocks of V
channels: products of several y components with the same (M, m1) are summed before they meet the channels.  P: two channels at a
time in packed instructions.

``generated/triple_specs.inc`` holds the blocks of a product of two channelled operands in the forms that its kernels take:
one component of the contracted operand at a time, and all of them from a pair of channels.

    python -m equitorch_b200.csrc.gen_path_specs        # rewrites generated/path_specs.inc and triple_specs.inc
"""
from __future__ import annotations

import os

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.join(HERE, "generated", "path_specs.inc")
TRIPLE_OUT = os.path.join(HERE, "generated", "triple_specs.inc")
MAX_L = 3
TRIPLE_MAX_L = 2


def triples(max_l: int = MAX_L):
    return [(lo, l1, l2) for lo in range(max_l + 1) for l1 in range(max_l + 1) for l2 in range(max_l + 1)
            if abs(l1 - l2) <= lo <= l1 + l2]


def _lit(v: float) -> str:
    return f"{v:.9g}f" if "." in f"{v:.9g}" or "e" in f"{v:.9g}" else f"{v:.9g}.f"


def _emit(lo: int, l1: int, l2: int) -> str:
    from ..constants import so3_clebsch_gordan
    cg = so3_clebsch_gordan(lo, l1, l2)
    pairs = {}                                          # (M, m1) -> [(m2, value)]
    for M, m1, m2 in zip(*cg.nonzero()):
        pairs.setdefault((int(M), int(m1)), []).append((int(m2), float(cg[M, m1, m2])))

    def coef(ts):
        expr = f"{_lit(ts[0][1])} * y[{ts[0][0]}]"
        for m2, v in ts[1:]:
            expr = f"fmaf({_lit(v)}, y[{m2}], {expr})"
        return expr
    no, n1, n2 = 2 * lo + 1, 2 * l1 + 1, 2 * l2 + 1
    out = [f"template <> struct CgPath<{lo}, {l1}, {l2}> {{",
           f"  // o[M] += sum_m1 (sum_m2 cg y[m2]) x[m1]",
           f"  template <int V, bool P = false> __device__ __forceinline__ static void forward(float (&o)[{no}][V], const float (&x)[{n1}][V], const float (&y)[{n2}]) {{"]
    for (M, m1), ts in pairs.items():
        out.append(f"    axpy<V, P>(o[{M}], {coef(ts)}, x[{m1}]);")
    out += ["  }",
            f"  // r[m1] += sum_M (sum_m2 cg y[m2]) g[M]",
            f"  template <int V, bool P = false> __device__ __forceinline__ static void adjoint(float (&r)[{n1}][V], const float (&g)[{no}][V], const float (&y)[{n2}]) {{"]
    for (M, m1), ts in pairs.items():
        out.append(f"    axpy<V, P>(r[{m1}], {coef(ts)}, g[{M}]);")
    out += ["  }",
            f"  // gy[m2] += sum_(M, m1) cg <g[M], x[m1]> over the V channels",
            f"  template <int V, bool P = false> __device__ __forceinline__ static void inner(float (&gy)[{n2}], const float (&g)[{no}][V], const float (&x)[{n1}][V]) {{",
            "    float d;"]
    for (M, m1), ts in pairs.items():
        out.append(f"    d = dot<V, P>(g[{M}], x[{m1}]);")
        out += [f"    gy[{m2}] = fmaf({_lit(v)}, d, gy[{m2}]);" for m2, v in ts]
    out += ["  }", "};"]
    return "\n".join(out)


def _emit_triple(lo: int, ls: int, lf: int) -> str:
    from ..constants import so3_clebsch_gordan
    cg = so3_clebsch_gordan(lo, ls, lf)
    no, ns, nf = 2 * lo + 1, 2 * ls + 1, 2 * lf + 1
    out = [f"template <> struct CgTriple<{lo}, {ls}, {lf}> {{",
           "  // o[a] += (sum_b cg[a, b, C] s[b]) z for component C of the contracted operand, 2 V columns",
           f"  template <int C, int V> __device__ __forceinline__ static void column(Two (&o)[{no}][V], const float (&s)[{ns}], const Two (&z)[V]) {{"]
    for c in range(nf):
        out.append(f"    if constexpr (C == {c}) {{")
        for a in range(no):
            ts = [(b, float(cg[a, b, c])) for b in range(ns) if cg[a, b, c]]
            if ts:
                expr = f"{_lit(ts[0][1])} * s[{ts[0][0]}]"
                for b, v in ts[1:]:
                    expr = f"fmaf({_lit(v)}, s[{b}], {expr})"
                out.append(f"      axpy<V>(o[{a}], {expr}, z);")
        out.append("    }")
    out += ["  }",
            "  // q[c] = sum_(a, b) cg[a, b, c] s[b] g[a], 2 V samples side by side",
            f"  template <int V> __device__ __forceinline__ static void pair(Two (&q)[{nf}][V], const Two (&s)[{ns}][V], const Two (&g)[{no}][V]) {{",
            "    Two d[V];"]
    seen = set()
    for a in range(no):
        for b in range(ns):
            cs = [(c, float(cg[a, b, c])) for c in range(nf) if cg[a, b, c]]
            if not cs:
                continue
            out.append(f"    times<V>(d, s[{b}], g[{a}]);")
            for c, v in cs:
                out.append(f"    axpy<V>(q[{c}], {_lit(v)}, d);" if c in seen else f"    scaled<V>(q[{c}], {_lit(v)}, d);")
                seen.add(c)
    out += ["  }", "};"]
    return "\n".join(out)


def _write(path: str, text: str) -> str:
    os.makedirs(os.path.dirname(path), exist_ok=True)
    if not os.path.exists(path) or open(path).read() != text:
        with open(path, "w") as fh:
            fh.write(text)
    return path


def generate_triples(path: str = TRIPLE_OUT) -> str:
    body = ["// AUTO-GENERATED by equitorch_b200/csrc/gen_path_specs.py - do not edit.", "#pragma once",
            "template <int LO, int LS, int LF> struct CgTriple;", ""]
    body += [_emit_triple(*t) for t in triples(TRIPLE_MAX_L)]
    body.append(f"constexpr int TRIPLE_MAX_L = {TRIPLE_MAX_L};")
    return _write(path, "\n".join(body) + "\n")


def generate(path: str = OUT) -> str:
    body = ["// AUTO-GENERATED by equitorch_b200/csrc/gen_path_specs.py - do not edit.", "#pragma once",
            "template <int LO, int L1, int L2> struct CgPath;", ""]
    body += [_emit(*t) for t in triples()]
    body.append(f"constexpr int PATH_MAX_L = {MAX_L};")
    return _write(path, "\n".join(body) + "\n")


if __name__ == "__main__":
    print(generate(), generate_triples())
