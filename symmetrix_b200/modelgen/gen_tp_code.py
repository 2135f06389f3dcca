"""Generates the straight-line inner loops of the tensor-product kernels and the canonical coupling table.

    python -m symmetrix_b200.modelgen.gen_tp_code      # rewrites symmetrix_b200/csrc/generated/*

For each highest feature degree L (0, 1, 2) the layer-1 tensor product
``Phi1[(l m e_p)] += R_p * sum_{m1 m2} C^{l m}_{l1 m1, l2 m2} Y[l1 m1] H[l2 m2]`` (reference form:
libsymmetrix/source/mace.cpp:453-502) has a fixed sparsity pattern in the real-harmonics basis. Writing
the non-zeros out as straight-line code keeps every accumulator in a register and lets the coupling
constants be instruction immediates. The files written:

* ``tp_L{L}_forward.inc``  per (edge, channel): uses ``Y[16]``, ``h[nLM]``, ``R[P]``; updates ``acc[Q]``.
* ``tp_L{L}_reverse.inc``  per (edge, channel): uses ``d[Q]``, ``Y[16]``, ``h[nLM]``, ``R[P]``, ``Rd[P]``;
  updates ``msg[nLM]`` (adjoint of the sender features), ``W[16]`` (adjoint of the harmonics) and ``fr``
  (adjoint of the edge length).
* ``tp_scale.hpp``         the factor of every output component that this code leaves out, see :func:`scaled`.
* ``cg_canon.hpp``         the same non-zeros as a table; the model loader checks a model file's
  Clebsch-Gordan COO against it path by path and folds the per-path scale into the radial tables.

The constants come from :func:`symmetrix_b200.modelgen.harmonics.coupling` (unit-normalised per output
component, sign fixed), in the path order of ``csrc/tp_tables.hpp``.
"""
from __future__ import annotations

import math
from fractions import Fraction
from pathlib import Path

from .generate import tp_paths
from .harmonics import coupling

OUT = Path(__file__).resolve().parents[1] / "csrc" / "generated"
L_MAX = 3


def tables(L: int):
    paths = tp_paths(L_MAX, L)
    ls = [p[0] for p in paths]
    n_e = [sum(1 for x in ls if x == l) for l in range(L_MAX + 1)]
    lme_off = [sum((2 * ll + 1) * n_e[ll] for ll in range(l)) for l in range(L_MAX + 1)]
    e_of = []
    seen = [0] * (L_MAX + 1)
    for l, _, _ in paths:
        e_of.append(seen[l]); seen[l] += 1
    nz = []   # (p, m, lm1, lm2, c)
    for p, (l, l1, l2) in enumerate(paths):
        cg = coupling(l1, l2, l)
        for m in range(2 * l + 1):
            for m1 in range(2 * l1 + 1):
                for m2 in range(2 * l2 + 1):
                    c = snap(float(cg[m, m1, m2]))
                    if abs(c) > 1e-12:
                        nz.append((p, m, l1 * l1 + m1, l2 * l2 + m2, c))
    lme = lambda p, m: lme_off[paths[p][0]] + m * n_e[paths[p][0]] + e_of[p]   # noqa: E731
    return paths, nz, lme


def snap(c: float) -> float:
    """Coupling constants are square roots of small rationals; remove the 1e-16 noise of their numerical derivation."""
    if abs(c) < 1e-12:
        return 0.0
    frac = Fraction(c * c).limit_denominator(20000)
    if abs(float(frac) - c * c) < 1e-12:
        return math.copysign(math.sqrt(frac.numerator / frac.denominator), c)
    return c


def lit(c: float) -> str:
    return f"T({c!r})"


def scaled(L: int):
    """The non-zeros with every output component (path, m) rescaled so that most of its constants are one.

    Returns ``(nz, scale)``: entries ``(p, m, lm1, lm2, c')`` with ``c = scale[p, m] * c'``. The kernels multiply the receiver's
    adjoint by ``scale`` when they load it and the accumulators when they store them, once per receiver; per edge, a constant
    of one costs nothing (L_max = 1: 59 of 86 entries) and -1 is a sign (9 more)."""
    _, nz, _ = tables(L)
    rows: dict = {}
    for (p, m, a, b, c) in nz:
        rows.setdefault((p, m), []).append((a, b, c))
    out, scale = [], {}
    for (p, m), terms in rows.items():
        sizes = [round(abs(c), 9) for _, _, c in terms]
        common = max(sorted(set(sizes)), key=sizes.count)
        t = next(abs(c) for _, _, c in terms if round(abs(c), 9) == common)
        if 2 * sum(c < 0 for _, _, c in terms) > len(terms):
            t = -t
        scale[p, m] = t
        out += [(p, m, a, b, 1.0 if abs(c / t - 1.0) < 1e-12 else -1.0 if abs(c / t + 1.0) < 1e-12 else c / t) for (a, b, c) in terms]
    return out, scale


class Multiples:
    """Names of the constant multiples ``c * source`` used in one block of code; ``c = 1`` is the source itself."""

    def __init__(self):
        self.lines, self.names = [], {}

    def of(self, source: str, stem: str, c: float) -> str:
        if c == 1.0:
            return source
        key = (source, c)
        if key not in self.names:
            name = f"{stem}_{len(self.names)}"
            self.names[key] = name
            self.lines.append(f"        const T {name} = " + (f"-{source};" if c == -1.0 else f"{lit(c)} * {source};"))
        return self.names[key]


def gen_forward(L: int) -> str:
    paths, _, lme = tables(L)
    nz, _ = scaled(L)
    out = [f"// generated by symmetrix_b200/modelgen/gen_tp_code.py -- tensor product forward, L_max = {L}",
           "// acc[] are in units of TPScale (applied when they are stored)", "{"]
    for p, (l, l1, l2) in enumerate(paths):
        mine = [(m, a, b, c) for (pp, m, a, b, c) in nz if pp == p]
        out.append(f"    {{   // path {p}: l = {l}, harmonics degree {l1}, feature degree {l2}")
        if l1 == 0 and all(c == 1.0 for (_, _, _, c) in mine):      # the harmonic of degree zero is 1
            out += [f"        acc[{lme(p, m)}] = fma(R[{p}], h[{b}], acc[{lme(p, m)}]);" for (m, _, b, _) in mine] + ["    }"]
            continue
        for b in sorted({x[2] for x in mine}):
            out.append(f"        const T x{b} = R[{p}] * h[{b}];")
        mult = Multiples()
        body = [f"        acc[{lme(p, m)}] = fma(Y[{a}], {mult.of(f'x{b}', f'x{b}', c)}, acc[{lme(p, m)}]);" for (m, a, b, c) in mine]
        out += mult.lines + body + ["    }"]
    out.append("}")
    return "\n".join(out) + "\n"


def gen_reverse(L: int, by_path: bool = False) -> str:
    """`by_path`: the receiver's adjoint is not a register array `d[Q]` but is fetched path by path -- the kernel
    defines TP_PATH_D(p, n, dp), which fills `T dp[n]` with the 2l+1 values of path p (from tensor memory)."""
    paths, _, lme = tables(L)
    nz, _ = scaled(L)
    out = [f"// generated by symmetrix_b200/modelgen/gen_tp_code.py -- tensor product reverse, L_max = {L}"
           + (", receiver adjoint fetched path by path" if by_path else ""),
           "// W[16] and msg[nLM] are ASSIGNED by their first contribution (every entry has one): no zero-fill is needed; W[0] is the",
           "// adjoint of the edge length (the harmonic of degree zero is 1 everywhere, its adjoint meets a zero gradient); the receiver's",
           "// adjoint has been multiplied by TPScale", "{"]
    touched = set()     # accumulators that already hold a contribution

    def accumulate(name: str, x: str, y: str) -> str:
        if name in touched:
            return f"        {name} = fma({x}, {y}, {name});"
        touched.add(name)
        return f"        {name} = {x} * {y};"

    for p, (l, l1, l2) in enumerate(paths):
        mine = [(m, a, b, c) for (pp, m, a, b, c) in nz if pp == p]
        bs = sorted({x[2] for x in mine})
        out.append(f"    {{   // path {p}: l = {l}, harmonics degree {l1}, feature degree {l2}")
        if by_path:
            out.append(f"        T dp[{2 * l + 1}];")
            out.append(f"        TP_PATH_D({p}, {2 * l + 1}, dp);")
        if l1 > 0:
            for b in bs:
                out.append(f"        const T x{b} = R[{p}] * h[{b}];")
        mult, body, begun = Multiples(), [], set()
        for (m, a, b, c) in mine:
            d = mult.of(f"dp[{m}]" if by_path else f"d[{lme(p, m)}]", f"d{m}", c)
            if l1 == 0:         # one harmonic, equal to 1
                body.append(f"        u{b} = u{b} + {d};" if b in begun else f"        T u{b} = {d};")
                begun.add(b)
                continue
            # u[m2] = sum d * Y[m1]: adjoint of the sender features before the radial factor
            body.append(f"        u{b} = fma({d}, Y[{a}], u{b});" if b in begun else f"        T u{b} = {d} * Y[{a}];")
            begun.add(b)
            # adjoint of the harmonics
            body.append(accumulate(f"W[{a}]", d, f"x{b}"))
        out += mult.lines + body
        for b in bs:
            out.append(accumulate(f"msg[{b}]", f"R[{p}]", f"u{b}"))
        sexpr = f"u{bs[0]} * h[{bs[0]}]"
        for b in bs[1:]:
            sexpr = f"fma(u{b}, h[{b}], {sexpr})"
        out.append(accumulate("W[0]", f"Rd[{p}]", f"({sexpr})"))
        out.append("    }")
    nlm_feat = (L + 1) ** 2
    missing = [n for n in [f"W[{a}]" for a in range(16)] + [f"msg[{b}]" for b in range(nlm_feat)] if n not in touched]
    if missing:
        raise RuntimeError(f"reverse code for L_max = {L} leaves {missing} without a contribution")
    out.append("}")
    return "\n".join(out) + "\n"


def gen_scale() -> str:
    out = ["// generated by symmetrix_b200/modelgen/gen_tp_code.py -- factor of every tensor-product output component that the",
           "// generated code leaves out (forward: of the accumulators; reverse: of the receiver's adjoint); used as a local constexpr object", "#pragma once", "",
           "namespace smx {", "template <int LF> struct TPScale;"]
    for L in range(4):
        paths, _, lme = tables(L)
        _, scale = scaled(L)
        q = sum(2 * p[0] + 1 for p in paths)
        vals = [1.0] * q
        for (p, m), t in scale.items():
            vals[lme(p, m)] = t
        out.append(f"template <> struct TPScale<{L}> {{")
        out.append(f"    double q[{q}] = {{")
        for i in range(0, q, 5):
            out.append("        " + " ".join(f"{v!r}," for v in vals[i:i + 5]))
        out.append("    };")
        out.append("};")
    out.append("}  // namespace smx")
    return "\n".join(out) + "\n"


def gen_table() -> str:
    out = ["// generated by symmetrix_b200/modelgen/gen_tp_code.py -- canonical non-zeros of the real Clebsch-Gordan map",
           "// entries: path, m index (0..2l), harmonics index lm1, feature index lm2, value", "#pragma once", "",
           "namespace smx {", "struct CanonCG { int p, m, lm1, lm2; double c; };", "template <int LF> struct CanonCGTable;"]
    for L in range(4):
        _, nz, _ = tables(L)
        out.append(f"template <> struct CanonCGTable<{L}> {{")
        out.append(f"    static constexpr int n = {len(nz)};")
        out.append(f"    static constexpr CanonCG e[{len(nz)}] = {{")
        for (p, m, a, b, c) in nz:
            out.append(f"        {{{p}, {m}, {a}, {b}, {c!r}}},")
        out.append("    };")
        out.append("};")
    out.append("}  // namespace smx")
    return "\n".join(out) + "\n"


def main():
    OUT.mkdir(parents=True, exist_ok=True)
    for L in range(4):
        (OUT / f"tp_L{L}_forward.inc").write_text(gen_forward(L))
        (OUT / f"tp_L{L}_reverse.inc").write_text(gen_reverse(L))
        (OUT / f"tp_L{L}_reverse_bypath.inc").write_text(gen_reverse(L, by_path=True))
        _, nz, _ = tables(L)
        print(f"L_max = {L}: {len(nz)} non-zeros")
    (OUT / "cg_canon.hpp").write_text(gen_table())
    (OUT / "tp_scale.hpp").write_text(gen_scale())


if __name__ == "__main__":
    main()
