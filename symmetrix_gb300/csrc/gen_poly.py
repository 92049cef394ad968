"""Generate poly_canon.h: straight-line CUDA for the symmetric-contraction polynomials.

The monomials of a MACE symmetric contraction (degree <= 3 in the 16 A-basis
components, l_max = 3) are fixed by the equivariance of each output component LM:
every species and channel uses the same monomial set, only the coefficients differ
(extract_mace_data.py:239-304 folds U tensors and weights into exactly these
coefficients).  This script writes those sets, in the order symmetrix_gb300.synth
emits them, as compile-time code: the A-basis values and the gradient live in
registers, and the nested form sum_a x_a (c_a + sum_b x_b (c_ab + sum_c c_abc x_c)) costs
one coalesced coefficient load and one FMA per cubic monomial, two with its gradient,
without products of pairs kept in registers.

    python symmetrix_gb300/csrc/gen_poly.py      # rewrites poly_canon.h next to it
"""
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(os.path.dirname(HERE)))

from symmetrix_gb300.synth.equivariant import equivariant_polynomial_basis  # noqa: E402

L_MAX = 2  # hidden irreps up to 0e + 1o + 2e: LM = 0..8 (an L_max = 1 model uses LM = 0..3)


def canonical(L, M):
    keys = []
    for d in (1, 2, 3):
        mono, U = equivariant_polynomial_basis(L, d, 3)
        for t, key in enumerate(mono):
            if (U[:, M, t] != 0.0).any():
                keys.append(tuple(key))
    return keys


def pack(m):
    idx = list(m) + [16] * (3 - len(m))
    return idx[0] | (idx[1] << 8) | (idx[2] << 16)


def tree(monos):
    """{a: (t of x_a, {b: (t of x_a x_b, [(c, t of x_a x_b x_c)])})}, t = None where there is no such
    monomial: the polynomial as sum_a x_a (c_a + sum_b x_b (c_ab + sum_c c_abc x_c))."""
    out = {}
    for t, m in enumerate(monos):
        node = out.setdefault(m[0], [None, {}])
        if len(m) == 1:
            node[0] = t
            continue
        leaf = node[1].setdefault(m[1], [None, []])
        if len(m) == 2:
            leaf[0] = t
        else:
            leaf[1].append((m[2], t))
    return out


def coef(t):
    return f"ld(cf + {t} * S)"


def inner(leaf, grad):
    """r = c_ab + sum_c c_abc x_c, with the gradient terms of the x_c."""
    t, cubic = leaf
    first = t is None
    out = [] if first else [f"r = {coef(t)};"]
    for c, u in cubic:
        if grad:
            out.append(f"k = {coef(u)}; g[{c}] = fm(wab, k, g[{c}]);")
        k = "k" if grad else coef(u)
        out.append(f"r = ml({k}, x[{c}]);" if first else f"r = fm({k}, x[{c}], r);")
        first = False
    return out


def value_fn(name, monos):
    out = ["template <typename V>", f"__device__ __forceinline__ V {name}(const V* x, const V* __restrict__ cf, int S) {{",
           "  V f, q, r;"]
    started = False
    for a, (t, bs) in tree(monos).items():
        first = t is None
        if not first:
            out.append(f"  q = {coef(t)};")
        for b, leaf in bs.items():
            out.append("  " + " ".join(inner(leaf, False) + [f"q = ml(x[{b}], r);" if first else f"q = fm(x[{b}], r, q);"]))
            first = False
        out.append(f"  f = fm(x[{a}], q, f);" if started else f"  f = ml(x[{a}], q);")
        started = True
    out += ["  return f;", "}"]
    return "\n".join(out)


def grad_body(monos, value):
    """g[v] += w dP/dx_v, and with `value` f = P."""
    out, started = [], False
    for a, (t, bs) in tree(monos).items():
        out.append(f"  wa = ml(w, x[{a}]);")
        first = t is None
        if not first:
            out.append(f"  q = {coef(t)};")
        for b, leaf in bs.items():
            line = [f"wab = ml(wa, x[{b}]);"] if leaf[1] else []
            line += inner(leaf, True)
            line += [f"q = ml(x[{b}], r);" if first else f"q = fm(x[{b}], r, q);", f"g[{b}] = fm(wa, r, g[{b}]);"]
            out.append("  " + " ".join(line))
            first = False
        out.append(f"  g[{a}] = fm(w, q, g[{a}]);")
        if value:
            out.append(f"  f = fm(x[{a}], q, f);" if started else f"  f = ml(x[{a}], q);")
            started = True
    return out


def grad_fn(name, monos):
    out = ["template <typename V>",
           f"__device__ __forceinline__ void {name}(const V* x, V w, const V* __restrict__ cf, int S, V* g) {{",
           "  V q, r, k, wa, wab;"]
    return "\n".join(out + grad_body(monos, False) + ["}"])


def value_grad_fn(name, monos):
    # (the gradient unweighted: w = 1, whose products the compiler drops)
    out = ["template <typename V>",
           f"__device__ __forceinline__ V {name}(const V* x, const V* __restrict__ cf, int S, V* g) {{",
           "  V f, q, r, k, wa, wab;"]
    body = [l.replace("  wa = ml(w, ", "  wa = (").replace("fm(w, q, g[", "ad(q, g[") for l in grad_body(monos, True)]
    return "\n".join(out + body + ["  return f;", "}"])


def main(out_dir=HERE):
    lists = []
    for L in range(L_MAX + 1):
        for M in range(2 * L + 1):
            lists.append(canonical(L, M))
    nLM = len(lists)
    flat = [pack(m) for lst in lists for m in lst]
    offs = [0]
    for lst in lists:
        offs.append(offs[-1] + len(lst))
    t = ["// Generated by gen_poly.py: canonical symmetric-contraction monomial tables (l_max 3,",
         "// degree <= 3), shared by host and device code.  Do not edit; rerun the script.",
         "#pragma once", "", "namespace smx {", "namespace poly {", "",
         f"constexpr int kNumLM = {nLM};  // LM = 0 .. (L_max + 1)^2 - 1 for L_max up to {L_MAX}",
         f"constexpr int kOffset[{nLM + 1}] = {{{', '.join(map(str, offs))}}};",
         "// packed a | b << 8 | c << 16, 16 = constant one; LM-major, canonical order",
         f"constexpr int kMono[{len(flat)}] = {{{', '.join(map(str, flat))}}};", "",
         "}  // namespace poly", "}  // namespace smx", ""]
    with open(os.path.join(out_dir, "poly_canon_tables.h"), "w") as f:
        f.write("\n".join(t))
    h = ["// Generated by gen_poly.py: canonical symmetric-contraction monomials (l_max 3,",
         "// degree <= 3) as straight-line code, for one channel (float) or two (float2, packed FMAs).",
         "// Do not edit; rerun the script.",
         "#pragma once", "", '#include "poly_canon_tables.h"', "", "namespace smx {", "namespace poly {", "",
         "__device__ __forceinline__ float ld(const float* p) { return __ldg(p); }",
         "__device__ __forceinline__ float2 ld(const float2* p) { return __ldg(p); }",
         "__device__ __forceinline__ float fm(float a, float b, float c) { return fmaf(a, b, c); }",
         "__device__ __forceinline__ float2 fm(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }",
         "__device__ __forceinline__ float ml(float a, float b) { return a * b; }",
         "__device__ __forceinline__ float2 ml(float2 a, float2 b) { return __fmul2_rn(a, b); }",
         "__device__ __forceinline__ float ad(float a, float b) { return a + b; }",
         "__device__ __forceinline__ float2 ad(float2 a, float2 b) { return __fadd2_rn(a, b); }", ""]
    for LM, lst in enumerate(lists):
        h.append(value_fn(f"value_LM{LM}", lst))
        h.append("")
        h.append(grad_fn(f"grad_LM{LM}", lst))
        h.append("")
    h.append("// the layer-1 contraction is the LM = 0 set")
    h.append(value_grad_fn("value_grad_M1", lists[0]))
    h += ["", "}  // namespace poly", "}  // namespace smx", ""]
    path = os.path.join(out_dir, "poly_canon.h")
    with open(path, "w") as f:
        f.write("\n".join(h))
    print(f"wrote {path}: {[len(x) for x in lists]} monomials")


if __name__ == "__main__":
    main()
