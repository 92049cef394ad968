"""Generate cg_canon.h: which output components each layer-1 tensor-product path reaches.

The real Clebsch-Gordan coefficients of (l1, l2) -> l in the evaluator's Y_lm basis are
fixed up to a factor, so their zero pattern is too: path (q, m1, m2) of instruction q
contributes to none, one or two of the 2 l + 1 output components, whatever the model.
The layer-1 kernels are compiled for this pattern (paths without a component are left
out); the values come from the model, and a model with another pattern runs the general
form.

    python symmetrix_gb300/csrc/gen_cg.py      # rewrites cg_canon.h next to it
"""
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(os.path.dirname(HERE)))

from symmetrix_gb300.synth.equivariant import phi1_tables  # noqa: E402


def pattern(L_max):
    """Per path the output components m it reaches, in ascending order."""
    phi, num_e = phi1_tables(3, L_max)
    n_p = sum((2 * a + 1) * (2 * b + 1) for a, b in zip(phi["Phi1_l1"], phi["Phi1_l2"]))
    off = [sum((2 * l + 1) * num_e[l] for l in range(q)) for q in range(5)]
    out = [set() for _ in range(n_p)]
    for lme, p in zip(phi["Phi1_lme"], phi["Phi1_lelm1lm2"]):
        l = max(q for q in range(4) if off[q] <= lme)
        out[p].add((lme - off[l]) // num_e[l])
    assert all(len(m) <= 2 for m in out)
    return [sorted(m) for m in out]


def main(out_dir=HERE):
    lines = ["// Generated by gen_cg.py: do not edit.", "#pragma once", "", "namespace smx {", "",
             "// output component of the t-th term (t = 0, 1) of layer-1 path p, or -1",
             "__host__ __device__ constexpr int cg_m(int LMAX, int p, int t) {"]
    for L in (1, 2):
        flat = [v for m in pattern(L) for v in (m + [-1, -1])[:2]]
        lines.append(f"  constexpr signed char t{L}[{len(flat)}] = {{")
        for i in range(0, len(flat), 30):
            lines.append("      " + ", ".join(str(v) for v in flat[i:i + 30]) + ",")
        lines[-1] = lines[-1].rstrip(",") + "};"
    lines += ["  return LMAX == 1 ? t1[2 * p + t] : t2[2 * p + t];", "}", "", "}  // namespace smx", ""]
    with open(os.path.join(out_dir, "cg_canon.h"), "w") as f:
        f.write("\n".join(lines))


if __name__ == "__main__":
    main()
