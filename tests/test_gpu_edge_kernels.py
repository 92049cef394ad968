"""The edge kernels of both layers (k_edge.cu, k_layer1.cu, k_layer1_rev.cu): edge counts around
the adjoints' sum batches (4 edges) and the staging chunks (4 to 32 edges), nodes of one and
of several warps, channel counts that leave lanes idle or need several channel blocks, every
instruction group, the Clebsch-Gordan tables (the canonical zero pattern, its general form, a
table outside the pattern) and contraction polynomials outside the canonical set; the
pattern's generated source and the fixed-point conversion of the H1_adj terms (CPU)."""
import importlib.util
import os
import sys

import numpy as np
import pytest

from helpers import edge_args


def clusters(sizes, seed, S):
    """Far-apart clusters whose atoms all see each other: an atom of a cluster of m has m - 1 edges."""
    rng = np.random.default_rng(seed)
    pos = []
    for c, m in enumerate(sizes):
        p = np.zeros((0, 3))
        while len(p) < m:
            v = rng.uniform(-2.4, 2.4, 3)
            if np.linalg.norm(v) < 2.4 and (len(p) == 0 or np.linalg.norm(p - v, axis=1).min() > 0.55):
                p = np.concatenate([p, v[None]])
        pos.append(p + np.array([30.0 * c, 0.0, 0.0]))
    n = sum(sizes)
    return np.concatenate(pos), rng.integers(0, S, n).astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("C,L_max,table", [(32, 1, "canonical"), (96, 1, "rows"), (128, 1, "canonical"),
                                           (64, 2, "canonical"), (32, 2, "rows"), (64, 1, "other"), (96, 2, "other"),
                                           (192, 1, "canonical"), (32, 1, "poly"), (64, 2, "poly")])
def test_edge_counts_and_splits(engine_lib, tmp_path, C, L_max, table):
    from oracle.pyoracle import Evaluator
    from symmetrix_gb300 import MACE
    from symmetrix_gb300.synth.model import make_model, write_model
    from symmetrix_gb300.synth.structures import neighbor_list
    model = make_model(num_channels=C, species=("H", "C", "O"), r_cut=5.0, L_max=L_max, num_knots=60, seed=5,
                       avg_num_neighbors=40.0)
    if table == "other":  # one term on a path that reaches no output in the canonical pattern
        unused = sorted(set(range(max(model["Phi1_lelm1lm2"]) + 1)) - set(model["Phi1_lelm1lm2"]))[0]
        model["Phi1_lme"].append(0)
        model["Phi1_lelm1lm2"].append(unused)
        model["Phi1_clebsch_gordan"].append(0.3)
    if table == "poly":  # one monomial more than the canonical set of output 0
        model["M0_monomials"]["0"].append([0, 1])
        for w in model["M0_weights"].values():
            for k in w["0"]:
                w["0"][k].append(0.1)
    path = write_model(model, str(tmp_path / "m.json"))
    pos, species = clusters([1, 2, 4, 5, 6, 9, 10, 17, 18, 33, 34], 3, 3)
    nl = neighbor_list(pos, 5.0)
    a = edge_args(species, nl)
    m = MACE(path)
    m.set_option("cg_padded", 0 if table == "rows" else 1)
    m.compute_node_energies_forces(*a)
    stages = ("A0", "M0", "Phi1", "H1_adj", "A0_adj")
    ref = Evaluator(path, "port")
    ref.compute_node_energies_forces(*a)
    # float32 sums of a few hundred terms against float64: 1e-5 of the largest component
    for got, want in [(m.node_energies, ref.node_energies), (m.node_forces, ref.node_forces)] + [
            (m.stage(s), ref.get(s)) for s in stages]:
        assert np.abs(got - want).max() <= 1e-5 * max(1.0, np.abs(want).max())
    # many copies: the edges of a node stay with one warp
    n, E = len(species), len(nl["r"])
    copies = 1 + 4 * 12 * 152 // (n * max(C // 64, 1))
    rep = np.tile(nl["neigh_indices"], copies) + np.repeat(np.arange(copies) * n, E)
    m.compute_node_energies_forces(n * copies, np.tile(species, copies), np.tile(nl["num_neigh"], copies), rep,
                                   np.tile(a[4], copies), np.tile(nl["xyz"], (copies, 1)), np.tile(nl["r"], copies))
    for got, want in [(m.node_forces, ref.node_forces)] + [(m.stage(s), ref.get(s)) for s in stages]:
        assert np.abs(got.reshape(copies, -1) - want).max() <= 1e-5 * max(1.0, np.abs(want).max())


def test_generated_pattern_is_current(tmp_path):
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "symmetrix_gb300", "csrc")
    spec = importlib.util.spec_from_file_location("gen_cg", os.path.join(csrc, "gen_cg.py"))
    gen = importlib.util.module_from_spec(spec)
    keep, sys.dont_write_bytecode = sys.dont_write_bytecode, True
    try:
        spec.loader.exec_module(gen)
    finally:
        sys.dont_write_bytecode = keep
    gen.main(out_dir=str(tmp_path))
    with open(os.path.join(csrc, "cg_canon.h")) as f, open(tmp_path / "cg_canon.h") as g:
        assert f.read() == g.read()


def test_to_fixed_is_the_rounding_of_v_2_to_34():
    """to_fixed (device.cuh) restated: the three words with their bias 0x4B400000 taken off as one
    64-bit constant give round-half-even(v 2^34) exactly."""
    rng = np.random.default_rng(4)
    v = (rng.uniform(-1, 1, 200000) * 2.0 ** rng.integers(-36, 29, 200000)).astype(np.float32)
    f32, magic = np.float32, np.float32(12582912.0)

    def fma(x, y, z):  # exact in float64 here (products of 24-bit values by powers of two), one rounding
        return (x.astype(np.float64) * y + np.float64(z)).astype(f32)

    ta = fma(v, 2.0 ** -10, magic)
    va = (v.astype(np.float64) - (ta - magic).astype(np.float64) * 1024.0).astype(f32)
    tb = fma(va, 4096.0, magic)
    vb = (va.astype(np.float64) - (tb - magic).astype(np.float64) / 4096.0).astype(f32)
    tc = fma(vb, 2.0 ** 34, magic)
    a, b, c = (t.view(np.uint32).astype(np.uint64) for t in (ta, tb, tc))
    k = 0x4B400000
    bias = np.uint64(((k << 44) + (k << 22) + k) % 2 ** 64)
    with np.errstate(over="ignore"):
        q = (((a << np.uint64(12)) & np.uint64(0xFFFFFFFF)) << np.uint64(32)) + ((b << np.uint64(22)) + c) - bias
    assert np.array_equal(q.view(np.int64), np.rint(v.astype(np.float64) * 2.0 ** 34).astype(np.int64))
