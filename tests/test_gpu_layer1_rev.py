"""The layer-1 adjoint (k_layer1_rev.cu): edge counts around its sum batches (4 edges) and
staging chunks (8, 16 and 32 edges), both edge splits, both CG tables, every instruction
group; and the fixed-point conversion it adds H1_adj terms with (CPU)."""
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
@pytest.mark.parametrize("C,L_max,padded", [(32, 1, 1), (96, 1, 0), (128, 1, 1), (64, 2, 1), (32, 2, 0)])
def test_edge_counts_and_splits(engine_lib, tmp_path, C, L_max, padded):
    from oracle.pyoracle import Evaluator
    from symmetrix_gb300 import MACE
    from symmetrix_gb300.synth.model import make_model, write_model
    from symmetrix_gb300.synth.structures import neighbor_list
    path = write_model(make_model(num_channels=C, species=("H", "C", "O"), r_cut=5.0, L_max=L_max, num_knots=60,
                                  seed=5, avg_num_neighbors=40.0), str(tmp_path / "m.json"))
    pos, species = clusters([1, 2, 4, 5, 6, 9, 10, 17, 18, 33, 34], 3, 3)
    nl = neighbor_list(pos, 5.0)
    a = edge_args(species, nl)
    m = MACE(path)
    m.set_option("cg_padded", padded)
    m.compute_node_energies_forces(*a)
    e, f, h = m.node_energies, m.node_forces, m.H1_adj
    ref = Evaluator(path, "port")
    ref.compute_node_energies_forces(*a)
    # float32 sums of a few hundred terms against float64: 1e-5 of the largest component
    for got, want in ((e, ref.node_energies), (f, ref.node_forces), (h, ref.get("H1_adj"))):
        assert np.abs(got - want).max() <= 1e-5 * max(1.0, np.abs(want).max())
    # many copies: the edges of a node stay with one warp; the same bits
    n, E = len(species), len(nl["r"])
    copies = 1 + 3000 // (n * C // 32)
    rep = [np.tile(nl["neigh_indices"], copies) + np.repeat(np.arange(copies) * n, E)]
    m.compute_node_energies_forces(n * copies, np.tile(species, copies), np.tile(nl["num_neigh"], copies), rep[0],
                                   np.tile(a[4], copies), np.tile(nl["xyz"], (copies, 1)), np.tile(nl["r"], copies))
    assert np.array_equal(m.node_forces.reshape(copies, -1), np.tile(f, (copies, 1)))
    assert np.array_equal(m.H1_adj.reshape(copies, -1), np.tile(h, (copies, 1)))


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
