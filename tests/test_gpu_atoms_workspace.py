"""The atom-level calls keep their buffers in the engine: growing and shrinking systems,
periodic, non-periodic and molecule calls and failed calls in between leave no trace in the
results; node counts around the scan's tiles (1024 x 8) and a neighbour list's reverse edges."""
import numpy as np
import pytest

from symmetrix_gb300.synth.structures import neighbor_list, random_box

pytestmark = pytest.mark.gpu


def test_calls_in_any_order_give_a_fresh_engines_results(engine_lib, small_model_path):
    from symmetrix_gb300 import MACE
    rng = np.random.default_rng(3)
    big, L, sp_big = random_box(300, 0.07, 0.9, 3, seed=4)
    small, Ls, sp_small = random_box(20, 0.05, 0.9, 3, seed=5)
    cluster = rng.normal(size=(30, 3)) * 3.0
    sp_cluster = rng.integers(0, 3, 30).astype(np.int32)
    mols = [(small[:7], sp_small[:7]), (cluster, sp_cluster), (small[7:], sp_small[7:])]
    calls = [lambda m: m.compute_atoms(small, sp_small, Ls), lambda m: m.compute_atoms(big, sp_big, L),
             lambda m: m.compute_molecules(mols), lambda m: m.compute_atoms(cluster, sp_cluster),
             lambda m: m.compute_molecules(mols[:1]), lambda m: m.compute_atoms(small, sp_small, Ls),
             lambda m: m.compute_atoms(np.zeros((0, 3)), np.zeros(0, np.int32)),
             lambda m: m.compute_atoms(big, sp_big, L)]

    def flat(r):
        return np.concatenate([np.concatenate([np.ravel(y) for y in x]) if isinstance(x, list) else np.ravel(x) for x in r])

    def fresh(c):
        m = MACE(small_model_path)
        m.set_option("autotune", 0)
        return flat(c(m))

    want = [fresh(c) for c in calls]
    m = MACE(small_model_path)
    m.set_option("autotune", 0)
    for c, w in zip(calls, want):
        assert np.array_equal(flat(c(m)), w)
        with pytest.raises(ValueError):
            m.compute_atoms(small, sp_small + 3, Ls)  # species out of range
        with pytest.raises(ValueError):
            m.compute_atoms(small, sp_small, -1.0)  # a box without a volume
    for c, w in zip(calls[::-1], want[::-1]):
        assert np.array_equal(flat(c(m)), w)


@pytest.mark.parametrize("n", [1, 8, 1023, 8191, 8192, 8193, 16385])
def test_node_offsets_around_the_scan_tiles(engine_lib, small_model_path, n):
    """Dimers and one odd atom: every node's offset is needed for its own edge and energy."""
    from symmetrix_gb300 import MACE
    m = MACE(small_model_path)
    pairs = n // 2
    num = np.ones(n, np.int32)
    if n % 2:
        num[-1] = 0
    nb = (np.arange(2 * pairs) ^ 1).astype(np.int32)
    sp = (np.arange(n) // 2 % 3).astype(np.int32)
    d = np.zeros((2 * pairs, 3))
    d[:, 0] = 2.0 * (1 - 2 * (np.arange(2 * pairs) % 2))
    m.compute_node_energies_forces(n, sp, num, nb, sp[nb] if pairs else sp[:0], d, np.abs(d[:, 0]))
    e, f = m.node_energies, m.node_forces.reshape(-1, 3)
    for s in range(3):  # all dimers of one species pair agree, to the bit
        same = np.nonzero(sp[:2 * pairs] == s)[0]
        assert np.ptp(e[same]) == 0.0 if len(same) else True
        assert np.ptp(f[same[::2]], axis=0).max() == 0.0 if len(same) else True
    nl = neighbor_list(np.array([[0.0, 0.0, 0.0], [2.0, 0.0, 0.0]]), m.r_cut)
    assert len(nl["r"]) == 2
