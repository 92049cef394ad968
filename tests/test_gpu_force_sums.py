"""Per-edge forces are summed in float64 above the float32 sums over lanes: the layer-1 adjoint's three
instruction groups at L_max = 2 (an infinite force stays one), the layer-0 adjoint's 64-channel sums."""
import numpy as np
import pytest

from helpers import edge_args
from symmetrix_gb300.synth.model import make_model, write_model
from symmetrix_gb300.synth.structures import neighbor_list, random_box

pytestmark = pytest.mark.gpu

# (l1, l2, l) of the groups of l2 = 2; the first group has the instructions of l2 = 0, 1
GROUPS = [{(0, 2, 2), (1, 2, 3), (2, 2, 0), (3, 2, 3)}, {(1, 2, 1), (2, 2, 2), (3, 2, 1)}]


def test_instruction_groups_of_l_max_2(engine_lib, tmp_path):
    """The edge forces of dPhi1 are the float64 sum of those of its rows of each group."""
    from symmetrix_gb300 import MACE
    C = 32  # one slice
    model = make_model(num_channels=C, species=("H", "C", "O"), r_cut=4.0, L_max=2, num_knots=40, seed=4)
    m = MACE(write_model(model, str(tmp_path / "m.json")))
    pos, L, species = random_box(40, 0.08, 0.9, 3, seed=6)
    nl = neighbor_list(pos, 4.0, L)
    a = edge_args(species, nl)
    n = len(species)
    m.compute_node_energies_forces(*a)
    ins = list(zip(model["Phi1_l1"], model["Phi1_l2"], model["Phi1_l"]))
    group, at = np.zeros(m.stage("Phi1_adj").size // (n * C), int), 0
    for l in range(4):
        of_l = [q for q in ins if q[2] == l]
        for k in range((2 * l + 1) * len(of_l)):
            q = of_l[k % len(of_l)]
            group[at + k] = 1 if q in GROUPS[0] else (2 if q in GROUPS[1] else 0)
        at += (2 * l + 1) * len(of_l)
    assert at == len(group)
    dPhi1 = np.random.default_rng(1).normal(size=(n, len(group), C)).astype(np.float32)
    m.compute_R1(n, species, a[2], a[4], a[6])
    m.compute_Y(a[5])

    def forces(mask):
        m.set_stage("Phi1_adj", dPhi1 * mask[None, :, None])
        m.reverse_Phi1(n, a[2], a[3], a[5], a[6], True, True)
        return np.array(m.node_forces)

    parts = [forces(group == g) for g in range(3)]
    for p in parts:  # float32 sums, one slice
        assert np.abs(p).max() > 1e-3 and np.array_equal(p, p.astype(np.float32))
    err = np.abs(forces(group >= 0) - (parts[0] + parts[1] + parts[2])).max()
    assert err <= 1e-13 * max(np.abs(p).max() for p in parts)


@pytest.mark.parametrize("L_max", [1, 2])
def test_infinite_layer_1_forces(engine_lib, tmp_path, L_max):
    """One channel's scalar row whose product with H1 is beyond float32: the edge forces are infinite,
    with the signs of a finite row's, at L_max = 2 through the sum of the three groups too."""
    from symmetrix_gb300 import MACE
    C, c = 32, 5
    model = make_model(num_channels=C, species=("H", "C", "O"), r_cut=4.0, L_max=L_max, num_knots=40, seed=4)
    assert (model["Phi1_l1"][0], model["Phi1_l2"][0], model["Phi1_l"][0]) == (0, 0, 0)  # row 0
    m = MACE(write_model(model, str(tmp_path / "m.json")))
    pos, L, species = random_box(40, 0.08, 0.9, 3, seed=6)
    a = edge_args(species, neighbor_list(pos, 4.0, L))
    n = len(species)
    m.compute_node_energies_forces(*a)
    H1, dPhi1 = np.zeros(m.stage("H1").shape, np.float32), np.zeros(m.stage("Phi1_adj").shape, np.float32)
    H1.reshape(n, -1, C)[:, 0, c] = 1.0
    dPhi1.reshape(n, -1, C)[:, 0, c] = 1.0
    m.compute_R1(n, species, a[2], a[4], a[6])
    m.compute_Y(a[5])

    def forces(scale):
        m.set_stage("H1", H1 * np.float32(scale))
        m.set_stage("Phi1_adj", dPhi1 * np.float32(scale))
        m.reverse_Phi1(n, a[2], a[3], a[5], a[6], True, True)
        return np.array(m.node_forces)

    want = forces(1.0)
    big = np.abs(want) > 1e-12
    assert big.any()
    assert np.array_equal(forces(1e30)[big], np.sign(want[big]) * np.inf)


@pytest.mark.parametrize("C", [64, 96, 128, 256])
def test_channels_of_layer_0(engine_lib, tmp_path, C):
    """With the readout of the first layer alone the energy is linear in the layer-0 contraction's
    channels: the edge forces are the float64 sum of those of each 64 channels by themselves."""
    from symmetrix_gb300 import MACE
    model = make_model(num_channels=C, species=("H", "C"), r_cut=4.0, L_max=1, num_knots=40, seed=4)
    model["readout_2_weights_2"] = [0.0] * len(model["readout_2_weights_2"])
    pos, L, species = random_box(40, 0.08, 0.9, 2, seed=6)
    nl = neighbor_list(pos, 4.0, L)

    def forces(channels):
        d = dict(model)
        d["M0_weights"] = {z: {LM: {k: c if int(k) in channels else [0.0] * len(c) for k, c in by_k.items()}
                               for LM, by_k in w.items()} for z, w in model["M0_weights"].items()}
        m = MACE(write_model(d, str(tmp_path / "m.json")))
        m.compute_node_energies_forces(*edge_args(species, nl))
        return np.array(m.node_forces)

    parts = [forces(range(k, min(k + 64, C))) for k in range(0, C, 64)]
    for p in parts:  # float32 sums
        assert np.abs(p).max() > 1e-3 and np.array_equal(p, p.astype(np.float32))
    assert np.abs(forces(range(C)) - sum(parts)).max() <= 1e-14 * max(np.abs(p).max() for p in parts)
