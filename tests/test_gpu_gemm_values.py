"""The float32 tensor-core GEMMs on values that a split in bf16 terms cannot hold: the results are those
of the SIMT kernel, which the per-stage calls run on the same rows."""
import numpy as np
import pytest

from helpers import edge_args
from symmetrix_gb300.synth.model import make_model, write_model
from symmetrix_gb300.synth.structures import neighbor_list, random_box

pytestmark = pytest.mark.gpu

C = 64


def system():
    pos, L, species = random_box(150, 0.08, 0.9, 2, seed=6)  # rows of two tiles
    return edge_args(species, neighbor_list(pos, 4.0, L))


def linear(model, channel, c):
    """M0 of one channel becomes c times A0's l = 0 row, read by H1 with weights that bring it back."""
    d = dict(model)
    d["M0_weights"] = {z: {LM: {k: ([c if LM == "0" else 0.0] + [0.0] * (len(w) - 1)) if int(k) == channel else w
                                for k, w in by_k.items()} for LM, by_k in by.items()}
                       for z, by in model["M0_weights"].items()}
    W = np.array(model["H1_weights"]).reshape(2, C, C)
    W[:, channel] *= 1e-30
    d["H1_weights"] = W.reshape(-1).tolist()
    return d


def compare(m, a):
    m.compute_node_energies_forces(*a)
    got = m.stage("H1")
    m.compute_H1(a[0])
    want = m.stage("H1")
    for q in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(q(got), q(want))
    ok = np.isfinite(want)
    assert np.abs(got[ok] - want[ok]).max() <= 1e-6 * np.abs(want)[ok].max()
    return want


def test_rows_beyond_bf16(engine_lib, tmp_path):
    """One node's value just below float32's largest, which rounds to infinity in bf16, two infinite."""
    from symmetrix_gb300 import MACE
    a = system()
    model = make_model(num_channels=C, species=("H", "C"), r_cut=4.0, L_max=1, num_knots=40, seed=4)
    m = MACE(write_model(model, str(tmp_path / "m.json")))
    m.compute_node_energies_forces(*a)
    assert model["M0_monomials"]["0"][0] == [0]
    A0 = np.abs(m.stage("A0").reshape(a[0], 16, C)[:, 0])
    channel = int(A0.max(axis=0).argmax())
    third = np.sort(A0[:, channel])[-3]
    assert third > 1.0
    m = MACE(write_model(linear(model, channel, 3.4e38 / third), str(tmp_path / "m.json")))
    want = compare(m, a).reshape(a[0], -1)
    M0 = m.stage("M0").reshape(a[0], -1)
    assert ((np.abs(M0) > 3.3895313892515355e38) & np.isfinite(M0)).any() and np.isinf(M0).any()
    rows = np.isfinite(want).all(axis=1)
    assert rows.any() and not rows.all()


def test_weights_beyond_bf16(engine_lib, tmp_path):
    from symmetrix_gb300 import MACE
    a = system()
    for w in (3.4e38, 1e39):  # finite in float32, infinite in float32
        model = make_model(num_channels=C, species=("H", "C"), r_cut=4.0, L_max=1, num_knots=40, seed=4)
        model["H1_weights"][5] = w
        model = {**model, "M0_weights": {z: {LM: {k: [1e-8 * x for x in c] for k, c in by_k.items()}
                                             for LM, by_k in by.items()} for z, by in model["M0_weights"].items()}}
        m = MACE(write_model(model, str(tmp_path / "m.json")))
        compare(m, a)
