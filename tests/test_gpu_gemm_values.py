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


@pytest.mark.parametrize("channels,L_max", [(64, 1), (128, 1), (160, 1), (128, 2)])
def test_single_products_and_one_sign(engine_lib, tmp_path, channels, L_max):
    """Columns with one nonzero weight, a power of two: each result is a row's element, which the split
    holds to 2^-25 of the largest contribution of its 64 elements.  Then rows of one sign."""
    from symmetrix_gb300 import MACE
    a = system()
    n, N = channels, a[0]
    model = make_model(num_channels=n, species=("H", "C"), r_cut=4.0, L_max=L_max, num_knots=40, seed=4)
    rng = np.random.default_rng(3)
    ne = [model["Phi1_l"].count(l) for l in range(4)]

    def one_per_column(K):
        W = np.zeros((K, n))
        W[rng.permutation(K)[:n], np.arange(n)] = rng.choice([-1, 1], n) * 2.0 ** rng.integers(-3, 4, n)
        return W.astype(np.float32)

    H1W = [one_per_column(n) for _ in range(L_max + 1)]
    A1W = [one_per_column(k * n) for k in ne]
    d = {**model, "H1_weights": np.concatenate([w.ravel() for w in H1W]).tolist(),
         "A1_weights": [w.ravel().tolist() for w in A1W]}
    m = MACE(write_model(d, str(tmp_path / "m.json")))
    m.compute_node_energies_forces(*a)
    get = {s: m.stage(s).reshape(N, -1, n) for s in ("M0", "H1", "H1_adj", "M0_adj", "Phi1", "A1", "A1_adj", "Phi1_adj")}

    def products(got, x, W):
        want = x @ W.astype(np.float64)
        K = len(W)
        part = np.zeros((*x.shape[:-1], -(-K // 64) * 64))
        part[..., :K] = np.abs(x) * np.abs(W).max(axis=1)
        block = part.reshape(*x.shape[:-1], -1, 64).max(axis=-1)[..., np.abs(W).argmax(axis=0) // 64]
        bound = 1.001 * 2.0 ** -24 * np.abs(want) + 2.0 ** -25 * block * (np.abs(W).max(axis=0) > 0)
        assert np.abs(want).max() > 0 and (np.abs(got - want) <= bound).all()

    for L in range(L_max + 1):
        r = slice(L * L, (L + 1) ** 2)
        products(get["H1"][:, r], get["M0"][:, r], H1W[L])
        products(get["M0_adj"][:, r], get["H1_adj"][:, r], H1W[L].T)
    at = 0
    for l in range(4):
        rows, r = slice(at, at + (2 * l + 1) * ne[l]), slice(l * l, (l + 1) ** 2)
        at += (2 * l + 1) * ne[l]
        products(get["A1"][:, r], get["Phi1"][:, rows].reshape(N, 2 * l + 1, ne[l] * n), A1W[l])
        products(get["Phi1_adj"][:, rows].reshape(N, 2 * l + 1, ne[l] * n), get["A1_adj"][:, r], A1W[l].T)

    # one sign: weights that follow the signs of one node's rows, column by column
    node = 17
    sign = np.sign(get["Phi1"][node])
    at, W1 = 0, []
    for l in range(4):
        x = sign[at:at + (2 * l + 1) * ne[l]].reshape(2 * l + 1, ne[l] * n)[0]
        W1.append((np.abs(rng.normal(size=(ne[l] * n, n))) * x[:, None]).astype(np.float32))
        at += (2 * l + 1) * ne[l]
    m = MACE(write_model({**d, "A1_weights": [w.ravel().tolist() for w in W1]}, str(tmp_path / "m.json")))
    m.compute_node_energies_forces(*a)
    A1, Phi1 = m.stage("A1").reshape(N, 16, n), m.stage("Phi1").reshape(N, -1, n)
    at = 0
    for l in range(4):
        K = ne[l] * n
        x = Phi1[node, at:at + (2 * l + 1) * ne[l]].reshape(2 * l + 1, K)[0]
        at += (2 * l + 1) * ne[l]
        want = x @ W1[l].astype(np.float64)
        assert (np.sign(x) * x @ np.abs(W1[l].astype(np.float64)) == np.abs(want)).all()
        # the leading terms' sum is exact; the other terms' accumulator, below 2^-6 of it, is cut by at
        # most one unit of 2^-23 at each of its 7 adds per 16-wide step; one rounding at the end
        steps = 4 * -(-K // 64)
        assert (np.abs(A1[node, l * l] - want) <= (7 * steps / 64 + 2) * 2.0 ** -23 * np.abs(want)).all()


@pytest.mark.parametrize("channels,L_max", [(64, 1), (96, 1), (128, 1), (256, 1), (128, 2)])
def test_no_mean_loss(engine_lib, tmp_path, channels, L_max):
    """Sums over many results keep what every one of them loses.  The errors' sum along the results is within
    8 standard deviations of that of errors of either sign (2 would be one in 20; sums of the leading
    products that the tensor core cuts: 20 and more)."""
    from symmetrix_gb300 import MACE
    a = system()
    n, N = channels, a[0]
    model = make_model(num_channels=n, species=("H", "C"), r_cut=4.0, L_max=L_max, num_knots=40, seed=4)
    ne = [model["Phi1_l"].count(l) for l in range(4)]
    m = MACE(write_model(model, str(tmp_path / "m.json")))
    m.compute_node_energies_forces(*a)
    get = {s: m.stage(s).reshape(N, -1, n) for s in ("M0", "H1", "H1_adj", "M0_adj", "Phi1", "A1", "A1_adj", "Phi1_adj")}

    def check(got, x, W):
        want = x @ W
        along = (got - want) * want
        assert abs(along.sum()) <= 8 * np.sqrt((along * along).sum())

    at = 0
    for l in range(4):
        W = np.array(model["A1_weights"][l]).astype(np.float32).astype(np.float64).reshape(ne[l] * n, n)
        rows, r = slice(at, at + (2 * l + 1) * ne[l]), slice(l * l, (l + 1) ** 2)
        at += (2 * l + 1) * ne[l]
        check(get["A1"][:, r], get["Phi1"][:, rows].reshape(N, 2 * l + 1, ne[l] * n), W)
        check(get["Phi1_adj"][:, rows].reshape(N, 2 * l + 1, ne[l] * n), get["A1_adj"][:, r], W.T)
    W = np.array(model["H1_weights"]).astype(np.float32).astype(np.float64).reshape(-1, n, n)
    for L in range(L_max + 1):
        r = slice(L * L, (L + 1) ** 2)
        check(get["H1"][:, r], get["M0"][:, r], W[L])
        check(get["M0_adj"][:, r], get["H1_adj"][:, r], W[L].T)


def test_units_of_the_channels(engine_lib, tmp_path):
    """M0's channels in units 2^-40 to 2^40 apart, taken back by H1's weights: the same H1 to the bit."""
    from symmetrix_gb300 import MACE
    a = system()
    model = make_model(num_channels=C, species=("H", "C"), r_cut=4.0, L_max=1, num_knots=40, seed=4)
    unit = 2.0 ** np.random.default_rng(5).integers(-40, 41, C)
    d = {**model, "M0_weights": {z: {LM: {k: [unit[int(k)] * x for x in c] for k, c in by_k.items()}
                                     for LM, by_k in by.items()} for z, by in model["M0_weights"].items()}}
    d["H1_weights"] = (np.array(model["H1_weights"]).reshape(2, C, C) / unit[None, :, None]).ravel().tolist()
    H1 = []
    for q in (model, d):
        m = MACE(write_model(q, str(tmp_path / "m.json")))
        m.compute_node_energies_forces(*a)
        H1.append(m.stage("H1"))
    assert np.abs(H1[0]).max() > 0 and np.array_equal(*H1)
