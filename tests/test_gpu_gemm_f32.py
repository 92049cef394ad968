"""The float32 tensor-core GEMMs (k_umma_f32 in k_umma.cu): A1, Phi1_adj, H1 and M0_adj of an
evaluation against float64 products of the stage rows they read, at row counts around the
128-row tile (per l: N (2 l + 1) rows), padded and whole k-blocks and every N-tile width."""
import numpy as np
import pytest

from helpers import edge_args
from symmetrix_gb300.synth.model import make_model, write_model
from symmetrix_gb300.synth.structures import neighbor_list

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,L_max,N", [(64, 1, 1), (64, 1, 43), (96, 1, 128), (128, 1, 19), (128, 1, 129), (96, 2, 26),
                                       (64, 2, 64)])
def test_gemms_against_float64_products(engine_lib, tmp_path, C, L_max, N):
    from symmetrix_gb300 import MACE
    model = make_model(num_channels=C, species=("H", "C", "O"), r_cut=5.0, L_max=L_max, num_knots=40, seed=7)
    m = MACE(write_model(model, str(tmp_path / "m.json")))
    rng = np.random.default_rng(2)
    pos = rng.uniform(0, (N / 0.08) ** (1 / 3) + 1.0, (N, 3))
    species = rng.integers(0, 3, N).astype(np.int32)
    m.compute_node_energies_forces(*edge_args(species, neighbor_list(pos, 5.0)))
    ne = [model["Phi1_l"].count(l) for l in range(4)]
    A1, A1_adj = (m.stage(s).reshape(N, 16, C) for s in ("A1", "A1_adj"))
    Phi1, Phi1_adj = (m.stage(s).reshape(N, -1, C) for s in ("Phi1", "Phi1_adj"))
    M0, H1, H1_adj, M0_adj = (m.stage(s).reshape(N, -1, C) for s in ("M0", "H1", "H1_adj", "M0_adj"))

    def check(got, x, w):
        # a float32 result cannot be nearer than its rounding (3e-8); 4e-7 is the error of a
        # chain of 640 float32 FMAs on random terms, which the split sums must not exceed
        want = x @ w
        assert np.linalg.norm(got - want) <= 4e-7 * max(np.linalg.norm(want), 1e-30)

    at = 0
    for l in range(4):
        W = np.array(model["A1_weights"][l]).astype(np.float32).astype(np.float64).reshape(ne[l] * C, C)
        rows = slice(at, at + (2 * l + 1) * ne[l])
        check(A1[:, l * l:(l + 1) ** 2], Phi1[:, rows].reshape(N, 2 * l + 1, ne[l] * C), W)
        check(Phi1_adj[:, rows].reshape(N, 2 * l + 1, ne[l] * C), A1_adj[:, l * l:(l + 1) ** 2], W.T)
        at += (2 * l + 1) * ne[l]
    H1W = np.array(model["H1_weights"]).astype(np.float32).astype(np.float64).reshape(-1, C, C)
    for L in range(L_max + 1):
        check(H1[:, L * L:(L + 1) ** 2], M0[:, L * L:(L + 1) ** 2], H1W[L])
        check(M0_adj[:, L * L:(L + 1) ** 2], H1_adj[:, L * L:(L + 1) ** 2], H1W[L].T)
