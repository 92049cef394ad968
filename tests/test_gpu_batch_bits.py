"""A molecule's energies and forces do not depend on the molecules beside it: the bits of a batch
that is large enough for every size rule of the kernels (edges per warp, contraction per
output) are those of the molecule alone."""
import numpy as np
import pytest

from symmetrix_gb300.synth.model import make_model, write_model
from symmetrix_gb300.synth.structures import random_molecule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,L_max,more,precision", [(32, 1, {}, "float32"), (64, 1, {}, "bfloat16"),
                                                    (96, 1, dict(zbl=True, density_scaled=True), "float32"),
                                                    (32, 2, {}, "float32"), (64, 2, dict(density_scaled=True), "bfloat16"),
                                                    (32, 1, dict(poly=True), "float32"), (64, 2, dict(poly=True), "float32")])
def test_alone_as_in_a_batch(engine_lib, tmp_path, C, L_max, more, precision):
    from symmetrix_gb300 import MACE
    more = dict(more)
    poly = more.pop("poly", False)
    d = make_model(num_channels=C, species=("H", "C", "O"), r_cut=4.0, L_max=L_max, num_knots=40, seed=6, **more)
    if poly:  # one monomial more than the canonical set of output 0
        d["M0_monomials"]["0"].append([0, 1])
        for w in d["M0_weights"].values():
            for k in w["0"]:
                w["0"][k].append(0.1)
    m = MACE(write_model(d, str(tmp_path / "m.json")), precision=precision)
    rng = np.random.default_rng(8)
    mols = [random_molecule(k, 0.08, 0.95, 3, rng) for k in (1, 2, 9, 23, 40)]
    alone = [m.compute_atoms(p, s, None) for p, s in mols]
    copies = 1 + 3100 // sum(len(p) for p, _ in mols)
    E, node_e, F = m.compute_molecules(mols * copies)
    for q in range(len(mols) * copies):
        e, ne, f, _ = alone[q % len(mols)]
        assert np.array_equal(F[q], f)
        assert np.array_equal(node_e[q], ne)
