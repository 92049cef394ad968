"""Several engines of different width or polynomials in one process: creating one narrows nothing
for those that are alive.  The kernels' shared-memory limit belongs to the function, and models
share instantiations of the layer-0 contraction adjoint (per pair: the one that needs more
shared memory first, then one that needs less)."""
import numpy as np
import pytest

from helpers import edge_args
from symmetrix_gb300.synth.model import make_model, write_model
from symmetrix_gb300.synth.structures import neighbor_list, random_box

pytestmark = pytest.mark.gpu


def model(path, C, L_max, data_driven):
    d = make_model(num_channels=C, species=("H", "C", "O"), r_cut=4.0, L_max=L_max, num_knots=40, seed=3)
    if data_driven:  # one monomial more than the canonical set of output 0
        d["M0_monomials"]["0"].append([0, 1])
        for w in d["M0_weights"].values():
            for k in w["0"]:
                w["0"][k].append(0.1)
    return write_model(d, str(path))


@pytest.mark.parametrize("L_max,first,second", [(1, (96, False), (32, False)), (2, (96, False), (64, False)),
                                                (1, (64, True), (64, False)), (1, (128, True), (128, False)),
                                                (1, (256, False), (96, True)), (2, (128, True), (128, False))])
def test_an_older_engine_still_evaluates(engine_lib, tmp_path, L_max, first, second):
    from symmetrix_gb300 import MACE
    pos, L, species = random_box(24, 0.08, 0.9, 3, seed=9)
    args = edge_args(species, neighbor_list(pos, 4.0, L))
    a = MACE(model(tmp_path / "a.json", first[0], L_max, first[1]))
    a.compute_node_energies_forces(*args)
    e, f = a.node_energies.copy(), a.node_forces.copy()
    b = MACE(model(tmp_path / "b.json", second[0], L_max, second[1]))
    a.compute_node_energies_forces(*args)
    assert np.array_equal(a.node_energies, e) and np.array_equal(a.node_forces, f)
    b.compute_node_energies_forces(*args)
    a.compute_node_energies_forces(*args)
    assert np.array_equal(a.node_energies, e) and np.array_equal(a.node_forces, f)
