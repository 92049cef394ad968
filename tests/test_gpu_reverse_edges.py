"""Atomic forces of the atom-level calls against the per-edge forces of the evaluator's own call, added on
the host (F_j += f_e, F_i -= f_e): a wrong reverse of an edge shows, whichever search found the list
(non-periodic lists: a binary search in the neighbour's ascending list; periodic: cell segments, or
all pairs with images)."""
import numpy as np
import pytest

from helpers import atomic_forces, edge_args
from symmetrix_gb300.synth.structures import neighbor_list, random_box, random_molecule

pytestmark = pytest.mark.gpu


def want(m, pos, species, box=None):
    nl = neighbor_list(pos, m.r_cut, box)
    if len(nl["r"]) == 0:
        return np.zeros((len(pos), 3))
    m.compute_node_energies_forces(*edge_args(species, nl))
    return atomic_forces(len(pos), nl["i"], nl["neigh_indices"], m.node_forces)


def close(got, ref):
    # the same float32 edge forces up to the last bit of an edge's length
    return np.abs(got - ref).max() <= 2e-6 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("n,density", [(1, 0.08), (2, 0.08), (33, 0.08), (400, 0.08), (150, 0.6)])
def test_atoms_without_a_box(engine_lib, small_model_path, n, density):
    """(The last one: neighbour lists of more than 32 atoms.)"""
    from symmetrix_gb300 import MACE
    m = MACE(small_model_path)
    pos, species = random_molecule(n, density, 0.6 if density > 0.5 else 0.95, 3, np.random.default_rng(n))
    F = m.compute_atoms(pos, species, None)[2]
    assert close(F, want(m, pos, species))


@pytest.mark.parametrize("n,density", [(40, 0.08), (700, 0.08)])
def test_atoms_in_a_box(engine_lib, small_model_path, n, density):
    """All pairs with images, then cells."""
    from symmetrix_gb300 import MACE
    m = MACE(small_model_path)
    pos, L, species = random_box(n, density, 0.9, 3, seed=n)
    F = m.compute_atoms(pos, species, L)[2]
    assert close(F, want(m, pos, species, L))


def test_molecules(engine_lib, small_model_path):
    from symmetrix_gb300 import MACE
    m = MACE(small_model_path)
    rng = np.random.default_rng(5)
    mols = [random_molecule(n, 0.08, 0.95, 3, rng) for n in (1, 2, 1, 17, 64, 3, 40, 2, 90)]
    F = m.compute_molecules(mols)[2]
    for (pos, species), f in zip(mols, F):
        assert close(f, want(m, pos, species))
