"""The energy reduction's sum over blocks is compensated from the first block to the last: energies
of opposite sign and a size that swallows all others leave the others' sum (each block's own
sum is exact here)."""
import math

import numpy as np
import pytest

from symmetrix_gb300.synth.model import make_model, write_model

pytestmark = pytest.mark.gpu


def test_energy_sum_over_blocks_keeps_small_terms(engine_lib, tmp_path):
    from symmetrix_gb300 import MACE
    model = make_model(num_channels=32, species=("H", "C", "O"), r_cut=4.0, L_max=1, num_knots=30, seed=2)
    model["atomic_energies"][:2] = [2.0 ** 60, -2.0 ** 60]  # an atom's other terms are below half an ulp
    m = MACE(write_model(model, str(tmp_path / "m.json")))
    n = 5000  # isolated atoms, 256 to a block: the first two blocks cancel
    species = np.full(n, 2, np.int32)
    species[:256], species[256:512] = 0, 1
    i = np.arange(n)
    pos = 6.0 * np.stack([i % 20, i // 20 % 20, i // 400], 1).astype(float)
    energy, node_energies, _, _ = m.compute_atoms(pos, species, None)
    want = math.fsum(node_energies)
    assert abs(want) > 100.0
    # float64 trees over 256 terms of some eV in each block
    assert abs(energy - want) <= 1e-12 * abs(want)
