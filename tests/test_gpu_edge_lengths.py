"""Edge lengths of a skin list: an atom whose position is no number has no edges inside the cut-off,
so the other atoms' forces stay those of the system without it."""
import numpy as np
import pytest

from symmetrix_gb300.synth.structures import random_box, species_masses

pytestmark = pytest.mark.gpu


def test_undefined_positions_leave_the_other_atoms_alone(engine_lib, small_model_path):
    from symmetrix_gb300 import MACE
    from symmetrix_gb300.md import MD
    m = MACE(small_model_path)
    pos, L, species = random_box(200, 0.08, 0.9, 3, seed=5)
    masses = species_masses(m.atomic_numbers, species)

    def after_a_step(p, s, w, v):
        md = MD(m, p, s, w, box=L, velocities=v, dt=1e-6, skin=1.0, rebuild_every=10)
        md.run(1)  # the list is of the start's positions
        md.sync()
        return md.state()

    vel = np.zeros((200, 3))
    vel[7] = np.nan
    with_it = after_a_step(pos, species, masses, vel)
    rest = np.arange(200) != 7
    without = after_a_step(pos[rest], species[rest], masses[rest], np.zeros((199, 3)))
    assert np.isnan(with_it["positions"][7]).all()
    f = with_it["forces"][rest]
    assert np.isfinite(f).all() and np.isfinite(with_it["potential_energy"])
    # the same sums in another order of the edges: float32 rounding
    assert np.abs(f - without["forces"]).max() <= 1e-5 * max(1.0, np.abs(without["forces"]).max())
