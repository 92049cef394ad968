"""The buffers that the atom-level calls keep are given back when the engine's own workspace does not fit
beside them: what fits an engine that has made no such call fits one that has."""
import numpy as np
import pytest

from symmetrix_gb300.synth.structures import random_box

pytestmark = pytest.mark.gpu


def test_evaluation_that_needs_the_kept_buffers(engine_lib, small_model_path):
    import torch

    from symmetrix_gb300 import MACE
    small, L, species = random_box(60, 0.07, 0.9, 3, seed=4)
    n = 45000
    args = (n, np.arange(n, dtype=np.int32) % 3, np.zeros(n, np.int32), np.zeros(0, np.int32), np.zeros(0, np.int32),
            np.zeros((0, 3)), np.zeros(0))
    fresh = MACE(small_model_path)
    fresh.compute_node_energies_forces(*args)
    want = np.array(fresh.node_energies)
    del fresh
    m = MACE(small_model_path)
    m.set_option("autotune", 0)
    rng = np.random.default_rng(3)
    # 3000 atoms of 1700 neighbours: 0.98 GB of list kept, 0.45 GB of workspace
    m.compute_atoms(rng.uniform(0, 9.7, (3000, 3)), rng.integers(0, 3, 3000).astype(np.int32), 9.7)
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
    m.compute_node_energies_forces(*args)  # 1.4 GB of workspace in all
    assert np.array_equal(m.node_energies, want)
    del hold
    torch.cuda.empty_cache()
    for got, w in zip(m.compute_atoms(small, species, L), MACE(small_model_path).compute_atoms(small, species, L)):
        assert np.allclose(got, w, rtol=1e-6, atol=1e-6)
