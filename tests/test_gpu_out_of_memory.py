"""A call whose buffers do not fit the GPU's free memory fails with an error and leaves the engine as it
was: the next call that fits gives the results of a fresh engine, and so does every other engine."""
import numpy as np
import pytest

from symmetrix_gb300.synth.structures import random_box

pytestmark = pytest.mark.gpu


def test_a_call_that_does_not_fit(engine_lib, small_model_path):
    import torch

    from symmetrix_gb300 import MACE
    small, Ls, sp_small = random_box(60, 0.07, 0.9, 3, seed=4)
    rng = np.random.default_rng(3)
    big = rng.uniform(0, 15.0, (20000, 3))  # 3,000 neighbours an atom: about 9 GB of list
    sp_big = rng.integers(0, 3, len(big)).astype(np.int32)
    m, other = MACE(small_model_path), MACE(small_model_path)
    for e in (m, other):
        e.set_option("autotune", 0)
    want = m.compute_atoms(small, sp_small, Ls)
    want_other = other.compute_atoms(small, sp_small, Ls)
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (3 << 30), dtype=torch.uint8, device="cuda")  # leave 3 GiB
    with pytest.raises(RuntimeError):
        m.compute_atoms(big, sp_big, 15.0)
    del hold
    torch.cuda.empty_cache()
    for _ in range(2):
        for got, w in ((m.compute_atoms(small, sp_small, Ls), want),
                       (other.compute_atoms(small, sp_small, Ls), want_other)):
            assert all(np.array_equal(x, y) for x, y in zip(got, w))
