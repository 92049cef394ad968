"""The timeout path of the float32 tensor-core GEMM (k_umma_f32), as test_gpu_timeout.py exercises that of
the bf16 one: no weights are loaded, so the bounded waits (2 ms here) of the thread that issues
the MMAs, and of the threads that split the rows where K is longer than the ring, run out with
nothing in flight.  The BF16 form runs this kernel where the bf16 GEMM does not take a shape."""
import numpy as np
import pytest

from helpers import edge_args
from symmetrix_gb300.synth.model import make_model, write_model
from symmetrix_gb300.synth.structures import neighbor_list, random_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,L_max,launches", [(64, 2, 1), (96, 1, 1), (96, 1, 2), (96, 1, 4)])
def test_wait_timeout_is_reported_and_recoverable(engine_lib, tmp_path, C, L_max, launches):
    """The first `launches` GEMM launches give up: H1 (one or two k-blocks), A1 (up to five), the adjoints."""
    from symmetrix_gb300 import MACE
    path = write_model(make_model(num_channels=C, species=("H", "C", "O"), r_cut=4.0, L_max=L_max, num_knots=40, seed=8),
                       str(tmp_path / "m.json"))
    pos, L, species = random_box(60, 0.08, 0.9, 3, seed=9)
    args = edge_args(species, neighbor_list(pos, 4.0, L))
    m = MACE(path, precision="bfloat16")
    m.compute_node_energies_forces(*args)
    e, f = m.node_energies.copy(), m.node_forces.copy()
    for _ in range(2):
        m.set_option("test_gemm_timeout", launches)
        with pytest.raises(TimeoutError):
            m.compute_node_energies_forces(*args)
        m.compute_node_energies_forces(*args)
        assert np.array_equal(m.node_energies, e) and np.array_equal(m.node_forces, f)
