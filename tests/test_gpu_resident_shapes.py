"""The resident time loop on FP64 tiles of 62 x 14 nodes (domains whose tiles of that shape
fit one to an SM, and two) and on FP32 tiles of 58 x 26 one to an SM: bit for bit the
host-driven loop's states, at ragged last tiles, with vector potential, holes and noise."""
import numpy as np
import pytest

from tests._pairs import gpu_state, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,shape", [(np.float64, s) for s in ((470, 230), (373, 337), (435, 421), (63, 1700))] +
                         [(np.float32, s) for s in ((449, 449), (465, 413), (60, 1690))])
@pytest.mark.parametrize("kappa", [np.inf, 4.0])
def test_equals_host_loop(dtype, shape, kappa):
    a, b = [make_pair(Nx=shape[0], Ny=shape[1], dx=0.5, dy=0.45, sigma=150.0, H=0.2, kappa=kappa, mask="holes", seed=7,
                      dtype=dtype, langevin=(0.02, 0.005))[0] for _ in range(2)]
    b._h.set_use_graphs(False)
    sa, sb = a._h.td(0.1, 3, 0), b._h.td(0.1, 3, 0)
    assert sa.sweep_launches == 1 and sb.used_graph == 0
    assert (sa.total_sweeps_psi, sa.total_sweeps_A) == (sb.total_sweeps_psi, sb.total_sweeps_A)
    assert all(np.array_equal(x, y) for x, y in zip(gpu_state(a), gpu_state(b)))
