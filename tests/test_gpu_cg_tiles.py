"""Device CG at the edges of its tiles (256 nodes times a depth that the instance's size
decides, 1 to 8): two iterations follow the oracle's CG, kappa infinite (the same
quartic roots).  FP64: 1e-9; FP32: rounding of sums over N terms, 2e-5."""
import numpy as np
import pytest

from tests._pairs import gpu_state, make_pair, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,shape", [(np.float64, s) for s in ((4, 4), (16, 16), (5, 52), (64, 65), (400, 390))] +
                         [(np.float32, s) for s in ((4, 4), (16, 33), (160, 122))])
def test_two_iterations_follow_oracle(dtype, shape):
    from svirl_gb300.batch import GLBatch
    gl, orc = make_pair(Nx=shape[0], Ny=shape[1], kappa=np.inf, H=0.2, mask="holes", seed=3, dtype=dtype)
    out = GLBatch([gl]).cg(n_iter=2, rtol=0.0)
    orc.convergence_rtol = 0.0
    orc.cg(n_iter=2)
    tol = 1e-9 if dtype == np.float64 else 2e-5
    assert abs(out["energy"][0] / orc.cg_energies[-1] - 1.0) < tol
    assert rel_err(gpu_state(gl)[0], orc.psi) < tol
