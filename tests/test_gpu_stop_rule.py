"""The stop rule of the Jacobi loops at its ends: (int)(1e4 residual / criterion) < 1e4 with
the reference's conversion (svirl/cuda/td.h: a NaN becomes 0)."""
import ctypes as C

import numpy as np
import pytest

from tests._pairs import make_pair

pytestmark = pytest.mark.gpu


def _sweeps(dtype, stop, value, route, steps=2):
    from svirl_gb300 import _lib
    gl = make_pair(Nx=40, Ny=33, dx=0.5, dy=0.5, H=0.2, landau=True, seed=2, dtype=dtype)[0]
    h = gl._h
    psi = h.get_psi()
    psi[20 + 40 * 16] = value
    h.set_psi(psi)
    h.set_params(stop_psi=stop)
    if route == "graph":
        h.set_loop_guard(1088)  # not the resident loop
    elif route == "host":
        h.set_use_graphs(False)
    st = _lib.TDStats()
    assert h.lib.glgpu_td(h.h, 0.1, steps, 0, C.byref(st)) in (_lib.GLGPU_OK, _lib.GLGPU_E_NAN)
    return st.total_sweeps_psi


@pytest.mark.parametrize("route", ["resident", "graph", "host"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_an_infinite_criterion_takes_any_residual(dtype, route):
    """One sweep a step, also where the residual is infinite."""
    assert _sweeps(dtype, np.inf, 0.5, route) == 2
    assert _sweeps(dtype, np.inf, np.inf, route) == 2
    assert _sweeps(dtype, 1e-6, 0.5, route) > 2
