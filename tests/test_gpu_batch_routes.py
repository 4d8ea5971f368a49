"""FP32 batches that do not fit on chip at once: films in waves of the resident loop where
these are faster, the loops over all films (a launch per Jacobi loop) where a film at a time
would leave much of the chip idle.  Either gives what single handles give, bit for bit."""
import numpy as np
import pytest

from tests._pairs import gpu_state, make_pair

pytestmark = pytest.mark.gpu


def _films(sizes, kappas):
    return [make_pair(Nx=n, Ny=n, dx=0.5, dy=0.5, sigma=150.0, H=0.2, kappa=k, mask="random30", seed=q, dtype=np.float32)[0]
            for q, (n, k) in enumerate(zip(sizes, kappas))]


@pytest.mark.parametrize("sizes,kappas,waves", [((512,) * 2, (np.inf,) * 2, True), ((512,) * 10, (np.inf,) * 10, False),
                                                ((512,) * 2, (4.0,) * 2, True), ((512,) * 6, (4.0,) * 6, False),
                                                ((450, 64) * 4, (np.inf,) * 8, True)])
def test_waves_or_loops(sizes, kappas, waves):
    from svirl_gb300.batch import HandleBatch
    many, one = _films(sizes, kappas), _films(sizes, kappas)
    batch = HandleBatch([g._h for g in many])
    st = batch.td_raw(0.1, 2)
    assert (st.sweep_launches == 1) == waves
    for a, b in zip(many, one):
        b._h.td(0.1, 2, 0)
        assert all(np.array_equal(x, y) for x, y in zip(gpu_state(a), gpu_state(b)))
    batch.close()


def test_selected_sweep_kernel_concerns_fp32_handles_alone():
    """The bulk-copy sweep exists in FP32 and for single handles: selecting it changes the
    route of nothing else."""
    from svirl_gb300.batch import HandleBatch
    for dtype, launch in ((np.float64, True), (np.float32, False)):
        gl = make_pair(Nx=97, Ny=64, H=0.2, dtype=dtype)[0]
        assert gl._h.td(0.1, 2).sweep_launches == 1
        gl._h.set_psi_sweep_kernel(1)
        assert (gl._h.td(0.1, 2).sweep_launches == 1) == launch
    films = _films((64, 97), (np.inf, 4.0))
    films[0]._h.set_psi_sweep_kernel(1)
    batch = HandleBatch([g._h for g in films])
    assert batch.td_raw(0.1, 2).sweep_launches == 1
    batch.close()


def test_td_resident_says_what_a_call_does():
    for dtype, n in ((np.float32, 97), (np.float64, 97), (np.float32, 900)):
        gl = make_pair(Nx=n, Ny=n - 3, H=0.2, dtype=dtype)[0]
        for guard in (0, 1000):
            gl._h.set_loop_guard(guard)
            assert gl._h.td_resident() == (gl._h.td(0.1, 2).sweep_launches == 1)
