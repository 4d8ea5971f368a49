"""TD calls of several handles from several threads at once: every call is a cooperative
launch on its handle's own stream, whose CTAs wait for one another and for no other
launch.  States and counts equal those of calls made one after the other."""
import threading

import numpy as np
import pytest

from tests._pairs import gpu_state, make_pair

pytestmark = pytest.mark.gpu

# on chip with one CTA per SM, two per SM, few CTAs; loops over the whole chip
KINDS = [((513, 500), np.float32, np.inf), ((385, 321), np.float32, 4.0), ((129, 129), np.float64, 5.0),
         ((1100, 900), np.float32, np.inf), ((700, 600), np.float64, np.inf), ((65, 65), np.float32, np.inf)]


def _solvers():
    out = []
    for q, ((nx, ny), dtype, kappa) in enumerate(KINDS):
        out.append(make_pair(Nx=nx, Ny=ny, dx=0.5, dy=0.5, sigma=150.0, H=0.2, kappa=kappa, seed=q, dtype=dtype)[0])
        out[-1]._h.set_wait_limit(1 << 20)
    return out


def test_handles_advance_from_threads():
    calls, steps = 6, 8
    alone, together = _solvers(), _solvers()
    for g in alone:
        for _ in range(calls):
            g._h.td(0.1, steps, 0)
    failed, start = [], threading.Barrier(len(together))

    def work(g):
        try:
            start.wait(30)
            for _ in range(calls):
                g._h.td(0.1, steps, 0)
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(g,)) for g in together]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not failed and not any(t.is_alive() for t in threads)
    for a, b in zip(alone, together):
        assert all(np.array_equal(x, y) for x, y in zip(gpu_state(a), gpu_state(b)))
        assert a._h.get_params().rand_t == b._h.get_params().rand_t
