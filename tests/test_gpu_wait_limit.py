"""The limit on the waits of the cooperative loops (glgpu_set_wait_limit), made to run out
by setting it to one poll: no GPU fault, every wait ends.  The call reports GLGPU_E_TIMEOUT
and does not go on to its remaining steps; once the state is set anew the handle gives what
a fresh one gives."""
import ctypes as C

import numpy as np
import pytest

from tests._pairs import gpu_state, make_pair

pytestmark = pytest.mark.gpu

STEPS = 12


def _pair(dtype, kappa, n=(150, 131), seed=4):
    return make_pair(Nx=n[0], Ny=n[1], dx=0.5, dy=0.45, sigma=150.0, H=0.2, kappa=kappa, mask="holes", seed=seed, dtype=dtype,
                     langevin=(0.02, 0.005))[0]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(gpu_state(a), gpu_state(b)))


@pytest.mark.parametrize("loop", ["resident", "graph", "host"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kappa", [np.inf, 4.0])
def test_wait_limit_ends_the_call(loop, dtype, kappa):
    from svirl_gb300 import _lib
    gl, ref = _pair(dtype, kappa), _pair(dtype, kappa)
    h = gl._h
    psi, ab, rand_t = h.get_psi(), h.get_ab(), h.get_params().rand_t
    if loop == "graph":  # a guard in launches: not the resident loop
        h.set_loop_guard(1000)
    elif loop == "host":
        h.set_use_graphs(False)
    h.set_wait_limit(1)
    st = _lib.TDStats()
    assert h.lib.glgpu_td(h.h, 0.1, STEPS, 0, C.byref(st)) == _lib.GLGPU_E_TIMEOUT
    assert b"barrier" in h.lib.glgpu_last_error(h.h) and st.steps < STEPS
    h.set_wait_limit(0)
    h.set_params(rand_t=rand_t)
    h.set_psi(psi)
    h.set_ab(ab)
    h.td(0.1, 3, 0)
    ref._h.td(0.1, 3, 0)
    assert _same(gl, ref) and h.get_params().rand_t == ref._h.get_params().rand_t


@pytest.mark.parametrize("sizes", [(60, 150, 97), (400, 300, 350, 420)])
def test_wait_limit_of_a_batch(sizes):
    """Films that fit on chip together, and in waves."""
    from svirl_gb300._lib import GLGPUError
    from svirl_gb300.batch import HandleBatch
    kw = dict(dtype=np.float32, kappa=np.inf)
    gls, refs = [[_pair(n=(n, n), seed=q, **kw) for q, n in enumerate(sizes)] for _ in range(2)]
    start = [(g._h.get_psi(), g._h.get_params().rand_t) for g in gls]
    batch = HandleBatch([g._h for g in gls])
    batch.set_wait_limit(1)
    with pytest.raises(GLGPUError, match="barrier"):
        batch.td_raw(0.1, STEPS)
    batch.set_wait_limit(0)
    for g, (psi, rand_t) in zip(gls, start):
        g._h.set_psi(psi)
        g._h.set_params(rand_t=rand_t)
    batch.td_raw(0.1, 3)
    for g, r in zip(gls, refs):
        r._h.td(0.1, 3, 0)
        assert _same(g, r)
    with pytest.raises(GLGPUError):
        batch.set_wait_limit(-1)
    batch.close()


def test_a_film_waits_for_the_films_before_it():
    """Films in waves, of which one takes many sweeps a step and its neighbours one: their
    CTAs wait at the next film's first barrier for nearly the whole call, far beyond the
    limit of a wait inside a film, and the call is none the worse for it."""
    from svirl_gb300.batch import HandleBatch
    # tiles of 58 x 26: 36 (random start), 260 (uniform, at rest in zero field: a sweep a step), 288
    shapes, steps, polls = [(348, 156), (754, 520), (696, 624)], 1500, 4000

    def films():
        out = []
        for q, (nx, ny) in enumerate(shapes):
            g = make_pair(Nx=nx, Ny=ny, dx=0.5, dy=0.5, sigma=150.0, H=0.0 if q else 0.3, kappa=np.inf, seed=q, dtype=np.float32)[0]
            if q:
                g._h.set_psi(np.ones(nx * ny, dtype=np.complex64))
            out.append(g)
        return out

    gls, refs = films(), films()
    batch = HandleBatch([g._h for g in gls])
    batch.set_wait_limit(polls)
    st, ms = batch.td_raw(0.1, steps, timed=True)
    assert st.sweep_launches == 1 and st.steps == steps
    for g, r in zip(gls, refs):
        r._h.td(0.1, steps, 0)
        assert _same(g, r)
    # the wait: the first film's time but for the second's, a poll being a microsecond or less
    alone = [r._h.td_timed(0.1, 100, 0)[1] * steps / 100 for r in refs]
    assert alone[0] - alone[1] > 2e-3 * polls, alone
    batch.close()
