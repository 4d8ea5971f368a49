"""The FP32 vector-potential loop in one cooperative launch (calls that the resident loop
does not take) against the resident loop: bit for bit the states and sweep counts, at the
edges of its strips of 60 columns, in full steps and for the vector potential alone, with
noise and holes, alone and in a batch; loops that stop after an odd and an even sweep, and
a guard that counts sweeps."""
import numpy as np
import pytest

from tests._pairs import gpu_state, make_pair

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4), (59, 9), (60, 24), (61, 25), (121, 70), (350, 301)]


def _gl(q, shape):
    return make_pair(Nx=shape[0], Ny=shape[1], dx=0.5, dy=0.45, sigma=150.0, H=0.2, kappa=2.0 + q, mask="holes" if q % 2 else "none",
                     seed=q, dtype=np.float32, langevin=(0.02, 0.005) if q % 3 else (0.0, 0.0))[0]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(gpu_state(a), gpu_state(b)))


@pytest.mark.parametrize("graphs", [True, False])
def test_loop_equals_resident_loop(graphs):
    from svirl_gb300.batch import HandleBatch
    ref, one, many = [[_gl(q, s) for q, s in enumerate(SHAPES)] for _ in range(3)]
    batch = HandleBatch([g._h for g in many])
    batch.set_loop_guard(1000)  # not the resident loop
    odd = set()
    for steps, eqn in ((3, 0), (2, 2), (1, 0)):
        total = 0
        for a, b in zip(ref, one):
            b._h.set_loop_guard(1000)
            b._h.set_use_graphs(graphs)
            w, st = a._h.td(0.1, steps, eqn), b._h.td(0.1, steps, eqn)
            for f in ("total_sweeps_psi", "total_sweeps_A", "last_sweeps_A", "max_sweeps_A"):
                assert getattr(w, f) == getattr(st, f), f
            assert _same(a, b)
            odd.add(w.last_sweeps_A % 2)
            total += w.total_sweeps_A
        assert batch.td_raw(0.1, steps, eqn).total_sweeps_A == total
        assert all(_same(a, b) for a, b in zip(ref, many))
    assert odd == {0, 1}
    batch.close()


def test_guard_counts_sweeps():
    from svirl_gb300._lib import GLGPUError
    n = _gl(1, (61, 40))._h.td(0.1, 1, 2).last_sweeps_A
    assert n > 1
    for guard in (n - 1, n):
        gl = _gl(1, (61, 40))
        gl._h.set_loop_guard(guard)
        if guard < n:
            with pytest.raises(GLGPUError, match="guard"):
                gl._h.td(0.1, 1, 2)
        else:
            assert gl._h.td(0.1, 1, 2).last_sweeps_A == n
