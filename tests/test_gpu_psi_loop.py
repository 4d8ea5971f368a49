"""The psi Jacobi loop in one cooperative launch (domains and calls that the resident loop
does not take): bit for bit the resident loop's states and sweep counts, alone and in a
batch, through the graph and from the host, at the edges of its tiles (FP64: 256 nodes,
a sweep per round) and strips (FP32: 56 columns, three sweeps per round, stops inside a
round that kept its sweeps or not); a guard of n launches stops it after 3 n sweeps."""
import numpy as np
import pytest

from tests._pairs import gpu_state, make_pair

pytestmark = pytest.mark.gpu

SHAPES = {np.float64: [(4, 4), (5, 51), (16, 16), (257, 4), (31, 33), (300, 241)],
          np.float32: [(4, 4), (55, 20), (56, 21), (57, 33), (60, 62), (113, 4), (129, 127), (400, 301)]}
KW = dict(dx=0.5, dy=0.45, sigma=150.0, H=0.2, langevin=(0.02, 0.005))


def _gl(q, shape, dtype):
    return make_pair(Nx=shape[0], Ny=shape[1], kappa=4.0 if q % 2 else np.inf, mask="holes" if q % 3 else "none", seed=q,
                     dtype=dtype, **KW)[0]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(gpu_state(a), gpu_state(b)))


@pytest.mark.parametrize("dtype", SHAPES)
@pytest.mark.parametrize("graphs", [True, False])
def test_loop_equals_resident_loop(dtype, graphs):
    from svirl_gb300.batch import HandleBatch
    ref, one, many = [[_gl(q, s, dtype) for q, s in enumerate(SHAPES[dtype])] for _ in range(3)]
    ref[1].params.linear_coefficient = one[1].params.linear_coefficient = many[1].params.linear_coefficient = \
        1.0 - 0.3 * np.random.default_rng(1).random(SHAPES[dtype][1])
    want = [g._h.td(0.1, 3, 0) for g in ref]
    for a, b, w in zip(ref, one, want):
        b._h.set_loop_guard(1000)  # not the resident loop
        b._h.set_use_graphs(graphs)
        st = b._h.td(0.1, 3, 0)
        assert w.sweep_launches == 1 and st.sweep_launches >= 3
        assert (st.total_sweeps_psi, st.last_sweeps_psi) == (w.total_sweeps_psi, w.last_sweeps_psi) and _same(a, b)
    batch = HandleBatch([g._h for g in many])
    batch.set_loop_guard(1000)
    st = batch.td_raw(0.1, 3)
    assert st.total_sweeps_psi == sum(w.total_sweeps_psi for w in want)
    assert all(_same(a, b) for a, b in zip(ref, many))
    batch.close()


@pytest.mark.parametrize("dtype", SHAPES)
def test_guard_counts_three_sweeps_a_launch(dtype):
    from svirl_gb300._lib import GLGPUError
    sweeps = _gl(0, (60, 41), dtype)._h.td(0.1, 1, 1).last_sweeps_psi
    for n in (1, -(-sweeps // 3)):
        gl = _gl(0, (60, 41), dtype)
        gl._h.set_loop_guard(n)
        if 3 * n < sweeps:
            with pytest.raises(GLGPUError, match="guard"):
                gl._h.td(0.1, 1, 1)
        else:
            assert gl._h.td(0.1, 1, 1).last_sweeps_psi == sweeps
    assert sweeps > 3
