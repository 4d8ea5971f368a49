"""The resident time loop (state on chip, one cooperative launch per call) against
the launch-per-sweep loop driven from the host: the same operations per node, so the
states, the sweep counts and the Langevin counter are equal bit for bit.  Sizes at the
edges of the tiles of every shape (one tile, one node more, ragged last tiles, the
smallest domain), both precisions, both equations, masks, noise, a spatial linear
coefficient, batches that fit at once and in waves."""
import numpy as np
import pytest

from tests._pairs import gpu_state, make_pair

pytestmark = pytest.mark.gpu

#: (Nx, Ny) by the shape that a single domain of that size takes
SIZES = {np.float32: [(4, 4), (16, 16), (17, 33), (129, 100), (270, 241), (385, 361), (500, 433), (701, 660)],
         np.float64: [(4, 5), (12, 12), (13, 25), (131, 120), (257, 181), (321, 290), (435, 391)]}


def _pair(Nx, Ny, **kw):
    return make_pair(Nx=Nx, Ny=Ny, dx=0.5, dy=0.45, sigma=150.0, H=0.2, **kw)[0]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(gpu_state(a), gpu_state(b)))


@pytest.mark.parametrize("dtype,shape", [(d, s) for d in SIZES for s in SIZES[d]])
@pytest.mark.parametrize("kappa", [np.inf, 4.0])
def test_resident_loop_equals_launch_per_sweep(dtype, shape, kappa):
    kw = dict(kappa=kappa, mask="holes" if min(shape) < 300 else "random30", seed=5, dtype=dtype, langevin=(0.02, 0.005))
    a, b = _pair(*shape, **kw), _pair(*shape, **kw)
    b._h.set_use_graphs(False)
    if shape == (17, 33):
        eps = 1.0 - 0.3 * np.random.default_rng(1).random(shape)
        a.params.linear_coefficient = eps
        b.params.linear_coefficient = eps
    sa, sb = [g._h.td(0.1, 3, 0) for g in (a, b)]
    assert sa.sweep_launches == 1 and sa.used_graph == 1 and sb.used_graph == 0
    assert _same(a, b)
    for f in ("steps", "total_sweeps_psi", "total_sweeps_A", "max_sweeps_psi", "last_sweeps_psi", "last_sweeps_A", "rand_t"):
        assert getattr(sa, f) == getattr(sb, f), f
    for eqn in (1, 2, 0):
        a._h.td(0.1, 2, eqn)
        b._h.td(0.1, 2, eqn)
    assert _same(a, b)


@pytest.mark.parametrize("sizes", [(40, 66, 97), (513, 257, 33, 481, 300, 520, 64)])
def test_batch_of_resident_loops_equals_single_handles(sizes):
    """All at once, and more tiles than resident CTAs (waves)."""
    from svirl_gb300.batch import HandleBatch
    kw = [dict(kappa=4.0 if q % 2 else np.inf, mask="holes" if n < 300 else "random30", seed=q, dtype=np.float32)
          for q, n in enumerate(sizes)]
    one, many = [[_pair(n, n - 1, **k) for n, k in zip(sizes, kw)] for _ in range(2)]
    batch = HandleBatch([g._h for g in many])
    st = batch.td_raw(0.1, 3)
    assert st.sweep_launches == 1
    for g in one:
        g._h.set_use_graphs(False)
        g._h.td(0.1, 3, 0)
    batch.td_raw(0.1, 1)
    for a, b in zip(one, many):
        a._h.td(0.1, 1, 0)
        assert _same(a, b)
    batch.close()
