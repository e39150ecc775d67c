"""The mixed solve as one graph (the second and later of a row of solves with the same parameters) against
the host-driven solve (the first): the same kernels on the same data, so the same iterations, status and
bits.  Sizes from one multigrid level to the tile kernels; budgets that end a sweep, a pair of iterations
and the solve; parameters that change and change back; a scene without fluid; a tuning change."""

import numpy as np
import pytest

import conftest
from helpers import make_sim

pytestmark = pytest.mark.gpu


def _solve(el, sim, vel, **kw):
    for f, a in vel.items():
        sim.upload(f, a)
    st = sim.solve_pressure(0.01, solver=el.SOLVER_MIXED, **kw)
    return st, [sim.download(f) for f in ("pressure", "u", "v", "w")]


def _same(a, b):
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(8, 7, 8), (20, 17, 33), (70, 64, 72)])
def test_graph_and_host_driven_solves_agree(el, dtype, shape):
    spec = dict(conftest.load_package().scenes.spheres_pool(32, 4), shape=shape)
    sim = make_sim(el, shape, dtype, spec)
    rng = np.random.default_rng(shape[0])
    vel = {f: rng.uniform(-1, 1, sim.shape(f)).astype(dtype) for f in "uvw"}
    for kw in (dict(tol=1e-6), dict(tol=1e-6, max_iter=1), dict(tol=1e-6, max_iter=4), dict(tol=1e-6, max_iter=5),
               dict(tol=1e-9, max_outer=1), dict(tol=1e-6)):
        first = _solve(el, sim, vel, **kw)
        _same(_solve(el, sim, vel, **kw), first)
        _same(_solve(el, sim, vel, **kw), first)
    sim.set_tuning(seg_blocks_per_sm=4)  # the graph holds launch shapes
    other = _solve(el, sim, vel, tol=1e-6)
    for _ in range(2):
        _same(_solve(el, sim, vel, tol=1e-6), other)
    # no fluid: the graph's loops end at once, and the call reports it as the host-driven one does
    sim.upload("phi", np.ones(sim.shape("phi"), dtype))
    for _ in range(3):
        with pytest.raises(el.ELError, match="(?i)fluid"):
            _solve(el, sim, vel, tol=1e-6)
    sim.close()
