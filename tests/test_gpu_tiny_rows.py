"""FP64 solvers on a system with a row whose reciprocal overflows: one fluid cell whose six face weights are
subnormal, so that its diagonal is 6e-310 and 1 / 6e-310 infinite.  The row weighs nothing in any other
row's sum: the solve converges, and every other cell has the pressure of the system without it.
Both solves stop at |r| <= 1e-12 |b|; as in test_gpu_mg64.py that leaves 1e-7 of the largest pressure at
sizes up to a hundred cells an axis, and these are a fifth of that."""

import numpy as np
import pytest

from helpers import make_sim

pytestmark = pytest.mark.gpu


def _solve(el, shape, solver, tiny):
    ni, nj, nk = shape
    sim = make_sim(el, shape, np.float64)
    phi = np.empty((nk, nj, ni))
    phi[:] = (np.arange(nj) + 0.5 - 0.7 * nj)[None, :, None] / ni
    weight = {}
    for axis, f in enumerate("uvw"):
        w = np.ones(sim.shape(f))
        d = 2 - axis
        w.swapaxes(0, d)[[0, -1]] = 0  # walls
        weight[f] = w
    k, j, i = nk // 2, nj // 3, ni // 2
    for f, at in (("u", ((k, j, i), (k, j, i + 1))), ("v", ((k, j, i), (k, j + 1, i))), ("w", ((k, j, i), (k + 1, j, i)))):
        for c in at:
            weight[f][c] = tiny
    rng = np.random.default_rng(ni)
    sim.upload("phi", phi)
    for f in "uvw":
        sim.upload("weight_" + f, weight[f])
        sim.upload(f, rng.uniform(-1, 1, sim.shape(f)))
    stats = sim.solve_pressure(0.01, solver=solver, tol=1e-12, max_iter=5000)
    p = sim.download("pressure")
    sim.close()
    p_cell = p[k, j, i]
    p[k, j, i] = 0
    return stats, p, p_cell


@pytest.mark.parametrize("solver", ["SOLVER_MG_FP64", "SOLVER_JACOBI_FP64"])
@pytest.mark.parametrize("shape", [(8, 7, 8), (20, 13, 16)])  # the coarsest level alone, and three levels
def test_a_subnormal_row(el, shape, solver):
    stats, p, p_cell = _solve(el, shape, getattr(el, solver), 1e-310)
    assert stats["status"] == 0 and stats["relres"] <= 1e-12
    assert np.isfinite(p_cell)
    without, want, _ = _solve(el, shape, getattr(el, solver), 0.0)
    assert stats["fluid_cells"] == without["fluid_cells"] + 1
    np.testing.assert_allclose(p, want, rtol=0, atol=1e-7 * np.max(np.abs(want)))
