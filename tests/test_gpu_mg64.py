"""The FP64 multigrid solver from one level (the coarsest sweeps alone) to five, with partial row
segments, empty cells and odd sizes, against the plain FP64 PCG: both stop at |r| <= 1e-13 |b|, so they
differ by at most 2e-13 times the condition number, about (2 n / pi)^2 < 5000 for n <= 100 cells and up
to 100 times that through the free surface's small thetas: 1e-7 of the largest pressure.  The V-cycle
reduces the residual several times an iteration: 13 digits within 40."""

import numpy as np
import pytest

import conftest
from conftest import rel_err
from helpers import make_sim, scene_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(8, 8, 8), (7, 5, 8), (9, 7, 5), (17, 9, 33), (31, 33, 18), (70, 40, 36), (100, 66, 50)])
def test_multigrid_solves_what_the_plain_pcg_solves(el, orc, dtype, shape):
    spec = dict(conftest.load_package().scenes.spheres_pool(32, 4), shape=shape)
    _, _, wts = scene_fields(orc, spec, dtype)
    rng = np.random.default_rng(shape[0])
    vel = [rng.uniform(-1, 1, a.shape).astype(dtype) for a in wts]
    got = []
    for solver in (el.SOLVER_MG_FP64, el.SOLVER_JACOBI_FP64):
        sim = make_sim(el, shape, dtype, spec)
        for f, a in zip(("u", "v", "w"), vel):
            sim.upload(f, a)
        stats = sim.solve_pressure(0.01, solver=solver, tol=1e-13, max_iter=5000)
        assert stats["relres"] <= 1e-13
        if solver == el.SOLVER_MG_FP64:
            assert stats["iterations"] <= 40
        got.append(sim.download("pressure"))
        sim.close()
    assert rel_err(got[0], got[1]) <= (1e-7 if dtype == np.float64 else 2e-7)
