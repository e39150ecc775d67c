"""The plain FP64 PCG iteration by iteration against the oracle's Jacobi PCG: grids with partial row
segments, fewer segments than warps and several segments a warp, and iteration counts that end
inside a batch, at its end and across several (the deferred dot products are summed by the next
iteration or by the batch's last kernel)."""

import numpy as np
import pytest

import conftest
from conftest import rel_err
from helpers import make_sim, scene_fields

pytestmark = pytest.mark.gpu

# the two run the same recurrences from the same start: after k iterations they differ by a few
# roundings (1.1e-16) an operation, grown by at most the k products of alpha and beta (each O(10))
TOL = 1e-11


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(33, 9, 8), (31, 33, 17), (64, 20, 20), (150, 70, 66)])
@pytest.mark.parametrize("iterations", [1, 4, 6, 9])
def test_iterates_match_oracle_jacobi_pcg(el, orc, dtype, shape, iterations):
    spec = dict(conftest.load_package().scenes.spheres_pool(32, 4), shape=shape)
    phi, _, wts = scene_fields(orc, spec, dtype)
    rng = np.random.default_rng(8)
    vel = [rng.uniform(-1, 1, a.shape).astype(dtype) for a in wts]
    sim = make_sim(el, shape, dtype, spec)
    for f, a in zip(("u", "v", "w"), vel):
        sim.upload(f, a)
    stats = sim.solve_pressure(0.01, solver=el.SOLVER_JACOBI_FP64, tol=1e-14, max_iter=iterations, check_every=4)
    assert stats["iterations"] == iterations
    mats = orc.build_matrix(phi, *vel, *wts, sim.dx, 0.01)
    x, _, _, rr = orc.pcg(*mats, precond=orc.PRE_JACOBI, tol=1e-14, maxit=iterations)
    got = sim.download("pressure")
    sim.close()
    # FP32 fields hold the pressure rounded to float
    assert rel_err(got, x) <= (TOL if dtype == np.float64 else 6e-8)
    assert abs(stats["relres"] - rr) <= 1e-9 * rr
