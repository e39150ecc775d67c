"""FP64 WENO6 of level sets far beyond a signed distance: the tiled kernel forms the nonlinear weights by one
reciprocal of a product of two smoothness terms (the eighth power of the values), which overflows from
about 4e37 on; there it gives the sample to the general path instead of dropping a weight.  The two paths
differ by the rounding of their weights and candidates: 1e-13 of the largest value where none overflow
(test_gpu_advection_tiles.py), and the bound is ten times that."""

import numpy as np
import pytest

from helpers import make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e30, 2e37, 4e37, 8e37, 1e39, 1e60])
def test_tiled_weno6_at_any_scale(el, scale):
    ni, nj, nk = 37, 18, 21
    rng = np.random.default_rng(11)
    phi = scale * rng.uniform(-1, 1, (nk, nj, ni))
    sim = make_sim(el, (ni, nj, nk), np.float64)
    vel = {f: rng.uniform(-0.9, 0.9, sim.shape(f)) for f in "uvw"}
    got = []
    for tiled in (1, 0):
        sim.set_tuning(advect_tiled=tiled)
        sim.upload("phi", phi)
        for f, a in vel.items():
            sim.upload(f, a)
        sim.advect_level_set(0.9 / ni, 0, 1)
        got.append(sim.download("phi"))
    sim.close()
    assert np.all(np.isfinite(got[1]))
    assert np.max(np.abs(got[0] - got[1])) <= 1e-12 * scale
