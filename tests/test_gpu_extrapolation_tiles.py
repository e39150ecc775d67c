"""Extrapolation at the edges of the layer kernel's tiles (64 x 8 x 8 cells; up to four a block on a large
grid): one cell more and less than a tile along each axis, a single cell of a seed in a corner, a seed
that crosses tiles, and a grid of enough tiles for several a block.  The cells, sums and divisions are
the oracle's: bit for bit."""

import numpy as np
import pytest

from helpers import make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(1, 1, 1), (63, 7, 9), (64, 8, 8), (65, 9, 7), (129, 17, 24), (200, 160, 150)])
@pytest.mark.parametrize("seed", ["corner", "plane"])
def test_layers_match_the_oracle(el, orc, dtype, shape, seed):
    ni, nj, nk = shape
    rng = np.random.default_rng(ni)
    sim = make_sim(el, shape, dtype)
    val = rng.standard_normal(sim.shape("u")).astype(dtype)
    valid = np.zeros(sim.shape("u"), np.uint8)
    if seed == "corner":
        valid[-1, -1, -1] = 1
    else:
        valid[:, nj // 2, 1::3] = 1
    for f in ("u", "v", "w"):
        sim.upload(f, val if f == "u" else np.zeros(sim.shape(f), dtype))
        sim.upload("valid_" + f, valid if f == "u" else np.zeros(sim.shape(f), np.uint8))
    sim.extrapolate_velocity(5)
    g, m = orc.extrapolate(val, valid, 5)
    np.testing.assert_array_equal(sim.download("u"), g)
    np.testing.assert_array_equal(sim.download("valid_u"), m)
    assert not sim.download("valid_v").any()
    sim.close()
