"""Samples that do not move, or move by whole cells, keep their values bit for bit in both precisions,
whatever their neighbours hold: a read of fraction zero takes its own value only.  A velocity of zero
displaces by -dt / dx * 0 = -0, and one cell against the axis by exactly -1.  Level sets carry the
largest float where they were cleared, so a neighbour's share of one part in 1e16 would already be
another sign.  Also: constant infinite regions stay infinite."""

import numpy as np
import pytest

from helpers import make_sim

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CLEARED = float(np.finfo(np.float32).max)


def _level_set(el, sim, phi, vel, dt, trace, sample, tiled):
    sim.set_tuning(advect_tiled=tiled)
    sim.upload("phi", phi)
    for f, a in zip("uvw", vel):
        sim.upload(f, a)
    sim.advect_level_set(dt, trace, sample)
    return sim.download("phi")


def _rough(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    phi = rng.uniform(-1, 1, shape).astype(dtype)
    phi[rng.random(shape) < 0.1] = CLEARED
    phi[phi == 0] = 0.5
    return phi


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("tiled", [1, 0])
@pytest.mark.parametrize("trace", [0, 1])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_level_set_at_rest_and_whole_cells(el, dtype, tiled, trace, sign):
    ni, nj, nk = 32, 17, 20
    sim = make_sim(el, (ni, nj, nk), dtype)
    phi = _rough((nk, nj, ni), dtype, 3)
    zero = [np.zeros(sim.shape(f), dtype) for f in "uvw"]
    np.testing.assert_array_equal(_level_set(el, sim, phi, zero, 0.01, trace, 0, tiled), phi)
    # one axis moves by one cell exactly (dt / dx a power of two), the others rest; by RK2, whose one
    # weight is 1 (the three of RK3 are rounded: in float their sum times dt / dx need not be)
    for axis in range(3 if trace == 0 else 0):
        vel = [np.zeros_like(a) for a in zero]
        vel[axis][:] = sign
        got = np.moveaxis(_level_set(el, sim, phi, vel, 1.0 / 32, trace, 0, tiled), 2 - axis, 0)
        want = np.moveaxis(phi, 2 - axis, 0)
        if sign > 0:
            np.testing.assert_array_equal(got[1:], want[:-1])
        else:
            np.testing.assert_array_equal(got[:-1], want[1:])
    sim.close()


@pytest.mark.parametrize("tiled", [1, 0])
def test_weno6_fp64_at_rest(el, tiled):
    """The middle candidate at its own node is that node's value, and the correction's weights are zero."""
    ni, nj, nk = 33, 17, 20
    sim = make_sim(el, (ni, nj, nk), np.float64)
    phi = np.random.default_rng(4).uniform(-1, 1, (nk, nj, ni))
    zero = [np.zeros(sim.shape(f)) for f in "uvw"]
    got = _level_set(el, sim, phi, zero, 0.01, 0, 1, tiled)
    # (the per-sample kernel divides three equal candidates by the sum of their weights)
    np.testing.assert_allclose(got, phi, rtol=0 if tiled else 2e-15, atol=0)
    sim.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_faces_at_rest(el, dtype):
    """Face fields: the velocity advecting itself (the tiled kernel) and another field on the same grid (the
    per-sample one), with w zero and u, v zero over a part of the domain."""
    ni, nj, nk = 40, 18, 19
    rng = np.random.default_rng(5)
    u, v, w = [rng.uniform(0.2, 0.9, s).astype(dtype) for s in ((nk, nj, ni + 1), (nk, nj + 1, ni), (nk + 1, nj, ni))]
    w[:] = 0
    u[:, :, 20:] = 0
    v[:, :, 20:] = 0
    code = el.EL_F64 if dtype == np.float64 else el.EL_F32
    dx = 1.0 / 40
    other = [_rough(a.shape, dtype, 6 + q) for q, a in enumerate((u, v, w))]
    dev = [torch.from_numpy(a).cuda() for a in (u, v, w)]
    fields = [torch.from_numpy(a).cuda() for a in other]
    for src in (dev, fields):
        out = [torch.empty_like(a) for a in src]
        el.advect_staggered_grid(ni, nj, nk, dx, code, [a.data_ptr() for a in out], [a.data_ptr() for a in src],
                                 [a.data_ptr() for a in dev], 0.7 * dx, 1, 0)
        torch.cuda.synchronize()
        for a, o in zip(src, out):  # beyond one cell from the moving part
            np.testing.assert_array_equal(o.cpu().numpy()[:, :, 22:], a.cpu().numpy()[:, :, 22:])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_infinite_regions_stay(el, dtype):
    """Moving samples inside a region of one infinite value return it."""
    ni, nj, nk = 32, 16, 16
    sim = make_sim(el, (ni, nj, nk), dtype)
    phi = np.full((nk, nj, ni), np.inf, dtype)
    vel = [np.full(sim.shape(f), c, dtype) for f, c in zip("uvw", (0.3, 0.7, -0.45))]
    np.testing.assert_array_equal(_level_set(el, sim, phi, vel, 0.5 / 32, 0, 0, 1), phi)
    sim.close()
