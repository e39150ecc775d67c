"""The tiled advection kernels, through the stateless operators, against the general per-sample path
(a context with advect_tiled = 0): grids at the tiles' edges (where the last tile also takes the
last faces), one cell thick, odd pitches, arrays that no box copy can stage (a pointer off the
16-byte boundary), steps inside and beyond the staged boxes, and velocities and level sets that
are infinite, NaN or cleared to the largest float."""

import numpy as np
import pytest

from conftest import rel_err
from helpers import RTOL_F32_WENO, make_sim, smooth_fields

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# the two paths share the displacement arithmetic and the lerps; the first stage differs in where its
# halves are rounded: a few roundings of 6e-8 on values and positions near 1 (FP32 WENO6: helpers.py)
TOL = {np.float32: 2e-6, np.float64: 1e-13}


def _stateless(el, dtype, dims, dx, fields, dt, trace, sample, offset):
    """phi and (trilinear) u, v, w by the stateless operators on arrays `offset` elements into theirs."""
    def put(a):
        t = torch.empty(a.size + offset, dtype=torch.float64 if dtype == np.float64 else torch.float32, device="cuda")
        t[offset:] = torch.from_numpy(a.reshape(-1))
        return t

    def at(t):
        return t.data_ptr() + offset * t.element_size()

    code = el.EL_F64 if dtype == np.float64 else el.EL_F32
    dev = [put(a) for a in fields]
    out = [put(np.zeros_like(a)) for a in fields]
    el.advect_collocated_grid(*dims, dx, code, at(out[0]), at(dev[0]), *[at(t) for t in dev[1:]], dt, trace, sample)
    el.advect_staggered_grid(*dims, dx, code, [at(t) for t in out[1:]], [at(t) for t in dev[1:]],
                             [at(t) for t in dev[1:]], dt, trace, el.SAMPLE_TRILINEAR)
    torch.cuda.synchronize()
    return [t[offset:].cpu().numpy().reshape(a.shape) for t, a in zip(out, fields)]


def _general(el, dtype, dims, fields, dt, trace, sample):
    sim = make_sim(el, dims, dtype)
    sim.set_tuning(advect_tiled=0)
    for f, a in zip(("phi", "u", "v", "w"), fields):
        sim.upload(f, a)
    sim.advect_level_set(dt, trace, sample)
    sim.advect_velocity(dt, trace, el.SAMPLE_TRILINEAR)
    out = [sim.download(f) for f in ("phi", "u", "v", "w")]
    sim.close()
    return out


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims,offset", [((32, 8, 8), 0), ((64, 16, 24), 1), ((33, 9, 17), 0), ((31, 7, 5), 0),
                                         ((96, 1, 8), 0), ((1, 8, 40), 0), ((20, 24, 1), 3)])
@pytest.mark.parametrize("cells", [0.6, 3.1])
@pytest.mark.parametrize("trace,sample", [(0, 1), (1, 0), (0, 0), (1, 1)])
def test_tiled_matches_per_sample(el, orc, dtype, dims, offset, cells, trace, sample):
    dx, *fields = smooth_fields(orc, *dims, dtype, seed=23)
    dt = float(dtype(cells) * dtype(dx))
    got = _stateless(el, dtype, dims, dx, fields, dt, trace, sample, offset)
    want = _general(el, dtype, dims, fields, dt, trace, sample)
    tol = TOL[dtype]
    assert rel_err(got[0], want[0]) <= (RTOL_F32_WENO if sample and dtype == np.float32 else 10 * tol if sample else tol)
    for g, w in zip(got[1:], want[1:]):
        assert rel_err(g, w) <= tol


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sample", [0, 1])
@pytest.mark.parametrize("bad", [np.nan, np.inf, np.finfo(np.float32).max])
def test_not_finite_values_match_per_sample(el, orc, dtype, sample, bad):
    """A velocity face and level-set cells that are NaN, infinite or the largest float (what a cleared
    level set holds), in a smooth flow.  The per-sample kernel also reads the neighbours that a
    first stage gives the weight zero (0 * NaN is NaN); the tiled ones read only what has a weight.
    So: not finite nowhere that the per-sample kernel is finite, the same values there, and not
    finite (NaN, inf) wherever the sample depends on the bad values, which a run with other finite
    numbers in their places shows."""
    dims = (40, 18, 19)

    def fields(value):
        dx, phi, u, v, w = smooth_fields(orc, *dims, dtype, seed=29)
        if value is not None:
            phi[4, 5, 6] = value
            phi[12:, :, 30:] = value
            v[15, 3, 9] = value
        return dx, [phi, u, v, w]

    dx, with_bad = fields(bad)
    dt = float(dtype(0.6) * dtype(dx))
    with np.errstate(all="ignore"):
        got = _stateless(el, dtype, dims, dx, with_bad, dt, 0, sample, 0)
        want = _general(el, dtype, dims, with_bad, dt, 0, sample)
        clean, other = (_stateless(el, dtype, dims, dx, fields(x)[1], dt, 0, sample, 0) for x in (None, 0.5))
        for g, r, c, o in zip(got, want, clean, other):
            fine = np.isfinite(r)
            assert np.all(np.isfinite(g[fine]))
            if not np.isfinite(bad):
                assert not np.any(np.isfinite(g[np.abs(c - o) > 1e-3]))
            small = fine & (np.abs(np.where(fine, r, 0)) < 1e3)
            tol = RTOL_F32_WENO if sample and dtype == np.float32 else 10 * TOL[dtype]
            assert np.max(np.abs(np.where(small, g, 0).astype(np.float64) - np.where(small, r, 0))) <= tol * 2
