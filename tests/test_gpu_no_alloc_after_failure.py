"""el_solve_pressure_noalloc keeps one scratch array for all calls.  Its PCG reads z and the direction at
neighbours in row segments without fluid, which no kernel of the call writes: what another call left there
meets zero couplings, so it has to be finite.  A call that met a NaN leaves the vectors cleared: the calls
after it, of its own shape and of others, have the bits they had before."""

import ctypes as C

import numpy as np
import pytest

import conftest
from helpers import make_sim
from test_zz_no_alloc import _declare

pytestmark = pytest.mark.gpu

SHAPES = [(40, 40, 40), (33, 20, 47), (64, 12, 9), (20, 61, 30)]


def _scene(torch, shape, seed):
    spec = dict(conftest.load_package().scenes.spheres_pool(32, seed), shape=shape)
    el = conftest.load_package()
    sim = make_sim(el, shape, np.float32, spec)
    rng = np.random.default_rng(seed)
    host = {f: sim.download(f) for f in ("phi", "weight_u", "weight_v", "weight_w")}
    host |= {f: rng.uniform(-1, 1, sim.shape(f)).astype(np.float32) for f in "uvw"}
    grid = el.Grid(*shape, sim.dx)
    sim.close()
    return grid, host


def _solve(torch, el, solve, scene, spoil=False):
    grid, host = scene
    dev = {f: torch.from_numpy(a.copy()).cuda() for f, a in host.items()}
    dev["pressure"] = torch.zeros_like(dev["phi"])
    if spoil:
        dev["v"][grid.nk // 2, 1, :] = float("nan")
    stats = el.SolveStats()
    rc = solve(C.byref(grid), *[dev[f].data_ptr() for f in ("phi", "u", "v", "w", "weight_u", "weight_v", "weight_w",
                                                            "pressure")],
               0.01, 1e-8, 20000, C.byref(stats), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return rc, stats.as_dict(), [dev[f].cpu().numpy() for f in ("pressure", "u", "v", "w")]


def test_calls_after_a_failed_one(el):
    torch = pytest.importorskip("torch")
    solve = _declare(el.load(), el)
    scenes = [_scene(torch, s, q + 3) for q, s in enumerate(SHAPES)]
    before = [_solve(torch, el, solve, s) for s in scenes]
    assert all(b[0] == el.EL_OK for b in before)
    for failing in range(len(SHAPES)):
        assert _solve(torch, el, solve, scenes[failing], spoil=True)[0] == el.EL_ERR_NAN
        for q, s in enumerate(scenes):
            rc, stats, fields = _solve(torch, el, solve, s)
            assert (rc, stats) == before[q][:2]
            for a, b in zip(fields, before[q][2]):
                np.testing.assert_array_equal(a, b)
