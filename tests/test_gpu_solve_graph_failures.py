"""The mixed solve as one graph (the second and later of a row) where it fails or its surroundings change: a NaN
is reported as the host-driven solve (the first of a context) reports it, the solves after it have the bits
of a context that never failed, and the graph runs on whichever stream the context has."""

import ctypes

import numpy as np
import pytest

import conftest
from helpers import make_sim

pytestmark = pytest.mark.gpu

SHAPES = [(8, 7, 8), (20, 17, 33), (70, 64, 72)]  # one multigrid level, row segments, the tile kernels


def _scene(shape, dtype):
    spec = dict(conftest.load_package().scenes.spheres_pool(32, 4), shape=shape)
    sim = make_sim(conftest.load_package(), shape, dtype, spec)
    rng = np.random.default_rng(shape[0])
    return sim, {f: rng.uniform(-1, 1, sim.shape(f)).astype(dtype) for f in "uvw"}


def _solve(el, sim, vel):
    """Status, the stats and the fields, by the C call: the Python one gives no stats with an error."""
    for f, a in vel.items():
        sim.upload(f, a)
    sim.upload("pressure", np.zeros(sim.shape("pressure"), sim.field_dtype("pressure")))
    stats = el.SolveStats()
    prm = el.solve_params(solver=el.SOLVER_MIXED, tol=1e-6)
    status = sim.lib.el_solve_pressure(sim.h, 0.01, ctypes.byref(prm), ctypes.byref(stats))
    return status, stats.as_dict(), [sim.download(f) for f in ("pressure", "u", "v", "w")]


def _same(a, b):
    assert a[:2] == b[:2]
    for x, y in zip(a[2], b[2]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_nan_by_graph_as_host_driven(el, dtype, shape):
    sim, vel = _scene(shape, dtype)
    bad = {f: a.copy() for f, a in vel.items()}
    bad["v"][shape[2] // 2, 2, shape[0] // 2] = np.nan
    good = _solve(el, sim, vel)
    assert good[0] == 0 and good[1]["fluid_cells"] > 0
    _same(_solve(el, sim, vel), good)
    by_graph = _solve(el, sim, bad)
    fresh, _ = _scene(shape, dtype)
    host_driven = _solve(el, fresh, bad)
    fresh.close()
    assert by_graph[0] == host_driven[0] != 0
    nan = lambda st: {k: v for k, v in st.items() if k != "relres"}  # noqa: E731 (NaN there, or what the sweep left)
    assert nan(by_graph[1]) == nan(host_driven[1])
    assert by_graph[1]["fluid_cells"] == good[1]["fluid_cells"]
    # every solver vector was cleared: the next solves have their bits, over other cells too
    for _ in range(2):
        _same(_solve(el, sim, vel), good)
    other = np.roll(sim.download("phi"), 3, axis=0)
    sim.upload("phi", other)
    _solve(el, sim, bad)
    fresh, _ = _scene(shape, dtype)
    fresh.upload("phi", other)
    _same(_solve(el, sim, vel), _solve(el, fresh, vel))
    fresh.close()
    sim.close()


@pytest.mark.parametrize("shape", SHAPES)
def test_graph_on_other_streams(el, shape):
    torch = pytest.importorskip("torch")
    sim, vel = _scene(shape, np.float32)
    good = _solve(el, sim, vel)
    streams = [torch.cuda.Stream() for _ in range(2)]
    for s in (None, streams[0], streams[1], streams[0], None):
        sim.set_stream(s.cuda_stream if s is not None else None)
        for _ in range(2):
            _same(_solve(el, sim, vel), good)
    sim.close()
