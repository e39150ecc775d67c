"""Runs the advection of a library built with cpp/advect_fakes.cuh (argv[1]) and prints what came of it as
JSON; launched by tests/test_gpu_tile_failures.py in a process of its own, since a process loads one
build of the library."""

import ctypes
import json
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

import conftest  # noqa: E402


def main():
    el = conftest.load_package()
    el._build_mod.LIB = sys.argv[1]
    el._build_mod.up_to_date = lambda *a, **k: True
    import torch
    lib = el.load()
    setup_fails = ctypes.c_int.in_dll(lib, "el_test_setup_fails")

    def stateless(dims=(40, 18, 20)):
        ni, nj, nk = dims
        shapes = [(nk, nj, ni), (nk, nj, ni + 1), (nk, nj + 1, ni), (nk + 1, nj, ni)]
        rng = np.random.default_rng(1)
        fields = [torch.from_numpy(rng.uniform(-0.5, 0.5, s).astype(np.float32)).cuda() for s in shapes]
        dx = 1.0 / ni
        out = [torch.zeros_like(a) for a in fields]
        vel = [a.data_ptr() for a in fields[1:]]
        status = []
        for call in (lambda: el.advect_collocated_grid(ni, nj, nk, dx, el.EL_F32, out[0].data_ptr(),
                                                       fields[0].data_ptr(), *vel, 0.7 * dx, 0, 1),
                     lambda: el.advect_staggered_grid(ni, nj, nk, dx, el.EL_F32, [a.data_ptr() for a in out[1:]], vel,
                                                      vel, 0.7 * dx, 0, 0)):
            try:
                call()
                status.append(0)
            except el.ELError as e:
                status.append(str(e))
        torch.cuda.synchronize()
        return status, [a.cpu().numpy() for a in out]

    said = {}
    _, want = stateless()
    setup_fails.value = 1
    said["setup_status"], got = stateless()
    setup_fails.value = 0
    said["setup_error"] = max(float(np.max(np.abs(g - w))) for g, w in zip(got, want))

    def step(tiled, nan):
        # 15 cells a row: u alone is staged by box copies, so that the level set keeps its fluid
        sim = el.Simulator(15, 12, 20, dtype=el.EL_F32)
        sim.set_tuning(advect_tiled=tiled)
        sim.init_scene(dict(el.scenes.spheres_pool(16, 4), shape=(15, 12, 20)))
        if nan:
            u = np.zeros(sim.shape("u"), np.float32)
            u[10, 2, 7] = np.nan
            sim.upload("u", u)
        try:
            sim.step(0.005, sample_phi=el.SAMPLE_WENO6, solver=el.SOLVER_MIXED, tol=1e-6)
            return "stepped"
        except el.ELError as e:
            return str(e)
        finally:
            sim.close()

    # the waits give up: NaN from the stateless operators and no other trace of it; a context's step reports its own
    assert lib.el_test_set_wait_fails(1) == 0
    said["wait_status"], got = stateless()
    said["wait_nan"] = [bool(np.all(np.isnan(a))) for a in got]
    _, got = stateless((64, 16, 24))
    said["wait_nan_full_tiles"] = [bool(np.all(np.isnan(a))) for a in got]
    said["wait_step_tiled"] = step(1, False)
    _, got = stateless()
    assert lib.el_test_set_wait_fails(0) == 0
    said["nan_step_per_sample"] = step(0, True)
    print(json.dumps(said))


if __name__ == "__main__":
    main()
