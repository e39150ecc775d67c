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
    rng = np.random.default_rng(1)
    ni, nj, nk = 40, 18, 20
    shapes = [(nk, nj, ni), (nk, nj, ni + 1), (nk, nj + 1, ni), (nk + 1, nj, ni)]
    fields = [torch.from_numpy(rng.uniform(-0.5, 0.5, s).astype(np.float32)).cuda() for s in shapes]
    dx = 1.0 / 40

    def stateless():
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
    print(json.dumps(said))


if __name__ == "__main__":
    main()
