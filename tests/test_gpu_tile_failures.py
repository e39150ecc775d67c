"""What the advection does when its tiled kernels cannot run: the library with el_advect.cu compiled
against cpp/advect_fakes.cuh, which makes the kernels' set-up, or their wait for box copies, fail on
the host's request."""

import glob
import importlib
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def said(el, tmp_path_factory):
    build = importlib.import_module("eulerian_liquid_gb300.build")
    build.build()
    out = str(tmp_path_factory.mktemp("fakes"))
    obj, lib = os.path.join(out, "el_advect.cu.o"), os.path.join(out, "libfakes.so")
    run = dict(capture_output=True, text=True, timeout=600)
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-include",
                        os.path.join(HERE, "cpp", "advect_fakes.cuh"), "-c",
                        os.path.join(build.CSRC, "el_advect.cu"), "-o", obj], **run)
    assert r.returncode == 0, r.stderr
    others = [o for o in glob.glob(os.path.join(build.OUT_DIR, "*.cu.o")) if os.path.basename(o) != "el_advect.cu.o"]
    r = subprocess.run([build.nvcc(), *build.ARCH, "-shared", "-o", lib, obj, *others, "-lcudart_static", "-lrt",
                        "-lpthread", "-ldl"], **run)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([sys.executable, os.path.join(HERE, "tile_failures_run.py"), lib], **run)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_setup_failure_falls_back(said):
    """The per-sample kernels take over, and the call succeeds."""
    assert said["setup_status"] == [0, 0]
    assert said["setup_error"] < 2e-4  # FP32 WENO6 by the two paths (helpers.py)


def test_wait_failure_is_nan_and_not_another_callers(said):
    """A context's step reports its own advection's wait as a timeout; a NaN in a step that no box copy had a
    part in stays a NaN, whatever became of a stateless call before it (arrays of 40 cells a row: phi, v
    and w by box copies, u by plain loads)."""
    assert said["wait_status"] == [0, 0]
    assert said["wait_nan"] == [True] * 4
    assert "gave up" in said["wait_step_tiled"]
    assert "gave up" not in said["nan_step_per_sample"] and "non-finite" in said["nan_step_per_sample"]


def test_wait_failure_is_nan_on_the_last_faces(said):
    """Grids of whole tiles: the last tiles also take the last faces along each axis."""
    assert said["wait_nan_full_tiles"] == [True] * 4
