"""The FP64 quotients of csrc/el_div.cuh (a float reciprocal and Newton steps) against the compiler's division:
within one ulp over 2^28 random operands a range.  The correction by the residual leaves an error of half an ulp
and 2^-88 of the quotient, so that it differs from the rounded quotient by at most one ulp."""

import importlib
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_quotients_within_an_ulp(el, tmp_path):
    build = importlib.import_module("eulerian_liquid_gb300.build")
    exe = str(tmp_path / "test_div")
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS,
                        os.path.join(HERE, "cpp", "test_div.cu"), "-o", exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    worst = [int(x) for line in r.stdout.split("\n") for x in line.split()]
    assert len(worst) == 6 and max(worst) <= 1, r.stdout
