"""The FP32 level set's advection, bit for bit.  The projection divides by distances to the surface down
to a hundredth of a cell, so another rounding of phi (1e-9 of it is enough) moves the velocity of
single faces by up to 5e-3: the roundings are part of the result.  golden/level_set_bits.json holds
the SHA-256 of phi after one advection, recorded before the WENO6 kernel was last rewritten, for
inputs made of integers (the same on every machine): both schemes, both traces, tiles of four and of
eight planes, rows that a box copy can and cannot stage, a step of one cell and one of three.

`python tests/test_gpu_level_set_bits.py` prints the file for the library as built."""

import hashlib
import json
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "level_set_bits.json")
SHAPES = [(37, 18, 21), (64, 64, 48), (97, 40, 53)]
CELLS = [1.0, 3.0]


def _mix(shape, salt):
    """Whole numbers below 2^16, scattered."""
    k, j, i = np.meshgrid(*(np.arange(n, dtype=np.uint64) for n in shape), indexing="ij")
    h = (i + np.uint64(977) * j + np.uint64(65537) * k + np.uint64(salt)) * np.uint64(2654435761)
    h ^= h >> np.uint64(15)
    h *= np.uint64(2246822519)
    return ((h >> np.uint64(13)) & np.uint64(0xFFFF)).astype(np.int64)


def _fields(ni, nj, nk):
    """A bowl with a rough surface, and a velocity below 1 with shear and noise; every value a
    multiple of 2^-20."""
    k, j, i = np.meshgrid(*(np.arange(n, dtype=np.int64) for n in (nk, nj, ni)), indexing="ij")
    bowl = (i - ni // 2) ** 2 + (j - nj // 3) ** 2 + (k - nk // 2) ** 2 - (min(ni, nj, nk) // 3) ** 2
    phi = (512 * bowl + (_mix((nk, nj, ni), 1) >> 6)) / 2.0 ** 20
    vel = []
    for c, shape in enumerate(((nk, nj, ni + 1), (nk, nj + 1, ni), (nk + 1, nj, ni))):
        k, j, i = np.meshgrid(*(np.arange(n, dtype=np.int64) for n in shape), indexing="ij")
        wave = ((i * (3 + c) + j * (5 - c) + k * 4) % 64 - 32) * 24576 // 32
        vel.append((wave * 32 + _mix(shape, 7 + c) * 2) / 2.0 ** 20)
    return [a.astype(np.float32) for a in (phi, *vel)]


def _advected(el, shape, cells, trace, sample):
    sim = el.Simulator(*shape, dtype=el.EL_F32)
    for f, a in zip(("phi", "u", "v", "w"), _fields(*shape)):
        sim.upload(f, a)
    sim.advect_level_set(float(np.float32(cells) * (np.float32(1) / np.float32(shape[0]))), trace, sample)
    phi = sim.download("phi")
    sim.close()
    return phi


def _key(shape, cells, trace, sample):
    return "%dx%dx%d, %g cells, RK%d, %s" % (*shape, cells, trace + 2, "WENO6" if sample else "trilinear")


@pytest.mark.parametrize("sample", [0, 1])
@pytest.mark.parametrize("trace", [0, 1])
@pytest.mark.parametrize("cells", CELLS)
@pytest.mark.parametrize("shape", SHAPES)
def test_level_set_bits(el, shape, cells, trace, sample):
    with open(GOLDEN) as f:
        want = json.load(f)
    phi = _advected(el, shape, cells, trace, sample)
    assert np.all(np.isfinite(phi))
    assert hashlib.sha256(phi.tobytes()).hexdigest() == want[_key(shape, cells, trace, sample)]


if __name__ == "__main__":
    from conftest import load_package
    print(json.dumps({_key(s, c, t, q): hashlib.sha256(_advected(load_package(), s, c, t, q).tobytes()).hexdigest()
                      for s in SHAPES for c in CELLS for t in (0, 1) for q in (0, 1)}, indent=1))
