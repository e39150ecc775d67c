"""The weight-gradient kernel at the edges of its tiles, all channel pairs: grids smaller than a tile,
ragged in x and y, of one plane, longer than a run.  References are float64 on bf16-representable
inputs; products are exact, and the FP32 accumulation of n <= 6120 voxels adds at most (n / 16) * 2^-23:
5e-5."""

import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_nn import _args, _rand, _ws, bf, dev, up2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

FWD = [(16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (128, 64), (96, 32), (48, 16)]
SHAPES = [(13, 19, 5), (16, 8, 1), (3, 2, 2), (17, 9, 40)]


def wgrad_ref(x, gm):
    """x (z, y, x, ci), gm (z, y, x, co) float64 -> dW [co][27][ci], db [co]"""
    nz, ny, nx, ci = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    gf = gm.reshape(-1, gm.shape[3])
    taps = [gf.T @ xp[dz:dz + nz, dy:dy + ny, dx:dx + nx].reshape(-1, ci)
            for dz in range(3) for dy in range(3) for dx in range(3)]
    return torch.stack(taps, 1), gf.sum(0)


@pytest.mark.parametrize("cin,cout", FWD)
@pytest.mark.parametrize("shape,up", [(s, 0) for s in SHAPES] + [((18, 10, 6), 1)])
def test_weight_gradient(cin, cout, shape, up):
    W = _ws()
    L = W.lib()
    nx, ny, nz = shape
    rng = np.random.default_rng(cin * 7 + cout + nx)
    ca = cin if not up else max(16, (2 * cin // 3) // 16 * 16)
    a = bf(_rand(rng, nz // 2, ny // 2, nx // 2, ca) if up else _rand(rng, nz, ny, nx, ca))
    b = bf(_rand(rng, nz, ny, nx, cin - ca)) if ca < cin else None
    y, g = bf(_rand(rng, nz, ny, nx, cout)), bf(_rand(rng, nz, ny, nx, cout))
    ad, bd, yd, gd = dev(a), dev(b) if b is not None else None, dev(y), dev(g)
    dw = torch.zeros(cout * 27 * cin, device="cuda")
    db = torch.zeros(cout, device="cuda")
    n = L.el_nn_conv3_backward_weight_workspace(nx, ny, nz, cin, cout)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    args = _args(W, shape, cin, cout, ad, ca, up, bd, cin - ca)
    args.out_a, args.out_a_channels = yd.data_ptr(), cout
    assert L.el_nn_conv3_backward_weight(C.byref(args), gd.data_ptr(), dw.data_ptr(), db.data_ptr(), ws.data_ptr(),
                                         n, None) == 0
    torch.cuda.synchronize()
    x = up2(a) if up else a
    x = x if b is None else torch.cat([x, b], 3)
    rw, rb = wgrad_ref(x, g * (y > 0))
    assert rel_err(dw.cpu().numpy(), rw.reshape(-1).numpy()) < 5e-5
    assert rel_err(db.cpu().numpy(), rb.numpy()) < 5e-5
