"""The weight-gradient and tcgen05 convolution kernels at the edges of their tiles, all channel pairs.

Both stage a column of planes and work on a run of units: grids smaller than a tile, ragged in x and y,
of one plane, longer than a run, and with more columns than blocks.  References are float64 on
bf16-representable inputs.

  - weight gradients (FP32 out): products are exact, at most (n / 16) * 2^-23 of accumulation for the
    n <= 6120 voxels here: 5e-5;
  - bf16 outputs, each element: half an ulp of rounding, 2^-8 |y| (8 significant bits), and the FP32
    accumulation's 27 * 128 / 16 steps of 2^-23 max |y|, doubled: 5e-5 max |y|;
  - tcgen05 against mma.sync on a large grid: FP32 sums in another order (< 2e-5 apart) round
    differently in a share 2e-5 * 2^8 of the outputs, by 2^-8 each: 5e-4."""

import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_nn import _args, _pack, _rand, _ws, bf, conv_ref, dev, up2

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


PAIRS = FWD + [(32, 16), (64, 32), (64, 128), (32, 96), (16, 48)]


def _run_conv(W, shape, cin, cout, xd, w, bias, mask, split, tc):
    L = W.lib()
    nx, ny, nz = shape
    fwd, _ = _pack(L, w.numpy(), cin, cout)
    args = _args(W, shape, cin, cout, xd, cin, 0)
    args.weights, args.relu = fwd.data_ptr(), 1 if bias is not None else 0
    args.bias = bias.data_ptr() if bias is not None else None
    args.mask = mask.data_ptr() if mask is not None else None
    if tc:
        pt = torch.empty_like(fwd)
        wd = torch.from_numpy(w.numpy().astype(np.float32)).cuda()
        assert L.el_nn_pack_weights_tc(cin, cout, wd.data_ptr(), pt.data_ptr(), None, None) == 0
        args.weights_tc = pt.data_ptr()
    out_a = torch.empty((nz, ny, nx, split), dtype=torch.bfloat16, device="cuda")
    out_b = torch.empty((nz, ny, nx, cout - split), dtype=torch.bfloat16, device="cuda")
    args.out_a, args.out_a_channels, args.out_b = out_a.data_ptr(), split, out_b.data_ptr()
    assert L.el_nn_conv3_forward(C.byref(args), None) == 0
    torch.cuda.synchronize()
    assert L.el_nn_take_error() == 0
    return torch.cat([out_a, out_b], 3)


def _within_rounding(got, ref):
    return bool(((got.double().cpu() - ref).abs() <= 2.0 ** -8 * ref.abs() + 5e-5 * ref.abs().max()).all())


@pytest.mark.parametrize("cin,cout", PAIRS)
@pytest.mark.parametrize("shape", SHAPES)
def test_tcgen05_convolution(cin, cout, shape):
    W = _ws()
    assert W.lib().el_nn_tc_supported(cin, cout) == 1
    nx, ny, nz = shape
    rng = np.random.default_rng(cin + 3 * cout + nz)
    x, m = bf(_rand(rng, nz, ny, nx, cin)), bf(_rand(rng, nz, ny, nx, cin))
    w = bf(_rand(rng, cout, 27, cin, scale=(2.0 / (27 * cin)) ** 0.5))
    bias = torch.from_numpy(_rand(rng, cout, scale=0.1))
    xd, md = dev(x), dev(m)
    got = _run_conv(W, shape, cin, cout, xd, w, bias.cuda(), None, cout - 8, True)
    assert _within_rounding(got, torch.relu(conv_ref(x, w, bias.double())))
    got = _run_conv(W, shape, cin, cout, xd, w, None, md, cout, True)
    assert _within_rounding(got, conv_ref(x * (m > 0), w))


@pytest.mark.parametrize("cin,cout", PAIRS)
def test_tcgen05_convolution_more_units_than_a_wave(cin, cout):
    W = _ws()
    shape = (40, 33, 330)  # 4950 units in 15 columns: several runs a block, across columns
    gen = torch.Generator(device="cuda").manual_seed(cin + cout)
    xd = torch.randn((330, 33, 40, cin), device="cuda", generator=gen).to(torch.bfloat16)
    w = bf(_rand(np.random.default_rng(cin), cout, 27, cin, scale=(2.0 / (27 * cin)) ** 0.5))
    tc = _run_conv(W, shape, cin, cout, xd, w, None, None, cout, True).float()
    mma = _run_conv(W, shape, cin, cout, xd, w, None, None, cout, False).float()
    assert float((tc - mma).norm() / mma.norm()) < 5e-4
