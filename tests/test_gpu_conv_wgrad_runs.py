"""The weight gradient where a block works through several columns, for every channel pair: more units (the
16 x 8 voxels of a brick of one plane) than eight a split, so that the ring of planes wraps, both gradient
buffers are refilled and a block changes column.  Reference: float64 on the GPU, bf16-representable
inputs.  Products are exact; an accumulator takes at most 8 steps a unit (4950 units in at least 38
splits: 1050 steps) and the reduction 64 more, 2^-23 of the largest partial sum each at most and with random
signs their square root: 34 * 2^-23 = 4e-6, ten times that for a partial sum above the total.

And a workspace that is aligned for a float and no more."""

import ctypes as C

import numpy as np
import pytest

from test_gpu_conv_tiles import FWD, wgrad_ref
from test_gpu_nn import _args, _rand, _ws, bf, dev

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _wgrad(W, shape, cin, cout, x, y, g, offset=0):
    L = W.lib()
    dw = torch.zeros(cout * 27 * cin, device="cuda")
    db = torch.zeros(cout, device="cuda")
    n = L.el_nn_conv3_backward_weight_workspace(*shape, cin, cout)
    ws = torch.full((n // 4 + 1 + offset,), float("nan"), device="cuda")
    args = _args(W, shape, cin, cout, x, cin, 0)
    args.out_a, args.out_a_channels = y.data_ptr(), cout
    assert L.el_nn_conv3_backward_weight(C.byref(args), g.data_ptr(), dw.data_ptr(), db.data_ptr(),
                                         ws.data_ptr() + 4 * offset, n, None) == 0
    torch.cuda.synchronize()
    return dw, db, n


@pytest.mark.parametrize("cin,cout", FWD)
def test_workspace_of_float_alignment(cin, cout):
    W = _ws()
    shape = nx, ny, nz = 17, 9, 6
    rng = np.random.default_rng(cin + cout)
    x, y, g = (dev(bf(_rand(rng, nz, ny, nx, c))) for c in (cin, cout, cout))
    want = _wgrad(W, shape, cin, cout, x, y, g)
    got = _wgrad(W, shape, cin, cout, x, y, g, offset=1)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("cin,cout", FWD)
def test_several_columns_a_block(cin, cout):
    W = _ws()
    shape = nx, ny, nz = 40, 33, 330
    gen = torch.Generator(device="cuda").manual_seed(cin + cout)
    x, y, g = (torch.randn((nz, ny, nx, c), device="cuda", generator=gen).to(torch.bfloat16) for c in (cin, cout, cout))
    dw, db, n = _wgrad(W, shape, cin, cout, x, y, g)
    units = -(-nx // 16) * -(-ny // 8) * nz
    assert units >= 8 * (n // (4 * (27 * cin * cout + cout)))
    rw, rb = wgrad_ref(x.double(), g.double() * (y > 0))
    for got, want in ((dw, rw.reshape(-1)), (db, rb)):
        assert float((got.double() - want).abs().max() / want.abs().max()) < 4e-5
