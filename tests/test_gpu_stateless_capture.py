"""The stateless advections inside a caller's stream capture: no allocation, no synchronisation, tensor maps by
value, so that a replay on new values in the same arrays gives what a call gives."""

import numpy as np
import pytest

from helpers import smooth_fields

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sample", [0, 1])
def test_capture_and_replay(el, orc, dtype, sample):
    dims = (52, 20, 27)
    dx, *first = smooth_fields(orc, *dims, dtype, seed=3)
    _, *second = smooth_fields(orc, *dims, dtype, seed=4)
    dt = float(dtype(0.8) * dtype(dx))
    code = el.EL_F64 if dtype == np.float64 else el.EL_F32
    src = [torch.from_numpy(a).cuda() for a in first]
    out = [torch.empty_like(a) for a in src]

    def calls():
        stream = torch.cuda.current_stream().cuda_stream
        vel = [a.data_ptr() for a in src[1:]]
        el.advect_collocated_grid(*dims, dx, code, out[0].data_ptr(), src[0].data_ptr(), *vel, dt, 1, sample, stream)
        el.advect_staggered_grid(*dims, dx, code, [a.data_ptr() for a in out[1:]], vel, vel, dt, 1, 0, stream)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    for fields in (first, second):
        for a, f in zip(src, fields):
            a.copy_(torch.from_numpy(f))
        graph.replay()
        torch.cuda.synchronize()
        got = [a.clone() for a in out]
        calls()
        torch.cuda.synchronize()
        for g, o in zip(got, out):
            assert torch.equal(g, o)
