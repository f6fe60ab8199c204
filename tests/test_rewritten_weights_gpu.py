"""Weights that an earlier kernel of the stream writes, for layers whose tables do not depend on them (input zero point 0)."""
import numpy as np
import pytest

from q8util import Cuda, gpu_pack, random_fc_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [256, 1024])
def test_written_by_the_kernel_before(built, m):
    """The writer runs for tens of microseconds after it has let its successor start; some of its SMs are idle for the last of it."""
    import torch
    from armnn_b200 import _abi, lib
    mem, stream = Cuda(), torch.cuda.Stream()
    writer, layer = random_fc_case(1, 4096, 4096, 4096), random_fc_case(2, m, 4096, 4096, x_q=(0.03, 0))
    w, _, _ = writer.params(mem)
    p, y, _ = layer.params(mem)
    w.y.data = p.w.data                                     # the first layer's output is the second one's weights
    for q in (w, p):
        c = _abi.Conv2dParams()
        c.w, c.oc, c.kh, c.kw, c.c = q.w, q.n, 1, 1, q.k
        q.packed = gpu_pack(mem, c)
    lib.call("fully_connected_q8", w)
    torch.cuda.synchronize()
    p.algo = 1
    lib.call("fully_connected_q8", p)
    want = mem.fetch(y).copy()
    p.algo = 0
    old = torch.from_numpy(layer.w).cuda()
    weights = [t for t in mem.keep if t.data_ptr() == p.w.data][0]
    for _ in range(5):
        weights.copy_(old)
        torch.cuda.synchronize()
        lib.call("fully_connected_q8", w, stream.cuda_stream)
        lib.call("fully_connected_q8", p, stream.cuda_stream)
        got = mem.fetch(y)
        assert np.array_equal(want, got), int((want != got).sum())
