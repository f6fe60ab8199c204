"""One kernel launched by several threads with different amounts of shared memory: none may take away what another has opted in to."""
import threading

import numpy as np
import pytest

from armnn_b200 import _abi, lib
from q8util import Cuda, random_fc_case
from test_shape_edges_gpu import softmax

pytestmark = pytest.mark.gpu

# the sizes of one instantiation: FullyConnected by K, softmax rows by axis (a CTA per row)
GROUPS = {
    "fc_mma": [lambda k=k: (random_fc_case(k, 40, k, 33), "fully_connected_q8") for k in (1023, 1301, 1603, 1901)],
    "softmax": [lambda n=n: (softmax(n, 3, n, _abi.S8), "softmax_q8") for n in (10500, 11000, 11500, 12200)],
}


@pytest.mark.parametrize("group", GROUPS)
def test_threads_with_different_sizes(built, group):
    l, work, keep = lib.load_library(), [], []
    for make in GROUPS[group]:
        case, entry = make()
        mem = Cuda()
        p, out = (case.params(mem) if hasattr(case, "params") else case.build(mem))[:2]
        out = out[0] if isinstance(out, list) else out
        lib.call(entry, p)
        mem.torch.cuda.synchronize()
        work.append((entry, p, out, out.clone(), mem.torch.cuda.Stream()))
        keep.append((mem, case))
    errors, start = [], threading.Barrier(len(work))

    def launches(entry, p, stream):
        start.wait()
        for _ in range(2000):
            try:
                lib.call(entry, p, stream.cuda_stream)
            except lib.B200KError as e:
                errors.append(str(e))
                return
    threads = [threading.Thread(target=launches, args=(e, p, s)) for e, p, _, _, s in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    mem.torch.cuda.synchronize()
    assert not errors, errors
    for _, _, out, want, _ in work:
        assert np.array_equal(out.cpu().numpy(), want.cpu().numpy())
