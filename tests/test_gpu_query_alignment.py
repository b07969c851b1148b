"""Device queries that start on any 4-byte boundary, in either scan order and form: the results of the same queries
on a 16-byte boundary, bit for bit."""
import numpy as np
import pytest

from tests import golden_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("order", ["lists", "queries", None])
def test_shifted_queries(shift, order):
    import torch

    from mestrado_gb300.engine import GpuIndex

    g = golden_cases.load("m16")
    nq, k, w = len(g.queries), 20, g.meta["w"]
    buf = torch.zeros(nq * 128 + 4, device="cuda")
    assert buf.data_ptr() % 16 == 0
    gi = GpuIndex(g.ix)
    for mixed in (False, True):
        out = []
        for s in (0, shift):
            d_q = buf[s:s + nq * 128]
            d_q.copy_(torch.from_numpy(np.ascontiguousarray(g.queries)).reshape(-1))
            ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
            dis = torch.empty((nq, k), dtype=torch.float32, device="cuda")
            gi.search_device(d_q.data_ptr(), nq, k, w, ids.data_ptr(), dis.data_ptr(), mixed_scan=mixed,
                             mixed_coarse=mixed, scan_order=order)
            torch.cuda.synchronize()
            out.append((ids.cpu().numpy(), dis.cpu().numpy().view(np.uint32)))
        for a, b in zip(*out):
            np.testing.assert_array_equal(a, b)
    gi.close()
