"""The plain coarse stage where the tensor-core screen's operands find no memory: the SIMT pass, same results; and the
screen again once there is room."""
import numpy as np
import pytest

from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu


def test_plain_stage_without_room_for_the_screen():
    import torch

    from mestrado_gb300._lib import GbivfError
    from mestrado_gb300.engine import GpuIndex

    C, nq, w = 262_144, 40, 16
    rng = np.random.default_rng(5)
    coa = rng.normal(0, 30, (C, 128)).astype(np.float32)
    q = (coa[rng.integers(0, C, nq)] + rng.normal(0, 10, (nq, 128))).astype(np.float32)

    def index():
        return GpuIndex(IVFPQData(coa=coa, pq=rng.normal(0, 1, (8, 256, 16)).astype(np.float32),
                                  list_off=np.zeros(C + 1, np.int64), ids=np.zeros(0, np.int32),
                                  codes=np.zeros((0, 8), np.uint8)))

    gi = index()
    want = gi.coarse_assign(q, w, full=True)
    gi.close()
    gi = index()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = torch.empty(torch.cuda.mem_get_info()[0] - (128 << 20), dtype=torch.uint8, device="cuda")
    try:  # the centroids' tiles alone take 168 MB
        got = gi.coarse_assign(q, w)
        with pytest.raises(GbivfError):
            gi.coarse_assign(q, w, mixed=True)
        again = gi.coarse_assign(q, w)
    finally:
        del room
        torch.cuda.empty_cache()
    results = [got, again, gi.coarse_assign(q, w), gi.coarse_assign(q, w, mixed=True)]
    gi.close()
    for idx, dis in results[:3]:
        np.testing.assert_array_equal(idx, want[0])
        np.testing.assert_array_equal(dis.view(np.uint32), want[1].view(np.uint32))
    np.testing.assert_array_equal(results[3][0], want[0])
