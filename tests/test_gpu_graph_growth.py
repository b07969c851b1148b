"""A captured search replayed after searches that made the index's buffers grow: the replay's own buffers must still
be there. They are given back with the last graph."""
import numpy as np
import pytest

from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("order", ["queries", "lists"])
@pytest.mark.parametrize("mixed", [False, True])
def test_replay_after_larger_searches(order, mixed):
    import torch

    from mestrado_gb300.engine import GpuIndex

    rng = np.random.default_rng(3)
    C, length, m = 256, 300, 8
    n = C * length
    ix = IVFPQData(coa=rng.uniform(0.0, 40.0, (C, 128)).astype(np.float32),
                   pq=rng.normal(0.0, 15.0, (m, 256, 128 // m)).astype(np.float32),
                   list_off=np.arange(C + 1, dtype=np.int64) * length, ids=rng.permutation(n).astype(np.int32),
                   codes=rng.integers(0, 256, (n, m), dtype=np.uint8))
    big = rng.uniform(0.0, 40.0, (6000, 128)).astype(np.float32)
    q, k, w = big[:64], 10, 8
    gi = GpuIndex(ix)
    d_q = torch.from_numpy(q).cuda()
    d_ids = torch.empty((64, k), dtype=torch.int32, device="cuda")
    d_dis = torch.empty((64, k), dtype=torch.float32, device="cuda")
    s = torch.cuda.Stream()
    graphs = [gi.capture_graph(d_q.data_ptr(), 64, k, w, d_ids.data_ptr(), d_dis.data_ptr(), mixed_scan=mixed,
                               scan_order=order, stream_ptr=s.cuda_stream) for _ in range(2)]
    graphs[0].launch(s.cuda_stream)
    s.synchronize()
    want = d_ids.cpu().numpy(), d_dis.cpu().numpy().view(np.uint32)
    for kk in (50, 1000):
        for o in ("queries", "lists"):
            gi.search(big, kk, 32, scan_order=o)
            gi.search(big, kk, 32, scan_order=o, mixed_scan=True)
    used = torch.full((200 << 20,), 255, dtype=torch.uint8, device="cuda")  # over whatever was freed
    for g in graphs:
        d_ids.fill_(-9)
        g.launch(s.cuda_stream)
        s.synchronize()
        np.testing.assert_array_equal(d_ids.cpu().numpy(), want[0])
        np.testing.assert_array_equal(d_dis.cpu().numpy().view(np.uint32), want[1])
    before = _free()
    graphs[0].close()
    assert _free() <= before + (1 << 20)
    graphs[1].close()
    assert _free() > before + (4 << 20)  # the outgrown buffers
    del used
    gi.close()
