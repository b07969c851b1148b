"""Device memory of the list scan: its workspace follows the lists there are, not the longest one times the batch,
and where it cannot be had the engine's own choice of order is the per-query scan."""
import numpy as np
import pytest

from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu


def _index(lens, m=8, seed=3):
    rng = np.random.default_rng(seed)
    C, n = len(lens), int(np.sum(lens))
    off = np.zeros(C + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    ix = IVFPQData(coa=rng.uniform(0.0, 40.0, (C, 128)).astype(np.float32),
                   pq=rng.normal(0.0, 15.0, (m, 256, 128 // m)).astype(np.float32), list_off=off,
                   ids=rng.permutation(n).astype(np.int32), codes=rng.integers(0, 256, (n, m), dtype=np.uint8))
    return ix, rng


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_one_long_list():
    """One list of a million rows among 1,023 short ones: 3,000 queries x 64 probes took 7.5 GB of item headers
    when every pair counted with the longest list's pieces."""
    from mestrado_gb300.engine import GpuIndex

    ix, rng = _index([1_000_000] + [40] * 1023)
    q = rng.uniform(0.0, 40.0, (3000, 128)).astype(np.float32)
    gi = GpuIndex(ix)
    want = gi.search(q, 10, 64, scan_order="queries")
    before = _free()
    got = gi.search(q, 10, 64, scan_order="lists")
    grown = before - _free()
    gi.close()
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    assert grown < 1 << 30, f"{grown / 2**30:.1f} GB"


@pytest.mark.parametrize("mixed", [False, True])
def test_no_room(mixed):
    """About 1.5 GB free: the list scan's buffers for 10,000 queries with 1,000 results take more, the per-query
    scan's less."""
    import torch

    from mestrado_gb300._lib import GbivfError
    from mestrado_gb300.engine import GpuIndex

    ix, rng = _index([150] * 2048)
    q = rng.uniform(0.0, 40.0, (10_000, 128)).astype(np.float32)
    gi = GpuIndex(ix)
    want = gi.search(q, 1000, 16, scan_order="queries", mixed_scan=mixed)
    want = [x.copy() for x in want]
    gi.close()
    gi = GpuIndex(ix)
    gi.search(q[:4], 1000, 16, mixed_scan=mixed)
    torch.cuda.empty_cache()
    room = torch.empty(_free() - (3 << 29), dtype=torch.uint8, device="cuda")
    try:
        got = gi.search(q, 1000, 16, mixed_scan=mixed)
        with pytest.raises(GbivfError):
            gi.search(q, 1000, 16, mixed_scan=mixed, scan_order="lists")
        again = gi.search(q, 1000, 16, mixed_scan=mixed)
    finally:
        del room
        torch.cuda.empty_cache()
    after = gi.search(q, 1000, 16, scan_order="lists")  # the memory is back
    gi.close()
    if not mixed:
        for g in (got, again, after):
            np.testing.assert_array_equal(g[0], want[0])
            np.testing.assert_array_equal(g[1].view(np.uint32), want[1].view(np.uint32))
    else:
        for g in (got, again):  # (the same per-query scan)
            np.testing.assert_array_equal(g[0], want[0])
            np.testing.assert_array_equal(g[1].view(np.uint32), want[1].view(np.uint32))


def test_row_norms_are_made_for_list_scans_only():
    """20 million rows: an index that is searched query by query holds its codes and ids, not the 80 MB of row norms."""
    import torch

    from mestrado_gb300.engine import GpuIndex

    C, n, m = 2048, 20_000_000, 4
    rng = np.random.default_rng(9)
    coa = rng.uniform(0.0, 40.0, (C, 128)).astype(np.float32)
    pq = rng.normal(0.0, 15.0, (m, 256, 128 // m)).astype(np.float32)
    off = np.linspace(0, n, C + 1).astype(np.int64)
    ids = torch.arange(n, dtype=torch.int32, device="cuda")
    codes = torch.randint(0, 256, (n, m), dtype=torch.uint8, device="cuda")
    q = rng.uniform(0.0, 40.0, (200, 128)).astype(np.float32)
    before = _free()
    gi = GpuIndex.from_device(coa, pq, off, ids, codes)
    want = gi.search(q, 10, 4, scan_order="queries")
    held = before - _free()
    assert held < n * (m + 4) + (60 << 20), f"{held / 2**20:.0f} MB"
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):  # the first list scan on one stream, the next on another
        s = torch.cuda.current_stream()
        d_q = torch.from_numpy(q).cuda()
        d_ids = torch.empty((200, 10), dtype=torch.int32, device="cuda")
        d_dis = torch.empty((200, 10), dtype=torch.float32, device="cuda")
        gi.search_device(d_q.data_ptr(), 200, 10, 4, d_ids.data_ptr(), d_dis.data_ptr(), stream_ptr=s.cuda_stream,
                         scan_order="lists")
        s.synchronize()
    got = gi.search(q, 10, 4, scan_order="lists")
    for ids_, dis_ in ((d_ids.cpu().numpy(), d_dis.cpu().numpy()), got):
        np.testing.assert_array_equal(ids_, want[0])
        np.testing.assert_array_equal(dis_.view(np.uint32), want[1].view(np.uint32))
    gi.close()
