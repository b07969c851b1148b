"""An index of more than 2^31 code rows: the hand-off between the kernels keeps rows in 32 bits, so every form that
re-scores or re-ranks rows must take them as unsigned. The list order, the precision form and the refinement re-rank
on the last lists, against the exact per-query scan, which hands base ids over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_last_lists():
    import torch

    from mestrado_gb300.engine import GpuIndex

    C, m, n = 1024, 4, (1 << 31) + (1 << 22)
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB of device memory")
    rng = np.random.default_rng(1)
    # the last 64 lists are short and lie beyond row 2^31; the queries are near them
    lens = np.full(C, 500, np.int64)
    lens[: C - 64] = (n - 64 * 500) // (C - 64)
    lens[0] += n - lens.sum()
    off = np.zeros(C + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    assert off[C - 64] > 1 << 31
    coa = rng.uniform(0.0, 40.0, (C, 128)).astype(np.float32)
    coa[: C - 64] += 1000.0
    pq = rng.normal(0.0, 15.0, (m, 256, 32)).astype(np.float32)
    pq2 = rng.normal(0.0, 4.0, (1, 256, 128)).astype(np.float32)
    ids = torch.arange(n, device="cuda", dtype=torch.int64).bitwise_and_(0x7FFFFFFF).to(torch.int32)
    codes = torch.randint(0, 256, (n, m), device="cuda", dtype=torch.uint8)
    codes2 = torch.randint(0, 256, (n, 1), device="cuda", dtype=torch.uint8)
    gi = GpuIndex.from_device(coa, pq, off, ids, codes, pq2=pq2, d_codes2=codes2)
    del ids, codes, codes2
    torch.cuda.empty_cache()
    q = (coa[C - 64 + np.arange(48)] + rng.normal(0.0, 15.0, (48, 128))).astype(np.float32)
    want = gi.search(q, 30, 8, scan_order="queries")
    assert want[0].min() >= 0
    got = gi.search(q, 30, 8, scan_order="lists")
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    for order in ("lists", "queries"):
        ids_, dis_ = gi.search(q, 30, 8, mixed_scan=True, scan_order=order)
        same = (ids_ == want[0]).all(1) & (dis_.view(np.uint32) == want[1].view(np.uint32)).all(1)
        assert (~same).sum() <= gi.last_unproven()
    refined = [gi.search(q, 10, 8, kl=30, refine=True, scan_order=o, mixed_scan=x)
               for o, x in (("queries", False), ("lists", False), ("queries", True))]
    gi.close()
    for r in refined[1:]:
        np.testing.assert_array_equal(r[0], refined[0][0])
        np.testing.assert_array_equal(r[1].view(np.uint32), refined[0][1].view(np.uint32))
    for i in range(48):
        assert set(refined[0][0][i]) <= set(want[0][i])
    torch.cuda.empty_cache()
