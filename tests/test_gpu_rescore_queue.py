"""The re-score with and without the staged codebook, around the batch size that decides (4 chunks of 32
candidates per SM) and with queues that end inside a chunk: the list scan's exact form and the precision form
against the oracle, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from tests.test_gpu_refine import built_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [4, 8, 16])
def test_rescore_queues(m):
    from mestrado_gb300.engine import GpuIndex

    ix, q, _ = built_index(m=m)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    gi = GpuIndex(ix)
    w = 12
    for nq, k in ((1, 33), (4 * sms - 1, 32), (4 * sms, 32), (4 * sms, 7), (2 * sms + 1, 65), (40, 1000)):
        qq = np.ascontiguousarray(q[np.arange(nq) % len(q)])
        o_ids, o_dis = oracle.ivfpq_search(ix, q, k=k, kl=k, w=w, rerank=False, ties=oracle.TIES_KEYED)
        for kw in (dict(scan_order="lists"), dict(mixed_scan=True)):
            ids, dis = gi.search(qq, k, w, **kw)
            np.testing.assert_array_equal(ids, o_ids[np.arange(nq) % len(q)])
            np.testing.assert_array_equal(dis.view(np.uint32), o_dis[np.arange(nq) % len(q)].view(np.uint32))
    gi.close()
