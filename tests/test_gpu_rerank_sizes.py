"""The re-rank at the sizes where its rounds, its sorts and its lane layouts end: exact results, as in
tests/test_gpu_refine.py (the refined distances in their defined order) and as the oracle's re-rank by the
raw vectors (every operation in its order)."""
import numpy as np
import pytest

import oracle
from tests.test_gpu_refine import built_index, refined_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,m2", [(8, 32), (4, 8), (16, 1), (8, 8)])
def test_refined_sizes(m, m2):
    """Candidate counts around a warp's four and the sorts' 256 and 512, refinement pieces of 4 to 128."""
    from mestrado_gb300.engine import GpuIndex

    ix, q, _ = built_index(m=m)
    rng = np.random.default_rng(17)  # (any refinement codes do: the order of the operations is defined)
    ix.pq2 = rng.normal(0, 4, (m2, 256, 128 // m2)).astype(np.float32)
    ix.codes2 = rng.integers(0, 256, (ix.n, m2), dtype=np.uint8)
    gi = GpuIndex(ix)
    for k, kl, w in ((1, 1, 3), (5, 5, 8), (3, 255, 8), (257, 257, 8), (100, 513, 12), (1000, 1000, 16), (1024, 1024, 1)):
        adc_ids, _ = oracle.ivfpq_search(ix, q, k=kl, kl=kl, w=w, rerank=False, ties=oracle.TIES_KEYED)
        for mixed in (False, True):
            ids, dis = gi.search(q, k, w, kl=kl, refine=True, mixed_scan=mixed)
            for i in range(len(q)):
                r_ids, r_dis = refined_reference(ix, q[i : i + 1], adc_ids[i : i + 1], k)
                n = r_ids.shape[1]
                np.testing.assert_array_equal(ids[i, :n], r_ids[0])
                np.testing.assert_array_equal(dis[i, :n].view(np.uint32), r_dis[0].view(np.uint32))
                assert (ids[i, n:] == -1).all() and np.isinf(dis[i, n:]).all()
    gi.close()


def test_raw_sizes():
    """Candidate counts around a round of the gather (32 rows) and the sorts' 256 and 512."""
    from mestrado_gb300.engine import GpuIndex

    ix, q, base = built_index()
    gi = GpuIndex(ix, base=base)
    for k, kl, w in ((1, 1, 3), (31, 33, 8), (64, 65, 8), (10, 256, 8), (257, 257, 8), (100, 513, 12), (1000, 1000, 16),
                     (1024, 1024, 1)):
        o_ids, o_dis = oracle.ivfpq_search(ix, q, k=k, kl=kl, w=w, base=base, rerank=True, ties=oracle.TIES_KEYED)
        for kw in (dict(scan_order="queries"), dict(scan_order="lists"), dict(mixed_scan=True)):
            ids, dis = gi.search(q, k, w, kl=kl, rerank=True, **kw)
            np.testing.assert_array_equal(ids, o_ids)
            np.testing.assert_array_equal(dis.view(np.uint32), o_dis.view(np.uint32))
    gi.close()
