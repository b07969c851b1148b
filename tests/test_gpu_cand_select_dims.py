"""The candidate selection's staged rows at dimensions where a chunk of 32 or a 16-byte load ends: the
filtered coarse stage against the full selection and the oracle, bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [4, 30, 36, 64, 100, 126])
@pytest.mark.parametrize("nq,w", [(3, 1), (20, 40)])
def test_dims(d, nq, w):
    from mestrado_gb300.engine import GpuIndex
    from mestrado_gb300.ivfdata import IVFPQData

    C = 16384
    rng = np.random.default_rng(d * 100 + w)
    coa = rng.normal(0, 30, (C, d)).astype(np.float32)
    q = (coa[rng.integers(0, C, nq)] + rng.normal(0, 5, (nq, d))).astype(np.float32)
    gi = GpuIndex(IVFPQData(coa=coa, pq=rng.normal(0, 10, (2, 256, d // 2)).astype(np.float32),
                            list_off=np.zeros(C + 1, np.int64), ids=np.zeros(0, np.int32),
                            codes=np.zeros((0, 2), np.uint8)))
    o_idx, o_dis = oracle.knn_full(coa, q, w, ties=oracle.TIES_KEYED)
    for full in (True, False):
        idx, dis = gi.coarse_assign(q, w, full=full)
        np.testing.assert_array_equal(idx, o_idx)
        np.testing.assert_array_equal(dis.view(np.uint32), o_dis.view(np.uint32))
    gi.close()
