"""Query norms (double, summed in order) through the coarse distances: rows whose products are exact in any
order, rows whose products spread too far for that, subnormal and zero rows, and dimensions around a warp's width
must all give the oracle's distances bit for bit."""
import numpy as np
import pytest

import oracle
from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [4, 32, 36, 128, 160])
def test_norms(d):
    from mestrado_gb300.engine import GpuIndex

    rng = np.random.default_rng(d)
    C, nq = 40, 37
    coa = rng.normal(0, 3, (C, d)).astype(np.float32)
    q = rng.integers(0, 256, (nq, d)).astype(np.float32)
    q[1] = 0.0
    q[2] = rng.normal(0, 1, d) * 10.0 ** rng.uniform(-12, 8, d)
    q[3] = rng.normal(0, 1e-22, d)
    q[4] = rng.normal(0, 1, d)
    q[5, 0], q[5, 1:] = 1e9, 1e-7
    q[6] = rng.uniform(0, 1, d) * 2.0 ** rng.integers(-15, 15, d)
    q = q.astype(np.float32)
    gi = GpuIndex(IVFPQData(coa=coa, pq=rng.normal(0, 1, (4, 256, d // 4)).astype(np.float32),
                            list_off=np.zeros(C + 1, np.int64), ids=np.zeros(0, np.int32),
                            codes=np.zeros((0, 4), np.uint8)))
    idx, dis = gi.coarse_assign(q, 9)
    gi.close()
    o_idx, o_dis = oracle.knn_full(coa, q, 9, ties=oracle.TIES_KEYED)
    np.testing.assert_array_equal(idx, o_idx)
    np.testing.assert_array_equal(dis.view(np.uint32), o_dis.view(np.uint32))
