"""The plain form's large-C coarse stage through its tensor-core screen (three products of split BF16 parts):
queries of any value, not bytes, at the edges of its 128-query tiles, must give the full selection's lists and
distances bit for bit -- with a zero query, and with queries so large or so small that the screen's error bound
does not hold and every centroid is taken exactly."""
import numpy as np
import pytest

from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [64, 127, 128, 129, 300])
@pytest.mark.parametrize("C,w,scale", [(16384, 40, 1.0), (16500, 1, 1e-3), (16384, 300, 1e9)])
def test_split_queries(nq, C, w, scale):
    from mestrado_gb300.engine import GpuIndex

    rng = np.random.default_rng(nq + C + w)
    coa = (rng.normal(0.0, 1.0, (C, 128)) * scale).astype(np.float32)
    q = (coa[rng.integers(0, C, nq)] + rng.normal(0.0, 0.7, (nq, 128)) * scale).astype(np.float32)
    q[0] = 0.0
    q[1] = q[1] * np.float32(1e17 / scale)
    q[2] = q[2] * np.float32(1e-17 / scale)
    gi = GpuIndex(IVFPQData(coa=coa, pq=rng.normal(0, 1, (8, 256, 16)).astype(np.float32),
                            list_off=np.zeros(C + 1, np.int64), ids=np.zeros(0, np.int32),
                            codes=np.zeros((0, 8), np.uint8)))
    full = gi.coarse_assign(q, w, full=True)
    idx, dis, _, fallbacks = gi.coarse_assign(q, w, stats=True)
    gi.close()
    np.testing.assert_array_equal(idx, full[0])
    np.testing.assert_array_equal(dis.view(np.uint32), full[1].view(np.uint32))
    assert 2 <= fallbacks
