"""The engine's choice of scan order for an uneven batch through the host entry point, which knows the counts: a
batch of equal counts is estimated at its full work, as the uniform entry point's is."""
import ctypes as C

import numpy as np
import pytest

from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu


def test_equal_counts_take_the_uniform_order():
    from mestrado_gb300 import _lib
    from mestrado_gb300.engine import GpuIndex

    rng = np.random.default_rng(2)
    C_, length, nq, w, k = 4096, 100, 1500, 12, 10
    n = C_ * length
    ix = IVFPQData(coa=rng.uniform(0.0, 40.0, (C_, 128)).astype(np.float32),
                   pq=rng.normal(0.0, 15.0, (16, 256, 8)).astype(np.float32),
                   list_off=np.arange(C_ + 1, dtype=np.int64) * length, ids=rng.permutation(n).astype(np.int32),
                   codes=rng.integers(0, 256, (n, 16), dtype=np.uint8))
    q = rng.uniform(0.0, 40.0, (nq, 128)).astype(np.float32)
    wq, kq = np.full(nq, w, np.int32), np.full(nq, k, np.int32)
    ids, dis = (np.empty((2, nq, k), t) for t in (np.int32, np.float32))
    gi = GpuIndex(ix)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    _lib.check(gi.lib.gbivf_ivfpq_search(gi.h, p(q), nq, k, k, w, _lib.GBIVF_PROFILE, p(ids[0]), p(dis[0])))
    uniform = gi.last_scan_parts()[1]["list_scan"]
    _lib.check(gi.lib.gbivf_search_batched(gi.h, p(q), nq, p(wq), p(kq), _lib.GBIVF_PROFILE, p(ids[1]), p(dis[1])))
    uneven = gi.last_scan_parts()[1]["list_scan"]
    gi.close()
    assert uniform == uneven == 1
    np.testing.assert_array_equal(ids[0], ids[1])
    np.testing.assert_array_equal(dis[0].view(np.uint32), dis[1].view(np.uint32))
