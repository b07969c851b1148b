"""The plain form's tensor-core screen for queries whose squared norm underflows to zero: its error bound is relative to
the norm, so every centroid is taken exactly, as for other queries out of its range; a query of zeros is in range."""
import numpy as np
import pytest

from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -60, 2.0 ** -70])
def test_norm_underflows(scale):
    from mestrado_gb300.engine import GpuIndex

    C, w = 16_384, 20
    rng = np.random.default_rng(8)
    coa = (rng.choice([-1.0, 1.0], (C, 128)) * scale * (1.0 + rng.integers(0, 8, (C, 1)) * 2.0 ** -18)).astype(np.float32)
    tiny = np.ldexp(rng.integers(-5, 6, (3, 128)).astype(np.float32), -78)
    gi = GpuIndex(IVFPQData(coa=coa, pq=rng.normal(0, 1, (8, 256, 16)).astype(np.float32),
                            list_off=np.zeros(C + 1, np.int64), ids=np.zeros(0, np.int32),
                            codes=np.zeros((0, 8), np.uint8)))
    for q, expected in ((tiny, 3), (np.zeros((2, 128), np.float32), None)):
        full = gi.coarse_assign(q, w, full=True)
        idx, dis, _, fallbacks = gi.coarse_assign(q, w, stats=True)
        np.testing.assert_array_equal(idx, full[0])
        np.testing.assert_array_equal(dis.view(np.uint32), full[1].view(np.uint32))
        assert expected is None or fallbacks == expected
    gi.close()
