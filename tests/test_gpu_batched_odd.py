"""Uneven batches through the host entry point with odd and even query counts: the 64-bit output offsets
follow two 32-bit arrays of the batch's length in one buffer."""
import numpy as np
import pytest

import oracle
from tests import golden_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 2, 5, 8])
def test_query_counts(nq):
    from mestrado_gb300.engine import GpuIndex

    g = golden_cases.load("cfg1")
    rng = np.random.default_rng(nq)
    q = np.ascontiguousarray(g.queries[:nq])
    assert len(q) == nq
    wq = rng.integers(1, min(8, g.ix.coarsek) + 1, nq).astype(np.int32)
    kq = rng.integers(1, 20, nq).astype(np.int32)
    gi = GpuIndex(g.ix)
    got = gi.search_batched(q, wq, kq)
    want = oracle.search_batched(g.ix, q, wq, kq)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(np.asarray(a), np.asarray(b))
    gi.close()
