"""core_gpu's packed outputs whatever the order and the gaps of their ranges: back to back, reversed, with
gaps (few and many queries): the written ranges hold the oracle's results, every other element is left alone."""
import numpy as np
import pytest

import oracle
from tests import golden_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 3, 60])
@pytest.mark.parametrize("layout", ["packed", "reversed", "gaps", "far"])
def test_ranges(nq, layout):
    from mestrado_gb300.engine import GpuIndex

    g = golden_cases.load("cfg1")
    w, k = 3, 20
    q = g.queries[:nq]
    coaidx = np.argsort(((q[:, None, :] - g.ix.coa[None]) ** 2).sum(-1), axis=1, kind="stable")[:, :w]
    res = (q[:, None, :] - g.ix.coa[coaidx]).reshape(-1, q.shape[1]).astype(np.float32)
    cnt = np.minimum(g.ix.list_sizes()[coaidx].sum(1), k)
    order = np.arange(nq)[::-1] if layout == "reversed" else np.arange(nq)
    gap = {"gaps": 5, "far": 400}.get(layout, 0)
    start, at = np.zeros(nq, np.int32), 7
    for i in order:
        start[i] = at
        at += int(cnt[i]) + gap
    gi = GpuIndex(g.ix)
    rid = coaidx.reshape(-1).astype(np.int32)
    idxs, dists = gi.core_gpu(res, rid, start, at + 9, k, w)
    gi.close()
    used = np.zeros(at + 9, bool)
    o_start = np.concatenate([[0], np.cumsum(cnt)[:-1]]).astype(np.int32)
    o_idxs, o_dists = oracle.core_cpu(g.ix, res, rid, o_start, int(cnt.sum()), k, w)
    for i in range(nq):
        used[start[i]:start[i] + cnt[i]] = True
        np.testing.assert_array_equal(idxs[start[i]:start[i] + cnt[i]], o_idxs[o_start[i]:o_start[i] + cnt[i]])
        np.testing.assert_array_equal(dists[start[i]:start[i] + cnt[i]], o_dists[o_start[i]:o_start[i] + cnt[i]])
    assert (idxs[~used] == -1).all() and np.isnan(dists[~used]).all()
