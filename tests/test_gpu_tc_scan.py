"""The tensor-core list scan of the precision form (scan_tc.cu) at the edges of its tiles: lists of 1 to
300 rows (128-row tiles), 1 to over 64 queries per work item (MMA columns in steps of 16, items of up to 32
or 64 queries), every m, and vectors whose scale takes the FP16 operands' power-of-two scaling away from 1.

Its approximate distances only choose candidates: every row that the form reports as proven must be the
oracle's exactly (ids and distance bits, keyed ties), so there is no tolerance; at most the unproven rows
may differ, and on this data (Gaussian residuals) at most 1% may be unproven."""
import numpy as np
import pytest

import oracle
from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu

LENGTHS = [300, 129, 128, 127, 1, 0, 33, 257, 64, 16, 8, 7]


def _index(m, scale, seed):
    rng = np.random.default_rng(seed)
    lens = np.array(LENGTHS * 2, np.int64)
    C, n = len(lens), int(lens.sum())
    coa = rng.uniform(0.0, 40.0, (C, 128)).astype(np.float32) * np.float32(scale)
    pq = rng.normal(0.0, 15.0, (m, 256, 128 // m)).astype(np.float32) * np.float32(scale)
    off = np.zeros(C + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    ix = IVFPQData(coa=coa, pq=pq, list_off=off, ids=rng.permutation(n).astype(np.int32),
                   codes=rng.integers(0, 256, (n, m), dtype=np.uint8))
    return ix, rng


@pytest.mark.parametrize("m", [4, 8, 16])
@pytest.mark.parametrize("nq,w,k,scale", [(1, 24, 1, 1.0), (15, 20, 10, 1.0), (33, 24, 1, 2.0 ** -9), (70, 24, 5, 300.0),
                                          (600, 7, 1, 1.0)])
def test_edges_against_oracle(m, nq, w, k, scale):
    from mestrado_gb300.engine import GpuIndex

    ix, rng = _index(m, scale, seed=m * 1000 + nq)
    q = (ix.coa[rng.integers(0, ix.coarsek, nq)] + rng.normal(0.0, 15.0, (nq, 128)) * scale).astype(np.float32)
    gi = GpuIndex(ix)
    ids, dis = gi.search(q, k, w, mixed_scan=True, scan_order="lists")
    unproven = gi.last_unproven()
    gi.close()
    o_ids, o_dis = oracle.ivfpq_search(ix, q, k=k, kl=k, w=w, rerank=False, ties=oracle.TIES_KEYED)
    differ = sum(not (np.array_equal(ids[i], o_ids[i]) and
                      np.array_equal(dis[i].view(np.uint32), o_dis[i].view(np.uint32))) for i in range(nq))
    assert differ <= unproven <= 0.01 * nq, f"{differ} rows differ, {unproven} not proven"
