"""The list order on long lists and the per-query order in ranges, at the sizes where their pieces end: a first
pass that ends inside a list (mean lists of 4,096 rows and more), lists around its least remainder of 512 rows, lists
cut in pieces of 1,024 and 8,192 rows, more than eight items of a list, a flat index, and queries that the error
bound leaves to a second scan. Everything is compared with the oracle bit for bit (keyed ties); the precision form
may differ on the queries that it does not report as proven."""
import ctypes as C

import numpy as np
import pytest

import oracle
from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu

CUT = [592, 593, 1023, 1024, 1025, 8191, 8192, 8193, 20_000, 5 * 1024 + 1, 4096, 591]
PIECES = [24_000, 8192, 8193, 16_385] + [5] * 1300


def _index(lens, m, seed, distinct=0):
    rng = np.random.default_rng(seed)
    C, n = len(lens), int(np.sum(lens))
    off = np.zeros(C + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    codes = rng.integers(0, 256, (n, m), dtype=np.uint8)
    if distinct:
        codes = np.ascontiguousarray(codes[rng.integers(0, distinct, n)])
    coa = rng.uniform(0.0, 40.0, (C, 128)).astype(np.float32) if C > 1 else np.zeros((1, 128), np.float32)
    ix = IVFPQData(coa=coa, pq=rng.normal(0.0, 15.0, (m, 256, 128 // m)).astype(np.float32), list_off=off,
                   ids=rng.permutation(n).astype(np.int32), codes=codes)
    return ix, rng


def _same(got, want):
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


def _lists_against_oracle(ix, q, k, w):
    from mestrado_gb300.engine import GpuIndex

    want = oracle.ivfpq_search(ix, q, k=k, kl=k, w=w, rerank=False, ties=oracle.TIES_KEYED)
    gi = GpuIndex(ix)
    _same(gi.search(q, k, w, scan_order="lists"), want)
    ids, dis = gi.search(q, k, w, mixed_scan=True, scan_order="lists")
    unproven = gi.last_unproven()
    gi.close()
    differ = sum(not (np.array_equal(ids[i], want[0][i]) and
                      np.array_equal(dis[i].view(np.uint32), want[1][i].view(np.uint32))) for i in range(len(q)))
    assert differ <= unproven, f"{differ} rows differ, {unproven} not proven"
    return unproven


@pytest.mark.parametrize("m", [4, 8, 16])
@pytest.mark.parametrize("nq,w,k", [(60, 1, 10), (17, 12, 1), (70, 5, 100), (9, 12, 1000)])
def test_first_pass_ends_inside_a_list(m, nq, w, k):
    ix, rng = _index(CUT, m, seed=m + nq)
    q = (ix.coa[np.arange(nq) % ix.coarsek] + rng.normal(0.0, 15.0, (nq, 128))).astype(np.float32)
    assert _lists_against_oracle(ix, q, k, w) <= 1 + nq // 20


def test_uneven_on_long_lists():
    from mestrado_gb300.engine import GpuIndex

    ix, rng = _index(CUT, 8, seed=1)
    nq = 50
    q = (ix.coa[np.arange(nq) % ix.coarsek] + rng.normal(0.0, 15.0, (nq, 128))).astype(np.float32)
    wq = rng.integers(1, ix.coarsek + 1, nq).astype(np.int32)
    kq = rng.choice([1, 10, 100, 1000], nq).astype(np.int32)
    gi = GpuIndex(ix)
    _same(gi.search_batched(q, wq, kq, scan_order="lists")[:2], oracle.search_batched(ix, q, wq, kq)[:2])
    gi.close()


@pytest.mark.parametrize("nq,w", [(40, 300), (600, 3)])
def test_pieces_of_8192_rows(nq, w):
    ix, rng = _index(PIECES, 8, seed=2)
    q = (ix.coa[np.arange(nq) % 4] + rng.normal(0.0, 15.0, (nq, 128))).astype(np.float32)
    _lists_against_oracle(ix, q, 10, w)


@pytest.mark.parametrize("n,nq", [(4095, 3), (10_000, 33), (33_000, 300)])
def test_flat(n, nq):
    ix, rng = _index([n], 8, seed=n)
    _lists_against_oracle(ix, rng.normal(0.0, 20.0, (nq, 128)).astype(np.float32), 10, 1)


def test_flat_order_is_the_engine_s_choice():
    """A flat index that 160 queries share goes list by list by itself, 4 queries go query by query."""
    from mestrado_gb300 import _lib
    from mestrado_gb300.engine import GpuPQ

    ix, rng = _index([300_000], 8, seed=4)
    gi = GpuPQ(ix.pq, ix.codes)
    flat = IVFPQData(coa=ix.coa, pq=ix.pq, list_off=ix.list_off, ids=np.arange(ix.n, dtype=np.int32), codes=ix.codes)
    for nq, order in ((160, 1), (4, 0)):
        q = rng.normal(0.0, 20.0, (nq, 128)).astype(np.float32)
        ids, dis = np.empty((nq, 20), np.int32), np.empty((nq, 20), np.float32)
        _lib.check(gi.lib.gbivf_ivfpq_search(gi.h, q.ctypes.data_as(C.c_void_p), nq, 20, 20, 1, _lib.GBIVF_PROFILE,
                                             ids.ctypes.data_as(C.c_void_p), dis.ctypes.data_as(C.c_void_p)))
        assert gi.last_scan_parts()[1]["list_scan"] == order
        _same((ids, dis), oracle.ivfpq_search(flat, q, k=20, kl=20, w=1, rerank=False, ties=oracle.TIES_KEYED))
    gi.close()


@pytest.mark.parametrize("lens", [CUT, [700] * 12])
def test_unproven_queries_are_scanned_again(lens):
    """Three distinct rows: the selection is full of equal distances, so the bound proves no query."""
    ix, rng = _index(lens, 8, seed=6, distinct=3)
    q = (ix.coa[np.arange(40) % ix.coarsek] + rng.normal(0.0, 15.0, (40, 128))).astype(np.float32)
    assert _lists_against_oracle(ix, q, 10, 12) > 20


@pytest.mark.parametrize("m", [4, 8, 16])
def test_ranges_of_a_small_batch(m):
    """Three queries over long lists are scanned in ranges: one kernel more than a large batch takes."""
    import torch

    from mestrado_gb300.engine import GpuIndex

    ix, rng = _index(CUT, m, seed=20 + m)
    gi = GpuIndex(ix)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    s = torch.cuda.Stream()
    for mixed in (False, True):
        kernels = {}
        for nq in (3, 8 * sms):
            q = (ix.coa[np.arange(nq) % ix.coarsek] + rng.normal(0.0, 15.0, (nq, 128))).astype(np.float32)
            d_q = torch.from_numpy(q).cuda()
            d_ids = torch.empty((nq, 100), dtype=torch.int32, device="cuda")
            d_dis = torch.empty((nq, 100), dtype=torch.float32, device="cuda")
            g = gi.capture_graph(d_q.data_ptr(), nq, 100, 12, d_ids.data_ptr(), d_dis.data_ptr(), mixed_scan=mixed,
                                 stream_ptr=s.cuda_stream, scan_order="queries")
            kernels[nq] = g.kernel_count()
            g.launch(s.cuda_stream)
            s.synchronize()
            want = oracle.ivfpq_search(ix, q[:3], k=100, kl=100, w=12, rerank=False, ties=oracle.TIES_KEYED)
            _same((d_ids[:3].cpu().numpy(), d_dis[:3].cpu().numpy()), want)
            g.close()
        assert kernels[3] == kernels[8 * sms] + 1, kernels
    for w, k in ((1, 1), (1, 1000), (5, 37), (12, 1000)):
        q = (ix.coa[np.arange(3)] + rng.normal(0.0, 15.0, (3, 128))).astype(np.float32)
        want = oracle.ivfpq_search(ix, q, k=k, kl=k, w=w, rerank=False, ties=oracle.TIES_KEYED)
        _same(gi.search(q, k, w, scan_order="queries"), want)
    gi.close()
