"""The list scan's error bound on values at the ends of the float range. Its screen proves a query or leaves it to
the per-query scan, so the exact form in list order must give that scan's results whatever the values are, and the
precision form may differ on the queries that it does not report as proven only. No tolerance."""
import numpy as np
import pytest

from mestrado_gb300.ivfdata import IVFPQData

pytestmark = pytest.mark.gpu


def _index(scale, seed, C=24, m=8, length=200):
    rng = np.random.default_rng(seed)
    n = C * length
    coa = (rng.uniform(0.0, 40.0, (C, 128)) * scale).astype(np.float32)
    pq = (rng.normal(0.0, 15.0, (m, 256, 128 // m)) * scale).astype(np.float32)
    ix = IVFPQData(coa=coa, pq=pq, list_off=np.arange(C + 1, dtype=np.int64) * length,
                   ids=rng.permutation(n).astype(np.int32), codes=rng.integers(0, 256, (n, m), dtype=np.uint8))
    return ix, rng


def _check(ix, q, k, w):
    """Both forms in list order against the exact per-query scan; the precision form's unproven queries."""
    from mestrado_gb300.engine import GpuIndex

    gi = GpuIndex(ix)
    want = gi.search(q, k, w, scan_order="queries")
    got = gi.search(q, k, w, scan_order="lists")
    mixed = gi.search(q, k, w, mixed_scan=True, scan_order="lists")
    unproven = gi.last_unproven()
    gi.close()
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    differ = sum(not (np.array_equal(mixed[0][i], want[0][i]) and
                      np.array_equal(mixed[1][i].view(np.uint32), want[1][i].view(np.uint32))) for i in range(len(q)))
    assert differ <= unproven, f"{differ} rows differ, {unproven} not proven"
    return want, unproven


@pytest.mark.parametrize("k,w", [(1, 3), (10, 24), (100, 20)])
def test_infinite_query_component(k, w):
    """x_0 infinite: rows whose centroid is negative there are infinitely far, the others' distances are not
    numbers. The first lists, which the first pass takes, hold rows of the second kind only."""
    ix, rng = _index(1.0, 5)
    ix.coa[:, 0] = -1.0  # every list infinitely far: probed in list order
    ix.pq[0, :128, 0], ix.pq[0, 128:, 0] = 3.0, -3.0
    near = np.searchsorted(ix.list_off, np.arange(ix.n), side="right") - 1 < 2
    ix.codes[near, 0] &= 127
    q = rng.uniform(0.0, 40.0, (40, 128)).astype(np.float32)
    q[::2, 0] = np.inf
    want, _ = _check(ix, q, k, w)
    assert (want[0][::2] >= 0).any()


@pytest.mark.parametrize("values", [(np.nan,), (np.inf, -np.inf), (1e19,), (3e38, -3e38), (np.nan, np.inf)])
def test_other_extreme_queries(values):
    ix, rng = _index(1.0, 6)
    q = rng.uniform(0.0, 40.0, (60, 128)).astype(np.float32)
    for i in range(0, len(q), 3):
        for j, v in enumerate(values):
            q[i, (7 * i + 40 * j) % 128] = v
    _check(ix, q, 10, 12)


@pytest.mark.parametrize("value", [np.inf, 1e19, 3e38])
def test_extreme_codebook(value):
    ix, rng = _index(1.0, 7)
    ix.pq[3, 5, 2] = value
    ix.pq[6, 9, 11] = -value
    q = rng.uniform(0.0, 40.0, (40, 128)).astype(np.float32)
    _check(ix, q, 10, 12)


def test_overflowed_infinite_queries_are_listed_once(monkeypatch):
    """An emission buffer of 16 keys: queries that overflow it and have infinite residuals too."""
    monkeypatch.setenv("GBIVF_LIST_SCAN_CAP", "16")
    ix, rng = _index(1.0, 5)
    ix.coa[:, 0] = -1.0
    ix.coa[0, 1] = np.inf  # one list infinitely far from every query
    q = rng.uniform(0.0, 40.0, (90, 128)).astype(np.float32)
    q[::3, 0] = np.inf
    _check(ix, q, 10, 24)


@pytest.mark.parametrize("exponent", [-14, -30, 20])
def test_scaled_data_is_proven(exponent):
    """A power of two times data of which every query is proven: the bound scales with the data."""
    ix, rng = _index(2.0 ** exponent, 8)
    q = (rng.uniform(0.0, 40.0, (200, 128)) * 2.0 ** exponent).astype(np.float32)
    _, unproven = _check(ix, q, 10, 12)
    assert unproven <= 0.01 * len(q), f"{unproven} of {len(q)} not proven"


@pytest.mark.parametrize("exponent", [-50, -66, -72, -80, -100])
def test_vanishing_data(exponent):
    """Products that underflow in the screen or in the reference's arithmetic."""
    ix, rng = _index(2.0 ** exponent, 9)
    q = (rng.uniform(0.0, 40.0, (60, 128)) * 2.0 ** exponent).astype(np.float32)
    q[::4] *= np.float32(2.0 ** -20)
    q[1::4] *= np.float32(2.0 ** 40)
    _check(ix, q, 10, 12)
