"""Training and encoding kernels at the edges of their blocks: row counts around a block's 512 rows (and one
row), every sub-vector length, rows that are not on 16-byte boundaries, duplicate centroids (ties keep the first),
clusters that stay empty. Codes must be numpy's in the same arithmetic exactly; one k-means iteration's centroids
are the FP64 means of that assignment rounded to FP32, within one FP32 rounding (FP64 sums in another order)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _nearest(v, c):
    """First nearest of c for each row of v: ||c||^2 - 2 <v, c>, every FP32 operation rounded, in order."""
    f = np.float32
    dot, n = np.zeros((len(v), len(c)), f), np.zeros(len(c), f)
    for l in range(v.shape[1]):
        dot = (dot + (v[:, l, None] * c[None, :, l]).astype(f)).astype(f)
        n = (n + (c[:, l] * c[:, l]).astype(f)).astype(f)
    return (n[None, :] - (f(2.0) * dot).astype(f)).astype(f).argmin(1)


@pytest.mark.parametrize("n", [1, 511, 512, 1025, 3000])
@pytest.mark.parametrize("ds,m,shift", [(8, 16, 0), (16, 8, 0), (32, 4, 1), (8, 3, 2)])
def test_encode(n, ds, m, shift):
    import torch

    from mestrado_gb300._lib import check, load

    lib, d = load(), ds * m
    rng = np.random.default_rng(n + ds)
    x = rng.normal(0, 20, (n, d)).astype(np.float32)
    pq = rng.normal(0, 20, (m, 256, ds)).astype(np.float32)
    pq[:, 7] = pq[:, 200]
    pq[:, 100:110] = pq[:, 90:100]
    coa = rng.normal(0, 30, (5, d)).astype(np.float32)
    a = rng.integers(0, 5, n).astype(np.int32)
    buf = torch.zeros(n * d + 4, device="cuda")  # rows `shift` floats past a 16-byte boundary
    buf[shift:shift + n * d] = torch.from_numpy(x.reshape(-1)).cuda()
    dpq, dcoa, da = torch.from_numpy(pq).cuda(), torch.from_numpy(coa).cuda(), torch.from_numpy(a).cuda()
    for coarse in (True, False):
        codes = torch.full((n, m), 255, dtype=torch.uint8, device="cuda")
        check(lib.gbivf_pq_encode(_p(buf[shift:]), n, d, _p(da) if coarse else C.c_void_p(0),
                                  _p(dcoa) if coarse else C.c_void_p(0), m, _p(dpq), _p(codes), C.c_void_p(0)))
        r = (x - coa[a]).astype(np.float32) if coarse else x
        want = np.stack([_nearest(r[:, s * ds:(s + 1) * ds], pq[s]) for s in range(m)], 1)
        np.testing.assert_array_equal(codes.cpu().numpy(), want)


def _means(x, assign, k, old):
    want = old.astype(np.float64)
    for c in range(k):
        if (assign == c).any():
            want[c] = x[assign == c].astype(np.float64).sum(0) / (assign == c).sum()
    return want


@pytest.mark.parametrize("n", [256, 511, 1025, 5000])
@pytest.mark.parametrize("ds,m", [(8, 2), (16, 8), (32, 3)])
def test_pq_train_iteration(n, ds, m):
    import torch

    from mestrado_gb300._lib import check, load

    lib, d = load(), ds * m
    rng = np.random.default_rng(n * ds)
    x = rng.normal(0, 20, (n, d)).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    c0, c1 = (torch.empty((m, 256, ds), device="cuda") for _ in range(2))
    check(lib.gbivf_pq_train(_p(dx), n, d, m, 0, 9, _p(c0), C.c_void_p(0)))
    check(lib.gbivf_pq_train(_p(dx), n, d, m, 1, 9, _p(c1), C.c_void_p(0)))
    c0, c1 = c0.cpu().numpy(), c1.cpu().numpy()
    for s in range(m):
        v = x[:, s * ds:(s + 1) * ds]
        a = _nearest(v, c0[s])
        filled = np.bincount(a, minlength=256) > 0
        np.testing.assert_allclose(c1[s][filled], _means(v, a, 256, c0[s])[filled], rtol=2.0 ** -23, atol=1e-30)
        assert all((v == row).all(1).any() for row in c1[s][~filled])  # re-seeded with points


@pytest.mark.parametrize("n,k,d", [(1, 1, 128), (63, 5, 128), (65, 64, 128), (4100, 700, 128), (4100, 5000, 16)])
def test_kmeans_iteration(n, k, d):
    import torch

    from mestrado_gb300._lib import check, load

    lib = load()
    rng = np.random.default_rng(n + k)
    x = np.rint(rng.uniform(0, 255, (n, d))).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    c0, c1 = (torch.empty((k, d), device="cuda") for _ in range(2))
    a = torch.empty(n, dtype=torch.int32, device="cuda")
    check(lib.gbivf_kmeans(_p(dx), n, d, k, 0, 9, _p(c0), C.c_void_p(0)))
    check(lib.gbivf_kmeans(_p(dx), n, d, k, 1, 9, _p(c1), C.c_void_p(0)))
    check(lib.gbivf_assign(_p(dx), n, d, _p(c0), k, _p(a), C.c_void_p(0)))
    a = a.cpu().numpy()
    filled = np.bincount(a, minlength=k) > 0
    np.testing.assert_allclose(c1.cpu().numpy()[filled], _means(x, a, k, c0.cpu().numpy())[filled], rtol=2.0 ** -23,
                               atol=1e-30)
