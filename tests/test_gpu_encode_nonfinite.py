"""Encoding with components that are infinite or not a number: the first centroid of the smallest distance below
infinity, in the defining arithmetic; without one the first centroid."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_train_encode import _p

pytestmark = pytest.mark.gpu


def _nearest(v, c):
    f = np.float32
    with np.errstate(all="ignore"):
        dot, n = np.zeros((len(v), len(c)), f), np.zeros(len(c), f)
        for l in range(v.shape[1]):
            dot = (dot + (v[:, l, None] * c[None, :, l]).astype(f)).astype(f)
            n = (n + (c[:, l] * c[:, l]).astype(f)).astype(f)
        d = (n[None, :] - (f(2.0) * dot).astype(f)).astype(f)
    return np.where(np.isnan(d), f(np.inf), d).argmin(1)


@pytest.mark.parametrize("ds,m", [(8, 16), (16, 8), (32, 4)])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3e38, 1e19])
def test_nonfinite(ds, m, value):
    import torch

    from mestrado_gb300._lib import check, load

    lib, d, n = load(), ds * m, 700
    rng = np.random.default_rng(ds)
    x = rng.normal(0, 20, (n, d)).astype(np.float32)
    pq = rng.normal(0, 20, (m, 256, ds)).astype(np.float32)
    x[::5, 3] = value
    x[1::7, d - 1] = -value
    pq[0, 17, 2] = pq[m - 1, 200, ds - 1] = pq[m // 2, 0, 0] = value
    pq[1, 31, 1] = -value
    dx, dpq = torch.from_numpy(x).cuda(), torch.from_numpy(pq).cuda()
    codes = torch.full((n, m), 255, dtype=torch.uint8, device="cuda")
    none = C.c_void_p(0)
    check(lib.gbivf_pq_encode(_p(dx), n, d, none, none, m, _p(dpq), _p(codes), none))
    want = np.stack([_nearest(x[:, s * ds:(s + 1) * ds], pq[s]) for s in range(m)], 1)
    np.testing.assert_array_equal(codes.cpu().numpy(), want)
