"""Encoding of rows so small that products of two components are subnormal: the screen's fused arithmetic and the
defining one then differ by roundings of 2^-149 each, whatever the norms are. Whole numbers times 2^-75 make those
roundings ties. Codes must be numpy's exactly."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_train_encode import _nearest, _p

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ds,m", [(8, 16), (16, 8), (32, 4)])
@pytest.mark.parametrize("most,exponent", [(5, -75), (40, -75), (5, -74), (3, -20), (100, -66)])
def test_tiny(ds, m, most, exponent):
    import torch

    from mestrado_gb300._lib import check, load

    lib, d, n = load(), ds * m, 2000
    rng = np.random.default_rng(ds + most - exponent)
    x, pq = (np.ldexp(rng.integers(-most, most + 1, s).astype(np.float32), exponent) for s in ((n, d), (m, 256, ds)))
    dx, dpq = torch.from_numpy(x).cuda(), torch.from_numpy(pq).cuda()
    codes = torch.full((n, m), 255, dtype=torch.uint8, device="cuda")
    none = C.c_void_p(0)
    check(lib.gbivf_pq_encode(_p(dx), n, d, none, none, m, _p(dpq), _p(codes), none))
    want = np.stack([_nearest(x[:, s * ds:(s + 1) * ds], pq[s]) for s in range(m)], 1)
    np.testing.assert_array_equal(codes.cpu().numpy(), want)
