"""Assignment and training whose workspace cannot be allocated: an error, nothing is read or launched, and the same
calls work afterwards."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

HUGE = 1 << 30  # centroids: 550 GB of operand tiles


def test_assign_and_kmeans_without_memory():
    import torch

    from mestrado_gb300._lib import check, load

    lib = load()
    x = torch.randn((300, 128), device="cuda")
    cent = torch.randn((64, 128), device="cuda")
    out = torch.full((300,), -7, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    none = C.c_void_p(0)
    check(lib.gbivf_assign(p(x), 300, 128, p(cent), 64, p(out), none))
    want = out.clone()
    out.fill_(-7)
    assert lib.gbivf_assign(p(x), 300, 128, p(cent), HUGE, p(out), none) == 3  # GBIVF_ERR_NOMEM
    assert lib.gbivf_kmeans(p(x), 300, 128, HUGE, 1, 1, p(cent), none) == 3
    torch.cuda.synchronize()
    assert (out == -7).all()
    check(lib.gbivf_assign(p(x), 300, 128, p(cent), 64, p(out), none))
    assert (out == want).all()
