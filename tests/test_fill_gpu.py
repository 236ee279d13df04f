"""stfttr into a full square: the stored triangle copied bit for bit and exact
zeros elsewhere, whatever the memory held before, at the edges of the 64 x 64
tiles, for every storage variant and both element types; nothing outside the
square is written and the triangle-only entry leaves the rest alone."""
import ctypes

import pytest
import torch

from conftest import VARIANTS


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 130, 257, 1000])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_fill(curfp, n, dtype, tr, ul):
    f = dtype == torch.float32
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    M = torch.randn(n, n, device="cuda", dtype=dtype)
    A = (curfp.strttf if f else curfp.dstrttf)(M, **lay)
    want = M.triu() if ul == 1 else M.tril()
    lda = n + 3
    buf = torch.full((n, lda), float("nan"), device="cuda", dtype=dtype)
    h = curfp._get_handle()
    fn = h._lib.curfpSstfttrFill if f else h._lib.curfpDstfttrFill
    assert fn(h.ptr, tr, ul, n, ctypes.c_void_p(A.data_ptr()), ctypes.c_void_p(buf.data_ptr()),
              lda) == 0
    torch.cuda.synchronize()
    assert torch.equal(buf[:, :n], want)
    assert bool(buf[:, n:].isnan().all())
    assert torch.equal((curfp.stfttr if f else curfp.dstfttr)(A, **lay), want)
    part = torch.full((n, n), float("nan"), device="cuda", dtype=dtype)
    (curfp.stfttr_raw if f else curfp.dstfttr_raw)(h, tr, ul, n, A, part, n)
    torch.cuda.synchronize()
    stored = torch.ones_like(part, dtype=torch.bool).triu() if ul == 1 else \
        torch.ones_like(part, dtype=torch.bool).tril()
    assert torch.equal(part[stored], want[stored]) and bool(part[~stored].isnan().all())
    assert fn(None, tr, ul, n, None, None, lda) == 1 and fn(h.ptr, tr, ul, n, None, None, n - 1) == 3
