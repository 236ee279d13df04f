"""The inverse's error against 64 bits: no larger than that of the recursion
down to 64-row blocks, whose partial sums are short.  Its errors on these
matrices (A = B B^T + I, B ~ N(0, 1) / sqrt(k), k = max(32, n // 32)) are the
limits: 1.33e-7 to 1.93e-7, |X - A^-1|_F / |A^-1|_F."""
import pytest
import torch

LIMIT = {200: 1.19e-7, 700: 1.33e-7, 1500: 1.33e-7, 2000: 1.39e-7, 2500: 1.46e-7, 4096: 1.53e-7,
         6001: 1.79e-7, 8192: 1.93e-7}


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bf16x3", "fp32"])
@pytest.mark.parametrize("n", sorted(LIMIT))
def test_inverse_error(curfp, n, mode):
    g = torch.Generator(device="cuda").manual_seed(10)
    k = max(32, n // 32)
    B = torch.randn(n, k, device="cuda", generator=g) / k ** 0.5
    K = B @ B.t()
    K.diagonal().add_(1.0)
    L = torch.linalg.cholesky((K + K.t()) / 2).contiguous()
    lay = dict(transr="T", uplo="L")
    C = curfp.strttf(L, **lay)
    prev = curfp.get_math_mode()
    curfp.set_math_mode(mode)
    try:
        curfp.spftri(C, **lay)
    finally:
        curfp.set_math_mode(prev)
    want = torch.cholesky_inverse(L.double()).tril()
    err = ((curfp.stfttr(C, **lay).double() - want).norm() / want.norm()).item()
    assert err <= LIMIT[n]
