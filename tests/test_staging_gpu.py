"""Operand staging of the split-BF16 contractions: an operand that the 16-byte
loads read (unit stride, base and leading dimension multiples of 16 bytes)
gives bit for bit the result of the same operand shifted by one element, which
the element-wise loads read, at ragged rows and depths and with zero, tiny and
huge rows (the row scales' limits).  The digits are exact, so no tolerance."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("trans", ["T", "N"])
@pytest.mark.parametrize("n,k,beta", [(2048, 256, 0.0), (2048, 260, 0.0), (2049, 259, 0.5), (2050, 513, 0.0),
                                      (2051, 1027, 0.5), (4161, 130, 0.0)])
def test_wide_staging_same_bits(curfp, trans, n, k, beta):
    from curfp_b200 import precision as P
    g = torch.Generator(device="cuda").manual_seed(n + k)
    M = torch.randn(n, k, device="cuda", generator=g)
    M[3] = 0.0
    M[5] *= 2.0 ** -126  # subnormal and smallest normal elements
    M[7] *= 1e17
    M[n - 1, k - 1] = 3.0e18
    if trans == "N":
        M = M.T
    rows, cols = M.shape
    out = []
    P.profile_enable(True)
    for shift in (0, 1):
        lda = (cols + 3) // 4 * 4 + shift
        buf = torch.full((rows * lda + 8,), float("nan"), device="cuda")
        assert buf.data_ptr() % 16 == 0
        buf[shift:shift + rows * lda].view(rows, lda)[:, :cols] = M
        C = torch.ones(n * (n + 1) // 2, device="cuda")
        curfp.ssfrk(buf[shift:], C, beta=beta, trans=trans, n=n, k=k, lda=lda)
        torch.cuda.synchronize()
        out.append(C)
    classes = P.profile_read()
    P.profile_enable(False)
    if (n // 2) ** 2 * k >= 2.7e8:  # smaller products stay on the SIMT cores
        assert classes["tc_gemm"]["launches"] >= 2
    assert bool(out[0].isfinite().all())
    assert torch.equal(out[0], out[1])
