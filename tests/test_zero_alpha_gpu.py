"""Symmetric products with alpha = 0: C := beta C with neither the array nor the
other operand read (NaN in both), at the orders whose RFP blocks are empty or
one element, every storage variant, both sides and both element types; and the
rank updates with k = 0, which also have an empty contraction.  Scalings by 0
and 2 are exact."""
import pytest
import torch

from conftest import VARIANTS

DTYPES = [torch.float32, torch.float64]


def nan(*shape, dtype):
    return torch.full(shape, float("nan"), device="cuda", dtype=dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 64, 130])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_products(curfp, n, dtype, tr, ul):
    f = dtype == torch.float32
    mv, mm = (curfp.ssfmv, curfp.ssfmm) if f else (curfp.dsfmv, curfp.dsfmm)
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    A = nan(n * (n + 1) // 2, dtype=dtype)
    for beta in (0.0, 2.0):
        y0 = nan(n, dtype=dtype) if beta == 0.0 else torch.randn(n, device="cuda", dtype=dtype)
        want = torch.zeros_like(y0) if beta == 0.0 else 2.0 * y0
        assert torch.equal(mv(A, nan(n, dtype=dtype), y0.clone(), alpha=0.0, beta=beta, **lay), want)
        for cols in (1, 5, 70):
            for side in "LR":
                shape = (n, cols) if side == "L" else (cols, n)
                c0 = nan(*shape, dtype=dtype) if beta == 0.0 else \
                    torch.randn(*shape, device="cuda", dtype=dtype)
                want = torch.zeros_like(c0) if beta == 0.0 else 2.0 * c0
                got = mm(A, nan(*shape, dtype=dtype), c0.clone(), alpha=0.0, beta=beta, side=side,
                         **lay)
                assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 64, 130])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_rank_updates_without_columns(curfp, n, dtype, tr, ul):
    f = dtype == torch.float32
    rk, r2k = (curfp.ssfrk_raw, curfp.ssfr2k_raw) if f else (curfp.dsfrk_raw, curfp.dsfr2k_raw)
    h = curfp._get_handle()
    A = nan(n, dtype=dtype)
    for trans in (0, 1):
        lda = n if trans == 0 else 1
        C = torch.randn(n * (n + 1) // 2, device="cuda", dtype=dtype)
        want = 2.0 * C
        rk(h, tr, ul, trans, n, 0, 1.0, A, lda, 2.0, C)
        assert torch.equal(C, want)
        r2k(h, tr, ul, trans, n, 0, 1.0, A, lda, A, lda, 2.0, C)
        assert torch.equal(C, 2.0 * want)
