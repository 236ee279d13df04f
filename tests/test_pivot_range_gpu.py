"""Cholesky of matrices near the ends of the number range: pivots whose
reciprocal is infinite (subnormal pivots) or subnormal.

A = 2^e M with M = B B^T / 4 + I (integers / 2^12, so that A is exact down to
2^e 2^-12).  Scaling by 4^h maps every rounding of the factorization onto that
of M, as long as nothing falls below the smallest subnormal number s = 2^-149
(2^-1074); what does is an absolute error of at most s / 2 in each of the n sums
of an element, at most n s relative to |A| >= 2^e in all, beside the backward
error 4 sqrt(n) u of the tile Cholesky.  The identity scaled by an even power
of two has a diagonal factor, to 4 u (two units in the last place of the
reciprocal square root)."""
import pytest
import torch

UNIT = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}
SMALLEST = {torch.float32: -149, torch.float64: -1074}
EXPONENTS = {torch.float32: [-140, -132, -128, -127, -126, -125, -64, 0, 118, 120],
             torch.float64: [-1060, -1040, -1024, -1023, -1022, -1021, -600, 0, 1014, 1016]}


def scaled(M, e):
    """M 2^e, in steps that stay in range."""
    h = e // 2
    return M * 2.0 ** h * 2.0 ** (e - h)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 20, 33, 64, 100, 300])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("at", range(10))
def test_scaled_factor(curfp, n, dtype, at):
    f = dtype == torch.float32
    pack, unpack, chol = (curfp.strttf, curfp.stfttr, curfp.spftrf) if f else \
        (curfp.dstrttf, curfp.dstfttr, curfp.dpftrf)
    e = EXPONENTS[dtype][at]
    g = torch.Generator(device="cuda").manual_seed(n + e)
    B = torch.randint(-8, 9, (n, 16), device="cuda", generator=g).double() / 32
    M = B @ B.t() / 4 + torch.eye(n, device="cuda", dtype=torch.float64)
    lay = dict(transr="T", uplo="L")
    A = scaled(M, e).to(dtype)
    C = pack(A, **lay)
    assert chol(C, check=False, **lay) == 0
    # both sides scaled back by powers of two: exact in FP64
    L = scaled(unpack(C, **lay).double(), -(e // 2))
    want = scaled(A.double(), -2 * (e // 2))
    err = (torch.linalg.norm(L @ L.t() - want) / torch.linalg.norm(want)).item()
    u = UNIT[dtype]
    bound = 4 * n ** 0.5 * u * (2 if dtype == torch.float64 else 1)
    assert err <= bound + n * 2.0 ** (SMALLEST[dtype] - e)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,e", [(torch.float32, e) for e in (-148, -140, -130, -128, 126)] +
                         [(torch.float64, e) for e in (-1074, -1030, -1024, 1022)])
def test_scaled_identity(curfp, dtype, e):
    f = dtype == torch.float32
    pack, unpack, chol = (curfp.strttf, curfp.stfttr, curfp.spftrf) if f else \
        (curfp.dstrttf, curfp.dstfttr, curfp.dpftrf)
    n = 150
    eye = torch.eye(n, device="cuda", dtype=torch.float64)
    C = pack(scaled(eye, e).to(dtype))
    assert chol(C, check=False) == 0
    L = unpack(C).double()
    assert torch.equal(L, torch.diag(L.diagonal()))
    assert (L.diagonal() * 2.0 ** -(e // 2) - 1.0).abs().max().item() <= 4 * UNIT[dtype]
