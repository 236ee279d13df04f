"""The inverse by waves of 64 x 64 tiles and one-product triangular blocks.

Orders whose RFP halves lie at the edges of tiles (64), of the one-product
blocks (1024) and of the one-wave inverse (2048), for every storage variant
and both element types: A A^-1 against the identity in FP64.  Each element of
the residual is a sum of n products of rounded terms; with condition number
kappa <= 46 (A = B B^T + I, n / k <= 32) its root mean square stays below
4 sqrt(n) u kappa (u the unit roundoff).
"""
import pytest
import torch

from conftest import VARIANTS

UNIT = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}
KAPPA = 46.0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 63, 64, 65, 127, 129, 255, 2046, 2050, 4097])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_inverse(curfp, n, dtype, tr, ul):
    f = dtype == torch.float32
    pack, unpack = (curfp.strttf, curfp.stfttr) if f else (curfp.dstrttf, curfp.dstfttr)
    chol, inv = (curfp.spftrf, curfp.spftri) if f else (curfp.dpftrf, curfp.dpftri)
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    g = torch.Generator(device="cuda").manual_seed(n + 7 * tr + 13 * ul)
    k = max(32, n // 32 + 1)
    B = torch.randn(n, k, device="cuda", dtype=dtype, generator=g) / k ** 0.5
    A = B @ B.t()
    A.diagonal().add_(1.0)
    C = pack(A, **lay)
    chol(C, **lay)
    inv(C, **lay)
    Z = unpack(C, **lay).double()
    Z = Z + (Z.triu(1) if ul == 1 else Z.tril(-1)).t()
    R = pack(A, **lay)
    S = unpack(R, **lay).double()
    S = S + (S.triu(1) if ul == 1 else S.tril(-1)).t()
    E = S @ Z
    E.diagonal().sub_(1.0)
    rms = (torch.linalg.norm(E) / n).item() * n ** 0.5
    assert rms <= 4 * n ** 0.5 * UNIT[dtype] * KAPPA
