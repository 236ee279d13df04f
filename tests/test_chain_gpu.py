"""Solves with few right-hand sides, whose chain of 64-row blocks runs inside
clusters of eight CTAs.

Orders whose RFP halves lie at the edges of blocks (64) and clusters (512),
right-hand sides at the edges of the chunks (8, 16, 32 columns) and of the
chunk rule, every storage variant and both element types.  The backward error
|A x - b| / (|A|_F |x| + |b|) per column is a sum of at most n rounded terms per
element in each of the two triangular solves, random in sign: below
4 sqrt(n) u (u the unit roundoff).
"""
import pytest
import torch

from conftest import VARIANTS

UNIT = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}


def check(curfp, n, nrhs, dtype, tr, ul):
    f = dtype == torch.float32
    pack = curfp.strttf if f else curfp.dstrttf
    solve = curfp.spftrs if f else curfp.dpftrs
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    g = torch.Generator(device="cuda").manual_seed(n + 1000 * nrhs + 7 * tr + 13 * ul)
    k = max(32, n // 32 + 1)
    A = torch.randn(n, k, device="cuda", dtype=torch.float64, generator=g) / k ** 0.5
    K = A @ A.t()
    K.diagonal().add_(1.0)
    L = torch.linalg.cholesky(K).to(dtype)  # the factor as stored: K is L L^T
    K = L.double() @ L.double().t()
    F = pack((L.t() if ul == 1 else L).contiguous(), **lay)
    B = torch.randn(n, nrhs, device="cuda", dtype=dtype, generator=g)
    X = B.clone()
    solve(F, X, **lay)
    Xd, Bd = X.double(), B.double()
    R = (K @ Xd - Bd).norm(dim=0) / (torch.linalg.norm(K) * Xd.norm(dim=0) + Bd.norm(dim=0))
    assert R.max().item() <= 4 * n ** 0.5 * UNIT[dtype]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 255, 257, 1022, 1023, 1025, 1153, 2500])
@pytest.mark.parametrize("nrhs", [1, 2, 8, 9, 65])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_few_columns(curfp, n, nrhs, dtype, tr, ul):
    check(curfp, n, nrhs, dtype, tr, ul)


@pytest.mark.gpu
@pytest.mark.parametrize("n,nrhs", [(4096, 33), (4096, 257), (9001, 16), (9001, 50), (9001, 150),
                                    (1500, 512), (1500, 513)])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_chunk_rule(curfp, n, nrhs, tr, ul):
    check(curfp, n, nrhs, torch.float32, tr, ul)


@pytest.mark.gpu
@pytest.mark.parametrize("n,nrhs", [(4096, 10), (2000, 128), (2000, 129)])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_chunk_rule_fp64(curfp, n, nrhs, tr, ul):
    check(curfp, n, nrhs, torch.float64, tr, ul)
