"""The tile Cholesky (one launch of 64 x 64 tiles that hand on through flags).

Orders at the edges of tiles (both blocks of the RFP split are cut into tiles
from their own first row), at the largest single launch and just above it,
where the recursion takes over, for every storage variant and both element
types, against the FP64 product of the factor: each stored element of L L^T
carries a sum of at most n rounded terms, whose errors add like a random
walk, so the Frobenius backward error stays below 4 sqrt(n) u of the matrix
(u the unit roundoff).  Non-positive pivots: info at the first and last
column of tiles, of 32-column halves and of blocks, and nothing after a
failure blocks the next call.
"""
import pytest
import torch

from conftest import VARIANTS

UNIT = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}


def spd(n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = max(32, n // 32)
    A = torch.randn(n, k, device="cuda", dtype=dtype, generator=g) / k ** 0.5
    M = A @ A.t()
    M.diagonal().add_(1.0)
    return (M + M.t()) / 2


def ops(curfp, dtype):
    if dtype == torch.float32:
        return curfp.strttf, curfp.stfttr, curfp.spftrf
    return curfp.dstrttf, curfp.dstfttr, curfp.dpftrf


SIZES = [1, 2, 3, 31, 33, 64, 65, 127, 128, 129, 191, 250, 257, 1000, 2047, 4095, 4096, 4097]


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_backward_error(curfp, n, dtype, tr, ul):
    pack, unpack, chol = ops(curfp, dtype)
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    M = spd(n, dtype, n + 7 * tr + 13 * ul)
    C = pack(M, **lay)
    guard = torch.full((C.numel() + 64,), -7.0, device="cuda", dtype=dtype)
    guard[32:32 + C.numel()] = C
    assert chol(guard[32:32 + C.numel()], **lay) == 0
    assert bool((guard[:32] == -7.0).all()) and bool((guard[32 + C.numel():] == -7.0).all())
    L = unpack(guard[32:32 + C.numel()].clone(), **lay).double()
    L = L if ul == 0 else L.t()
    err = torch.linalg.norm(L @ L.t() - M.double()) / torch.linalg.norm(M.double())
    bound = 4 * n ** 0.5 * UNIT[dtype]
    if dtype == torch.float64:  # the check's own product rounds in the same precision
        bound *= 2
    assert err.item() <= bound


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_info(curfp, dtype, tr, ul):
    pack, unpack, chol = ops(curfp, dtype)
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    n = 500  # blocks of 250: tiles of 64, 64, 64, 58 twice
    M = spd(n, dtype, 5)
    for col in (0, 31, 32, 63, 64, 200, 249, 250, 281, 282, 313, 499):
        for bad in (-1.0, 0.0, float("nan")):
            B = M.clone()
            B[col, col] = bad
            if bad == 0.0:  # a zero pivot
                B[col, :] = 0.0
                B[:, col] = 0.0
            assert chol(pack(B, **lay), check=False, **lay) == col + 1
    assert chol(pack(M, **lay), **lay) == 0
