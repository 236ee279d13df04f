"""An infinite last pivot: positive, so the factorization does not fail (info
0), whatever padding the last tile has; a negative infinite one fails at its
own column.  An infinite pivot further up leaves NaN below it: the failing
column lies inside the matrix."""
import pytest
import torch

from conftest import VARIANTS


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 63, 64, 65, 100, 127, 130, 257])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_info(curfp, n, dtype, tr, ul):
    pack, chol = (curfp.strttf, curfp.spftrf) if dtype == torch.float32 else \
        (curfp.dstrttf, curfp.dpftrf)
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    M = torch.full((n, n), 0.25, device="cuda", dtype=dtype) / n
    M.diagonal().add_(1.0)
    M[-1, -1] = float("inf")
    assert chol(pack(M, **lay), check=False, **lay) == 0
    M[-1, -1] = float("-inf")
    assert chol(pack(M, **lay), check=False, **lay) == n
    M[-1, -1] = 1.0
    for j in range(0, n - 1, 29):
        K = M.clone()
        K[j, j] = float("inf")
        assert j + 1 < chol(pack(K, **lay), check=False, **lay) <= n
    assert chol(pack(M, **lay), check=False, **lay) == 0
