"""Solves with so many right-hand sides that the leaves run as tiles made for
throughput: below, at and past the switch, ragged in rows and columns, from
one row on, and inside the Cholesky factorization (its panels below a large
diagonal block).  Backward errors against FP64, bound 2e-6 as for the other
solves."""
import pytest
import torch

from conftest import VARIANTS


def sym(curfp, C, lay):
    M = curfp.stfttr(C, **lay).double()
    return M + (M.triu(1).T if lay["uplo"] == "U" else M.tril(-1).T)


def matrix(curfp, n, k, lay):
    A = torch.randn(n, k, device="cuda") / k ** 0.5
    C = torch.empty(n * (n + 1) // 2, device="cuda")
    curfp.ssfrk(A, C, **lay)
    curfp.add_to_diagonal(C, 1.0, **lay)
    return C


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 63, 129, 500, 1025, 1400])
@pytest.mark.parametrize("m", [4095, 4096, 4133])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_solve_many(curfp, n, m, tr, ul):
    torch.manual_seed(n + m)
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    C = matrix(curfp, n, 64, lay)
    S = sym(curfp, C, lay)
    curfp.spftrf(C, **lay)
    B = torch.randn(n, m, device="cuda")
    X = B.clone()
    curfp.spftrs(C, X, **lay)
    R = B.double() - S @ X.double()
    scale = torch.linalg.norm(S) * X.double().norm(dim=0) + B.double().norm(dim=0)
    assert (R.norm(dim=0) / scale).max().item() <= 2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bf16x3", "fp32"])
@pytest.mark.parametrize("n", [8300, 8257])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_factor(curfp, mode, n, tr, ul):
    torch.manual_seed(n)
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    C = matrix(curfp, n, 256, lay)
    S = sym(curfp, C, lay)
    prev = curfp.get_math_mode()
    curfp.set_math_mode(mode)
    try:
        curfp.spftrf(C, **lay)
    finally:
        curfp.set_math_mode(prev)
    T = curfp.stfttr(C, **lay).double()
    L = T.T if ul == 1 else T
    assert (torch.linalg.norm(S - L @ L.T) / torch.linalg.norm(S)).item() <= 2e-6
