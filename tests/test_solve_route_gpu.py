"""Solves with hundreds of right-hand sides at orders where the route changes:
the recursion with tensor-core updates above 8192 rows, one launch below, in
both math modes.  The backward error |A x - b| / (|A|_F |x| + |b|) per column
against FP64, bound 2e-6 as for the other solves."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bf16x3", "fp32"])
@pytest.mark.parametrize("n,m", [(16390, 512), (18500, 256), (18500, 255), (9000, 481), (500, 300)])
@pytest.mark.parametrize("tr,ul", [(0, 0), (1, 1)])
def test_backward_error(curfp, n, m, mode, tr, ul):
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    g = torch.Generator(device="cuda").manual_seed(n + m)
    k = max(32, n // 32)
    A = torch.randn(n, k, device="cuda", generator=g) / k ** 0.5
    C = torch.empty(n * (n + 1) // 2, device="cuda")
    curfp.ssfrk(A, C, **lay)
    curfp.add_to_diagonal(C, 1.0, **lay)
    F = C.clone()
    curfp.spftrf(F, **lay)
    B = torch.randn(n, m, device="cuda", generator=g)
    X = B.clone()
    prev = curfp.get_math_mode()
    curfp.set_math_mode(mode)
    try:
        curfp.spftrs(F, X, **lay)
    finally:
        curfp.set_math_mode(prev)
    Ad, Xd, Bd = A.double(), X.double(), B.double()
    R = Ad @ (Ad.t() @ Xd) + Xd - Bd  # A itself is C to 1e-7
    scale = (Ad.t() @ Ad).norm() * Xd.norm(dim=0) + Bd.norm(dim=0)
    assert (R.norm(dim=0) / scale).max().item() <= 2e-6
