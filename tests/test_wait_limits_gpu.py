"""The waits of the kernels that hand tiles on through flags, made to run out:
the self-test launches each kernel without the CTAs that hold its first
ticket, so the others wait on a flag that nothing sets.  Each has to give up
after its limit (~2 s of globaltimer), report error code 5 and end, and the
same handle then computes correctly with the same kernels: solves with one
right-hand side (its chain goes on with what it has after a wait that ran out,
and its CTAs stay until what their peers sent them has arrived), with a few,
with hundreds and with thousands, an inverse and a factorization."""
import time

import pytest
import torch


def matrix(n, k=64, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.randn(n, k, device="cuda", generator=g) / k ** 0.5
    K = A @ A.t()
    K.diagonal().add_(1.0)
    return (K + K.t()) / 2


def backward_error(K, X, B):
    R = (K.double() @ X.double() - B.double()).norm(dim=0)
    return (R / (torch.linalg.norm(K.double()) * X.double().norm(dim=0) + B.double().norm(dim=0))).max().item()


@pytest.mark.gpu
def test_every_wait_gives_up_and_the_handle_survives(curfp):
    from curfp_b200 import precision as P
    n, lay = 2000, dict(transr="T", uplo="L")
    K = matrix(n)
    t0 = time.monotonic()
    assert P.diag_wait_timeout() == (4, 5)
    assert time.monotonic() - t0 < 60.0
    C = curfp.strttf(K, **lay)
    assert curfp.spftrf(C, **lay) == 0
    # the bound of the solves: at most n rounded terms an element, random in
    # sign, in the factor and in each of two triangular solves
    bound = 6 * n ** 0.5 * 2.0 ** -24
    for m in (1, 9, 600, 4096):
        B = torch.randn(n, m, device="cuda")
        X = B.clone()
        curfp.spftrs(C, X, **lay)
        assert backward_error(K, X, B) <= bound
    curfp.spftri(C, **lay)
    Z = curfp.stfttr(C, **lay)
    Z = Z + Z.tril(-1).t()
    B = torch.randn(n, 3, device="cuda")
    assert backward_error(K, Z.double() @ B.double(), B) <= 46 * bound  # 46: the condition number
