"""The waits of the kernels that hand tiles on through flags, made to run out:
the self-test launches each kernel without the CTAs that hold its first
ticket, so the others wait on a flag that nothing sets.  Each has to give up
after its limit (~2 s of globaltimer), report error code 5 and end, and the
same handle then computes correctly with the same kernels: a solve with one
right-hand side (its chain goes on with what it has after a wait that ran out,
and its CTAs stay until what their peers sent them has arrived)."""
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
    K = matrix(2000)
    C = curfp.strttf(K, transr="T", uplo="L")
    curfp.spftrf(C, transr="T", uplo="L")
    t0 = time.monotonic()
    assert P.diag_wait_timeout() == (4, 5)
    assert time.monotonic() - t0 < 60.0
    B = torch.randn(2000, 1, device="cuda")
    X = B.clone()
    curfp.spftrs(C, X, transr="T", uplo="L")
    # the bound of the solves: at most n rounded terms an element, random in
    # sign, in each of two triangular solves: below 4 sqrt(n) u
    assert backward_error(K, X, B) <= 4 * 2000 ** 0.5 * 2.0 ** -24
