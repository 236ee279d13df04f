"""ssfmv in FP32: strips along each RFP block's contiguous index.

Orders at the edges of groups (64), steps (128) and strips (128 to 1024), both
blocks of every storage variant, increments, alpha and beta, against the FP64
product: an element is a sum of n rounded products in short chains, so the
relative error stays below sqrt(n) u (u = 2^-24); the same call twice gives the
same bits.  An infinite x_j makes exactly the y_i infinite or NaN that the
dense product has, wherever the element (i, j) is stored.
"""
import pytest
import torch

from conftest import VARIANTS


def case(curfp, n, tr, ul, seed):
    lay = dict(transr="NT"[tr], uplo="LU"[ul])
    g = torch.Generator(device="cuda").manual_seed(seed)
    K = torch.randn(n, n, device="cuda", generator=g)
    K = K + K.t()
    return curfp.strttf(K, **lay), K.double(), torch.randn(n, device="cuda", generator=g), lay


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 129, 255, 257, 1000, 2049, 6001, 15000])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_product(curfp, n, tr, ul):
    A, K, x, lay = case(curfp, n, tr, ul, n + 3 * tr + 5 * ul)
    y0 = x.flip(0).contiguous()
    y = curfp.ssfmv(A, x, y0.clone(), alpha=-0.5, beta=2.0, **lay)
    want = -0.5 * (K @ x.double()) + 2.0 * y0.double()
    scale = 0.5 * (K.abs() @ x.double().abs()) + 2.0 * y0.double().abs()
    assert ((y.double() - want).norm() / scale.norm()).item() <= n ** 0.5 * 2.0 ** -24
    assert torch.equal(y, curfp.ssfmv(A, x, y0.clone(), alpha=-0.5, beta=2.0, **lay))


@pytest.mark.gpu
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_infinite_entry(curfp, tr, ul):
    n = 300
    A, K, x, lay = case(curfp, n, tr, ul, 9)
    for j in (0, 63, 149, 150, 299):
        z = x.clone()
        z[j] = float("inf")
        y = curfp.ssfmv(A, z, **lay)
        assert torch.equal(y, K[:, j].sign().float() * float("inf"))
