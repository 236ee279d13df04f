"""ssfmv with increments, at the edges of the groups (64), steps (128) and
strips (128 to 1024) of its kernel: the result is bit for bit that of the same
vectors packed, and the elements between the increments stay as they are."""
import pytest
import torch

from conftest import VARIANTS


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 64, 65, 127, 129, 257, 1000, 2049])
@pytest.mark.parametrize("incx,incy", [(2, 1), (1, 3), (-1, 2), (3, -2), (-2, -1)])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_increments(curfp, n, incx, incy, tr, ul):
    g = torch.Generator(device="cuda").manual_seed(n + 3 * tr + 5 * ul)
    A = torch.randn(n * (n + 1) // 2, device="cuda", generator=g)
    x = torch.randn(n, device="cuda", generator=g)
    y = torch.randn(n, device="cuda", generator=g)

    def spread(v, inc):  # BLAS: a negative increment walks the vector backwards
        buf = torch.full(((n - 1) * abs(inc) + 1,), -7.0, device="cuda")
        buf[::abs(inc)] = v if inc > 0 else v.flip(0)
        return buf

    h = curfp._get_handle()
    want = y.clone()
    curfp.ssfmv_raw(h, tr, ul, n, 1.5, A, x, 1, -0.5, want, 1)
    xs, ys = spread(x, incx), spread(y, incy)
    curfp.ssfmv_raw(h, tr, ul, n, 1.5, A, xs, incx, -0.5, ys, incy)
    assert torch.equal(ys, spread(want, incy)) and torch.equal(xs, spread(x, incx))
