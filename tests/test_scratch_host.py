"""The planner when scratch runs out (CPU executor): block operations that find
none have done nothing, and the recursions go on with smaller blocks, so that
factorization, solve and inverse end with the results they have otherwise."""
import ctypes

import numpy as np
import pytest

from conftest import VARIANTS

fp = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731


@pytest.mark.parametrize("n", [1, 2, 65, 129, 200, 257, 520])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_smaller_blocks(orc, hostsim, n, tr, ul):
    rng = np.random.default_rng(n + 2 * tr + ul)
    M = rng.standard_normal((n, max(1, n // 3)))
    M = M @ M.T / max(1, n // 3) + np.eye(n)
    C = orc.strttf(tr, ul, n, M)
    B = rng.standard_normal((4, n))
    F, X = C.astype(np.float32), B.astype(np.float32)
    refused = ctypes.c_long(0)
    assert hostsim.hs_scarce(tr, 1 - ul, n, fp(F), fp(X), ctypes.byref(refused)) == 0
    assert refused.value > 0
    Fo, info = orc.spftrf(tr, ul, n, C.copy())
    assert info == 0
    Xo = orc.spftrs(tr, ul, n, 4, Fo, B.ravel(), n)
    np.testing.assert_allclose(X.ravel(), Xo, atol=5e-5 * max(1, np.abs(Xo).max()))
    Io, rc = orc.spftri(tr, ul, n, Fo)
    np.testing.assert_allclose(F, Io, atol=5e-5 * max(1, np.abs(Io).max()))
