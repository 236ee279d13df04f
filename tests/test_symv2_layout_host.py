"""Index arithmetic of the ssfmv strips (curfp_b200/csrc/symv2_layout.h),
enumerated on the host: the CTAs visit every stored element exactly once, with
the element's row and column as the two y indices, and every partial sum has
a slot of its own inside the workspace, for every storage variant."""
import ctypes

import numpy as np
import pytest

from conftest import VARIANTS


def layout(hs, n, tr, ul):
    out = np.zeros(6, np.int64)
    assert hs.hs_symv2_layout(n, tr, 1 - ul, out.ctypes.data_as(ctypes.c_void_p)) == 0
    return out


@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 127, 128, 129, 130, 255, 256, 257, 513, 1000,
                               1025, 2300])
@pytest.mark.parametrize("tr,ul", VARIANTS)
def test_every_element_once(hostsim, n, tr, ul):
    total, visited, bad, wrong, slots, span = layout(hostsim, n, tr, ul)
    assert visited == n * (n + 1) // 2
    assert bad == wrong == slots == span == 0
    # a vector per group of 64 of the other index and block, one per strip
    h = (n + 1) // 2
    assert total <= 3 * ((h + 63) // 64) * h + 3 * ((h + 127) // 128) * h
