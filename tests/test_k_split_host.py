"""The split of a product's k range over CTAs (curfp_b200/csrc/gemm_route.h),
host code: every k from 0 on gives ranges that cover it, none of them empty,
in multiples of 32 columns; an empty k (a product with alpha = 0) is one
range."""
import ctypes

import pytest


def split(hs, few, size, k):
    out = (ctypes.c_int * 2)()
    assert hs.hs_k_split(few, size, k, out) == 0
    return out[0], out[1]


@pytest.mark.parametrize("few,least,sizes", [(0, 128, [1, 2, 31, 32, 147, 148, 149, 296, 297, 10000]),
                                             (1, 512, [1, 32, 1024, 37888, 37889, 1 << 20])])
def test_ranges_cover_k(hostsim, few, least, sizes):
    ks = list(range(0, 1100)) + [2047, 2048, 2049, 8192, 16383, 65537, 131072]
    for size in sizes:
        for k in ks:
            splits, kseg = split(hostsim, few, size, k)
            assert splits >= 1
            if splits == 1:
                assert kseg == k
                continue
            assert kseg % 32 == 0 and kseg >= least // 2
            assert (splits - 1) * kseg < k <= splits * kseg


def test_short_k_is_not_cut(hostsim):
    for k in (0, 1, 127, 255):
        assert split(hostsim, 0, 1, k) == (1, k)
    for k in (0, 1, 512):
        assert split(hostsim, 1, 1, k) == (1, k)
    assert split(hostsim, 0, 1, 256) == (2, 128)
    assert split(hostsim, 1, 8192, 8192) == (5, 1664)
