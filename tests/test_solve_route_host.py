"""The rules that choose a solve's kernel (curfp_b200/csrc/solve_route.h), host
code: what they give on both sides of each line, and that every order and
number of right-hand sides has a kernel whose limits it keeps."""
import ctypes

import pytest

CHAIN1, CHAIN8, CHAIN16, CHAIN32, WAVE64, TILES = range(6)


def route(hs, n, m, fp32=1, math=1):
    out = (ctypes.c_int * 3)()
    assert hs.hs_solve_route(fp32, n, m, math, out) == 0
    return list(out)


@pytest.mark.parametrize("n,m,math,one", [(8192, 512, 1, 1), (8193, 512, 1, 0), (8193, 128, 1, 1),
                                          (9215, 256, 1, 1), (9216, 256, 1, 0), (18431, 128, 1, 1),
                                          (18432, 128, 1, 0), (65536, 127, 1, 1),
                                          (65536, 128, 1, 0), (65536, 512, 0, 1), (100, 513, 0, 0),
                                          (100, 513, 1, 0), (1, 512, 1, 1)])
def test_one_launch_or_recursion(hostsim, n, m, math, one):
    assert route(hostsim, n, m, math=math)[0] == one


def test_leaves(hostsim):
    assert route(hostsim, 9000, 512)[1] == 2048 and route(hostsim, 9000, 513)[1] == 512


@pytest.mark.parametrize("n,m,kernel", [(64, 1, CHAIN1), (64, 2, CHAIN8), (512, 255, CHAIN8),
                                        (512, 256, CHAIN32), (513, 256, CHAIN16),
                                        (512, 480, CHAIN32), (512, 481, WAVE64), (2048, 64, CHAIN8),
                                        (2048, 65, CHAIN16), (2048, 257, CHAIN32),
                                        (4096, 480, CHAIN32), (4096, 481, WAVE64),
                                        (8192, 287, CHAIN32), (8192, 288, WAVE64),
                                        (16384, 256, CHAIN32), (16384, 257, WAVE64),
                                        (512, 4095, WAVE64), (512, 4096, TILES)])
def test_fp32_kernels(hostsim, n, m, kernel):
    assert route(hostsim, n, m)[2] == kernel


@pytest.mark.parametrize("n,m,kernel", [(64, 1, CHAIN8), (8192, 120, CHAIN8), (8192, 121, WAVE64),
                                        (16384, 56, CHAIN8), (16384, 57, WAVE64), (16384, 64, WAVE64),
                                        (16384, 65, CHAIN8), (16384, 72, CHAIN8), (16384, 73, WAVE64),
                                        (64, 128, CHAIN8), (64, 129, WAVE64), (512, 4096, WAVE64)])
def test_fp64_kernels(hostsim, n, m, kernel):
    assert route(hostsim, n, m, fp32=0, math=0)[2] == kernel
