"""Calls on a device whose memory is taken: the kernels that need tens of
megabytes of scratch give way to those that need little.  The handle has made a
smaller call before, so that it holds the scratch that every call needs; then
all but 24 MiB of the device is allocated (and given back afterwards).  The
results keep the bounds of the kernels' own tests."""
import ctypes
import gc

import pytest
import torch

LAY = dict(transr="T", uplo="L")
LEAVE = 24 << 20


class Filled:
    """Takes the device's free memory but LEAVE bytes."""

    def __enter__(self):
        self.rt = ctypes.CDLL("libcudart.so.12")
        self.blocks = []
        torch.cuda.synchronize()
        gc.collect()
        torch.cuda.empty_cache()
        size = torch.cuda.mem_get_info()[0]
        while size >= 1 << 20:
            free = torch.cuda.mem_get_info()[0]
            if free < LEAVE + (2 << 20):
                break
            size = min(size, free - LEAVE)
            p = ctypes.c_void_p()
            if self.rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
                self.blocks.append(p)
            else:
                self.rt.cudaGetLastError()
                size //= 2
        return self

    def __exit__(self, *exc):
        torch.cuda.synchronize()
        for p in self.blocks:
            self.rt.cudaFree(p)
        return False


def spd(n, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, 64, device="cuda", dtype=dtype, generator=g) / 8.0
    K = A @ A.t()
    K.diagonal().add_(1.0)
    return (K + K.t()) / 2


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.gpu
def test_solve_many_columns(curfp):
    n, m = 1000, 32768
    K = spd(n, torch.float32)
    F = curfp.strttf(K, **LAY)
    assert curfp.spftrf(F, **LAY) == 0
    B = torch.randn(m, n, device="cuda")  # column-major n x m
    X = B.clone()
    with curfp.Handle() as h:
        h.set_math_mode("fp32")
        assert h._lib.curfpSpftrs(h.ptr, 1, 0, n, 600, ptr(F), ptr(X), n) == 0
        X.copy_(B)
        with Filled():
            st = h._lib.curfpSpftrs(h.ptr, 1, 0, n, m, ptr(F), ptr(X), n)
    assert st == 0
    R = (X.double() @ K.double() - B.double()).norm(dim=1)
    scale = torch.linalg.norm(K.double()) * X.double().norm(dim=1) + B.double().norm(dim=1)
    assert (R / scale).max().item() <= 2e-6


@pytest.mark.gpu
def test_factor_fp64(curfp):
    n = 4096  # one launch takes 68 MB of tiles
    K = spd(n, torch.float64)
    F = curfp.dstrttf(K, **LAY)
    C = F.clone()
    x = torch.randn(n, device="cuda", dtype=torch.float64)
    info, count = ctypes.c_int(0), [ctypes.c_longlong(0), ctypes.c_longlong(0)]
    with curfp.Handle() as h:
        lib = h._lib

        def launches(i):
            assert lib.curfpGetKernelLaunchCount(h.ptr, ctypes.byref(count[i])) == 0

        assert lib.curfpDpftrf(h.ptr, 1, 0, n, ptr(F), ctypes.byref(info)) == 0  # loads kernels
        assert lib.curfpReleaseWorkspace(h.ptr) == 0
        assert lib.curfpDpftrs(h.ptr, 1, 0, n, 1, ptr(F), ptr(x), n) == 0
        F.copy_(C)
        with Filled():
            launches(0)
            st = lib.curfpDpftrf(h.ptr, 1, 0, n, ptr(F), ctypes.byref(info))
            launches(1)
    assert st == 0 and info.value == 0
    assert count[1].value - count[0].value > 4  # not the one launch
    L = curfp.dstfttr(F, **LAY)
    err = torch.linalg.norm(L @ L.t() - K) / torch.linalg.norm(K)
    assert err.item() <= 8 * n ** 0.5 * 2.0 ** -53
