"""A handle bound to another stream while work on its workspaces is in flight.

The workspaces are one set per handle, so what the second stream enqueues has to
start after the first stream's call: with the first stream held up (100 ms), the
second call must not have ended before the first could start.  Both results are
compared with those of a single stream, bit for bit (acc64 adds its FP64 sums
atomically: one unit in the last place).  A switch to a stream that captures
a graph stays possible, and so does one away from a stream that is destroyed."""
import ctypes

import pytest
import torch


def routines(curfp):
    """name -> (call with a factor and an output, a new output)"""
    from curfp_b200 import precision as P
    n = 3001
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn(n * (n + 1) // 2, device="cuda", generator=g)
    x = torch.randn(n, device="cuda", generator=g)
    B = torch.randn(n, 5, device="cuda", generator=g)
    Ad, xd = A.double(), x.double()
    return {
        "ssfmv": (lambda s, y: curfp.ssfmv(A, s * x, y), lambda: torch.zeros_like(x)),
        "dsfmv": (lambda s, y: curfp.dsfmv(Ad, s * xd, y), lambda: torch.zeros_like(xd)),
        "acc64": (lambda s, y: P.ssfmm_acc64(A, s * B, y), lambda: torch.zeros_like(B)),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["ssfmv", "dsfmv", "acc64"])
def test_second_stream_starts_after_the_first(curfp, name):
    f, new = routines(curfp)[name]
    want = [f(s, new()) for s in (1.0, -3.0)]
    first, second = new(), new()
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    start = torch.cuda.Event()
    try:
        curfp.set_stream(a)
        with torch.cuda.stream(a):
            torch.cuda._sleep(200_000_000)
            start.record(a)
            f(1.0, first)
        curfp.set_stream(b)
        with torch.cuda.stream(b):
            f(-3.0, second)
        b.synchronize()
        assert start.query()  # the first call was not held up any more
    finally:
        torch.cuda.synchronize()
        curfp.set_stream(None)
    for got, ref in zip((first, second), want):
        if name == "acc64":
            assert torch.allclose(got, ref, rtol=2.0 ** -22, atol=0.0)
        else:
            assert torch.equal(got, ref)


@pytest.mark.gpu
def test_capture_after_a_switch(curfp):
    f, new = routines(curfp)["ssfmv"]
    want, other, got = f(2.0, new()), new(), new()
    a = torch.cuda.Stream()
    try:
        curfp.set_stream(a)
        with torch.cuda.stream(a):
            f(1.0, other)  # leaves work on the workspace in flight
        a.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            curfp.set_stream(torch.cuda.current_stream())
            f(2.0, got)
            curfp.set_stream(a)
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    finally:
        torch.cuda.synchronize()
        curfp.set_stream(None)


@pytest.mark.gpu
def test_switch_away_from_a_destroyed_stream(curfp):
    """The old stream's handle is not used by the switch."""
    f, new = routines(curfp)["ssfmv"]
    want = f(2.0, new())
    rt = ctypes.CDLL("libcudart.so.12")
    s = ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
    h = curfp._get_handle()
    try:
        torch.cuda.synchronize()
        h.set_stream_ptr(s.value)
        with torch.cuda.stream(torch.cuda.ExternalStream(s.value)):
            f(1.0, new())
        assert rt.cudaStreamSynchronize(s) == 0 and rt.cudaStreamDestroy(s) == 0
    finally:
        curfp.set_stream(None)
    assert torch.equal(f(2.0, new()), want)
