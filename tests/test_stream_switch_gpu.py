"""A handle bound to another stream while work on its workspaces is in flight.

The workspaces are one set per handle, so what the second stream enqueues has to
start after the first stream's call: with the first stream held up (100 ms), the
second call's end has to come after the first call's.  Both results are compared
with those of a single stream, bit for bit.  A switch to a stream that captures
a graph stays possible, and so does one away from a stream that is destroyed."""
import ctypes

import pytest
import torch


def routines(curfp):
    from curfp_b200 import precision as P
    n = 3001
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn(n * (n + 1) // 2, device="cuda", generator=g)
    x = torch.randn(n, device="cuda", generator=g)
    B = torch.randn(n, 5, device="cuda", generator=g)
    y, C = torch.zeros_like(x), torch.zeros_like(B)
    Ad, xd, yd = A.double(), x.double(), y.double()
    return {
        "ssfmv": lambda s: curfp.ssfmv(A, s * x, y),
        "dsfmv": lambda s: curfp.dsfmv(Ad, s * xd, yd),
        "acc64": lambda s: P.ssfmm_acc64(A, s * B, C),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["ssfmv", "dsfmv", "acc64"])
def test_second_stream_starts_after_the_first(curfp, name):
    f = routines(curfp)[name]
    want = [f(s).clone() for s in (1.0, -3.0)]
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    done = torch.cuda.Event()
    try:
        curfp.set_stream(a)
        with torch.cuda.stream(a):
            torch.cuda._sleep(200_000_000)
            first = f(1.0).clone()  # y and C are shared: the copies are what counts
            done.record(a)
        curfp.set_stream(b)
        with torch.cuda.stream(b):
            second = f(-3.0).clone()
        b.synchronize()
        assert done.query()
    finally:
        torch.cuda.synchronize()
        curfp.set_stream(None)
    assert torch.equal(first, want[0])
    assert torch.equal(second, want[1])


@pytest.mark.gpu
def test_capture_after_a_switch(curfp):
    f = routines(curfp)["ssfmv"]
    want = f(2.0).clone()
    a = torch.cuda.Stream()
    try:
        curfp.set_stream(a)
        with torch.cuda.stream(a):
            f(1.0)  # leaves work on the workspace in flight
        a.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            curfp.set_stream(torch.cuda.current_stream())
            got = f(2.0)
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
    f = routines(curfp)["ssfmv"]
    want = f(2.0).clone()
    rt = ctypes.CDLL("libcudart.so.12")
    s = ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
    h = curfp._get_handle()
    try:
        torch.cuda.synchronize()
        h.set_stream_ptr(s.value)
        with torch.cuda.stream(torch.cuda.ExternalStream(s.value)):
            f(1.0)
        assert rt.cudaStreamSynchronize(s) == 0 and rt.cudaStreamDestroy(s) == 0
    finally:
        curfp.set_stream(None)
    assert torch.equal(f(2.0), want)
