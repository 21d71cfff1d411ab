"""Tables of constants that a transform makes at its first use: complete for whoever uses them next, on another stream
without a synchronisation between, and in eager calls after a first use that was only captured."""
import numpy as np
import pytest

import util
from cnet_b200.ops import Context
from test_kernels_gpu import _c, _dev, _host, _pair, _rand

pytestmark = pytest.mark.gpu

# the chirp form's tables take milliseconds to make; mixed radices; the pipelined kernel; the twiddle matrix, and packed
CASES = [("fft", 4093), ("fft", 6007), ("fft", 900), ("fft", 1024), ("product", 200), ("triangle", 136)]


def _call(ctx, kind, x):
    B, N = x[0].shape
    if kind == "triangle":
        y = ctx._new(B, N)
        assert ctx.lib.cnb_tdft_fwd(ctx.h, x[0].data_ptr(), x[1].data_ptr(), y[0].data_ptr(), y[1].data_ptr(), B, N, ctx._stream()) == 0
        return y
    return ctx.dft_fwd(x)


def _case(kind, N):
    ctx = Context(arena_bytes=256 << 20)
    if kind == "product":
        assert ctx.lib.cnb_set_dft_engine(ctx.h, 1) == 0
    x = _rand(np.random.default_rng(N), 64, N)
    if kind == "triangle":
        k = np.arange(N)
        f = np.where(k[None, :] <= k[:, None], np.exp(-2j * np.pi * (np.outer(k, k) % N) / N), 0) / np.sqrt(N)
        want = _c(x) @ f.T
    else:
        want = np.fft.fft(_c(x), axis=1) / np.sqrt(N)
    return ctx, _dev(x), _pair(want)


@pytest.mark.parametrize("kind,N", CASES)
def test_second_stream_right_after_the_first(kind, N):
    import torch
    ctx, x, want = _case(kind, N)
    torch.cuda.synchronize()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        y1 = _call(ctx, kind, x)
    if kind != "fft":
        first.synchronize()                 # these products also share the context's scratch, which is one stream's at a time
    with torch.cuda.stream(second):
        y2 = _call(ctx, kind, x)
        y3 = _call(ctx, kind, x)
    torch.cuda.synchronize()
    for y in (y1, y2, y3):
        assert util.relerr(_host(y), want) < 1e-5
    ctx.close()


@pytest.mark.parametrize("kind,N", CASES)
def test_first_use_under_capture(kind, N):
    import torch
    ctx, x, want = _case(kind, N)
    ctx.lib.cnb_reserve_scratch(ctx.h, 32 << 20)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = _call(ctx, kind, x)
    assert util.relerr(_host(_call(ctx, kind, x)), want) < 1e-5       # before any replay
    graph.replay()
    torch.cuda.synchronize()
    assert util.relerr(_host(y), want) < 1e-5
    ctx.close()


def test_captured_behind_an_unfinished_build():
    """A table still being made on the captured stream's own queue: the graph may be launched anywhere."""
    import torch
    ctx, x, want = _case("fft", 6007)
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        _call(ctx, "fft", x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = _call(ctx, "fft", x)
    with torch.cuda.stream(other):
        graph.replay()
    torch.cuda.synchronize()
    assert util.relerr(_host(y), want) < 1e-5
    ctx.close()
