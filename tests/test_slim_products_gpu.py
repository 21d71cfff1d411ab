"""Products of few outputs in fp32 FMAs (tiles of 8 x 8): one to many slabs of k, remainders of every size, each orientation of the
operands, planes of 4-byte alignment."""
import pytest

from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,n_in,n_out", [
    (1, 1, 17),            # one k
    (8, 32, 24), (9, 33, 25), (7, 31, 23),         # one slab, a k and a row beyond it, less of both
    (33, 161, 35),         # as many slabs as are on their way, and one k
    (53, 27, 993),         # a long K for dX*
    (993, 53, 27),         # and for dW*
    (16, 2000, 40),        # and forward
    (70, 199, 150),        # sums of sixteen (K between 48 and 256, more than two million multiplications): forward
    (1241, 204, 20),       # tiles of 16 a quarter empty
    (177, 35, 285),        # several to an SM
])
def test_few_outputs(B, n_in, n_out):
    import torch
    ctx = Context(arena_bytes=64 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B + n_in + n_out)

    def pair(rows, cols):
        return tuple(torch.randn(rows * cols + 1, generator=gen, device="cuda")[1:].view(rows, cols) for _ in range(2))
    x, w, g, r = pair(B, n_in), pair(n_out, n_in), pair(B, n_out), pair(B, n_out)
    full = lambda t: torch.complex(t[0].double(), t[1].double())
    X, W, G = full(x), full(w), full(g)

    def near(got, want, K):
        # K rounded terms, one after the other: sqrt(K) / 2 roundings of 2^-24 in the mean square, and twice that
        err = float((full(got) - want).norm() / want.norm())
        assert err < 6e-8 * (2 + K ** 0.5), (err, K)
    near(ctx.linear_fwd(x, w), X @ W.T, n_in)
    near(ctx.linear_fwd(x, w, res=r), X @ W.T + full(r), n_in)
    near(ctx.linear_bwd_x(g, w), G @ W.conj(), n_out)
    near(ctx.linear_bwd_w(g, x), G.T @ X.conj(), B)
    old = pair(B, n_in)
    near(ctx.linear_bwd_x(g, w, out=tuple(t.clone() for t in old)), G @ W.conj() + full(old), n_out)
    old = pair(n_out, n_in)
    near(ctx.linear_bwd_w(g, x, out=tuple(t.clone() for t in old)), G.T @ X.conj() + full(old), B)


def test_a_short_k_takes_no_longer_than_a_longer_one():
    """16 x 31, K = 3, is not the tiles of 8 x 8, whose set-up is for several slabs of K: 1.2 us, by those 1.4, as K = 20 takes."""
    import torch
    ctx = Context(arena_bytes=64 << 20)

    def least(k):
        g, x = [tuple(torch.randn(k, n, device="cuda") for _ in range(2)) for n in (16, 31)]
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            ctx.linear_bwd_w(g, x)
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(50):
                ctx.linear_bwd_w(g, x)
        times = []
        for _ in range(30):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert least(3) < 0.95 * least(20)
