"""The operators that go through ops_native.so: the values and errors of the C ABI calls that they make, results in place,
planes that are no tensors, another stream."""
import pytest

from cnet_b200.lib import CnetError
from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


class Plane:
    """Something with a shape and an address."""

    def __init__(self, t):
        self.t, self.shape = t, tuple(t.shape)

    def data_ptr(self):
        return self.t.data_ptr()


@pytest.mark.parametrize("wrap", [tuple, list, lambda p: (Plane(p[0]), Plane(p[1]))])
def test_the_same_as_the_c_calls(wrap):
    import torch
    ctx = Context(arena_bytes=32 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    pair = lambda *s: (torch.randn(*s, generator=gen, device="cuda"), torch.randn(*s, generator=gen, device="cuda"))
    x, w, g, r = pair(7, 20), pair(5, 20), pair(7, 5), pair(7, 5)
    p, st = lambda t: t.data_ptr(), torch.cuda.current_stream().cuda_stream
    like = lambda a: (torch.empty_like(a[0]), torch.empty_like(a[0]))
    same = lambda a, b: torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    lib = ctx.lib
    y = like(g)
    assert lib.cnb_linear_fwd(ctx.h, p(x[0]), p(x[1]), p(w[0]), p(w[1]), p(r[0]), p(r[1]), p(y[0]), p(y[1]), 7, 20, 5, st) == 0
    assert same(ctx.linear_fwd(wrap(x), wrap(w), res=wrap(r)), y)
    dx = like(x)
    assert lib.cnb_linear_bwd_x(ctx.h, p(g[0]), p(g[1]), p(w[0]), p(w[1]), p(dx[0]), p(dx[1]), 7, 20, 5, 0, st) == 0
    assert same(ctx.linear_bwd_x(wrap(g), wrap(w)), dx)
    out = (torch.ones_like(dx[0]), torch.ones_like(dx[0]))
    assert ctx.linear_bwd_x(wrap(g), wrap(w), out=out) is out and torch.equal(out[0], dx[0] + 1)
    dw = like(w)
    assert lib.cnb_linear_bwd_w(ctx.h, p(g[0]), p(g[1]), p(x[0]), p(x[1]), p(dw[0]), p(dw[1]), 7, 20, 5, 0, st) == 0
    assert same(ctx.linear_bwd_w(wrap(g), wrap(x)), dw)
    f = like(x)
    assert lib.cnb_dft_fwd(ctx.h, p(x[0]), p(x[1]), p(f[0]), p(f[1]), 7, 20, st) == 0
    assert same(ctx.dft_fwd(wrap(x)), f)
    back = (x[0].clone(), x[1].clone())
    assert ctx.dft_bwd(wrap(f), out=back) is back and torch.allclose(back[0], 2 * x[0], atol=1e-5)
    s, inv = ctx.softmax_fwd(wrap(g))
    assert s[0].shape == (7, 5) and inv.shape == (7,)
    labels = torch.arange(7, device="cuda", dtype=torch.int32) % 5
    loss, d = ctx.crossent(wrap(s), labels)
    only, none = ctx.crossent(wrap(s), labels, backward=False)
    assert torch.equal(loss, only) and none == (None, None)
    assert ctx.softmax_bwd(wrap(d), wrap(g), inv)[0].shape == (7, 5)


def test_errors_and_streams():
    import torch
    ctx = Context(arena_bytes=32 << 20)
    x = (torch.randn(64, 100, device="cuda"), torch.randn(64, 100, device="cuda"))
    want = ctx.dft_fwd(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        got = ctx.dft_fwd(x)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0])
    with pytest.raises(ValueError):
        ctx.dft_fwd((x[0][0], x[1][0]))
    with pytest.raises(CnetError, match="dft_fwd failed"):
        ctx.dft_fwd((torch.empty(0, 100, device="cuda"),) * 2)
    ctx.close()
    with pytest.raises(CnetError, match="null"):
        ctx.dft_fwd(x)


def test_a_tensor_of_two_planes_is_a_pair():
    import torch
    ctx = Context(arena_bytes=32 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    pair = lambda *s: (torch.randn(*s, generator=gen, device="cuda"), torch.randn(*s, generator=gen, device="cuda"))
    same = lambda a, b: torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    x, w, g = pair(7, 20), pair(5, 20), pair(7, 5)
    sx, sw, sg = torch.stack(x), torch.stack(w), torch.stack(g)
    assert same(ctx.linear_fwd(sx, sw), ctx.linear_fwd(x, w))
    assert same(ctx.linear_bwd_x(sg, sw), ctx.linear_bwd_x(g, w))
    assert same(ctx.linear_bwd_w(sg, sx), ctx.linear_bwd_w(g, x))
    assert same(ctx.dft_fwd(sx), ctx.dft_fwd(x))
    y, inv = ctx.softmax_fwd(g)
    assert same(ctx.softmax_fwd(sg)[0], y) and same(ctx.softmax_bwd(sx[:, :, :5].contiguous(), sg, inv), ctx.softmax_bwd((x[0][:, :5].contiguous(), x[1][:, :5].contiguous()), g, inv))
    labels = torch.arange(7, device="cuda", dtype=torch.int32) % 5
    assert torch.equal(ctx.crossent(torch.stack(y), labels)[0], ctx.crossent(y, labels)[0])
    for f, like in ((lambda out: ctx.linear_bwd_x(g, w, out=out), x), (lambda out: ctx.linear_bwd_w(g, x, out=out), w), (lambda out: ctx.dft_bwd(x, out=out), x)):
        planes, stacked = (torch.ones_like(like[0]), torch.ones_like(like[0])), torch.ones_like(torch.stack(like))
        assert f(stacked) is stacked and same(stacked, f(planes))
    with pytest.raises(IndexError):
        ctx.dft_fwd(sx[:1])


def test_a_missing_plane_is_the_c_calls_error():
    import torch
    ctx = Context(arena_bytes=32 << 20)
    x = (torch.randn(4, 6, device="cuda"), torch.randn(4, 6, device="cuda"))
    half = (x[0], None)
    inv, labels = torch.ones(4, device="cuda"), torch.zeros(4, device="cuda", dtype=torch.int32)
    for f in (lambda: ctx.linear_fwd(half, x), lambda: ctx.linear_fwd(x, half), lambda: ctx.linear_bwd_x(x, half), lambda: ctx.linear_bwd_w(half, x),
              lambda: ctx.dft_fwd(half), lambda: ctx.dft_bwd(x, out=half), lambda: ctx.dft_bwd(x, out=(None, None)), lambda: ctx.softmax_fwd(half),
              lambda: ctx.softmax_bwd(half, x, inv), lambda: ctx.softmax_bwd(x, x, None), lambda: ctx.crossent(half, labels),
              lambda: ctx.crossent(x, None)):
        with pytest.raises(CnetError, match="null"):
            f()
    with pytest.raises(CnetError, match="pair"):
        ctx.linear_fwd(x, x, res=(torch.zeros(4, 4, device="cuda"), None))


def test_the_other_operand_may_have_more_dimensions():
    import torch
    ctx = Context(arena_bytes=32 << 20)
    pair = lambda *s: (torch.randn(*s, device="cuda"), torch.randn(*s, device="cuda"))
    same = lambda a, b: a[0].shape == b[0].shape and torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    view = lambda a, *s: (a[0].view(*s), a[1].view(*s))
    x, w, g = pair(7, 20), pair(5, 20), pair(7, 5)
    assert same(ctx.linear_fwd(x, view(w, 5, 4, 5)), ctx.linear_fwd(x, w))
    assert same(ctx.linear_bwd_x(g, view(w, 5, 20, 1)), ctx.linear_bwd_x(g, w))
    assert same(ctx.linear_bwd_w(g, view(x, 7, 20, 1)), ctx.linear_bwd_w(g, x))
    with pytest.raises(IndexError):
        ctx.linear_bwd_x(g, view(w, 100))
