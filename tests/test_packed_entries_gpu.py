"""The entry points that pack what they produce, by themselves: the update of an arena and the FourierTrans with its tail."""
import ctypes as C

import numpy as np
import pytest

import util
from oracle import cnet_oracle as co
from test_kernels_gpu import _c, _dev, _host, _pair, _rand, ctx  # noqa: F401
from test_packed_args import Span

pytestmark = pytest.mark.gpu

PLAIN = 1 << 20      # the exponent of a pack that holds fp32 planes


def _new_pack(ctx, rows, cols):  # noqa: F811
    import torch
    p = torch.full((ctx.lib.cnb_pack_bytes(rows, cols) // 4,), float("nan"), device="cuda")
    p[:64] = 0
    return p


def _unpack(pack, rows, cols):
    """(exponent, re, im) that a pack stands for, in float64."""
    raw = pack.cpu().numpy()
    e, pitch = int(raw[:1].view(np.int32)[0]), -(-cols // 64) * 64
    assert not raw[1:4].view(np.uint32).any()                # ready for the next use
    if e == PLAIN:
        planes = raw[64:64 + 2 * rows * pitch].reshape(2, rows, pitch)[:, :, :cols].astype(np.float64)
        return e, planes[0], planes[1]
    h = raw[64:].view(np.float16)[:4 * rows * pitch].reshape(4, rows, pitch)[:, :, :cols].astype(np.float64)
    return e, (h[0] + h[2]) * 2.0 ** -e, (h[1] + h[3]) * 2.0 ** -e


def _check_pack(pack, re, im, plain=False):
    e, r, i = _unpack(pack, *re.shape)
    assert (e == PLAIN) == plain
    most = max(np.abs(re).max(), np.abs(im).max())
    for got, want in ((r, re.astype(np.float64)), (i, im.astype(np.float64))):
        # 22 bits of every component down to 2^-17 of the largest, 2^-39 of it below
        assert (np.abs(got - want) <= (0 if plain else np.maximum(np.abs(want) * 2.0 ** -22, most * 2.0 ** -39))).all()


# rows x cols of the matrices of one arena, floats before each plane: rows that are no multiples of 4, planes that start at any
# float, more matrices than one launch takes
@pytest.mark.parametrize("shapes,gap", [([(26, 900)], 0), ([(128, 256), (64, 64), (10, 33)], 0), ([(33, 7), (5, 129)], 3), ([(3, 20)] * 40, 0),
                                        ([(9, 13)] * 70, 1)])
def test_sgd_update_packed(ctx, shapes, gap):  # noqa: F811
    import torch
    rng = np.random.default_rng(len(shapes))
    spans, packs, at = [], [], 0
    for rows, cols in shapes:
        packs.append(_new_pack(ctx, rows, cols))
        re, im = at + gap, at + 2 * gap + rows * cols
        spans.append(Span(re, im, rows, cols, packs[-1].data_ptr()))
        at = im + rows * cols
    spans.append(spans[0])                                   # a shared weight: a second pack of the same planes
    packs.append(_new_pack(ctx, *shapes[0]))
    spans[-1] = Span(spans[0].re, spans[0].im, *shapes[0], packs[-1].data_ptr())
    n = at + 5
    w, g = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
    dw, dg = torch.from_numpy(w).cuda(), torch.from_numpy(g).cuda()
    for step in range(2):                                    # the heads come back ready for a second use
        arr = (Span * len(spans))(*spans)
        assert ctx.lib.cnb_sgd_update_packed(ctx.h, dw.data_ptr(), dg.data_ptr(), n, 0.25, 0, C.byref(arr), len(spans), ctx._stream()) == 0
        got = dw.cpu().numpy()
        want = w - np.float32(0.25 * (step + 1)) * g
        assert np.abs(got - want).max() < 1e-6
        for s, p in zip(spans, packs):
            planes = [got[k:k + s.rows * s.cols].reshape(s.rows, s.cols) for k in (s.re, s.im)]
            _check_pack(p, *planes)
    assert np.array_equal(dg.cpu().numpy(), g)
    assert ctx.lib.cnb_sgd_update_packed(ctx.h, dw.data_ptr(), dg.data_ptr(), n, 0.25, 1, None, 0, ctx._stream()) == 0
    assert not dg.cpu().numpy().any()


@pytest.mark.parametrize("B,N", [(1, 16), (7, 127), (300, 500), (33, 900), (64, 1024), (129, 784), (3, 4096)])
@pytest.mark.parametrize("plain", [False, True])
def test_fourier_tail_packed(ctx, B, N, plain):  # noqa: F811
    rng = np.random.default_rng(B + N)
    x, h = _rand(rng, B, N), _rand(rng, N)
    if plain:
        for p in x:
            p[0] *= 2.0 ** -40                               # one row of another scale than the others
        if B == 1:
            return
    dx, dh = _dev(x), _dev(h)
    u, y, a = ctx._new(B, N), ctx._new(B, N), ctx._new(B, N)
    pack = _new_pack(ctx, B, N)
    ptr = lambda *t: [p.data_ptr() for pair in t for p in pair]  # noqa: E731
    f = np.fft.fft(_c(x), axis=1) / np.sqrt(N)
    prod = f * _c(h)
    want = co._gelu(prod.real), co._gelu(prod.imag)
    for keep in (False, True):
        if keep and not ctx.lib.cnb_dft_keeps_product(N):
            continue
        if keep:
            rc = ctx.lib.cnb_dft_hadamard_gelu_fwd_keep(ctx.h, *ptr(dx, dh, u, a, y), pack.data_ptr(), B, N, ctx._stream())
            assert rc == 0 and util.relerr(_host(a), _pair(prod)) < 2e-6
        else:
            assert ctx.lib.cnb_dft_hadamard_gelu_fwd_packed(ctx.h, *ptr(dx, dh, u, y), pack.data_ptr(), B, N, ctx._stream()) == 0
        assert util.relerr(_host(u), _pair(f)) < 2e-6
        assert util.relerr(_host(y), want) < 2e-6
        _check_pack(pack, *_host(y), plain=plain)


def test_kernels_that_keep_no_product_say_so(ctx):  # noqa: F811
    z = ctx._new(4, 1024)
    p = [t.data_ptr() for t in z]
    assert not ctx.lib.cnb_dft_keeps_product(1024)
    assert ctx.lib.cnb_dft_hadamard_gelu_fwd_keep(ctx.h, *p, *p, *p, *p, *p, None, 4, 1024, ctx._stream()) < 0
    assert ctx.lib.cnb_dft_hadamard_gelu_fwd_keep(ctx.h, *p, *p, *p, p[0], None, *p, None, 4, 512, ctx._stream()) < 0
