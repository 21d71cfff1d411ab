"""The three Linear products on the tensor-core tiles at sizes that are multiples of nothing: operand rows at a padded
pitch, edge tiles, scalar write-out (N % 4 != 0) under every schedule, plain and accumulating, raw planes and operands
packed once."""
import numpy as np
import pytest

import util
from test_kernels_gpu import _c, _dev, _host, _pair, _rand, ctx  # noqa: F401

pytestmark = pytest.mark.gpu

# Operands to 2^-22 and as much for the dropped product of the low parts; the tensor core's accumulator truncates, which
# makes 3e-6 over a chain of 1024 products of balanced data and grows with the chain.
TOL = 1e-5


@pytest.mark.parametrize("B,n_in,n_out", [
    (17, 1356, 130),      # a batch below a quarter tile, K % 16 != 0
    (64, 1001, 77),       # one row of tiles, K-split clusters
    (130, 300, 129),      # one row and one column beyond a tile
    (257, 999, 1023),     # pairs with a part-empty last tile
    (777, 1333, 1001),    # stream-K, all sizes odd
    (2049, 515, 1027),    # whole tiles first, then a shared remainder
    (83, 13688, 102),     # one tile, a very long K
    (100, 5000, 70),      # capped accumulation chains (K > 4096) at odd sizes
])
def test_ragged_products(ctx, B, n_in, n_out):  # noqa: F811
    import torch
    rng = np.random.default_rng(B + n_in)
    x, w, g = _rand(rng, B, n_in), _rand(rng, n_out, n_in, scale=n_in ** -0.5), _rand(rng, B, n_out)
    r = _rand(rng, B, n_out)
    X, W, G = _c(x), _c(w), _c(g)
    y, dx, dw = _pair(X @ W.T), _pair(G @ np.conj(W)), _pair(G.T @ np.conj(X))
    yr = _pair(X @ W.T + _c(r))
    dX, dW, dG, dR = _dev(x), _dev(w), _dev(g), _dev(r)
    assert util.relerr(_host(ctx.linear_fwd(dX, dW)), y) < TOL
    assert ctx.last_gemm_engine() == 1
    assert util.relerr(_host(ctx.linear_fwd(dX, dW, res=dR)), yr) < TOL
    assert util.relerr(_host(ctx.linear_bwd_x(dG, dW)), dx) < TOL
    assert util.relerr(_host(ctx.linear_bwd_w(dG, dX)), dw) < TOL
    acc = ctx.linear_bwd_x(dG, dW)
    assert util.relerr(_host(ctx.linear_bwd_x(dG, dW, out=acc)), (2 * dx[0], 2 * dx[1])) < TOL
    acc = ctx.linear_bwd_w(dG, dX)
    assert util.relerr(_host(ctx.linear_bwd_w(dG, dX, out=acc)), (2 * dw[0], 2 * dw[1])) < TOL
    # packed once, used by every product; the padding of the rows holds NaNs, which must reach nothing
    lib = ctx.lib
    assert lib.cnb_linear_pack_ok(B, n_in, n_out)

    def pack(t):
        rows, cols = t[0].shape
        out = torch.full((lib.cnb_pack_bytes(rows, cols) // 4,), float("nan"), device="cuda")
        out[:64] = 0.0
        assert lib.cnb_pack_matrix(ctx.h, t[0].data_ptr(), t[1].data_ptr(), rows, cols, out.data_ptr(), 0, ctx._stream()) == 0
        return out.data_ptr(), out
    px, pw, pg = pack(dX), pack(dW), pack(dG)
    o = ctx._new(B, n_out)
    assert lib.cnb_linear_fwd_packed(ctx.h, px[0], pw[0], dR[0].data_ptr(), dR[1].data_ptr(), o[0].data_ptr(), o[1].data_ptr(),
                                     B, n_in, n_out, ctx._stream()) == 0
    assert util.relerr(_host(o), yr) < TOL
    o = ctx._new(B, n_in)
    assert lib.cnb_linear_bwd_x_packed(ctx.h, pg[0], pw[0], o[0].data_ptr(), o[1].data_ptr(), B, n_in, n_out, 0, ctx._stream()) == 0
    assert util.relerr(_host(o), dx) < TOL
    o = ctx._new(n_out, n_in)
    assert lib.cnb_linear_bwd_w_packed(ctx.h, pg[0], px[0], o[0].data_ptr(), o[1].data_ptr(), B, n_in, n_out, 0, ctx._stream()) == 0
    assert util.relerr(_host(o), dw) < TOL


@pytest.mark.parametrize("scale", [2.0 ** -90, 2.0 ** -20, 1.0, 2.0 ** 30, 2.0 ** 60])
def test_packed_range(ctx, scale):  # noqa: F811
    """The scale of a packed operand follows its largest component, and rows down to 2^-20 of the largest keep the
    precision of the split products they replace: 22 bits less the 2 that low loses below 2^-18, and less half a bit a
    doubling of the terms; 2^-18 for each row by itself."""
    rng = np.random.default_rng(3)
    B, n_in, n_out = 256, 320, 192
    x, w = _rand(rng, B, n_in), _rand(rng, n_out, n_in)
    rows = (2.0 ** rng.uniform(-20, 0, B)).astype(np.float32)[:, None]
    rows[0] = 1.0
    x = tuple((p * rows * np.float32(scale)).astype(np.float32) for p in x)
    want = _c(x) @ _c(w).T
    y = _host(ctx.linear_fwd(_dev(x), _dev(w)))
    got = y[0].astype(np.float64) + 1j * y[1]
    err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() < 2.0 ** -18, err.max()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_packed_nonfinite_row(ctx, bad):  # noqa: F811
    """A row with an infinity or a NaN makes its own results NaN and leaves every other row as it is without it."""
    rng = np.random.default_rng(5)
    x, w = _rand(rng, 200, 320), _rand(rng, 192, 320)
    want = _pair(_c(x) @ _c(w).T)
    x[0][7, 33] = bad
    y = _host(ctx.linear_fwd(_dev(x), _dev(w)))
    keep = np.arange(200) != 7
    assert util.relerr(tuple(p[keep] for p in y), tuple(p[keep] for p in want)) < TOL
    assert not np.isfinite(y[0][7]).any() and not np.isfinite(y[1][7]).any()


def test_packed_zero_matrix(ctx):  # noqa: F811
    x, w = (np.zeros((128, 128), np.float32),) * 2, _rand(np.random.default_rng(4), 128, 128)
    y = _host(ctx.linear_fwd(_dev(x), _dev(w)))
    assert not y[0].any() and not y[1].any()
