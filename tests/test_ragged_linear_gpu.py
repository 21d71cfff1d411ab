"""The three Linear products on the tensor-core tiles at sizes that are multiples of nothing: operand rows at a padded
pitch, edge tiles, scalar write-out (N % 4 != 0) under every schedule, plain and accumulating, raw planes and operands
split once."""
import numpy as np
import pytest

import util
from test_kernels_gpu import _c, _dev, _host, _pair, _rand, ctx  # noqa: F401

pytestmark = pytest.mark.gpu

# Operands to 2^-18 and 2^-20 for the dropped product of the low parts; the tensor core's accumulator truncates, about
# 2e-6 of its magnitude over 64 k-blocks of balanced data and growing as the square root of the chain.
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
    # split once, used by every product; the padding of the rows holds NaNs, which must reach nothing
    assert ctx.lib.cnb_linear_matrix_ok(B, n_in, n_out)

    def split(t):
        rows, cols = t[0].shape
        out = torch.full((ctx.lib.cnb_split_matrix_floats(rows, cols),), float("nan"), device="cuda")
        assert ctx.lib.cnb_split_matrix(ctx.h, t[0].data_ptr(), t[1].data_ptr(), rows, cols, out.data_ptr(), ctx._stream()) == 0
        return out
    sx, sw, sg = split(dX), split(dW), split(dG)
    assert util.relerr(_host(ctx.linear_fwd_split(sx, sw, B, n_in, n_out, res=dR)), yr) < TOL
    assert util.relerr(_host(ctx.linear_bwd_x_split(sg, sw, B, n_in, n_out)), dx) < TOL
    assert util.relerr(_host(ctx.linear_bwd_w_split(sg, sx, B, n_in, n_out)), dw) < TOL
