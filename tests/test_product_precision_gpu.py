"""The tensor-core tiles against fp32 FMAs at sizes that have both: the error against float64 of the three Linear products
must not be larger than that of the SIMT tiles, which a context without room for packed operands falls back to."""
import numpy as np
import pytest

from cnet_b200.ops import Context
from test_kernels_gpu import _c, _dev, _host, _rand, ctx  # noqa: F401

pytestmark = pytest.mark.gpu

# The errors are means over at least 1300 components each way, known to about 3 %.
SLACK = 1.1


@pytest.mark.parametrize("B,n_in,n_out", [
    (500, 900, 26),       # fewer outputs than a tile has rows: clusters along K
    (2000, 50, 50),       # one chain would hold all of K
    (300, 500, 500),      # no multiple of 8
    (300, 257, 2500),     # K one product beyond a block
    (777, 1333, 1001),    # long chains, CTA pairs
    (40, 4095, 513),      # stream-K
    (2049, 515, 1027),    # whole tiles, then a shared remainder
    (33, 9001, 70),       # capped segments (K > 4096)
])
def test_tiles_are_no_less_exact_than_fmas(ctx, B, n_in, n_out):  # noqa: F811
    rng = np.random.default_rng(B + n_out)
    x, w, g = _rand(rng, B, n_in), _rand(rng, n_out, n_in), _rand(rng, B, n_out)
    X, W, G = _c(x), _c(w), _c(g)
    dx, dw, dg = _dev(x), _dev(w), _dev(g)
    plain = Context(arena_bytes=1 << 20)
    calls = [(lambda c: c.linear_fwd(dx, dw), X @ W.T, n_in), (lambda c: c.linear_bwd_x(dg, dw), G @ W.conj(), n_out),
             (lambda c: c.linear_bwd_w(dg, dx), G.T @ X.conj(), B)]
    for call, want, K in calls:
        if K % 8 == 0 and K >= 32 and min(want.shape) >= 64:
            continue                                     # always split here, never fp32
        err = []
        for c, engine in ((ctx, (1, 2)), (plain, (2,))):
            y = _host(call(c))
            assert c.last_gemm_engine() in engine
            err.append(np.linalg.norm(y[0] + 1j * y[1].astype(np.float64) - want) / np.linalg.norm(want))
        print("%d x %d, K = %d: tiles %.2e, FMAs %.2e" % (*want.shape, K, *err))
        assert err[0] <= SLACK * err[1], (want.shape, K, err)
