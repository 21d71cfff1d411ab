"""TriangFourier's matrix is a constant: at lengths of which some batches run on the tensor core it is packed once, by whichever
batch comes first, and batches on both sides of the line between FMAs and the tensor core are right."""
import numpy as np
import pytest

import util
from cnet_b200.ops import Context
from test_kernels_gpu import _c, _dev, _host, _pair, _rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,packed", [(50, False), (64, True), (100, False), (128, True), (200, True), (203, True), (256, True)])
def test_packed_when_it_is_made(n, packed):
    import torch
    ctx = Context(arena_bytes=64 << 20)
    assert ctx.lib.cnb_reserve_scratch(ctx.h, 16 << 20) == 0           # what the products take is there before
    k = np.arange(n)
    f = np.where(k[None, :] <= k[:, None], np.exp(-2j * np.pi * (np.outer(k, k) % n) / n), 0) / np.sqrt(n)
    at_first = ctx.lib.cnb_arena_used(ctx.h)
    engines = []
    line = 8e6 / n / n                                                 # rows from which the tensor core takes the product
    for rows in (17, int(line), int(line) + 1):
        x, g = (_rand(np.random.default_rng(rows + i), rows, n) for i in range(2))
        dx, dg = _dev(x), _dev(g)
        y = ctx._new(rows, n)
        p = lambda t: t.data_ptr()
        assert ctx.lib.cnb_tdft_fwd(ctx.h, p(dx[0]), p(dx[1]), p(y[0]), p(y[1]), rows, n, ctx._stream()) == 0
        engines.append(ctx.last_gemm_engine())
        assert util.relerr(_host(y), _pair(_c(x) @ f.T)) < 1e-5
        assert ctx.lib.cnb_tdft_bwd(ctx.h, p(dg[0]), p(dg[1]), p(y[0]), p(y[1]), rows, n, 0, ctx._stream()) == 0
        assert util.relerr(_host(y), _pair(_c(g) @ f.conj())) < 1e-5
        pitch = (n + 7) // 8 * 8
        grown = 2 * -(-4 * n * n // 256) * 256 + (-(-(256 + 8 * n * pitch) // 256) * 256 if packed else 0)
        assert ctx.lib.cnb_arena_used(ctx.h) - at_first == grown
    assert engines == [2, 2, 1 if n >= 64 else 2]
    ctx.close()
