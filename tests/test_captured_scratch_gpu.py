"""Scratch of a captured product that is smaller than what an eager one before it grew: allocations that make the scratch give
way afterwards must not be given memory that the graph works on."""
import numpy as np
import pytest

import util
from cnet_b200.ops import Context
from test_arena_limits_gpu import _product, _transform
from test_kernels_gpu import _c, _dev, _host, _pair, _rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [900, 2000])
def test_smaller_captured_product(rows):
    import torch
    ctx = Context(arena_bytes=64 << 20)
    _product(ctx, 3900, 1000, 1000)                          # 39 MB of packed operands
    rng = np.random.default_rng(rows)
    x, w = _rand(rng, rows, 1000), _rand(rng, 1000, 1000)
    dx, dw = _dev(x), _dev(w)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ctx.linear_fwd(dx, dw)
    z, want = _transform(ctx, 2000)                          # 32 MB of matrix, for which the scratch has to shrink
    assert util.relerr(_host(z), want) < 1e-5
    graph.replay()
    torch.cuda.synchronize()
    assert util.relerr(_host(y), _pair(_c(x) @ _c(w).T)) < 1e-5
    z, want = _transform(ctx, 2000)                          # the same matrix again, after the replay
    assert util.relerr(_host(z), want) < 1e-5
    ctx.close()
