"""Arenas with little room: scratch that grows takes in what it had, packed operands of raw products give way to whatever has
no other form, and a net whose arena was sized without them runs on raw planes."""
import numpy as np
import pytest

import util
from cnet_b200 import configs
from cnet_b200 import lib as L
from cnet_b200.net import Net
from cnet_b200.ops import Context
from oracle import cnet_oracle as co
from test_kernels_gpu import _c, _dev, _host, _pair, _rand

pytestmark = pytest.mark.gpu


def _product(ctx, B, n_in, n_out):
    rng = np.random.default_rng(B)
    x, w = _rand(rng, B, n_in), _rand(rng, n_out, n_in)
    return ctx.linear_fwd(_dev(x), _dev(w)), _pair(_c(x) @ _c(w).T)


def _transform(ctx, N):
    x = _rand(np.random.default_rng(N), 4, N)
    assert ctx.lib.cnb_set_dft_engine(ctx.h, 1) == 0
    return ctx.dft_fwd(_dev(x)), _pair(np.fft.fft(_c(x), axis=1) / np.sqrt(N))


def test_scratch_grows_in_place_and_gives_way():
    ctx = Context(arena_bytes=64 << 20)
    for rows in (900, 1900, 2900, 3900):                     # up to 8 * 4900 * 1000 bytes of packed operands
        y, want = _product(ctx, rows, 1000, 1000)
        assert ctx.last_gemm_engine() == 1
        assert util.relerr(_host(y), want) < 1e-5
        used = ctx.lib.cnb_arena_used(ctx.h)
        assert used < 8 * (rows + 1000) * 1000 + (9 << 20)   # not the sum of what it was before
    y, want = _transform(ctx, 2000)                          # 32 MB of matrix, for which the scratch has to shrink
    assert util.relerr(_host(y), want) < 1e-5
    y, want = _product(ctx, 3900, 1000, 1000)                # no room any more: the SIMT tiles
    assert ctx.last_gemm_engine() == 2
    assert util.relerr(_host(y), want) < 1e-5
    ctx.close()


def test_captured_scratch_stays():
    import torch
    ctx = Context(arena_bytes=64 << 20)
    rng = np.random.default_rng(1)
    x, w = _rand(rng, 3900, 1000), _rand(rng, 1000, 1000)
    dx, dw = _dev(x), _dev(w)
    ctx.linear_fwd(dx, dw)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ctx.linear_fwd(dx, dw)
    with pytest.raises(L.CnetError, match="arena"):
        _transform(ctx, 2000)                                # 32 MB of matrix
    graph.replay()
    torch.cuda.synchronize()
    assert util.relerr(_host(y), _pair(_c(x) @ _c(w).T)) < 1e-5
    ctx.close()


def test_net_without_room_for_packed_operands():
    B, kw = 300, dict(n=500, blocks=2, m=40)
    ora = co.OracleNet()
    so = configs.build_mixer(ora, **kw)
    full, dev = Net(), Net()
    configs.build_mixer(full, **kw)
    pack = full.lib.cnb_pack_bytes
    packs = 2 * (pack(B, 500) + pack(500, 500)) + pack(B, 500) + pack(40, 500) + pack(B, 500)
    full_bytes = full.required_arena(B)
    dev = Net(arena_bytes=full_bytes - packs - (16 << 20) + (256 << 10))
    sd = configs.build_mixer(dev, **kw)
    for uid, (re, im) in configs.init_weights(sd, 5).items():
        dev.set_values(uid, re, im)
        ora.set_values(uid, re, im)
    dev.allocate(B)
    x, labels = configs.make_batch(sd, B, 6)
    for t in range(2):
        got, want = dev.run_batch(sd.main, x=x, labels=labels), ora.run_batch(so.main, x=x, labels=labels)
        assert np.linalg.norm(got - want) < 1e-4 * np.linalg.norm(want)
        for name in ("w0", "h1", "wh"):
            assert util.relerr(dev.get_wgrad(sd.layers[name]), ora.get_wgrad(so.layers[name])) < 1e-3, name
        dev.adam(0.01, B, 0.9, t)
        ora.adam(0.01, B, 0.9, t)
    for name in ("w0", "wh"):
        assert util.relerr(dev.get_values(sd.layers[name]), ora.get_values(so.layers[name])) < 1e-4, name
