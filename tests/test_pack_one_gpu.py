"""Packed operands against their definition: one launch (up to 16 tiles of 32 x 128), two, and the sizes between; whole and ragged
tiles, ranges that are too wide, infinities."""
import ctypes as C

import numpy as np
import pytest

from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu

PLAIN = 1 << 20


def _expected(re, im, spread):
    big = max(np.abs(a[np.isfinite(a)]).max(initial=0.0) for a in (re, im))
    if big == 0:
        return 0
    return PLAIN if spread else 14 - int(np.floor(np.log2(big)))


@pytest.mark.parametrize("rows,cols", [
    (1, 1), (31, 127), (32, 128), (33, 129), (7, 500), (300, 4),       # a tile, remainders
    (256, 128), (128, 256),            # eight tiles
    (257, 128), (130, 257), (128, 512), (500, 100), (512, 65),         # up to sixteen
    (513, 65), (512, 129), (128, 516),  # more
])
@pytest.mark.parametrize("what", ["plain numbers", "a small row", "infinities", "zeros"])
def test_pack(rows, cols, what):
    import torch
    ctx = Context(arena_bytes=64 << 20)
    rng = np.random.default_rng(rows * 1000 + cols)
    re, im = [rng.standard_normal((rows, cols)).astype(np.float32) * np.float32(3.7) for _ in range(2)]
    spread = what == "a small row" and rows > 1
    if spread:
        re[rows // 2] *= np.float32(2.0 ** -30)
        im[rows // 2] *= np.float32(2.0 ** -30)
    if what == "infinities":
        re[0, 0], im[-1, -1] = np.inf, -np.inf
    if what == "zeros":
        re[:], im[:] = 0, 0
    dr, di = torch.from_numpy(re).cuda(), torch.from_numpy(im).cuda()
    size = ctx.lib.cnb_pack_bytes(rows, cols)
    pack = torch.zeros(size, dtype=torch.uint8, device="cuda")
    for _ in range(2):                                   # the head is ready for a second use
        assert ctx.lib.cnb_pack_matrix(ctx.h, dr.data_ptr(), di.data_ptr(), rows, cols, pack.data_ptr(), 0, ctx._stream()) == 0
    host = pack.cpu().numpy()
    head = host[:16].view(np.int32)
    e = _expected(re, im, spread)
    assert head[0] == e and (head[1:4] == 0).all(), (head, e)
    body = host[256:]
    pitch = -(-cols // 64) * 64
    if e == PLAIN:
        planes = body[:8 * rows * pitch].view(np.float32).reshape(2, rows, pitch)[:, :, :cols]
        assert (planes[0] == re).all() and (planes[1] == im).all()
        return
    planes = body[:8 * rows * pitch].view(np.float16).reshape(4, rows, pitch)[:, :, :cols]
    with np.errstate(over="ignore", invalid="ignore"):
        for k, a in enumerate((re, im)):
            scaled = a * np.float32(2.0) ** e
            high = scaled.astype(np.float16)
            low = (scaled - high.astype(np.float32)).astype(np.float16)
            assert np.array_equal(planes[k], high, equal_nan=True) and np.array_equal(planes[2 + k], low, equal_nan=True)
