"""Packs of matrices whose rows go four columns at a time and of others, alone, mixed in one launch and beside a plain one: the
parts that the scale makes of every value, whatever the launch."""
import ctypes as C

import numpy as np
import pytest

from cnet_b200.ops import Context
from test_adam_packed_gpu import Span

pytestmark = pytest.mark.gpu


def _parts(pack, r, c):
    """Head's exponent and the planes of a pack, as numpy."""
    pitch = (c + 63) // 64 * 64
    raw = pack.cpu().numpy()
    e = int(raw[:4].view(np.int32)[0])
    if e == 1 << 20:
        return e, raw[256:256 + 8 * r * pitch].view(np.float32).reshape(2, r, pitch)[:, :, :c]
    return e, raw[256:256 + 8 * r * pitch].view(np.float16).reshape(4, r, pitch)[:, :, :c]


def _check(pack, re, im):
    r, c = re.shape
    e, planes = _parts(pack, r, c)
    for k, x in enumerate((re.cpu().numpy(), im.cpu().numpy())):
        if e == 1 << 20:
            assert np.array_equal(planes[k], x)
            continue
        scaled = x * np.float32(2.0) ** e
        high = scaled.astype(np.float16)
        assert np.array_equal(planes[k], high)
        assert np.array_equal(planes[2 + k], (scaled - high.astype(np.float32)).astype(np.float16))
    return e


# 700 x 1024 and 699 x 1023: several pieces a thread; one column; one row; rows of 4 at an address that is no multiple of 16
@pytest.mark.parametrize("shapes", [[(64, 64)], [(33, 129)], [(1, 1)], [(5, 2)], [(1, 4096)], [(4000, 1)], [(2900, 1024)], [(2900, 1023)],
                                    [(64, 64), (65, 63)], [(2900, 1024), (3, 4)], [(2899, 1023), (3, 5)], [(17, 48), (9, 9), (64, 64)] * 12])
@pytest.mark.parametrize("shift", [0, 1])
def test_parts_of_every_value(shapes, shift):
    import torch
    ctx = Context(arena_bytes=16 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(len(shapes))
    pad = lambda n: (n + 3) // 4 * 4                          # planes start on 16 bytes, or `shift` floats behind
    n = shift + sum(2 * pad(r * c) for r, c in shapes)
    w, g = torch.randn(n, generator=gen, device="cuda"), torch.zeros(n, device="cuda")
    spans, packs, planes, at = (Span * len(shapes))(), [], [], shift
    for k, (r, c) in enumerate(shapes):
        packs.append(torch.zeros(ctx.lib.cnb_pack_bytes(r, c), dtype=torch.uint8, device="cuda"))
        a, b = at, at + pad(r * c)
        spans[k] = Span(a, b, r, c, packs[k].data_ptr())
        planes.append((w[a:a + r * c].view(r, c), w[b:b + r * c].view(r, c)))
        at = b + pad(r * c)
    if len(shapes) > 1:
        planes[-1][0][0, 0] = 1e12                             # a range that no scale covers: fp32 planes, beside scaled ones
    st = torch.cuda.current_stream().cuda_stream
    for _ in range(2):                                         # the heads are ready for the next use
        assert ctx.lib.cnb_sgd_update_packed(ctx.h, w.data_ptr(), g.data_ptr(), n, 0.0, 1, spans, len(shapes), st) == 0
        kinds = [_check(p, *xy) for p, xy in zip(packs, planes)]
        if len(shapes) > 1:
            assert kinds[-1] == 1 << 20 and kinds[0] != 1 << 20
