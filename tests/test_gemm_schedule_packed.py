"""The schedule of products on packed operands, which is what everything but the C ABI's split buffers runs on: the checks of
the split form's schedule at k-blocks of 32, and products whose K is shorter than a CTA's least run."""
import ctypes as C

import pytest

from cnet_b200 import lib as L
from test_gemm_schedule import LIMITS, SHAPES, SMS


def _schedule(M, N, K, acc, limit):
    out = (C.c_int * 8)()
    assert L.load().cnb_gemm_schedule_packed(M, N, K, acc, SMS, limit, out) == 0
    return dict(zip(("pair", "ctas", "cluster_ctas", "run", "whole_per_cta", "segments", "atomics", "clear_from_row"), out))


@pytest.mark.parametrize("limit", LIMITS)
@pytest.mark.parametrize("M,N,K,acc", SHAPES)
def test_products_fill_the_sms_they_may_use(M, N, K, acc, limit):
    s = _schedule(M, N, K, acc, limit)
    may_use = limit if limit > 0 else SMS
    tiles = -(-M // 128) * -(-N // 128)
    k_blocks = -(-K // 32)
    if s["whole_per_cta"] == 0 and s["segments"] == 0 and s["ctas"] > may_use:
        assert s["ctas"] in (tiles, 2 * -(-M // 256) * -(-N // 128)), s
    assert s["ctas"] >= min(0.4 * may_use, tiles * max(1, k_blocks // 4) * 0.4), (s, may_use)
    assert s["cluster_ctas"] in (1, 2, 4, 8)
    if s["pair"]:
        assert s["ctas"] % 2 == 0 and s["cluster_ctas"] in (2, 4) and M >= 256
    if s["segments"]:
        assert k_blocks > 128 and s["run"] <= 32 and s["run"] * s["segments"] >= k_blocks     # capped accumulation chains


@pytest.mark.parametrize("limit", LIMITS)
@pytest.mark.parametrize("M,N,K", [(500, 900, 26), (250, 1500, 20), (777, 1001, 60), (2000, 50, 50), (128, 1333, 77), (4096, 17, 33),
                                   (4096, 4096, 17), (2100, 1200, 64), (17, 8000, 48)])
def test_whole_tiles_of_a_short_k_are_dealt_to_all_ctas(M, N, K, limit):
    s = _schedule(M, N, K, 0, limit)
    tiles = 2 * -(-M // 256) * -(-N // 128) if s["pair"] else -(-M // 128) * -(-N // 128)
    may_use = limit if limit > 0 else SMS
    assert s["ctas"] >= min(tiles, 0.8 * may_use), (s, tiles)


def test_refusals():
    out = (C.c_int * 8)()
    for bad in ((0, 8, 8), (8, 0, 8), (8, 8, 0)):
        assert L.load().cnb_gemm_schedule_packed(*bad, 0, SMS, 0, out) < 0
