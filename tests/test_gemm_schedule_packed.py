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
        _check_segments(s, M, N, K)


def _check_segments(s, M, N, K):
    """The segments of a tile cover its k-blocks, none of them empty, one CTA (or pair) each."""
    tiles = -(-M // (256 if s["pair"] else 128)) * -(-N // 128)
    k_blocks = -(-K // 32)
    assert s["ctas"] == tiles * s["segments"] * (2 if s["pair"] else 1), s
    assert k_blocks > 128 and (s["segments"] - 1) * s["run"] < k_blocks <= s["segments"] * s["run"], s


@pytest.mark.parametrize("limit", LIMITS)
@pytest.mark.parametrize("M,N,K", [(2000, 2000, 60000), (130, 1030, 9000), (700, 515, 8200), (1024, 8192, 16384), (100, 2048, 16384), (64, 64, 100000),
                                   (1000, 2050, 4104), (4096, 4096, 8192), (1500, 1500, 4100), (700, 1301, 9001), (1069, 38, 4215)])
def test_a_long_k_is_cut_into_chains(M, N, K, limit):
    """Whatever the form of the launch (segments, whole tiles, short runs), no more than 1024 products are summed in tensor
    memory at sizes of multiples of 8, and 4.28 sqrt(K) at others; a chain is no shorter than an equal cut at that length makes
    it, of K or (others, where a run is longer than 1024 products) of the runs that K was once cut into; a block less where pairs
    sum five chains or more."""
    s = _schedule(M, N, K, 0, limit)
    chain = L.load().cnb_gemm_chain_packed(M, N, K, 0, SMS, limit)
    k_blocks = -(-K // 32)
    if K % 8 == 0:
        assert chain == -(-k_blocks // -(-k_blocks // 32)), (chain, s)
    else:
        most = int(4.28 * K ** 0.5 / 32)
        former = -(-k_blocks // -(-k_blocks // 32))
        cluster = s["cluster_ctas"] // (2 if s["pair"] else 1)
        run = -(-k_blocks // cluster) if cluster > 1 else k_blocks if s["whole_per_cta"] else min(s["run"], k_blocks)
        c = -(-former // -(-former // most)) if run > 32 else most
        assert chain == (c - 1 if s["pair"] and most >= 3 and run > 4 * c else c), (chain, s)
    if s["segments"]:
        _check_segments(s, M, N, K)
    elif s["whole_per_cta"] and not s["atomics"]:
        tiles = -(-M // (256 if s["pair"] else 128)) * -(-N // 128)
        assert s["ctas"] // (2 if s["pair"] else 1) * s["whole_per_cta"] >= tiles


def test_segments_of_known_launches():
    assert {(2000, 2000, 60000): 4, (130, 1030, 9000): 8} == {k: _schedule(*k, 0, 0)["segments"] for k in ((2000, 2000, 60000), (130, 1030, 9000))}


@pytest.mark.parametrize("M,N,K,chain", [
    (4096, 1024, 1024, 16),        # 128 tiles on 74 pairs, whole: two chains of 16 where one of 32 would pass 24
    (4096, 1024, 512, 8),          # the same tiles, short of the cap: two chains all the same
    (4096, 1024, 96, 2),
    (4096, 1024, 64, 2),           # two blocks: one chain
    (512, 1024, 1024, 32),         # clusters along K: one chain
    (4096, 4096, 4096, 128),       # whole tiles of K <= 4096: one chain
    (777, 1001, 1333, 3),          # K of no multiple of 8: 4.28 sqrt(1333) = 156 products, and a block less for six chains by pairs
    (77, 1001, 1333, 4),           # single CTAs
    (777, 1001, 500, 2),           # two blocks at most
    (50, 70, 50, 1),
    (1500, 1500, 4100, 6),         # 129 blocks in one run, cut as the 26 of a fifth were: four chains, and a block less
    (700, 1301, 9001, 10),         # as 32 blocks in three chains, and a block less
    (1069, 38, 4215, 8),           # short runs: 4.28 sqrt(4215) = 277 products
])
def test_chains(M, N, K, chain):
    assert L.load().cnb_gemm_chain_packed(M, N, K, 0, SMS, 0) == chain


def test_chain_refusals():
    for bad in ((0, 8, 8), (8, 0, 8), (8, 8, 0)):
        assert L.load().cnb_gemm_chain_packed(*bad, 0, SMS, 0) < 0


def test_whole_tiles_of_a_long_k():
    s = _schedule(1000, 2050, 4104, 0, 0)
    assert s["whole_per_cta"] > 0 and s["segments"] == 0 and not s["atomics"]


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
