"""The schedule of products of few tiles (cnb_gemm_schedule_packed: host arithmetic, no GPU)."""
import ctypes as C
import random

import pytest

from cnet_b200 import lib as L
from test_gemm_schedule import SMS
from test_gemm_schedule_packed import _schedule


@pytest.mark.parametrize("limit", [0, 74])
def test_narrow_tiles_fit_the_device(limit):
    """Products of few tiles: as many CTAs as one of the two tile widths asks for, in no more clusters than are resident at once
    (15 of eight CTAs and 33 of four on 148 SMs) where the order of the sums is free; a chain is no longer than in a run of wide tiles."""
    rng = random.Random(3)
    narrow = 0
    for _ in range(400):
        M, N, K = rng.randint(1, 700), rng.randint(1, 700), rng.randint(96, 4000)
        s = _schedule(M, N, K, 0, limit)
        if s["pair"] or s["atomics"] or s["segments"] or s["whole_per_cta"]:
            continue
        c, rows = s["cluster_ctas"], -(-M // 128)
        assert s["ctas"] in (rows * -(-N // 64) * c, rows * -(-N // 128) * c), (M, N, K, s)
        narrow += s["ctas"] == rows * -(-N // 64) * c and N > 64
        sms = limit or SMS
        fit = {1: sms, 2: sms // 2, 4: sms * 33 // 148, 8: sms * 15 // 148}[c]
        if s["ctas"] // c > fit:
            assert N <= 128 and s["ctas"] == rows * c, (M, N, K, s)
        chain = L.load().cnb_gemm_chain_packed(M, N, K, 0, SMS, limit)
        if K % 8 or M < 64 or N < 64:
            assert chain <= max(1, int(4.28 * K ** 0.5 / 32)), (M, N, K, chain)
    assert narrow > 100


def _form(M, N, K, acc, limit=0):
    out = (C.c_int * 4)()
    assert L.load().cnb_gemm_form_packed(M, N, K, acc, SMS, limit, out) == 0
    return dict(zip(("tile_n", "first", "rest", "form"), out))


def test_runs_that_are_cut_are_launched_so():
    """A launch of the form that makes one chain of every run has no run that is longer than its chains: not the longest, and not the
    one that holds a tile's first blocks, whose first chain may be shorter."""
    rng = random.Random(4)
    sizes = [(785, 1218, 616, 1), (282, 2355, 696, 1), (280, 2320, 640, 0), (1136, 1008, 1008, 0), (363, 2393, 640, 1)]
    sizes += [(8 * rng.randint(8, 350), 8 * rng.randint(8, 350), 8 * rng.randint(8, 512), rng.randint(0, 1)) for _ in range(4000)]
    shorter = 0
    for M, N, K, acc in sizes:
        s, f = _schedule(M, N, K, acc, 0), _form(M, N, K, acc)
        c = s["cluster_ctas"] // (2 if s["pair"] else 1)
        k_blocks = -(-K // 32)
        if c == 1:
            continue
        shorter += f["first"] < k_blocks // c
        if k_blocks // c > f["first"] or -(-k_blocks // c) > f["rest"]:
            assert f["form"] != 0, (M, N, K, acc, s, f)
    assert shorter > 3


@pytest.mark.parametrize("M,N,K,acc,pair,atomics", [
    (1820, 552, 163, 1, 1, 1),     # six chains of a block each either way: 1.16e-7 off float64 as runs of pairs, 1.18e-7 as one run
    (2622, 482, 206, 0, 1, 1),
])
def test_as_many_cubes_in_another_order_are_left(M, N, K, acc, pair, atomics):
    s = _schedule(M, N, K, acc, 0)
    assert (s["pair"], s["atomics"]) == (pair, atomics), s


@pytest.mark.parametrize("M,N,K,acc,ctas,cluster_ctas", [
    (1013, 1747, 366, 1, 136, 2),      # a CTA that adds to its whole tile reads it four bytes a lane: 43.4 us as runs with atomics, 55.6
    (2734, 478, 258, 1, 132, 2),
    (171, 2961, 192, 1, 96, 2),
    (824, 240, 680, 1, 112, 8),        # clusters half as wide read twice as many rows a CTA: 20.0 us, 21.6
    (1022, 107, 2390, 0, 120, 2),      # runs with atomics 33.6 us, clusters of eight 35.0
])
def test_products_that_smaller_clusters_slow_down(M, N, K, acc, ctas, cluster_ctas):
    s, f = _schedule(M, N, K, acc, 0), _form(M, N, K, acc)
    assert (s["ctas"], s["cluster_ctas"], f["tile_n"]) == (ctas, cluster_ctas, 128), (s, f)


def test_the_choice_takes_little_of_the_host():
    """A launch decides anew: 14 us a time where every chain of every candidate was walked, a microsecond or two now (least of many
    calls, beside a size with nothing to choose)."""
    import time
    lib, out = L.load(), (C.c_int * 8)()

    def least(M, N, K):
        best = 1.0
        for _ in range(300):
            t = time.perf_counter()
            lib.cnb_gemm_schedule_packed(M, N, K, 0, SMS, 0, out)
            best = min(best, time.perf_counter() - t)
        return best

    for M, N, K in [(437, 89, 3952), (411, 110, 3952), (506, 124, 3888), (281, 203, 2560), (159, 4070, 3377)]:
        assert least(M, N, K) - least(4096, 4096, 64) < 6e-6, (M, N, K)


def test_the_same_chains_in_fewer_slices_are_as_exact():
    """Eight slices of two blocks as four of two chains each: the same cuts and no more in any sum, so no chain need be shorter."""
    s, f = _schedule(300, 500, 500, 0, 0), _form(300, 500, 500, 0)
    assert (s["cluster_ctas"], f["tile_n"], f["first"], f["rest"]) == (4, 64, 2, 2), (s, f)
