"""What a product truncates (cnb_gemm_truncation_packed: host arithmetic), by which dX* and dW* are kept on halves of the device."""
import pytest

from cnet_b200 import lib as L
from test_gemm_schedule import SMS


def _cubes(M, N, K, acc, limit):
    return L.load().cnb_gemm_truncation_packed(M, N, K, acc, SMS, limit)


@pytest.mark.parametrize("M,N,K,acc,limit,cubes", [
    (4096, 512, 512, 0, 0, 16 ** 3),                     # a chain a tile
    (4096, 512, 512, 0, 74, 2 * 8 ** 3),                 # whole tiles in two chains
    (512, 1024, 1024, 0, 0, 4 * 8 ** 3),                 # slices of a cluster of four
    (4096, 4096, 4096, 0, 0, 128 ** 3),
    (785, 1218, 616, 1, 0, (9 ** 3 + 9 ** 3 + 1)),       # slices of 9 and 10 blocks, chains of 9 in the first, 10 in the other
])
def test_cubes_of_known_launches(M, N, K, acc, limit, cubes):
    got = _cubes(M, N, K, acc, limit)
    if (M, N, K) == (785, 1218, 616):
        assert got < 1765.1                              # what runs of pairs, summed with atomics, had
    else:
        assert got == cubes


def test_sizes_that_are_none():
    for bad in ((0, 1, 1), (1, 0, 1), (1, 1, 0)):
        assert _cubes(*bad, 0, 0) == -1.0 and L.load().cnb_gemm_share_packed(*bad, 0, SMS) == -1.0


@pytest.mark.parametrize("M,N,K,acc,share", [
    (512, 1024, 1024, 0, 32 / 33),                       # clusters of four
    (512, 320, 512, 0, 20 / 33),
    (512, 320, 512, 1, 12 / 15),                         # added to what is there: clusters of eight
    (4096, 512, 512, 0, 64 / 74),                        # pairs
])
def test_shares_of_known_launches(M, N, K, acc, share):
    assert L.load().cnb_gemm_share_packed(M, N, K, acc, SMS) == pytest.approx(share)
