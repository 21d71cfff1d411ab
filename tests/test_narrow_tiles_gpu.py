"""Products of few tiles on tiles of 128 x 64: widths around a narrow tile, one and several rows of tiles, every size of cluster
and none, chains that are cut inside a slice of K, residuals, accumulation, and operands that run as fp32 FMAs."""
import ctypes as C

import pytest

from cnet_b200 import lib as L
from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,cluster,tile_n", [
    (128, 64, 1024, 8, 64),       # one narrow tile, whole
    (130, 65, 1000, 8, 64),       # one row and one column beyond it
    (40, 1, 60000, 1, 128),       # (stream-K as before: the tiles are not what such a K is short of)
    (64, 784, 784, 8, 64),        # 13 of them
    (500, 26, 900, 8, 64),        # half empty
    (300, 500, 500, 4, 64),       # smaller clusters than wide tiles had, two chains a slice
    (130, 1001, 700, 4, 64),      # rows that are not 16-byte aligned
    (512, 512, 1024, 4, 64),      # K % 8 == 0, two chains a slice
    (260, 1030, 300, 2, 64),
    (700, 400, 300, 2, 64),
    (442, 69, 1281, 8, 64),       # runs of pairs before, summed with atomics
    (200, 1000, 100, 2, 64),
    (257, 999, 52, 1, 64),        # a CTA to a tile
    (785, 1218, 616, 2, 128),     # wide tiles in clusters of two, in the place of runs of pairs
    (2041, 643, 552, 1, 128),     # a CTA to a wide tile, a first chain of 11 blocks and the others of 12; as a gradient runs of pairs
    (1041, 1329, 277, 1, 128),    # chains of one block
])
def test_narrow_tiles(M, N, K, cluster, tile_n):
    import torch
    lib = L.load()
    out, form = (C.c_int * 8)(), (C.c_int * 4)()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert lib.cnb_gemm_schedule_packed(M, N, K, 0, sms, 0, out) == 0 and lib.cnb_gemm_form_packed(M, N, K, 0, sms, 0, form) == 0
    if sms == 148:
        assert out[2] == cluster and form[0] == tile_n, (list(out), list(form))
        if K < 60000:
            assert out[1] == -(-M // 128) * -(-N // tile_n) * cluster, list(out)
    # what a chain of C blocks of 32 products truncates, 4.2e-9 of the result a product, for all chains of a tile, of the schedule that
    # adds to what is there or of the one that does not
    blocks = -(-K // 32)
    chains = [4.2e-9 * 32 * (lib.cnb_gemm_truncation_packed(M, N, K, acc, sms, 0) / blocks) ** 0.5 for acc in (0, 1)]
    ctx = Context(arena_bytes=(64 << 20) + 24 * (M * K + N * K + 64 * (M + N + K)))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N + K)
    planes = lambda *n: (torch.randn(*n, generator=gen, device="cuda"), torch.randn(*n, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())

    def near(got, want, acc, spread):
        # two parts of 22 bits; as FMAs 1.8e-8 of the root of K; 1.3 times that for a mean over few values
        tol = 1.3 * (2.4e-7 + (1.8e-8 * K ** 0.5 if spread else chains[acc]))
        err = float((full(got) - want).norm() / want.norm())
        assert err < tol, (err, tol)

    for spread in (0, 40):                               # with rows 2^40 apart the product runs as FMAs
        x, w, r, g = planes(M, K), planes(N, K), planes(M, N), planes(M, N)
        if spread:
            x[0][M // 2] *= 2.0 ** -spread
            x[1][M // 2] *= 2.0 ** -spread
        X, W, G = full(x), full(w), full(g)
        near(ctx.linear_fwd(x, w), X @ W.T, 0, spread)
        near(ctx.linear_fwd(x, w, res=r), X @ W.T + full(r), 0, spread)
        # the same sizes as gradients: of x ([M, K] @ [K, N]) and of w, both added to what is there
        near(ctx.linear_bwd_x(x, tuple(t.T.contiguous() for t in w), out=tuple(t.clone() for t in r)), X @ W.conj().T + full(r), 1, spread)
        near(ctx.linear_bwd_w(tuple(t.T.contiguous() for t in x), tuple(t.T.contiguous() for t in w), out=tuple(t.clone() for t in r)),
             X @ W.conj().T + full(r), 1, spread)
    assert lib.cnb_check_device_status(ctx.h, ctx._stream()) == 0


@pytest.mark.parametrize("M,N,K,acc,former", [
    # a shorter first chain: cut, though the longest run is a single chain
    (785, 1218, 616, 1, 1.0849e-06),
    (282, 2355, 696, 1, 1.1950e-06),
    (280, 2320, 640, 0, 1.0843e-06),
    (1136, 1008, 1008, 0, 1.7386e-06),
    # as many cubes in other runs
    (1820, 552, 163, 1, 1.1584e-07),
    (2622, 482, 206, 0, 1.1640e-07),
    (450, 591, 144, 0, 2.8908e-07),
])
def test_no_further_off_than_the_former_schedule(M, N, K, acc, former):
    """Sums in another order than runs of pairs, summed with atomics, had: `former` is what those were off float64 by on these inputs."""
    import torch
    ctx = Context(arena_bytes=(64 << 20) + 24 * (M * K + N * K + 64 * (M + N + K)))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000003 + M * 31 + N * 17 + K)
    planes = lambda *n: (torch.randn(*n, generator=gen, device="cuda"), torch.randn(*n, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    a, b = planes(M, K), planes(K, N) if acc else planes(N, K)
    if acc:
        got = ctx.linear_bwd_x(a, b, out=(torch.zeros(M, N, device="cuda"), torch.zeros(M, N, device="cuda")))
        want = full(a) @ full(b).conj()
    else:
        got, want = ctx.linear_fwd(a, b), full(a) @ full(b).T
    err = float((full(got) - want).norm() / want.norm())
    assert err <= 1.002 * former, (err, former)          # (atomics add in any order)
