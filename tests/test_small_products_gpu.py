"""fp32 SIMT products at the edges of their tiles and slabs, every operand orientation, on top of a residual or of what is
there, against float64; and on both sides of the lines to larger tiles and to the tensor core."""
import pytest

from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (1, 17, 1), (16, 17, 31), (17, 33, 32), (33, 18, 33), (64, 64, 64), (20, 300, 65),     # tiles of 16
    (200, 190, 257), (1000, 40, 300),                                                      # more than an SM's worth, long K: 32
    (900, 517, 20), (1031, 1001, 19),                                                      # more than six to an SM: 32
    (200, 200, 200), (201, 200, 200), (128, 128, 256), (128, 128, 264),                    # about the line to the tensor core
])
def test_products(M, N, K):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N + K)
    planes = lambda *s: (torch.randn(*s, generator=gen, device="cuda"), torch.randn(*s, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    off = lambda y, want: float(torch.linalg.vector_norm(full(y) - want) / torch.linalg.vector_norm(want))
    x, w, r = planes(M, K), planes(N, K), planes(M, N)
    wt, g, xt = planes(K, N), planes(K, M), planes(K, N)
    for ctx in (Context(arena_bytes=1 << 20), Context(arena_bytes=64 << 20)):              # without room for packs, and with
        def close(y, want):
            # Twice what rounded sums of K products show, and the roundings of the last additions; where the tensor core took the
            # product, twice what it loses in its chains and by the operands' 22 bits.  (skinny kernels sum as FMAs do.)
            tol = 2 * 1.8e-8 * K ** 0.5 + 2.0 ** -23
            if ctx.last_gemm_engine() == 1:
                assert ctx.lib.cnb_arena_size(ctx.h) > 1 << 20
                tol = 2 * (4.2e-9 * K + 2.0 ** -22) + 2.0 ** -23
            e = off(y, want)
            assert e < tol, (e, tol, ctx.last_gemm_engine())
        close(ctx.linear_fwd(x, w), full(x) @ full(w).T)
        close(ctx.linear_fwd(x, w, res=r), full(x) @ full(w).T + full(r))
        out = (r[0].clone(), r[1].clone())
        ctx.linear_bwd_x(x, wt, out=out)
        close(out, full(r) + full(x) @ full(wt).conj())
        out = (r[0].clone(), r[1].clone())
        ctx.linear_bwd_w(g, xt, out=out)
        close(out, full(r) + full(g).T @ full(xt).conj())


@pytest.mark.parametrize("M,N,K", [(268, 117, 213), (49, 891, 124), (19, 1879, 209), (2310, 19, 126), (35, 520, 231), (900, 61, 97)])
def test_small_products_of_ragged_sizes_are_as_exact_as_in_chains(M, N, K):
    """The tensor core cuts these into chains of one or two blocks, 1.13e-7 to 2.5e-7 off float64; FMAs in sums of sixteen are
    1.12e-7 off at most up to K = 256 (the same roundings in numpy), one by one 1.9e-7 to 2.8e-7."""
    import torch
    ctx = Context(arena_bytes=64 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N + K)
    planes = lambda *s: (torch.randn(*s, generator=gen, device="cuda"), torch.randn(*s, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    off = lambda y, want: float(torch.linalg.vector_norm(full(y) - want) / torch.linalg.vector_norm(want))
    x, w, wt, g, xt = planes(M, K), planes(N, K), planes(K, N), planes(K, M), planes(K, N)
    for y, want in ((ctx.linear_fwd(x, w), full(x) @ full(w).T), (ctx.linear_bwd_x(x, wt), full(x) @ full(wt).conj()),
                    (ctx.linear_bwd_w(g, xt), full(g).T @ full(xt).conj())):
        assert off(y, want) < 1.16e-7
    assert ctx.last_gemm_engine() == 2


@pytest.mark.parametrize("M,N,K", [(1000, 500, 64), (1000, 500, 63), (1031, 1001, 65), (777, 1333, 95), (2000, 641, 80), (64, 9000, 128), (7103, 65, 79)])
def test_large_products_without_room(M, N, K):
    """Tiles of 64 x 64 (and K = 63, just below them), every operand orientation, on top of a residual or of what is there; the
    same bits as in smaller tiles, which take some of the rows alone."""
    import torch
    ctx = Context(arena_bytes=1 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N + K)
    planes = lambda *s: (torch.randn(*s, generator=gen, device="cuda"), torch.randn(*s, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    tol = 2 * 1.8e-8 * K ** 0.5 + 2.0 ** -23
    off = lambda y, want: float(torch.linalg.vector_norm(full(y) - want) / torch.linalg.vector_norm(want))
    x, w, r = planes(M, K), planes(N, K), planes(M, N)
    wt, g, xt = planes(K, N), planes(K, M), planes(K, N)
    copy = lambda: (r[0].clone(), r[1].clone())
    part = lambda a, k: (a[0][:k].contiguous(), a[1][:k].contiguous())
    few = min(M, 40)
    y = ctx.linear_fwd(x, w)
    assert ctx.last_gemm_engine() == 2 and off(y, full(x) @ full(w).T) < tol
    z = ctx.linear_fwd(part(x, few), w)
    assert torch.equal(y[0][:few], z[0]) and torch.equal(y[1][:few], z[1])
    assert off(ctx.linear_fwd(x, w, res=r), full(x) @ full(w).T + full(r)) < tol
    assert off(ctx.linear_bwd_x(x, wt, out=copy()), full(r) + full(x) @ full(wt).conj()) < tol
    assert off(ctx.linear_bwd_w(g, xt, out=copy()), full(r) + full(g).T @ full(xt).conj()) < tol
