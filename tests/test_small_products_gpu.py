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
        tol = 4 * 1.8e-8 * K ** 0.5 + 2.4e-7             # four times what rounded sums of K products show; a few roundings
        if ctx.lib.cnb_arena_size(ctx.h) > 1 << 20:
            tol += 4.2e-9 * K + 2.0 ** -21               # or the tensor core's chains and the operands' 22 bits
        assert off(ctx.linear_fwd(x, w), full(x) @ full(w).T) < tol
        assert off(ctx.linear_fwd(x, w, res=r), full(x) @ full(w).T + full(r)) < tol
        out = (r[0].clone(), r[1].clone())
        ctx.linear_bwd_x(x, wt, out=out)
        assert off(out, full(r) + full(x) @ full(wt).conj()) < tol
        out = (r[0].clone(), r[1].clone())
        ctx.linear_bwd_w(g, xt, out=out)
        assert off(out, full(r) + full(g).T @ full(xt).conj()) < tol
