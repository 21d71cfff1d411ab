"""FourierTrans with its fused tail (Hadamard, CGelu): the tail in a loop over shared memory and by the threads of the last
butterflies, on both sides of the line between them, at one pass and several, in the chirp form, on planes of any alignment."""
import pytest

from test_kernels_gpu import ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,offset", [
    (1, 2, 0), (3, 7, 0), (5, 16, 0),          # one pass
    (1, 256, 0), (33, 100, 0), (300, 77, 1),   # several rows to a CTA
    (9, 784, 0), (700, 748, 0), (702, 748, 0),  # up to half a million elements, and more
    (5, 17, 0), (40, 137, 1), (1900, 137, 0), (1920, 137, 0),     # chirp form, both sides
    (4, 1009, 0), (4, 1031, 0), (5, 2048, 0),  # both sides of 1024 points
    (1, 1024, 0), (31, 1024, 0), (1300, 1024, 0), (31, 1024, 1),  # its own kernel; planes of 4-byte alignment
])
@pytest.mark.parametrize("keep", [False, True])
def test_tail(ctx, B, N, offset, keep):  # noqa: F811
    import torch
    if keep and N == 1024:
        pytest.skip("the product is not stored at 1024 points")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B * N)

    def plane(*n):
        size = 1
        for k in n:
            size *= k
        return torch.randn(size + 4, generator=gen, device="cuda")[offset:offset + size].view(*n)
    x, h = (plane(B, N), plane(B, N)), (plane(N), plane(N))

    def result(at):
        return tuple(torch.full((B * N + 4,), float("nan"), device="cuda")[at:at + B * N].view(B, N) for _ in range(2))
    # the transform at the offset only where its own kernel does not want 16 bytes
    u, a, y = result(0 if N == 1024 else offset), result(offset), result(offset)
    if N == 1024:
        x = tuple(t.clone() for t in x)
    p = lambda t: t.data_ptr()
    rc = ctx.lib.cnb_dft_hadamard_gelu_fwd_keep(ctx.h, p(x[0]), p(x[1]), p(h[0]), p(h[1]), p(u[0]), p(u[1]), p(a[0]) if keep else None,
                                                p(a[1]) if keep else None, p(y[0]), p(y[1]), None, B, N, ctx._stream())
    assert rc == 0
    U = torch.fft.fft(torch.complex(x[0].double(), x[1].double()), norm="ortho")
    A = U * torch.complex(h[0].double(), h[1].double())
    gelu = lambda t: torch.nn.functional.gelu(t, approximate="tanh")
    Y = torch.complex(gelu(A.real), gelu(A.imag))
    # rounding of log2(N) passes (three times that in the chirp form), magnitudes of 1: well below 1e-6
    for got, want in ((u, U), (y, Y)) + (((a, A),) if keep else ()):
        err = float((torch.complex(got[0].double(), got[1].double()) - want).norm() / want.norm())
        assert err < 1e-6, err
