"""FourierTrans at lengths whose buffers are spread and at others that are not, plain, adding and with the fused tail, at
batches of a CTA to an SM (more threads) and above, against float64."""
import pytest

from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [10, 16, 100, 256, 500, 784, 1000, 1500, 2500, 4096])
@pytest.mark.parametrize("rows", [1, 3, 149, 700])
def test_against_float64(n, rows):
    import torch
    ctx = Context(arena_bytes=32 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + rows)
    planes = lambda *s: (torch.randn(*s, generator=gen, device="cuda"), torch.randn(*s, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    off = lambda y, want: float(torch.linalg.vector_norm(full(y) - want) / torch.linalg.vector_norm(want))
    x, h = planes(rows, n), planes(n)
    want = torch.fft.fft(full(x), norm="ortho")
    tol = 2e-6                                               # some dozen roundings of 6e-8 an element, through three passes
    assert off(ctx.dft_fwd(x), want) < tol
    out = (x[0].clone(), x[1].clone())
    ctx.dft_bwd(x, out=out)
    assert off(out, full(x) + torch.fft.ifft(full(x), norm="ortho")) < tol
    y = (torch.empty_like(x[0]), torch.empty_like(x[0]))
    u = (torch.empty_like(x[0]), torch.empty_like(x[0]))
    p = lambda a: a.data_ptr()
    assert ctx.lib.cnb_dft_hadamard_gelu_fwd_keep(ctx.h, p(x[0]), p(x[1]), p(h[0]), p(h[1]), p(u[0]), p(u[1]), None, None, p(y[0]), p(y[1]),
                                                  None, rows, n, ctx._stream()) == 0
    assert off(u, want) < tol
    a = want * full(h)
    gelu = lambda v: 0.5 * v * (1 + torch.tanh(0.7978845608028654 * (v + 0.044715 * v ** 3)))
    assert off(y, torch.complex(gelu(a.real), gelu(a.imag))) < 2 * tol
