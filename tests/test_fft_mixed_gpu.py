"""FourierTrans at lengths of the mixed-radix kernel against numpy's float64 FFT: one pass, two and more, primes up to
13 as radices, larger ones through the chirp form, the longest rows that fit, batches that leave the last CTA part
empty; plain, accumulating, and with the fused Hadamard -> CGelu tail."""
import numpy as np
import pytest

import util
from oracle import cnet_oracle as co
from test_kernels_gpu import _c, _dev, _host, _pair, _rand, ctx  # noqa: F401

pytestmark = pytest.mark.gpu

# A pass rounds every element a few times (a butterfly of 16 points is 4 additions deep, 2 more roundings in the
# twiddle product) at 2^-24 each, at random; 4 passes, 8 in the chirp form: 8 * sqrt(6) * 2^-24 * ~2 = 2e-6 at worst.
TOL = 2e-6


@pytest.mark.parametrize("B,N", [(1, 2), (5, 13), (300, 16), (7, 17), (1, 31), (129, 60), (1000, 64), (33, 127), (700, 143), (2, 500),
                                 (601, 784), (3, 1009), (4, 2048), (1, 4093), (299, 4096), (2, 6007), (1, 12000)])
def test_mixed_radix_lengths(ctx, B, N):  # noqa: F811
    rng = np.random.default_rng(B + N)
    x, h = _rand(rng, B, N), _rand(rng, N)
    f = np.fft.fft(_c(x), axis=1) / np.sqrt(N)
    b = np.fft.ifft(_c(x), axis=1) * np.sqrt(N)
    assert util.relerr(_host(ctx.dft_fwd(_dev(x))), _pair(f)) < TOL
    assert ctx.last_gemm_engine() in (3, 5)
    assert util.relerr(_host(ctx.dft_bwd(_dev(x))), _pair(b)) < TOL
    assert util.relerr(_host(ctx.dft_bwd(_dev(x), out=_dev(x))), _pair(b + _c(x))) < TOL
    u, split = ctx.dft_hadamard_gelu_fwd(_dev(x), _dev(h))
    assert util.relerr(_host(u), _pair(f)) < TOL
    a = f * _c(h)
    want = co._gelu(a.real), co._gelu(a.imag)
    # the split keeps the value to 2^-18 beside the transform's own error
    assert util.relerr(_unsplit(split, B, N), want) < TOL + 2.0 ** -18


def _unsplit(split, B, N):
    """hi + l16 of both planes of a split buffer."""
    import torch
    np_ = split.numel() // 4
    lo = split[3 * np_:].view(torch.bfloat16).float()
    return tuple((split[q * np_:(q + 1) * np_] + lo[q * np_:(q + 1) * np_])[:B * N].view(B, N).cpu().numpy() for q in range(2))
