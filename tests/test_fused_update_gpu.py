"""The fused FourierTrans tail reads the Hadamard vector that the update just before it in the stream has written."""
import numpy as np
import pytest

import util
from oracle import cnet_oracle as co
from test_kernels_gpu import _c, _dev, _host, _rand, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N", [(1, 13), (40, 16), (3, 127), (40, 784), (2000, 60), (300, 1024)])
def test_updated_vector_reaches_the_tail(ctx, B, N):  # noqa: F811
    import torch
    rng = np.random.default_rng(N)
    x, h, g = _rand(rng, B, N), _rand(rng, N), _rand(rng, N)
    flat = lambda p: torch.from_numpy(np.concatenate(p)).cuda()  # noqa: E731
    dx, dh, dg = _dev(x), flat(h), flat(g)
    hr, hi = dh.data_ptr(), dh.data_ptr() + 4 * N
    out = [(ctx._new(B, N), ctx._new(B, N)) for _ in range(8)]
    torch.cuda.synchronize()
    for u, y in out:
        assert ctx.lib.cnb_sgd_update(ctx.h, dh.data_ptr(), dg.data_ptr(), 2 * N, 0.5, 0, ctx._stream()) == 0
        assert ctx.lib.cnb_dft_hadamard_gelu_fwd(ctx.h, dx[0].data_ptr(), dx[1].data_ptr(), hr, hi, u[0].data_ptr(), u[1].data_ptr(),
                                                 y[0].data_ptr(), y[1].data_ptr(), None, B, N, ctx._stream()) == 0
    f = np.fft.fft(_c(x), axis=1) / np.sqrt(N)
    for k, (u, y) in enumerate(out):
        a = f * (_c(h) - 0.5 * (k + 1) * _c(g))
        assert util.relerr(_host(y), (co._gelu(a.real), co._gelu(a.imag))) < 2e-6, k
