"""The skinny Linear forward on either side of its line between rows over threads and a staged W: one row and two rows
per CTA, an odd last row, rows shorter and longer than a CTA's threads take at once, every bound of the outputs."""
import numpy as np
import pytest

import util
from test_kernels_gpu import _c, _dev, _host, _pair, _rand, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 296, 297, 511, 512, 513])
@pytest.mark.parametrize("n_in,n_out", [(32, 1), (33, 4), (256, 5), (784, 10), (1024, 8), (1027, 9), (1500, 16)])
def test_skinny_forward(ctx, B, n_in, n_out):  # noqa: F811
    rng = np.random.default_rng(B + n_in)
    x, w = _rand(rng, B, n_in), _rand(rng, n_out, n_in, scale=n_in ** -0.5)
    y = _host(ctx.linear_fwd(_dev(x), _dev(w)))
    assert ctx.last_gemm_engine() == 4
    # fp32 sums of at most 2 * 1500 products: 2^-24 a rounding, some sqrt(3000) of them along a chain
    assert util.relerr(y, _pair(_c(x) @ _c(w).T)) < 2.0 ** -24 * 3000 ** 0.5
