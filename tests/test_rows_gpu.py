"""Row reductions at the edges of their forms: lanes per row, 16-byte and single accesses, clusters, the two-pass kernels
beyond them; rows that leave the last group of a warp or CTA empty."""
import numpy as np
import pytest

import util
from test_kernels_gpu import _c, _dev, _host, _pair, _rand, ctx  # noqa: F401

pytestmark = pytest.mark.gpu

# a sum of M products in fp32 over a tree: about log2(M) + M / (threads) roundings of 2^-24, then three more
TOL = 2e-6


@pytest.mark.parametrize("B,M", [(1, 1), (33, 7), (70, 32), (9, 33), (17, 128), (5, 129), (11, 512), (3, 513), (4, 2047), (2, 2048), (3, 2052),
                                 (2, 8192), (3, 8193), (2, 16388), (1, 32770), (2, 65536), (1, 65537)])
def test_row_forms(ctx, B, M):  # noqa: F811
    import torch
    rng = np.random.default_rng(M)
    z, g = _rand(rng, B, M), _rand(rng, B, M)
    labels = rng.integers(0, M, B).astype(np.int32)
    labels[-1] = M - 1
    Z, G = _c(z), _c(g)
    n = np.sqrt((np.abs(Z) ** 2).sum(1, keepdims=True))
    y, inv = ctx.softmax_fwd(_dev(z))
    assert util.relerr(_host(y), _pair(Z / n)) < TOL
    assert util.relerr(inv.cpu().numpy(), 1 / n[:, 0]) < TOL
    # the gradient along z is taken out: of two terms of the size of G / n, what stays is at least a tenth of them here
    want = G / n - Z * (G * np.conj(Z)).sum(1, keepdims=True).real / n ** 3
    if M > 1:
        assert util.relerr(_host(ctx.softmax_bwd(_dev(g), _dev(z), inv)), _pair(want)) < 10 * TOL
    S = (np.abs(Z) ** 2).sum(1)
    zl = Z[np.arange(B), labels]
    m = np.abs(zl) ** 2
    d = Z / S[:, None]
    d[np.arange(B), labels] = -zl * (S - m) / (m * S)
    loss, dz = ctx.crossent(_dev(z), torch.from_numpy(labels).cuda())
    if M > 1:
        assert util.relerr(loss.cpu().numpy(), -np.log(m / S)) < 10 * TOL
        assert util.relerr(_host(dz), _pair(d)) < 10 * TOL
    # planes that are not 16-byte aligned take the single-access form
    pad = torch.zeros(2, B * M + 1, device="cuda")
    zz = tuple(pad[q, 1:].view(B, M) for q in range(2))
    for q in range(2):
        zz[q].copy_(torch.from_numpy(z[q]))
    y2, _ = ctx.softmax_fwd(zz)
    assert util.relerr(_host(y2), _pair(Z / n)) < TOL
    # L2Out
    out, dd = torch.empty(B, device="cuda"), ctx._new(B, M)
    zd = _dev(z)
    assert ctx.lib.cnb_l2out_fwd_bwd(ctx.h, zd[0].data_ptr(), zd[1].data_ptr(), out.data_ptr(), dd[0].data_ptr(), dd[1].data_ptr(),
                                     B, M, ctx._stream()) == 0
    assert util.relerr(out.cpu().numpy(), S) < TOL
    assert util.relerr(_host(dd), z) == 0.0
