"""A training step whose gradients are ill-conditioned, against float64 and beside the same step in fp32 FMAs.

The gradient of a sample's scores goes with 1 / z_l, z_l the score of its class, so where a z_l is small against its row's
other scores, every rounding of the forward pass comes back |z| / |z_l| times as large; an update of that size then moves the
weights by as much as they are, and after a few steps two correct fp32 implementations agree in a few digits only.  What can be
asked is that the step is no further from float64 than one whose products and transform are sums of fp32 FMAs."""
import numpy as np
import pytest

import util
from cnet_b200 import configs
from cnet_b200.net import Net
from cnet_b200.ops import Context
from oracle import cnet_oracle as co
from test_kernels_gpu import _dev, _host, ctx  # noqa: F401

pytestmark = pytest.mark.gpu

SEEDS = range(8)


def _fma_gradients(ctx, rest, x, h, w, labels, B, n, m):
    """dL/dh* and dL/dW* of the classifier, operator by operator; `ctx` has no room for packed operands and takes products as fp32 FMAs."""
    import torch
    X, H, W = _dev(x), _dev(h), _dev(tuple(p.reshape(m, n) for p in w))
    lab = torch.from_numpy(labels).cuda()
    u = ctx.dft_fwd(X)
    assert ctx.last_gemm_engine() == 2
    a, y = ctx.hadamard_gelu_fwd(u, H)
    z = ctx.linear_fwd(y, W)
    assert ctx.last_gemm_engine() == 2
    _, g = ctx.crossent(z, lab)
    dw = ctx.linear_bwd_w(g, y)
    _, dh = rest.hadamard_gelu_bwd(ctx.linear_bwd_x(g, W), a, u, H)
    return _host(dh), tuple(p.ravel() for p in _host(dw))


@pytest.mark.parametrize("B,n,m", [(500, 900, 26), (130, 250, 40)])
def test_first_gradients_beside_fp32(ctx, B, n, m):  # noqa: F811
    fma = Context(arena_bytes=(7 << 20) + 8 * n * n)         # the twiddle matrix, and too little for packed operands
    assert fma.lib.cnb_set_dft_engine(fma.h, 1) == 0
    ratio, bound = [], []
    for seed in SEEDS:
        dev, ora = Net(), co.OracleNet()
        sd, so = configs.build_classifier(dev, n=n, m=m), configs.build_classifier(ora, n=n, m=m)
        weights = configs.init_weights(sd, seed)
        for uid, (re, im) in weights.items():
            dev.set_values(uid, re, im)
            ora.set_values(uid, re, im)
        dev.allocate(B)
        x, labels = configs.make_batch(sd, B, seed)
        dev.run_batch(sd.main, x=x, labels=labels)
        ora.run_batch(so.main, x=x, labels=labels)
        want = [ora.get_wgrad(so.layers[k]) for k in ("h", "w")]
        got = [dev.get_wgrad(sd.layers[k]) for k in ("h", "w")]
        ref = _fma_gradients(fma, ctx, x, weights[sd.layers["h"]], weights[sd.layers["w"]], labels, B, n, m)
        err, err32 = (max(util.relerr(a, b) for a, b in zip(v, want)) for v in (got, ref))
        z = np.abs(ora.act[so.layers["lin"]])
        spread = (np.linalg.norm(z, axis=1) / z[np.arange(B), labels]).max()
        print("seed %d: %.2e, in FMAs %.2e, |z| / |z_l| up to %.0f" % (seed, err, err32, spread))
        ratio.append(err / err32)
        # forward: 2^-22 a product and as much a sum of up to 900; the same twice more on the way back
        bound.append(err / (3 * 2.0 ** -21 * spread))
    assert max(bound) < 1, bound
    assert np.exp(np.mean(np.log(ratio))) < 1, ratio
    fma.close()
