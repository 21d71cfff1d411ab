"""Products of matrices whose rows or columns differ in scale by more than two fp16 parts hold: every row (forward, dX*) and
every column (dW*) of the result keeps its own relative precision, under every schedule and form of the tile kernel."""
import numpy as np
import pytest

import util
from cnet_b200 import configs
from cnet_b200.net import Net
from oracle import cnet_oracle as co
from test_kernels_gpu import _c, _dev, _host, _rand, ctx  # noqa: F401

pytestmark = pytest.mark.gpu

# per row or column by itself: 22-bit operands (2^-22), fp32 sums of at most 4096 products (2^-22 at worst), and what a
# line's own norm lies below the norms of what went into it (balanced lines: a factor of two)
TOL = 2.0 ** -18


def _scaled(pair, exponents, axis):
    s = np.exp2(np.asarray(exponents, np.float64)).astype(np.float32)
    return tuple((p * (s[:, None] if axis == 0 else s[None, :])).astype(np.float32) for p in pair)


def _err(got, want, axis):
    """the worst relative error of a row (axis 1) or of a column (axis 0)"""
    z = got[0].astype(np.float64) + 1j * got[1]
    return (np.linalg.norm(z - want, axis=axis) / np.linalg.norm(want, axis=axis)).max()


@pytest.mark.parametrize("B,n_in,n_out", [
    (256, 320, 192),      # clusters
    (512, 1024, 1024),    # clusters of four
    (4096, 256, 1024),    # CTA pairs, whole tiles
    (300, 1001, 130),     # nothing a multiple of anything
    (2500, 520, 1064),    # pairs with a part-empty tile, stream-K remainder
    (83, 9000, 102),      # capped chains
    (500, 900, 26),       # fewer outputs than a tile has rows
])
def test_lines_of_any_scale(ctx, B, n_in, n_out):  # noqa: F811
    rng = np.random.default_rng(B + n_out)
    x, w, g, r = _rand(rng, B, n_in), _rand(rng, n_out, n_in), _rand(rng, B, n_out), _rand(rng, B, n_out)
    # one line at 2^-60, one at 2^-25, the others between 2^-16 and 1
    span = lambda n: np.concatenate([[0, -60, -25], rng.uniform(-16, 0, n - 3)])  # noqa: E731
    xs, gs, ws, wt = _scaled(x, span(B), 0), _scaled(g, span(B), 0), _scaled(w, span(n_out), 0), _scaled(w, span(n_in), 1)
    dev = {k: _dev(v) for k, v in dict(x=x, w=w, g=g, r=r, xs=xs, gs=gs, ws=ws, wt=wt).items()}
    assert _err(_host(ctx.linear_fwd(dev["xs"], dev["w"])), _c(xs) @ _c(w).T, 1) < TOL
    assert ctx.last_gemm_engine() == 1
    assert _err(_host(ctx.linear_fwd(dev["x"], dev["ws"])), _c(x) @ _c(ws).T, 0) < TOL
    assert _err(_host(ctx.linear_fwd(dev["xs"], dev["ws"])), _c(xs) @ _c(ws).T, 1) < TOL
    assert _err(_host(ctx.linear_bwd_x(dev["gs"], dev["w"])), _c(gs) @ _c(w).conj(), 1) < TOL
    assert _err(_host(ctx.linear_bwd_x(dev["g"], dev["wt"])), _c(g) @ _c(wt).conj(), 0) < TOL
    gc, xc = _scaled(g, span(n_out), 1), _scaled(x, span(n_in), 1)
    assert _err(_host(ctx.linear_bwd_w(_dev(gc), dev["x"])), _c(gc).T @ _c(x).conj(), 1) < TOL
    assert _err(_host(ctx.linear_bwd_w(dev["g"], _dev(xc))), _c(g).T @ _c(xc).conj(), 0) < TOL
    # with a residual, and added to what is there
    want = _c(xs) @ _c(w).T + _c(r)
    assert _err(_host(ctx.linear_fwd(dev["xs"], dev["w"], res=dev["r"])), want, 1) < TOL
    acc = _dev(x)
    want = _c(gs) @ _c(w).conj() + _c(x)
    assert _err(_host(ctx.linear_bwd_x(dev["gs"], dev["w"], out=acc)), want, 1) < TOL


def test_one_huge_gradient_row(ctx):  # noqa: F811
    """A row of G 2^40 above the others (a loss near zero on one sample) whose inputs are zero in half of the features:
    dW* of these features comes from the other rows alone."""
    rng = np.random.default_rng(11)
    x, g = _rand(rng, 256, 320), _rand(rng, 256, 192)
    for p in x:
        p[7, :160] = 0
    for p in g:
        p[7] *= 2.0 ** 40
    want = _c(g).T @ _c(x).conj()
    got = _host(ctx.linear_bwd_w(_dev(g), _dev(x)))
    assert _err(tuple(p[:, :160] for p in got), want[:, :160], 0) < TOL
    assert _err(tuple(p[:, 160:] for p in got), want[:, 160:], 0) < TOL


@pytest.mark.parametrize("exponent", [-126, -115, -90, 60])
def test_whole_matrix_scale(ctx, exponent):  # noqa: F811
    rng = np.random.default_rng(12)
    x, w = _scaled(_rand(rng, 128, 256), [exponent] * 128, 0), _rand(rng, 192, 256)
    # the largest component is about 4 * 2^exponent; below 2^-126 fp32 itself has no 24 bits
    bound = TOL if exponent > -120 else 2.0 ** -14
    assert _err(_host(ctx.linear_fwd(_dev(x), _dev(w))), _c(x) @ _c(w).T, 1) < bound


def test_zero_lines_and_lone_elements(ctx):  # noqa: F811
    """Lines of zeros have no scale; a lone tiny element in an otherwise balanced line is within its line's precision."""
    rng = np.random.default_rng(13)
    x, w = _rand(rng, 200, 320), _rand(rng, 192, 320)
    for p in x:
        p[5] = 0
        p[:, 17] = 0
        p[9, 30] = 1e-30
    y = _host(ctx.linear_fwd(_dev(x), _dev(w)))
    want = _c(x) @ _c(w).T
    assert not y[0][5].any() and not y[1][5].any()
    keep = np.arange(200) != 5
    assert _err(tuple(p[keep] for p in y), want[keep], 1) < TOL


@pytest.mark.parametrize("B,n_in,n_out", [(480, 256, 128), (480, 250, 37),
                                          (160, 250, 37), (160, 250, 10)])     # SIMT tiles, skinny kernels
def test_net_with_rows_of_any_scale(B, n_in, n_out):
    """Through Net, in a captured step: the form is chosen on the device, for each batch anew, and every kernel reads what
    the kernel before it wrote for this batch."""
    import torch
    dev, ora = Net(), co.OracleNet()
    sd, so = configs.build_linear(dev, n_in, n_out), configs.build_linear(ora, n_in, n_out)
    for uid, (re, im) in configs.init_weights(sd, 3).items():
        dev.set_values(uid, re, im)
        ora.set_values(uid, re, im)
    stream = torch.cuda.Stream()
    dev.allocate(B, stream=stream.cuda_stream)
    x, labels = configs.make_batch(sd, B, 1, kind="fanin")
    rng = np.random.default_rng(4)
    wide = _scaled(x, np.concatenate([[0, -40], rng.uniform(-30, 0, B - 2)]), 0)
    pin = lambda t: tuple(torch.from_numpy(p).pin_memory() for p in t)  # noqa: E731
    lab = torch.from_numpy(labels).pin_memory()
    dev.upload(x=pin(x), labels=lab)
    dev.forward()
    dev.backward()
    dev.update_inputs(0.0)
    dev.sync()
    dev.capture_begin()
    dev.forward()
    dev.backward()
    dev.update_inputs(0.0)
    dev.capture_end()
    lin = sd.layers["lin"]
    for batch in (wide, x, wide):
        ora.zero_wgrads()
        ora.run_batch(so.main, x=batch, labels=labels)
        dev.upload(x=pin(batch), labels=lab)
        dev.graph_launch()
        dev.sync()
        want = ora.act[so.layers["lin"]]
        assert _err(dev.get_record(lin, 0), want, 1) < TOL
        # a row's gradient goes with 1 / z: the label's component carries z's error times |z| / |z_l|
        z, k = np.abs(want), np.arange(B)
        spread = np.linalg.norm(want, axis=1) / z[k, labels]
        got, dx = dev.get_record(sd.layers["x"], 1), ora.gstar[so.layers["x"]]
        err = np.linalg.norm(got[0] + 1j * got[1].astype(np.float64) - dx, axis=1) / np.linalg.norm(dx, axis=1)
        assert (err < TOL * np.maximum(1, spread)).all(), err.max()
    assert util.relerr(dev.get_values(sd.layers["w"]), ora.get_values(so.layers["w"])) == 0


@pytest.mark.parametrize("rows,cols", [(33, 900), (65, 129), (97, 257), (4097, 130), (32, 128), (500, 1025)])
def test_remainders_are_not_mistaken_for_small_lines(ctx, rows, cols):  # noqa: F811
    """Values of a CGelu of heavy-tailed products, of which many lone ones are tiny: at sizes one beyond a group the
    matrix is still packed, not kept plain."""
    import torch
    rng = np.random.default_rng(rows + cols)
    a = _c(_rand(rng, rows, cols)) * _c(_rand(rng, rows, cols)) * 2
    y = tuple(co._gelu(p).astype(np.float32) for p in (a.real, a.imag))
    pack = torch.zeros(ctx.lib.cnb_pack_bytes(rows, cols) // 4, device="cuda")
    d = _dev(y)
    assert ctx.lib.cnb_pack_matrix(ctx.h, d[0].data_ptr(), d[1].data_ptr(), rows, cols, pack.data_ptr(), 0, ctx._stream()) == 0
    assert pack[:1].view(torch.int32).item() < 1 << 20
