"""Linear layers of few outputs at every number of them: weights requested without asking which outputs exist, sums that share
shuffles, weight gradients written out four outputs at a time."""
import pytest

from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_out", range(1, 17))
@pytest.mark.parametrize("B,n_in", [(5, 1025), (310, 260), (700, 132)])     # a row a CTA, two rows, W staged; 4-byte and 16-byte rows
def test_every_number_of_outputs(B, n_in, n_out):
    import torch
    ctx = Context(arena_bytes=64 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B + n_in + n_out)
    pair = lambda *n: tuple(torch.randn(*n, generator=gen, device="cuda") for _ in range(2))
    full = lambda t: torch.complex(t[0].double(), t[1].double())
    x, w, g = pair(B, n_in), pair(n_out, n_in), pair(B, n_out)
    X, W, G = full(x), full(w), full(g)
    for got, want, k in ((ctx.linear_fwd(x, w), X @ W.T, n_in), (ctx.linear_bwd_x(g, w), G @ W.conj(), n_out),
                         (ctx.linear_bwd_w(g, x), G.T @ X.conj(), B)):
        assert torch.isfinite(got[0]).all() and torch.isfinite(got[1]).all()
        # at most K rounded terms, one after the other
        assert float((full(got) - want).norm() / want.norm()) < 6e-8 * (2 + k ** 0.5)
