"""How the chains of a product are added up: the difference of a chain's two accumulators is rounded at the chain's magnitude."""
import pytest

from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


# sizes whose chains are few, of one or two blocks, or summed by single CTAs
@pytest.mark.parametrize("M,N,K", [(5003, 2100, 399),          # whole tiles by pairs that stay, chains of two blocks
                                   (130, 30000, 1001),         # whole tiles by single CTAs, chains of four
                                   (777, 1001, 399)])          # shared runs
def test_accumulators_that_cancel(M, N, K):
    """1 in the first chain; in a later one A_re B_re = A_im B_im = 2^26, exact in tensor memory: their difference is 0, and 1
    stays 1.  Added to the running sum one after the other, the first takes it to 2^26 and the second to 0."""
    import torch
    ctx = Context(arena_bytes=(64 << 20) + 24 * (M * K + N * K + 64 * (M + N + K)))
    planes = lambda r: (torch.zeros(r, K, device="cuda"), torch.zeros(r, K, device="cuda"))
    x, w = planes(M), planes(N)
    for p in (x[0], w[0]):
        p[:, 0] = 1
    for p in x + w:
        p[:, 300] = 2.0 ** 13                                 # (chains of 64 and 128 products at these sizes)
    y = ctx.linear_fwd(x, w)
    assert ctx.last_gemm_engine() == 1
    assert bool((y[0] == 1).all()) and bool((y[1] == 2.0 ** 27).all())


# ragged sizes, whose chains are as short as fp32 FMAs make them: a dozen roundings of running sums are seen beside the chains'
@pytest.mark.parametrize("M,N,K,bound", [
    (466, 2805, 97, 1.16e-7),          # 1.14e-7; 1.19e-7 with the accumulators added one by one
    (2297, 1147, 500, 2.32e-7),        # 2.30e-7; 2.34e-7
    (777, 1001, 1333, 4.50e-7),        # pairs: shorter chains, added one by one, 3.75e-7
    (5273, 857, 785, 3.45e-7),         # 3.38e-7 in chains of three; of two, one by one, 2.7e-7
])
def test_no_further_off_than_with_one_rounding_a_chain(M, N, K, bound):
    import torch
    ctx = Context(arena_bytes=(64 << 20) + 24 * (M * K + N * K + 64 * (M + N + K)))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N + K)
    planes = lambda *n: (torch.randn(*n, generator=gen, device="cuda"), torch.randn(*n, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    x, w = planes(M, K), planes(N, K)
    y, want = full(ctx.linear_fwd(x, w)), full(x) @ full(w).T
    assert ctx.last_gemm_engine() == 1
    assert float(torch.linalg.vector_norm(y - want) / torch.linalg.vector_norm(want)) < bound
