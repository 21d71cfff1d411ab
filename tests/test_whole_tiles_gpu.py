"""Products on packed operands whose CTAs go through several tiles or cut long runs into chains: whole tiles by persistent
CTAs and CTA pairs, a remainder that is nearly a wave, segments of a long K, each with remainders in every size."""
import ctypes as C

import pytest

from cnet_b200 import lib as L
from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


def _schedule(M, N, K):
    import torch
    out = (C.c_int * 8)()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert L.load().cnb_gemm_schedule_packed(M, N, K, 0, sms, 0, out) == 0
    return dict(zip(("pair", "ctas", "cluster_ctas", "run", "whole_per_cta", "segments", "atomics", "clear_from_row"), out))


# kind: what the schedule must be for the case to test it (on 148 SMs)
@pytest.mark.parametrize("M,N,K,kind", [
    (4000, 1001, 72, "whole"),         # pairs, two tiles each and one for some: nearly a wave left over
    (5003, 2100, 40, "whole"),         # pairs, more than four waves of tiles, a chain of two blocks
    (200, 38001, 65, "whole"),         # single CTAs, rows that are not 16-byte aligned
    (1000, 2050, 4104, "whole"),       # K > 4096, one wave of tiles: chains of a long K
    (130, 1030, 9000, "segments"),     # K > 4096, segments of several chains, single CTAs
    (700, 515, 8200, "segments"),      # the same by pairs
    (300, 140, 4800, "runs"),          # short runs
])
def test_products_of_several_tiles_and_chains(M, N, K, kind):
    import torch
    s = _schedule(M, N, K)
    assert s["pair"] == (M >= 256), s
    assert {"whole": s["whole_per_cta"] > 0 and not s["atomics"], "segments": s["segments"] > 0, "runs": not s["whole_per_cta"]}[kind], s
    ctx = Context(arena_bytes=(64 << 20) + 24 * (M * K + N * K + 64 * (M + N + K)))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N + K)
    planes = lambda *n: (torch.randn(*n, generator=gen, device="cuda"), torch.randn(*n, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    off = lambda y, want: float(torch.linalg.vector_norm(full(y) - want) / torch.linalg.vector_norm(want))
    # what the tensor core loses in a chain of at most 1024 products (4.2e-9 each, cgemm_tc.cu) and the operands' 22 bits, twice
    tol = 2 * (4.2e-9 * min(K, 1024) + 2.0 ** -22)
    x, w, r = planes(M, K), planes(N, K), planes(M, N)
    want = full(x) @ full(w).T
    assert off(ctx.linear_fwd(x, w), want) < tol
    assert off(ctx.linear_fwd(x, w, res=r), want + full(r)) < tol
    g = planes(K, M)                                         # dW* [M, N] = sum over K rows, on top of what is there
    xt = planes(K, N)
    out = (r[0].clone(), r[1].clone())
    ctx.linear_bwd_w(g, xt, out=out)
    assert off(out, full(r) + full(g).T @ full(xt).conj()) < tol
    again = ctx.linear_fwd(x, w)                             # the barriers' phases start over with every launch
    first = ctx.linear_fwd(x, w)
    if not s["atomics"]:
        assert torch.equal(again[0], first[0]) and torch.equal(again[1], first[1])


@pytest.mark.parametrize("M,N,K", [(4096, 1024, 128), (4096, 1024, 512), (3840, 1152, 256), (4096, 1024, 768)])
def test_whole_tiles_that_used_to_be_shared_are_no_further_off(M, N, K):
    """Two chains: 4.2e-9 (cgemm_tc.cu) of half the products, and the operands' 22 bits.  As one chain K = 512 was 1.83e-6 off."""
    import torch
    s = _schedule(M, N, K)
    assert s["whole_per_cta"] == 2 and not s["atomics"], s
    ctx = Context(arena_bytes=(64 << 20) + 24 * (M * K + N * K + 64 * (M + N + K)))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K)
    planes = lambda *n: (torch.randn(*n, generator=gen, device="cuda"), torch.randn(*n, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    x, w = planes(M, K), planes(N, K)
    y, want = full(ctx.linear_fwd(x, w)), full(x) @ full(w).T
    assert float(torch.linalg.vector_norm(y - want) / torch.linalg.vector_norm(want)) < 4.2e-9 * K / 2 + 2.0 ** -23


@pytest.mark.parametrize("M,N,K,before", [(4089, 1019, 777, 3.357e-7), (3321, 1275, 250, 2.218e-7), (3577, 1915, 1001, 4.444e-7), (5113, 1275, 500, 2.298e-7)])
def test_whole_tiles_of_ragged_sizes_are_no_further_off_than_shared_runs(M, N, K, before):
    """`before`: measured with the remainder of tiles in shared runs (the same distributions; a million values and more, which
    puts the figure down to a part in a thousand)."""
    import torch
    s = _schedule(M, N, K)
    assert s["whole_per_cta"] > 1 and not s["atomics"], s
    ctx = Context(arena_bytes=(64 << 20) + 24 * (M * K + N * K + 64 * (M + N + K)))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K)
    planes = lambda *n: (torch.randn(*n, generator=gen, device="cuda"), torch.randn(*n, generator=gen, device="cuda"))
    full = lambda a: torch.complex(a[0].double(), a[1].double())
    x, w = planes(M, K), planes(N, K)
    y, want = full(ctx.linear_fwd(x, w)), full(x) @ full(w).T
    assert float(torch.linalg.vector_norm(y - want) / torch.linalg.vector_norm(want)) < 1.003 * before
