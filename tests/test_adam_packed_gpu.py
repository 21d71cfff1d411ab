"""Adam's update that leaves matrices packed: the same update, and the same packs as packing them one by one; in a net, more
than one launch's worth of matrices."""
import ctypes as C

import pytest

from cnet_b200.ops import Context

pytestmark = pytest.mark.gpu


class Span(C.Structure):
    _fields_ = [("re", C.c_size_t), ("im", C.c_size_t), ("rows", C.c_int), ("cols", C.c_int), ("pack", C.c_void_p)]


@pytest.mark.parametrize("shapes", [[(3, 5)], [(17, 48), (64, 64), (33, 129)], [(8, 12)] * 35])
def test_packs_after_the_update(shapes):
    import torch
    ctx = Context(arena_bytes=16 << 20)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(len(shapes))
    n = sum(2 * r * c for r, c in shapes)
    w, m, g = (torch.randn(n, generator=gen, device="cuda") for _ in range(3))
    w1, m1, g1 = w.clone(), m.clone(), g.clone()
    stream = torch.cuda.current_stream().cuda_stream
    new = lambda r, c: torch.zeros(ctx.lib.cnb_pack_bytes(r, c), dtype=torch.uint8, device="cuda")
    packs = [new(r, c) for r, c in shapes]
    spans, at = (Span * len(shapes))(), 0
    for k, (r, c) in enumerate(shapes):
        spans[k] = Span(at, at + r * c, r, c, packs[k].data_ptr())
        at += 2 * r * c
    assert ctx.lib.cnb_adam_update_packed(ctx.h, w.data_ptr(), m.data_ptr(), g.data_ptr(), n, 0.01, 0.9, 3, spans, len(shapes), stream) == 0
    assert ctx.lib.cnb_adam_update(ctx.h, w1.data_ptr(), m1.data_ptr(), g1.data_ptr(), n, 0.01, 0.9, 3, stream) == 0
    for a, b in ((w, w1), (m, m1), (g, g1)):
        assert torch.equal(a, b)
    for s, p, (r, c) in zip(spans, packs, shapes):
        q = new(r, c)
        assert ctx.lib.cnb_pack_matrix(ctx.h, w[s.re:].data_ptr(), w[s.im:].data_ptr(), r, c, q.data_ptr(), 0, stream) == 0
        assert torch.equal(p, q)
    bad = Span(n, 0, 1, 1, packs[0].data_ptr())
    assert ctx.lib.cnb_adam_update_packed(ctx.h, w.data_ptr(), m.data_ptr(), g.data_ptr(), n, 0.01, 0.9, 3, C.byref(bad), 1, stream) < 0
    assert torch.equal(w, w1)
