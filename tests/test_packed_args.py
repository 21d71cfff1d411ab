"""Arguments that the packed and split products must refuse before they touch anything (no GPU: the pointers are not real)."""
import ctypes as C

import pytest

from cnet_b200 import lib as L

FAKE = 4096          # never dereferenced: every call here is refused by its argument checks


class Span(C.Structure):
    _fields_ = [("re", C.c_size_t), ("im", C.c_size_t), ("rows", C.c_int), ("cols", C.c_int), ("pack", C.c_void_p)]


@pytest.mark.parametrize("entry", ["cnb_linear_fwd_packed", "cnb_linear_fwd_split"])
@pytest.mark.parametrize("res", [(FAKE, None), (None, FAKE)])
def test_residual_planes_come_as_a_pair(entry, res):
    lib = L.load()
    assert getattr(lib, entry)(FAKE, FAKE, FAKE, *res, FAKE, FAKE, 128, 128, 128, None) < 0
    assert b"pair" in lib.cnb_last_error()


@pytest.mark.parametrize("re,im,rows,cols", [(0, 65, 8, 8), (65, 0, 8, 8), (0, 64, 16, 16), (0, 0, 0, 8), (2 ** 64 - 8, 0, 8, 8), (0, 2 ** 64 - 64, 8, 8),
                                             (0, 0, 65536, 65536)])
def test_matrices_lie_inside_the_arena(re, im, rows, cols):
    lib = L.load()
    span = Span(re, im, rows, cols, FAKE)
    assert lib.cnb_sgd_update_packed(FAKE, FAKE, FAKE, 128, 0.1, 1, C.byref(span), 1, None) < 0
    assert b"not inside the arena" in lib.cnb_last_error()
