"""How a transform of mixed radices is launched (cnb_fft_form: host arithmetic, no GPU), at the registers that the kernels have here."""
import ctypes as C

import pytest

from cnet_b200 import lib as L
from test_gemm_schedule import SMS


def _form(B, N, tail):
    out = (C.c_int * 4)()
    assert L.load().cnb_fft_form(N, B, tail, SMS, 108 if tail else 96, 80, out) == 0
    return dict(zip(("ctas", "threads", "loop", "fewer"), out))


@pytest.mark.parametrize("B,N,tail,fewer", [
    (2282, 396, 0, 1), (4096, 784, 0, 1), (2000, 2000, 0, 1),
    (500, 900, 0, 0), (4096, 512, 0, 0),                     # no wave saved
    (2500, 1600, 0, 0), (39267, 50, 0, 0), (12361, 208, 0, 0), (1605, 2048, 0, 0),       # five CTAs to an SM where there were four
    (1000, 1500, 1, 1), (4096, 784, 1, 1), (2000, 2000, 1, 1), (28360, 32, 1, 1), (19809, 117, 1, 0),
    (47095, 50, 1, 0), (82001, 50, 1, 0), (48007, 72, 1, 0), (64750, 49, 1, 0), (40000, 100, 1, 0), (12361, 208, 1, 0),
])
def test_fewer_registers_where_they_are_faster(B, N, tail, fewer):
    assert _form(B, N, tail)["fewer"] == fewer


def test_no_form_for_what_has_no_kernel():
    out = (C.c_int * 4)()
    assert L.load().cnb_fft_form(1, 16, 0, SMS, 96, 80, out) < 0
    assert L.load().cnb_fft_form(100, 0, 0, SMS, 96, 80, out) < 0


@pytest.mark.parametrize("B,N,loop", [
    (16, 256, 1), (296, 500, 1), (512, 784, 1), (359, 273, 1),
    (4096, 512, 0), (86, 2000, 0),                       # half a million elements, more than 1024 points
])
def test_the_tail_in_a_loop(B, N, loop):
    assert _form(B, N, 1)["loop"] == loop
