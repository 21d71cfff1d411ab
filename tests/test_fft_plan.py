"""The plans of the mixed-radix FourierTrans kernel (cnb_fft_plan: host arithmetic, no GPU): the passes they describe,
carried out in numpy with the kernel's index formulas, give the DFT, and every index stays inside its buffer."""
import ctypes as C

import numpy as np
import pytest

from cnet_b200 import lib as L


@pytest.fixture(scope="module")
def lib():
    return L.load()


def plan(lib, n, b, sms=148):
    out = (C.c_int * 12)()
    passes = lib.cnb_fft_plan(n, b, sms, out, 12)
    assert passes >= 0
    return dict(m=out[0], rows=out[1], threads=out[2], buffers=out[3], stride=out[4], smem=out[5], radices=list(out[6:6 + passes]))


def stockham(x, radices, stride):
    m, L_ = x.shape[-1], 1
    for r in radices:
        nb = m // r
        j = np.arange(nb)
        k = j % L_
        v = np.stack([x[..., j + q * nb] * np.exp(-2j * np.pi * k * q / (L_ * r)) for q in range(r)], axis=-1)
        v = v @ np.exp(-2j * np.pi * np.outer(np.arange(r), np.arange(r)) / r)
        x = np.empty_like(x)
        for q in range(r):
            at = (j - k) * r + k + q * L_
            assert at.max() < m and (at + (at >> 4)).max() < stride
            x[..., at] = v[..., q]
        L_ *= r
    assert L_ == m
    return x


@pytest.mark.parametrize("n", [2, 3, 13, 16, 17, 31, 64, 100, 117, 257, 500, 784, 900, 1000, 1024, 1237, 1500, 2048, 4096, 5003])
def test_plan_is_the_dft(lib, n):
    p = plan(lib, n, 3)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((2, n)) + 1j * rng.standard_normal((2, n))
    if p["m"] == n:
        y = stockham(x, p["radices"], p["stride"])
    else:
        m = p["m"]
        assert m >= 2 * n - 1
        c = np.exp(-1j * np.pi * (np.arange(n, dtype=np.int64) ** 2 % (2 * n)) / n)
        b = np.zeros(m, complex)
        b[:n] = np.conj(c)
        b[m - n + 1:] = np.conj(c[1:][::-1])
        pad = np.zeros((2, m), complex)
        pad[:, :n] = x * c
        t = stockham(pad, p["radices"], p["stride"]) * np.fft.fft(b) / m
        t = stockham(t.imag + 1j * t.real, p["radices"], p["stride"])
        y = (t.imag + 1j * t.real)[:, :n] * c
    assert np.abs(y - np.fft.fft(x, axis=1)).max() < 1e-9 * n


def test_launch_shapes_stay_within_the_device(lib):
    for n in list(range(2, 300)) + [784, 1500, 2048, 4093, 4096, 6000, 8192, 12000, 16384]:
        for b in (1, 7, 500, 100000):
            p = plan(lib, n, b)
            if not p["radices"]:
                assert n > 6000                          # only long rows have no kernel
                continue
            assert 1 <= p["rows"] and p["threads"] % 32 == 0 and 64 <= p["threads"] <= 256
            assert p["smem"] <= 224 * 1024 and p["smem"] >= 8 * p["buffers"] * p["rows"] * p["stride"]
            assert all(2 <= r <= 16 for r in p["radices"]) and np.prod(p["radices"]) == p["m"]
            # the reciprocal division of the kernel: rows * nb items, exact below 2^32 / divisor
            assert all(p["rows"] * (p["m"] // r) * (p["m"] // r) < 2 ** 32 for r in p["radices"])
