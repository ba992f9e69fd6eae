"""The line transforms as the engines run them (psg_fft.cuh, psg_fft2.cuh): plain and
with the twiddles merged into the butterflies, FP64, FP32 and two FP32 lines packed,
against 80-bit transforms.

Tolerances: a line's RMS error is some sqrt(log2 N) roundings, 4 eps at most (eps
2^-53, 2^-24); and the merged form may not err by more than the plain one whose place
it takes, in the RMS over 301 random lines."""
import ctypes as C

import numpy as np
import pytest

import psgpu_b200 as P

pytestmark = pytest.mark.gpu

PLAIN, MERGED, PACKED, PACKED_MERGED, PACKED_MERGED_WIDE = range(5)


def _lines(n, prec, lines=301):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((lines, n)) + 1j * rng.standard_normal((lines, n))
    return x.astype(np.complex64).astype(np.complex128) if prec == 32 else x


def _run(n, sign, swap, form, prec, x):
    y = np.zeros_like(x)
    dp = C.POINTER(C.c_double)
    L = P.lib()
    assert L.psg_debug_line_form(n, sign, swap, form, prec, x.ctypes.data_as(dp), y.ctypes.data_as(dp), len(x)) == 0, \
        L.psg_last_error()
    return y


def _rms(y, ref):
    return float(np.sqrt((np.abs(y - ref) ** 2).sum() / (np.abs(ref) ** 2).sum()))


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("sign,swap", [(1, 0), (-1, 0), (-1, 1)])
@pytest.mark.parametrize("prec", [64, 32])
def test_line_forms(n, sign, swap, prec):
    x = _lines(n, prec)
    xl = x.astype(np.clongdouble)
    ref = np.fft.fft(xl, axis=1) if sign < 0 else np.fft.ifft(xl, axis=1) * n
    assert ref.dtype == np.clongdouble
    eps = 2.0 ** (-53 if prec == 64 else -24)
    plain = _rms(_run(n, sign, swap, PLAIN, prec, x), ref)
    assert plain < 4 * eps
    forms = [MERGED] if prec == 64 else [PACKED, MERGED, PACKED_MERGED, PACKED_MERGED_WIDE]
    got = {f: _rms(_run(n, sign, swap, f, prec, x), ref) for f in forms}
    assert got.pop(PACKED, plain) < 4 * eps
    for f, e in got.items():
        assert e <= plain, (f, e / eps, plain / eps)


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256])
def test_the_quarter_turn(n):
    """a line with one nonzero point: each output is that point times a root of unity,
    so every single factor of the merged tables is seen (1.5 eps a factor, at most
    eight factors in a row, 12 eps)"""
    x = np.zeros((n, n), np.complex128)
    x[np.arange(n), np.arange(n)] = 1.0 + 0.5j
    for prec, eps in ((64, 2.0 ** -53), (32, 2.0 ** -24)):
        for sign, swap in ((1, 0), (-1, 0), (-1, 1)):
            ref = np.fft.fft(x.astype(np.clongdouble), axis=1)
            if sign > 0:
                ref = np.fft.ifft(x.astype(np.clongdouble), axis=1) * n
            for f in [MERGED] if prec == 64 else [MERGED, PACKED_MERGED, PACKED_MERGED_WIDE]:
                err = np.abs(_run(n, sign, swap, f, prec, x) - ref).max()
                assert err < 12 * eps * abs(1.0 + 0.5j), (prec, sign, swap, f, float(err) / eps)
