"""Operator digits of the tensor-core axis passes, decoded on the CPU: every axis
kind and length the passes take must give back the dense operator to the last
digit (FP64 and FP32x2: 59 or 60 bits below 1, FP32: 39 or 40)."""
import ctypes as C

import numpy as np
import pytest

LENGTHS = (8, 9, 15, 16, 17, 30, 31, 32, 33, 48, 62, 64, 75, 96, 97, 128, 150, 192)


@pytest.mark.parametrize("prec,bits", ((0, 59), (1, 39)))
@pytest.mark.parametrize("wall", (0, 1))
@pytest.mark.parametrize("n", LENGTHS)
def test_operator_digits(srn, n, wall, prec, bits):
    import importlib
    L = importlib.import_module(srn.__name__ + "._lib").lib()
    f = L.scft_tc_operator
    dp = C.POINTER(C.c_double)
    f.restype, f.argtypes = C.c_int, [C.c_int, C.c_double, C.c_int, C.c_int, dp, dp]
    for alpha in (0.02, 0.5, 3.0):
        eff, ref = np.empty((n, n)), np.empty((n, n))
        assert f(n, alpha, wall, prec, eff.ctypes.data_as(dp), ref.ctypes.data_as(dp)) == 0
        # nb blocks of entries rounded to half a unit each, and the FP64 results' own rounding
        assert np.max(np.abs(eff - ref)) <= 2.0 * 2.0 ** -bits + 2.0 ** -53
        assert np.max(np.abs(ref - ref[::-1, ::-1])) <= 2.0 ** -53


def test_dense_operator_matches_modes(srn):
    """The operator itself against the reference's modes in NumPy (SCFT.c:983-1023)."""
    import importlib
    L = importlib.import_module(srn.__name__ + "._lib").lib()
    f = L.scft_tc_operator
    dp = C.POINTER(C.c_double)
    f.restype, f.argtypes = C.c_int, [C.c_int, C.c_double, C.c_int, C.c_int, dp, dp]
    for n in (9, 24, 75):
        for wall in (0, 1):
            eff, ref = np.empty((n, n)), np.empty((n, n))
            assert f(n, 0.4, wall, 0, eff.ctypes.data_as(dp), ref.ctypes.data_as(dp)) == 0
            i = np.arange(n)
            if wall:
                m = np.arange(1, n + 1)
                S = np.sin(np.pi * (np.outer(i + 1, m) % (2 * (n + 1))) / (n + 1))  # reduced exactly
                K = (S * np.exp(-0.4 * (np.pi * m / (n + 1)) ** 2)) @ S.T * (2.0 / (n + 1))
            else:
                k = 2.0 * np.pi * (n / 2.0 - np.abs(i - n / 2.0)) / n
                K = np.real(np.fft.ifft(np.exp(-0.4 * k * k)))[(i[:, None] - i[None, :]) % n]
            assert np.max(np.abs(ref - K)) <= 8 * 2.0 ** -53
