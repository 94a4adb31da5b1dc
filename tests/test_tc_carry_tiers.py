"""Which operators have their level sums carried, on the CPU: all levels where the operator is
wide enough to meet a flat line with digits of one sign, so that every level is exact."""
import ctypes as C
import importlib

import numpy as np
import pytest

LIMIT = 2.0 ** 24


@pytest.mark.parametrize("prec", (0, 1, 2))
@pytest.mark.parametrize("wall", (0, 1))
def test_tiers(srn, wall, prec):
    L = importlib.import_module(srn.__name__ + "._lib").lib()
    dp = C.POINTER(C.c_double)
    L.scft_tc_level_sums.argtypes = [C.c_int, C.c_double, C.c_int, C.c_int, dp, dp]
    L.scft_tc_carry.restype, L.scft_tc_carry.argtypes = C.c_int, [C.c_int, C.c_double, C.c_int, C.c_int]
    top = 3 if prec == 1 else 5
    seen = set()
    for n in list(range(8, 161, 3)) + ([] if wall else [192, 256]):
        for alpha in (0.02, 0.5, 3.0, 100.0, 3e3, 1e5):
            row, step = np.zeros(6), np.zeros(6)
            L.scft_tc_level_sums(n, alpha, wall, prec, row.ctypes.data_as(dp), step.ctypes.data_as(dp))
            how = L.scft_tc_carry(n, alpha, wall, prec)
            seen.add(how)
            if row[top] <= LIMIT:
                assert how == 0
            elif row[1] > LIMIT / 4:
                assert how == 2
                # after 16 points and, on levels 4 and 5, after half of the pairs: at most three
                # pairs of digits up to 512, and what carries leave and bring
                assert min(step[3], 3 * 16 * 2.0 ** 18) + 2.0 ** 9 + 2.0 ** 15 <= LIMIT
            else:
                # narrow: what a row has beyond its first two digits has mixed signs
                assert how == (1 if prec != 1 and row[3] > LIMIT else 0)
            if alpha <= 3.0:
                assert how < 2
    assert seen == ({0, 2} if prec == 1 else {0, 1, 2})
