"""Exactness of the tensor-core passes' level sums on the CPU: whatever the lines hold, levels
0 to 3 of FP64 and FP32x2 stay within the 2^24 that an FP32 accumulator holds exactly, over
whole rows or, where the operator's digits call for carries, over 16 points at a time."""
import ctypes as C
import importlib

import numpy as np
import pytest

LIMIT = 2.0 ** 24
# what a carry leaves behind and what it brings: 2^9, and 2^24 / 2^10
LEFT = 2.0 ** 9 + 2.0 ** 14


def sums(srn, n, alpha, wall, prec):
    f = importlib.import_module(srn.__name__ + "._lib").lib().scft_tc_level_sums
    row, step = np.zeros(6), np.zeros(6)
    dp = C.POINTER(C.c_double)
    f.restype, f.argtypes = C.c_int, [C.c_int, C.c_double, C.c_int, C.c_int, dp, dp]
    rc = f(n, alpha, wall, prec, row.ctypes.data_as(dp), step.ctypes.data_as(dp))
    assert rc in (0, 1)
    return rc, row, step


@pytest.mark.parametrize("wall", (0, 1))
def test_levels_below_the_accumulators_limit(srn, wall):
    carried = set()
    for n in range(8, 161 if wall else 257):
        for alpha in (0.005, 0.1, 0.5, 3.0, 100.0, 3e3, 1e5):
            rc, row, step = sums(srn, n, alpha, wall, 0)
            assert np.all(np.diff(row) >= 0) and row[0] + row[0] / 1024 <= LIMIT
            if rc:
                carried.add(alpha)
                assert step[3] + LEFT <= LIMIT
            else:
                assert row[3] <= LIMIT
    # flat operators of wide boxes, and long lines, are among them
    assert 3e3 in carried


def test_sums_are_those_of_the_digits(srn):
    """The bound itself, from digits taken apart again here."""
    for n, wall, alpha in ((64, 0, 0.5), (150, 0, 0.02), (75, 1, 0.64), (205, 0, 3e3)):
        _, row, step = sums(srn, n, alpha, wall, 0)
        i, ld = np.arange(n), np.longdouble
        pi = ld("3.14159265358979323846264338327950288")
        if wall:
            m = np.arange(1, n + 1)
            S = np.sin(pi * (np.outer(i + 1, m) % (2 * (n + 1))).astype(ld) / (n + 1))
            K = (S * np.exp(-ld(alpha) * (pi * m / (n + 1)) ** 2)) @ S.T * (ld(2) / (n + 1))
        else:
            k = 2 * pi * (ld(n) / 2 - np.abs(i - ld(n) / 2)) / n
            c = np.cos(2 * pi * (np.outer(i, i) % n).astype(ld) / n) @ np.exp(-ld(alpha) * k * k) / n
            K = c[(i[:, None] - i[None, :]) % n]
        if not wall and n % 4 == 0:
            h, m = n // 4, n // 2
            q = [K[:h, :h], K[:h, m - h:m][:, ::-1], K[:h, m:m + h], K[:h, n - h:][:, ::-1]]
            M = [(q[0] + q[2] + s * (q[1] + q[3])) / 4 for s in (1, -1)] + [(q[0] - q[2] + s * (q[1] - q[3])) / 4 for s in (1, -1)]
            scale = ld(2) ** 60
        else:
            h = (n + 1) // 2
            A, B = K[:h, :h], K[:h, ::-1][:, :h]
            M = [(A + B) / 2, (A - B) / 2]
            if n % 2:
                M[0][:, h - 1] /= 2
            scale = ld(2) ** 59
        worst_row, worst_step = np.zeros(6), np.zeros(6)
        for blk in M:
            v = np.rint(blk * scale).astype(np.int64)
            size = np.zeros((6,) + v.shape)
            for d in range(5, -1, -1):
                e = ((v + 512) & 1023) - 512 if d else v
                v = (v - e) >> 10
                size[d] = 512.0 * np.abs(e)
            level = np.cumsum(size, 0)
            worst_row = np.maximum(worst_row, level.sum(2).max(1))
            pad = np.pad(level, ((0, 0), (0, 0), (0, -v.shape[1] % 16)))
            worst_step = np.maximum(worst_step, pad.reshape(6, v.shape[0], -1, 16).sum(3).max((1, 2)))
        # the last digits come from sums in another order
        assert np.allclose(row[:4], worst_row[:4], rtol=0.02) and np.allclose(step[:4], worst_step[:4], rtol=0.02)
