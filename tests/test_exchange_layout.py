"""Shared memory of the 2D contour loop whose lines pass between the CTAs of a cluster,
on the CPU: warps of a CTA may be a phase apart across a change of axis, so what one
axis' outputs still read must lie where the other axis' digits do not."""
import ctypes as C
import importlib

import pytest

CLUSTERS = (1, 2, 3, 4, 6, 8, 12, 16)
GRIDS = ((32, 16), (64, 64), (96, 64), (128, 96), (192, 96), (192, 128), (150, 75), (130, 66), (150, 100), (9, 11), (17, 33), (108, 100))


@pytest.mark.parametrize("prec", (0, 1, 2))
@pytest.mark.parametrize("wall", (0, 1))
@pytest.mark.parametrize("grid", GRIDS)
def test_sums_behind_the_digits_of_either_axis(srn, grid, wall, prec):
    f = importlib.import_module(srn.__name__ + "._lib").lib().scft_tc_exchange_layout
    f.restype, f.argtypes = C.c_int, [C.c_int] * 5 + [C.POINTER(C.c_long), C.POINTER(C.c_long)]
    fits = 0
    for cluster in CLUSTERS:
        at, total = (C.c_long * 8)(), C.c_long()
        rc = f(prec, *grid, wall, cluster, at, C.byref(total))
        assert rc in (0, 1)
        if rc:
            continue
        fits += 1
        x, z = list(at[:4]), list(at[4:])
        for a in (x, z):
            assert a[0] < a[1] and a[2] < a[3] <= total.value
            for o in (x, z):
                assert a[3] <= o[0] or o[1] <= a[2], (cluster, x, z)
    assert fits or grid[0] * grid[1] > 96 * 64


def test_outputs_read_exponents_that_no_peer_writes(srn):
    """A CTA whose lines of the other axis are complete sends the next exponents while
    warps of the receiver may still be scaling outputs by the last ones."""
    f = importlib.import_module(srn.__name__ + "._lib").lib().scft_tc_exchange_exponents
    f.restype, f.argtypes = None, [C.POINTER(C.c_long)]
    at = (C.c_long * 8)()
    f(at)
    sets = sorted(zip(at[0::2], at[1::2]))
    assert all(b - a >= 128 * 4 for a, b in sets)
    assert all(p[1] <= q[0] for p, q in zip(sets, sets[1:]))
