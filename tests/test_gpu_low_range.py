"""Lines at the bottom of a form's range, where q of long chains in strong fields ends up: the
tensor-core passes against dense operators in extended precision, down to the smallest
normal numbers."""
import numpy as np
import pytest

from test_gpu_pass_tc import operator

pytestmark = pytest.mark.gpu

STEPS = 2
ULP = {"fp64": 2.0 ** -53, "fp32x2": 2.0 ** -46, "fp32": 2.0 ** -24}
SMALLEST = {"fp64": 2.0 ** -1022, "fp32x2": 2.0 ** -126, "fp32": 2.0 ** -126}
# the largest values, down to the smallest normal number's neighbourhood
TOP = {"fp64": (2.0 ** -957, 2.0 ** -961, 2.0 ** -990, 2.0 ** -1010, 2.0 ** -1019),
       "fp32x2": (2.0 ** -61, 2.0 ** -90, 2.0 ** -110, 2.0 ** -123),
       "fp32": (2.0 ** -93, 2.0 ** -97, 2.0 ** -110, 2.0 ** -123)}


@pytest.mark.parametrize("prec", ("fp64", "fp32x2", "fp32"))
@pytest.mark.parametrize("grid", [(30, 1, 15, 1), (40, 1, 20, 0), (16, 10, 12, 1)])
def test_low_lines(srn, grid, prec):
    nx, ny, nz, wall = grid
    s = srn.configs.film2d(ns=48) if wall else srn.configs.bulk2d()
    s.LX, s.LY, s.LZ = nx * s.DR_TARGET, (ny * s.DR_TARGET if ny > 1 else 1.0), nz * s.DR_TARGET
    rng = np.random.default_rng(nx * 100 + nz)
    u, w = rng.uniform(0.1, 1.0, (nx, ny, nz)), rng.uniform(-3.0, 3.0, nx * ny * nz)
    u[:, :, nz // 3] = 0.0
    naxes = 2 + (ny > 1)
    with srn.Solver(s, precision=prec) as one, srn.Solver(s, precision=prec, kernel_path="passes") as two:
        d = one.derived[0]
        assert d.grid == (nx, ny, nz)
        K = [operator(n, a, wall and i == 2) for i, (n, a) in enumerate(zip(grid[:3], (d.c.alphax, d.c.alphay, d.c.alphaz)))]
        b = np.exp(np.longdouble(d.c.ds) * (-w / 2)).reshape(nx, ny, nz)
        for top in TOP[prec]:
            q0 = (u * top).astype(np.float64 if prec == "fp64" else np.float32).astype(float)
            got = one.propagate(q0.ravel(), w, STEPS)
            assert np.array_equal(got, two.propagate(q0.ravel(), w, STEPS))
            q = q0.astype(np.longdouble)
            for t in range(STEPS):
                q = np.tensordot(K[0], q * b, (1, 0))
                if ny > 1:
                    q = np.moveaxis(np.tensordot(K[1], q, (1, 1)), 0, 1)
                q = (q @ K[2]) * b
                # relative as elsewhere in the range (test_gpu_pass_tc.py); and on every axis what
                # is below the smallest normal number, in a row of up to twice unit size, and in
                # the products with b (two terms each in FP32x2)
                most = (t + 1) * ((4 + 4 * naxes) * ULP[prec] * np.max(np.abs(q)) + (4 + 2 * naxes) * np.longdouble(SMALLEST[prec]))
                assert np.max(np.abs(got[t + 1].astype(np.longdouble) - q.ravel())) <= most, (top, t)
