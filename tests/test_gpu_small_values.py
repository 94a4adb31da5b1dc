"""Small values beside large ones on a line across a film: a grafted chain far from its wall.
The tensor-core passes hold a line in fixed point under its largest value, so the error of
every value is that of the line, whatever its own size (scft_gpu.h): about 8 digits in FP64
and FP32x2 are left at 1e-9 of the largest, none in the FP32 passes."""
import numpy as np
import pytest

from test_gpu_pass_tc import operator

pytestmark = pytest.mark.gpu

STEPS = 12
ULP = {"fp64": 2.0 ** -53, "fp32x2": 2.0 ** -46, "fp32": 2.0 ** -24}
LEVEL = {"fp64": 2.0 ** -56, "fp32x2": 2.0 ** -56, "fp32": 2.0 ** -27}


@pytest.mark.parametrize("prec", ("fp64", "fp32x2", "fp32"))
@pytest.mark.parametrize("nz", (33, 40, 75, 150))
def test_tail_of_a_grafted_chain(srn, nz, prec):
    nx = 12
    s = srn.configs.film2d(ns=64)
    s.LX, s.LZ = nx * s.DR_TARGET, nz * s.DR_TARGET
    rng = np.random.default_rng(nz)
    q0 = np.zeros((nx, nz))
    q0[:, 0] = 1.0
    w = np.tile(rng.uniform(-3.0, 3.0, nz), nx)  # the same on every line across the film
    got = {}
    for path in ("auto", "passes"):
        with srn.Solver(s, precision=prec, kernel_path=path) as sv:
            d = sv.derived[0]
            assert d.grid == (nx, 1, nz)
            got[path] = sv.propagate(q0.ravel(), w, STEPS).reshape(STEPS + 1, nx, nz)
    assert np.array_equal(got["auto"], got["passes"])
    K = operator(nz, d.c.alphaz, 1)
    b = np.exp(np.longdouble(d.c.ds) * (-w[:nz] / 2))
    q, scale = q0[0].astype(np.longdouble), np.longdouble(0)
    for t in range(STEPS):
        before = float(np.max(np.abs(q)))
        q = ((q * b) @ K) * b
        # of the line a step starts from: its split (a unit of 2^-57 a value, rows of up to twice
        # unit size), the operator's digits (half of 2^-60 for each of up to 150 values) and the
        # levels left out; passed on by the next steps. Of the value itself: the products with b
        # and the roundings of both axes
        scale = scale + 8 * LEVEL[prec] * before
        most = scale + (t + 1) * 12 * ULP[prec] * np.abs(q)
        assert np.all(np.abs(got["auto"][t + 1] - q) <= most), t
    # long lines go down to far less than that error, and what is at 1e-9 keeps these digits
    size = np.abs(q) / np.max(np.abs(q))
    assert nz < 75 or np.min(size) < 1e-12
    kept = (size > 3e-10) & (size < 3e-9)
    if prec != "fp32" and kept.any():
        err = np.max(np.abs(got["auto"][STEPS] - q) / np.max(np.abs(q)), axis=0)
        assert np.all(err[kept] / size[kept] < 1e-6)
