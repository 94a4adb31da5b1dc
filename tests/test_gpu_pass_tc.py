"""Tensor-core axis passes (scft_pass_tc.cu) against the same contour steps with
dense operators in extended precision: both symmetry splits (periodic lengths of
four, the others, walls), tile and chunk remainders, the shortest and longest
lines, zero lines; launched per pass and as one loop, with equal bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 3
# half an ulp of each form; its products with b count as four of them in FP32x2
ULP = {"fp64": 2.0 ** -53, "fp32x2": 2.0 ** -46, "fp32": 2.0 ** -24}

GRIDS = [  # nx, ny, nz, wall
    (8, 1, 9, 0),
    (9, 1, 11, 1),
    (17, 1, 33, 0),
    (30, 1, 15, 1),
    (36, 1, 31, 1),
    (150, 1, 75, 1),
    (144, 1, 112, 1),
    (256, 1, 16, 0),
    (16, 10, 12, 1),
    (12, 21, 20, 0),
]


def operator(n, alpha, wall):
    ld, pi = np.longdouble, np.longdouble("3.14159265358979323846264338327950288")
    i = np.arange(n)
    if wall:
        m = np.arange(1, n + 1)
        S = np.sin(pi * (np.outer(i + 1, m) % (2 * (n + 1))).astype(ld) / (n + 1))
        return (S * np.exp(-ld(alpha) * (pi * m / (n + 1)) ** 2)) @ S.T * (ld(2) / (n + 1))
    k = 2 * pi * (ld(n) / 2 - np.abs(i - ld(n) / 2)) / n
    c = np.cos(2 * pi * (np.outer(i, i) % n).astype(ld) / n) @ np.exp(-ld(alpha) * k * k) / n
    return c[(i[:, None] - i[None, :]) % n]


@pytest.mark.parametrize("prec", ("fp64", "fp32x2", "fp32"))
@pytest.mark.parametrize("grid", GRIDS)
def test_steps_against_dense_operators(srn, grid, prec):
    nx, ny, nz, wall = grid
    s = srn.configs.film2d(ns=48) if wall else srn.configs.bulk2d()
    s.LX, s.LY, s.LZ = nx * s.DR_TARGET, (ny * s.DR_TARGET if ny > 1 else 1.0), nz * s.DR_TARGET
    if nx == 8:
        s.LX *= 1.02  # a length of exactly 1 is one point
    rng = np.random.default_rng(nx * 1000 + nz)
    q0, w = rng.uniform(0.1, 1.5, (nx, ny, nz)), rng.uniform(-3.0, 3.0, nx * ny * nz)
    q0[:, :, nz // 2:] *= 1e-9
    q0[nx // 2] = 0.0
    if prec == "fp32":
        q0 = q0.astype(np.float32).astype(float)
    got = {}
    for path in ("auto", "passes"):
        with srn.Solver(s, precision=prec, kernel_path=path) as sv:
            d = sv.derived[0]
            assert d.grid == (nx, ny, nz)
            got[path] = sv.propagate(q0.ravel(), w, STEPS)
            alpha, ds = (d.c.alphax, d.c.alphay, d.c.alphaz), d.c.ds
    assert np.array_equal(got["auto"], got["passes"])
    K = [operator(n, a, wall and i == 2) for i, (n, a) in enumerate(zip(grid[:3], alpha))]
    b = np.exp(np.longdouble(ds) * (-w / 2)).reshape(nx, ny, nz)
    q = q0.astype(np.longdouble)
    naxes = 2 + (ny > 1)
    for t in range(STEPS):
        q = np.tensordot(K[0], q * b, (1, 0))
        if ny > 1:
            q = np.moveaxis(np.tensordot(K[1], q, (1, 1)), 0, 1)
        q = (q @ K[2]) * b
        err = float(np.max(np.abs(got["auto"][t + 1] - q.ravel())) / np.max(np.abs(q)))
        # per step: b and its two products, and per axis the line's split, the left-out
        # levels and the rounding of the result, half an ulp of the largest value each
        # (their sums over blocks in FP32: as much again)
        assert err <= (t + 1) * (4 + 4 * naxes) * ULP[prec]


@pytest.mark.parametrize("prec", ("fp64", "fp32x2", "fp32"))
@pytest.mark.parametrize("grid", [(8, 9), (9, 11), (17, 33), (30, 15), (60, 64), (75, 26), (150, 75), (108, 100)])
def test_solve_in_one_loop_equals_passes(srn, grid, prec):
    """Whole iterations (two blocks' factors, both directions of a chain, a batch) with
    the contour loop chosen by rule: ragged tiles of both axes, lines passed between
    clusters of several sizes. The same integers are summed, so the bits are equal."""
    nx, nz = grid
    s = srn.configs.film2d(ns=32) if nx % 2 else srn.configs.bulk2d()
    s.LX, s.LZ = nx * s.DR_TARGET * (1.02 if nx == 8 else 1.0), nz * s.DR_TARGET
    out = {}
    for path in ("auto", "passes"):
        with srn.Solver([s, s], precision=prec, kernel_path=path, autotune=False) as sv:
            assert sv.grid == (nx, 1, nz)
            rng = np.random.default_rng(nx + nz)
            for b in range(2):
                sv.set_fields(rng.uniform(-1.0, 1.0, 14 * sv.M), b)
                if nx % 2:
                    sv.set_masks(srn.configs.substrate_mask(s), b)
                sv.set_iteration(1, b)
            res = sv.iterate(2)
            out[path] = [sv.get_fields(b) for b in range(2)], [[r.free_energy for r in step] for step in res]
    assert np.isfinite(out["auto"][0]).all()
    assert np.array_equal(out["auto"][0], out["passes"][0]) and out["auto"][1] == out["passes"][1]
