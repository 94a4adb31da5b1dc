"""Operators wider than the line on lines that are flat or nearly so: the digits of both add
up with one sign, and the tensor-core passes carry between levels. Against dense operators
in extended precision, and as one loop against passes, bit for bit."""
import numpy as np
import pytest

from test_gpu_pass_tc import operator

pytestmark = pytest.mark.gpu

STEPS = 2
ULP = {"fp64": 2.0 ** -53, "fp32x2": 2.0 ** -46, "fp32": 2.0 ** -24}


@pytest.mark.parametrize("prec", ("fp64", "fp32x2", "fp32"))
@pytest.mark.parametrize("grid", [(146, 1, 16, 0), (93, 1, 30, 1), (150, 1, 93, 0), (16, 30, 150, 0)])
def test_flat_lines_under_wide_operators(srn, grid, prec):
    nx, ny, nz, wall = grid
    s = srn.configs.film2d(ns=48) if wall else srn.configs.bulk2d()
    s.NS, s.DR_TARGET = 48, 0.002
    s.LX, s.LY, s.LZ = nx * s.DR_TARGET, (ny * s.DR_TARGET if ny > 1 else s.DR_TARGET), nz * s.DR_TARGET
    rng = np.random.default_rng(nx + nz)
    for smooth in (0.0, 0.2):
        # flat along y and z, flat or nearly so along x
        x = 1.0 + smooth * np.cos(2 * np.pi * np.arange(nx) / nx)[:, None, None]
        q0 = np.ones((nx, ny, nz)) * x * rng.uniform(0.5, 1.0)
        w = np.full(nx * ny * nz, rng.uniform(-3.0, 3.0))
        if prec == "fp32":
            q0 = q0.astype(np.float32).astype(float)
        got = {}
        for path in ("auto", "passes"):
            with srn.Solver(s, precision=prec, kernel_path=path) as sv:
                d = sv.derived[0]
                assert d.grid == (nx, ny, nz) and d.c.alphax > 1e3
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
            err = float(np.max(np.abs(got["auto"][t + 1] - q.ravel())))
            # walls take nearly all of it away: relative to what a step started from
            base = float(np.max(np.abs(q0))) if wall else float(np.max(np.abs(q)))
            # as for narrow operators (test_gpu_pass_tc.py)
            assert err / base <= (t + 1) * (4 + 4 * naxes) * ULP[prec]


def test_slot_takes_a_wide_operator_between_iterations(srn):
    """A context whose operators need no carries, its iterations captured as a graph, is given
    one that does: from then on the bits of a context made with it."""
    nx, nz = 92, 93
    narrow = srn.configs.bulk2d()
    narrow.NS, narrow.LX, narrow.LZ = 48, nx * narrow.DR_TARGET, nz * narrow.DR_TARGET
    wide = narrow.copy()
    wide.DR_TARGET = 0.002
    wide.LX, wide.LY, wide.LZ = nx * wide.DR_TARGET, wide.DR_TARGET, nz * wide.DR_TARGET
    assert narrow.grid() == wide.grid() == (nx, 1, nz)
    w = np.repeat(np.linspace(-0.3, 0.4, 14), nx * nz)

    def last(sv):
        sv.set_fields(w, 0)
        sv.set_iteration(1, 0)
        r = sv.iterate(2)[-1][0]
        return r.free_energy, tuple(r.q), sv.get_fields(0)

    with srn.Solver([wide], precision="fp64", use_graph=True) as sv:
        fresh = last(sv)
    with srn.Solver([narrow], precision="fp64", use_graph=True) as sv:
        before = last(sv)
        sv.set_surface(0, wide)
        after = last(sv)
    assert np.isfinite(fresh[2]).all() and before[0] != after[0]
    assert after[:2] == fresh[:2] and np.array_equal(after[2], fresh[2])
