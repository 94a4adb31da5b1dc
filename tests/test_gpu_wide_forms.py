"""Wide operators on flat lines: passes, loops and batches give the same bits, as every level
of their sums is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def surface(srn, nx, nz, dr):
    s = srn.configs.bulk2d()
    s.NS, s.DR_TARGET = 48, dr
    s.LX, s.LY, s.LZ = nx * dr, dr, nz * dr
    assert s.grid() == (nx, 1, nz)
    return s


@pytest.mark.parametrize("prec", ("fp64", "fp32x2", "fp32"))
@pytest.mark.parametrize("nx,nz", [(93, 93), (146, 93), (150, 75), (150, 150), (110, 90), (134, 93)])
def test_forms_give_the_same_bits(srn, nx, nz, prec):
    rng = np.random.default_rng(5)
    s = surface(srn, nx, nz, 0.002)
    starts = [np.full(nx * nz, c) for c in rng.uniform(0.5, 1.0, 6).astype(np.float32).astype(float)]
    fields = [np.full(nx * nz, c) for c in rng.uniform(-3.0, 3.0, 6)]
    got = []
    for path, tune in (("passes", False), ("auto", False), ("auto", True)):
        with srn.Solver(s, precision=prec, kernel_path=path, autotune=tune) as sv:
            got.append([sv.propagate(q, w, 4) for q, w in zip(starts, fields)])
    for other in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.parametrize("prec", ("fp64", "fp32x2", "fp32"))
def test_narrow_and_wide_in_one_batch(srn, prec):
    nx, nz = 150, 93
    both = [surface(srn, nx, nz, 0.125), surface(srn, nx, nz, 0.002)]
    w = [np.repeat(np.linspace(-0.3, 0.4 + 0.1 * b, 14), nx * nz) for b in range(2)]

    def solve(which):
        with srn.Solver([both[b] for b in which], precision=prec) as sv:
            for slot, b in enumerate(which):
                sv.set_fields(w[b], slot)
                sv.set_iteration(1, slot)
            r = sv.iterate(2)
            return [([(x[k].free_energy, tuple(x[k].q)) for x in r], sv.get_fields(k)) for k in range(len(which))]

    together = solve([0, 1])
    for b in (0, 1):
        (rec, fields), = solve([b])
        assert rec == together[b][0] and np.array_equal(fields, together[b][1]) and np.isfinite(fields).all()
