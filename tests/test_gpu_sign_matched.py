"""Lines made against one row of an operator: every data digit that meets the row's digits on
level 3 of the sums has full size and their sign, so that the sum is the largest that the
accumulators can be given. Against the operator in extended precision."""
import numpy as np
import pytest

from test_gpu_pass_tc import ULP, operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ("fp64", "fp32x2"))
@pytest.mark.parametrize("nx", (54, 110, 150))
def test_level_three_at_its_bound(srn, nx, prec):
    nz = 16
    s = srn.configs.bulk2d()
    s.NS, s.LX, s.LZ = 128, nx * s.DR_TARGET, nz * s.DR_TARGET
    with srn.Solver(s, precision=prec) as sv:
        d = sv.derived[0]
        assert d.grid == (nx, 1, nz)
        K = operator(nx, d.c.alphax, 0)
        h = nx // 2
        assert nx % 4 == 2  # two blocks: mirror sums and differences
        v = np.rint((K[:h, :h] + K[:h, ::-1][:, :h]) / 2 * np.longdouble(2) ** 59).astype(np.int64)
        e = np.zeros((6, h, h), dtype=np.int64)
        for k in range(5, -1, -1):
            e[k] = ((v + 512) & 1023) - 512 if k else v
            v = (v - e[k]) >> 10
        row = int(np.argmax(np.abs(e[:4]).sum((0, 2))))
        if nx == 150:
            assert 512 * int(np.abs(e[:4, row]).sum()) > 2 ** 24
        # mirror sums u with digits 0 to 3; x from 1/4 to 1/2, so that u is x 2^60
        u = sum((500 if k == 0 else 511) * np.where(e[3 - k, row] < 0, -1, 1).astype(np.int64) << 10 * (5 - k) for k in range(4))
        half = u.astype(np.longdouble) * np.longdouble(2) ** -60
        x = np.concatenate([half, half[::-1]]).astype(float)
        assert np.all((np.abs(x) >= 0.25) & (np.abs(x) < 0.5)) and np.array_equal(x[:h], half)
        q0 = np.repeat(x, nz)
        got = sv.propagate(q0, np.zeros(nx * nz), 1)[1].reshape(nx, nz)
    want = K @ x.astype(np.longdouble)
    # both axes' split, left-out levels and rounding, and b = 1 twice, as in test_gpu_pass_tc.py
    assert np.max(np.abs(got - want[:, None])) <= 12 * ULP[prec] * np.max(np.abs(want))
