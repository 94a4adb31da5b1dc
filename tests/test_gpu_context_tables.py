"""Operator tables at context creation: axes of one length, kind and diffusion factor share
theirs, and come out as they do with tables of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,digits", (("fp64", 6), ("fp32", 4)))
def test_axes_alike_share_a_table(srn, prec, digits):
    n, hp = 60, 16  # blocks of 15 points, padded to 16
    s = srn.configs.bulk2d(nx=n, nz=n)
    other = s.copy()
    other.LX *= 1.005
    assert s.grid() == other.grid() == (n, 1, n)
    rng = np.random.default_rng(1)
    q0, w = rng.uniform(0.5, 1.0, n * n), rng.uniform(-1.0, 1.0, n * n)
    with srn.Solver([s], precision=prec) as one, srn.Solver([other], precision=prec) as two:
        assert two.device_bytes - one.device_bytes == 4 * hp * hp * digits * 2
        a = one.propagate(q0, w, 3).reshape(4, n, n)
        b = one.propagate(q0.reshape(n, n).T.ravel(), w.reshape(n, n).T.ravel(), 3).reshape(4, n, n)
    # x and z are the same operator: the transposed start gives the transposed steps, but for the
    # order of the two axes' roundings (half an ulp each, as many again for b's two products)
    ulp = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    assert np.max(np.abs(a - b.transpose(0, 2, 1))) <= 3 * 12 * ulp * np.max(np.abs(a))
