"""The launches after the contour loop: instances of a batch that fills the GPU
against the same instances alone (fields side by side or in turn in the Boltzmann
launch, the last CTA of each instance finishing Q and the record), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ("fp64", "fp32x2", "fp32"))
@pytest.mark.parametrize("grid,batch", (((32, 16), 80), ((9, 11), 160), ((75, 26), 24)))
def test_large_batch_equals_solo(srn, grid, batch, prec):
    s = srn.configs.film2d(nx=grid[0], nz=grid[1], ns=32)
    m = srn.configs.substrate_mask(s)
    w = [srn.configs.droplet_fields(s, seed=b, radius=1.0) for b in range(batch)]

    def solve(which):
        with srn.Solver([s] * len(which), precision=prec) as sv:
            for slot, b in enumerate(which):
                sv.set_fields(w[b], slot)
                sv.set_masks(m, slot)
                sv.set_iteration(1, slot)
            res = sv.iterate(3)
            return [([(r[k].free_energy, r[k].rms, tuple(r[k].q), tuple(r[k].mu)) for r in res], sv.get_fields(k),
                     sv.get_densities(k)) for k in range(len(which))]

    together = solve(range(batch))
    for b in (0, batch // 2, batch - 1):
        (rec, fields, phi), = solve([b])
        assert rec == together[b][0] and np.isfinite(fields).all()
        assert np.array_equal(fields, together[b][1])
        assert all(np.array_equal(x, y) for x, y in zip(phi, together[b][2]))
