"""The launches of an iteration around the contour loop: instances of a batch that fills the GPU
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


@pytest.mark.parametrize("graph", (False, True))
@pytest.mark.parametrize("what,prec,batch", (("bulk3d", "fp32", 8), ("bulk3d", "fp32", 10), ("film", "fp64", 33), ("film", "fp32x2", 17)))
def test_chains_in_parts_equal_solo(srn, what, prec, batch, graph):
    """More chains than clusters fit at once run part by part in several launches (also
    the next step after a stop criterion has put them back into one): the bits of an
    instance alone."""
    if what == "film":
        s = srn.configs.film2d(ns=40)
        m = srn.configs.substrate_mask(s)
        w = [srn.configs.droplet_fields(s, seed=b) for b in range(batch)]
    else:
        s = srn.configs.bulk3d_point(20.0, 40.0, srn.configs.PLANES[0], ns=31)
        m = None
        w = [srn.configs.uniform_fields(s.grid(), seed=b, amp=0.1, fields=(0, 1, 2)) for b in range(batch)]

    def solve(which):
        with srn.Solver([s] * len(which), precision=prec, use_graph=graph) as sv:
            for slot, b in enumerate(which):
                sv.set_fields(w[b], slot)
                if m is not None:
                    sv.set_masks(m, slot)
                sv.set_iteration(1, slot)
            res = sv.iterate(2)
            sv.set_stop(1e-30)
            res += sv.iterate(1)
            return [([(r[k].free_energy, r[k].rms, tuple(r[k].q)) for r in res], sv.get_fields(k)) for k in range(len(which))]

    together = solve(range(batch))
    for b in (0, batch - 1):
        (rec, fields), = solve([b])
        assert rec == together[b][0] and np.isfinite(fields).all()
        assert np.array_equal(fields, together[b][1])
