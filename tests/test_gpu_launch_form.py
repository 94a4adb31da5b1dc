"""The reported launch form of the contour steps: two threads per line and a cluster of CTAs
per chain are different forms of the fused 2D loop."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what,batch,prec,path,ctas", [
    ("film", 1, "fp32", "auto", 8), ("film", 5, "fp32", "auto", 4), ("film", 20, "fp32", "auto", 1),
    ("film", 40, "fp32", "auto", 1), ("film", 1, "fp64", "passes", 0), ("bulk3d", 1, "fp32", "auto", 8)])
def test_ctas_per_chain(srn, what, batch, prec, path, ctas):
    s = srn.configs.film2d(ns=40) if what == "film" else srn.configs.bulk3d_point(20.0, 40.0, srn.configs.PLANES[0], ns=31)
    with srn.Solver([s] * batch, precision=prec, kernel_path=path, autotune=False) as sv:
        t = sv.timing()
    assert t["ctas_per_chain"] == ctas
    if what == "film" and prec == "fp32":
        # 5 chains an instance: two threads per line or a cluster while the chains fit the SMs
        assert t["threads_per_line"] == (2 if 5 * batch <= 152 else 1)


def test_tensor_core_loop_reports_its_cluster(srn):
    with srn.Solver([srn.configs.film2d(nx=32, nz=16, ns=40)], precision="fp64") as sv:
        t = sv.timing()
        sv.enable_timing()
        assert t["fused_chain"] == 0 and (t["ctas_per_chain"] == 0 or 1 <= t["ctas_per_chain"] <= 16)
