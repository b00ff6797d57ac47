"""The solid solve as one persistent launch gives the bits of the captured
graphs it stands in for (ESF_SOLID_SOLVE=graph): the same sums in the same
order, so there is no tolerance. FP64 blocks, the FP32 matrix-free operator and
the FP32 blocks; a ball of a few dozen nodes, one whose rows are no multiple of
a warp, and one of more than two warps of rows a block (over 9728 nodes)."""
import numpy as np
import pytest

from eulersf_gb300 import abi
from eulersf_gb300.scene import SceneDesc, SolidDesc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,radius", [(12, 0.13), (33, 0.15), (64, 0.24)])
@pytest.mark.parametrize("precision,assembled", [(abi.ESF_FP64, False), (abi.ESF_MIXED, False),
                                                 (abi.ESF_MIXED, True)])
def test_persistent_solve_gives_the_bits_of_the_graphs(N, radius, precision, assembled, gpu_lib, monkeypatch):
    import eulersf_gb300 as E
    desc = SceneDesc(N=N, mass_sample_dh=(1 / N) / 4, noise_seed=N, eps=1e-6, solids=[SolidDesc(radius=radius)])
    if assembled:
        monkeypatch.setenv("ESF_SOLID_ASSEMBLED", "1")
    got = {}
    for how in ("graph", "persistent"):
        monkeypatch.setenv("ESF_SOLID_SOLVE", how)
        scene = E.make_scene(desc, precision=precision)
        report = scene.stepImplicit()
        assert all(report["converged"])
        got[how] = (report["iterations"], [scene.get(n) for n in ("solidVelocityAtDt0", "solidPressureCorrection",
                                                                   "velocity")])
        scene.close()
    assert got["graph"][0] == got["persistent"][0]
    for a, b in zip(got["graph"][1], got["persistent"][1]):
        assert np.array_equal(a, b)
