"""A served scene that runs alone takes its own loops, whatever scenes of its
grid shape ran before it and whether their results are still held."""
import pytest

from eulersf_gb300 import abi
from eulersf_gb300.scene import SceneDesc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("released", [True, False])
def test_a_scene_alone_is_not_batched(released, gpu_lib):
    from eulersf_gb300.serve import ESF_REQ_DONE, Server
    desc = SceneDesc(N=16, mass_sample_dh=(1.0 / 16) / 4, noise_seed=1)
    with Server(max_active=2) as srv:
        first = srv.submit(desc, 1, abi.ESF_MIXED)
        assert srv.wait(first)["state"] == ESF_REQ_DONE
        if released:
            srv.release(first)
        second = srv.submit(desc, 2, abi.ESF_MIXED)
        assert srv.wait(second)["state"] == ESF_REQ_DONE
        assert srv.batch_stats()["inner_solves"] == 0
