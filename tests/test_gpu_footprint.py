"""The server's admission estimate covers the device memory that a scene takes
(a 0.2-radius ball, as it was fitted, and one of few particles, whose sweeps'
buffers are the larger ones)."""
import ctypes as C

import pytest

from eulersf_gb300 import abi
from eulersf_gb300.scene import SceneDesc, SolidDesc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.ESF_FP64, abi.ESF_MIXED])
@pytest.mark.parametrize("N,particles", [(48, 32), (96, 32), (160, 32), (96, 4)])
def test_estimate_covers_a_scene(N, particles, precision, gpu_lib):
    import torch
    import eulersf_gb300 as E
    from eulersf_gb300.serve import request_for
    desc = SceneDesc(N=N, mass_sample_dh=0.25 / N, particles_per_cell=particles, eps=0.02, max_iters=30,
                     solids=[SolidDesc(center=(0.5, 0.5, 0.5), radius=0.2)])
    q, keep = request_for(desc, 1, precision)
    estimate = gpu_lib.esf_scene_footprint(C.byref(q.grid), C.byref(q.params), q.num_solids, q.solids)
    gpu_lib.esf_release_workspaces()
    torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    scene = E.make_scene(desc, precision=precision)
    for _ in range(2):
        scene.stepImplicit()
    used = before - torch.cuda.mem_get_info()[0]
    scene.close()
    print(f"N={N} precision={precision} particles={particles}: {estimate / used:.3f} of {used / 1e6:.0f} MB")
    assert 0.98 * used <= estimate <= 1.6 * used
