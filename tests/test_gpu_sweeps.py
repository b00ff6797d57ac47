"""The Gauss-Seidel sweeps (sweepPhi as a march of warps, the velocity
extension over level lists) give the bits of the cooperative hyperplane wave,
which walks every node of every pass: both visit each node after its three
upwind neighbours, so there is no tolerance. Boxes of a few nodes, boxes cut by
the walls, sides that are no multiple of a patch's 8 x 4 columns, and levels of
more entries than a block has threads."""
import numpy as np
import pytest

from eulersf_gb300.scene import SceneDesc, SolidDesc

pytestmark = pytest.mark.gpu

SCENES = {
    "small": SceneDesc(N=12, mass_sample_dh=(1 / 12) / 4, noise_seed=1),
    "at a corner": SceneDesc(N=29, mass_sample_dh=(1 / 29) / 4, noise_seed=2,
                             solids=[SolidDesc(center=(0.2, 0.21, 0.83), radius=0.12)]),
    "stretched": SceneDesc(N=45, mass_sample_dh=(1 / 45) / 4, noise_seed=3,
                           solids=[SolidDesc(center=(0.45, 0.5, 0.55), radius=0.1, scaling=(1.6, 0.8, 1.1))]),
    "wide levels": SceneDesc(N=72, mass_sample_dh=(1 / 72) / 4, noise_seed=4,
                             solids=[SolidDesc(center=(0.5, 0.5, 0.5), radius=0.3)]),
}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_sweeps_give_the_bits_of_the_wave(name, gpu_lib, monkeypatch):
    import eulersf_gb300 as E
    got = {}
    for schedule in ("wave", None):
        if schedule:
            monkeypatch.setenv("ESF_SWEEP", schedule)
        else:
            monkeypatch.delenv("ESF_SWEEP")
        scene = E.make_scene(SCENES[name])
        for _ in range(2):
            scene.stepImplicit()
        got[schedule] = {n: scene.get(n) for n in ("solid.phi", "solid.velocity", "solid.boxes", "solid.u")}
        scene.close()
    for n in got[None]:
        assert np.array_equal(got["wave"][n], got[None][n]), n
