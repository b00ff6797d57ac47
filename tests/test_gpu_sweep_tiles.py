"""The velocity extension by tiles, which large octants take: the bits of the
cooperative hyperplane wave, and taken where it is the faster schedule."""
import numpy as np
import pytest

from eulersf_gb300 import abi
from eulersf_gb300.scene import SceneDesc, SolidDesc
from test_gpu_sweeps import SCENES

pytestmark = pytest.mark.gpu
FIELDS = ("solid.phi", "solid.velocity", "solid.boxes", "solid.u")


def _run(lib, desc, schedule, monkeypatch, steps, precision=abi.ESF_FP64):
    """Fields after the steps, kernel launches of the last one."""
    import eulersf_gb300 as E
    monkeypatch.delenv("ESF_SWEEP", raising=False)
    if schedule:
        monkeypatch.setenv("ESF_SWEEP", schedule)
    scene = E.make_scene(desc, precision=precision)
    for _ in range(steps):
        before = lib.esf_kernel_launches()
        scene.stepImplicit()
    launches = lib.esf_kernel_launches() - before
    got = {n: scene.get(n) for n in FIELDS}
    scene.close()
    return got, launches


@pytest.mark.parametrize("name", sorted(SCENES))
def test_tiles_give_the_bits_of_the_wave(name, gpu_lib, monkeypatch):
    wave, _ = _run(gpu_lib, SCENES[name], "wave", monkeypatch, 2)
    tiles, by_tiles = _run(gpu_lib, SCENES[name], "tiles", monkeypatch, 2)
    _, by_lists = _run(gpu_lib, SCENES[name], None, monkeypatch, 2)
    assert by_tiles > by_lists  # 32 passes of several launches each
    for n in FIELDS:
        assert np.array_equal(wave[n], tiles[n]), n


def test_large_solid_takes_tiles(gpu_lib, monkeypatch):
    """A ball of 113 nodes across, whose octants' planes are more than a block's
    shared memory holds."""
    N = 256
    desc = SceneDesc(N=N, mass_sample_dh=0.5 / N, noise_seed=1, particles_per_cell=2, eps=0.02, max_iters=20,
                     solids=[SolidDesc(center=(0.5, 0.5, 0.5), radius=0.22)])
    default, launches = _run(gpu_lib, desc, None, monkeypatch, 1, abi.ESF_MIXED)
    tiles, by_tiles = _run(gpu_lib, desc, "tiles", monkeypatch, 1, abi.ESF_MIXED)
    wave, by_wave = _run(gpu_lib, desc, "wave", monkeypatch, 1, abi.ESF_MIXED)
    assert launches == by_tiles and launches > by_wave + 1000  # 32 passes of 46 launches each
    for n in FIELDS:
        assert np.array_equal(default[n], tiles[n]), n
        assert np.array_equal(default[n], wave[n]), n
