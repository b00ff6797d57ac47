"""Closed meshes on grids fine enough for the cubes: overlapping solids, cavities,
needles, triangles without area and corners written twice, as in
test_gpu_bake_cubes."""
import numpy as np
import pytest

from eulersf_gb300.scene import icosphere
from test_gpu_bake_cubes import _cavity, _dented, _join, _margin_and_solid, _pair

pytestmark = pytest.mark.gpu


def _overlap():  # winding number 2 in the lens
    v, f = icosphere(2, 0.06)
    return _join((v - [0.03, 0.0, 0.0], f), (v + [0.03, 0.01, 0.0], f))


def _twice():  # every triangle with corners of its own
    v, f = _dented()
    return v[f].reshape(-1, 3), np.arange(3 * len(f)).reshape(-1, 3)


def _split(at):
    """Every fifth triangle's first edge cut at a corner `at` of its height off
    it; at 0, the corner lies on the edge and a triangle without area closes the
    gap."""
    v, f = _dented()
    verts, faces = list(v), []
    for k, (a, b, c) in enumerate(f):
        if k % 5:
            faces.append((a, b, c))
            continue
        m = len(verts)
        verts.append((0.5 - 0.5 * at) * (v[a] + v[b]) + at * v[c])
        faces += [(a, m, c), (m, b, c), (a, b, m)]
    return np.array(verts), np.array(faces)


def _needles():
    return _split(1e-4)


def _no_area():
    return _split(0.0)


@pytest.mark.parametrize("mesh,dh", [(_dented, 0.0018), (_cavity, 0.0019), (_pair, 0.0014), (_overlap, 0.0016),
                                     (_twice, 0.0018), (_needles, 0.0019), (_no_area, 0.0019)])
def test_baked_nodes_match_every_distance(mesh, dh, gpu_lib):
    from eulersf_gb300.bake import rasterize_solid
    verts, faces = mesh()
    res, _, origin, mass, total = rasterize_solid(verts, faces, dh, 700.0)
    assert np.prod(res) * len(faces) >= 2e8  # by cubes
    area = np.linalg.norm(np.cross(*(verts[faces[:, k]] - verts[faces[:, 0]] for k in (1, 2))), axis=1)
    solid, margin = _margin_and_solid(verts, faces[area > 1e-12], res, origin, dh)
    got = mass.reshape(-1)
    assert np.all((got == 0.0) | (got == 700.0))
    assert not np.any(((got > 0) != solid) & (margin > 1e-6 * max(res) * dh))
    assert total == np.count_nonzero(got) * 700.0 * dh * dh * dh
