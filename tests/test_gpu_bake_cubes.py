"""Mass baking of closed meshes by cubes against the signed distance of every
node to every triangle in FP64 (plain torch): the same nodes are solid, but for
nodes within 1e-6 of the mesh's extent of the threshold, where the library's
FP32 positions (rounded at 2^-24 of the extent, a few operations each) may fall
either way. A dented ball, a ball with a cavity (winding number 0 inside it),
two balls, and an open mesh, which keeps the general kernel; grids whose sides
are no multiple of a cube."""
import math

import numpy as np
import pytest

from eulersf_gb300.scene import icosphere

pytestmark = pytest.mark.gpu


def _dented():
    v, f = icosphere(2, 0.1)
    return v * (1.0 + 0.1 * np.sin(40.0 * v[:, :1] + 25.0 * v[:, 1:2])), f


def _join(a, b):
    return np.concatenate([a[0], b[0]]), np.concatenate([a[1], b[1] + len(a[0])])


def _cavity():
    v, f = icosphere(2, 0.05)
    return _join(icosphere(2, 0.1), (v, f[:, ::-1]))


def _pair():
    v, f = icosphere(2, 0.05)
    return _join((v - [0.06, 0.0, 0.01], f), (v * 0.8 + [0.05, 0.01, 0.0], f))


def _open():
    v, f = icosphere(2, 0.1)
    return v, f[:-5]


def _margin_and_solid(verts, faces, res, origin, dh):
    import torch
    tri = torch.tensor(verts[faces], dtype=torch.float64, device="cuda")
    a, b, c = (tri[None, :, k] for k in range(3))
    normal = torch.linalg.cross(b - a, c - a)
    normal = normal / normal.norm(dim=-1, keepdim=True)
    axes = [torch.arange(n, dtype=torch.float64, device="cuda") * dh + o for n, o in zip(res, origin)]
    grid = torch.stack(torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")[::-1], -1).reshape(-1, 1, 3)
    solid, margin = [], []
    for p in grid.split(8192):
        best, over = None, None
        for u, v in ((a, b), (b, c), (c, a)):
            e, w = v - u, p - u
            t = ((w * e).sum(-1) / (e * e).sum(-1)).clamp(0, 1)
            d2 = (w - t[..., None] * e).square().sum(-1)
            best = d2 if best is None else torch.minimum(best, d2)
            side = (torch.linalg.cross(normal, e.expand_as(normal)) * w).sum(-1) >= 0
            over = side if over is None else over & side
        plane = ((p - a) * normal).sum(-1).square()
        dist = torch.where(over, torch.minimum(best, plane), best).amin(1).sqrt()
        x, y, z = a - p, b - p, c - p
        lx, ly, lz = x.norm(dim=-1), y.norm(dim=-1), z.norm(dim=-1)
        det = (x * torch.linalg.cross(y, z)).sum(-1)
        den = lx * ly * lz + (x * y).sum(-1) * lz + (y * z).sum(-1) * lx + (z * x).sum(-1) * ly
        angle = 2.0 * torch.atan2(det, den).sum(1)
        signed = torch.where(angle.abs() > 2.0 * math.pi, -dist, dist)
        solid.append(signed <= 0.5 * dh)
        margin.append(torch.minimum((signed - 0.5 * dh).abs(), (angle.abs() - 2.0 * math.pi).abs()))
    return torch.cat(solid).cpu().numpy(), torch.cat(margin).cpu().numpy()


@pytest.mark.parametrize("mesh", [_dented, _cavity, _pair, _open])
@pytest.mark.parametrize("dh", [0.0021, 0.0034])
def test_baked_nodes_match_every_distance(mesh, dh, gpu_lib):
    from eulersf_gb300.bake import rasterize_solid
    verts, faces = mesh()
    res, _, origin, mass, total = rasterize_solid(verts, faces, dh, 700.0)
    solid, margin = _margin_and_solid(verts, faces, res, origin, dh)
    got = mass.reshape(-1)
    assert np.all((got == 0.0) | (got == 700.0))
    assert not np.any(((got > 0) != solid) & (margin > 1e-6 * max(res) * dh))
    assert total == np.count_nonzero(got) * 700.0 * dh * dh * dh
