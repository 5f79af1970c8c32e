"""Hits exactly on edges and vertices: the barycentrics are the oracle's bit for bit, the signs of
their zeros included, for directions of either sign along every axis."""
import numpy as np
import pytest
import torch

import orc
import torch_psdr_b200 as dr
from torch_psdr_b200 import synth
from helpers import to_torch_scene
from test_gpu_parity import gpu_intersect

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("flip", [False, True])
def test_zero_barycentrics(cuda, axis, sign, flip):
    """A square of two triangles across `axis`; rays through a grid of its points with coordinates
    that fp32 holds exactly: its edges, diagonal and corners among them."""
    u, v = (axis + 1) % 3, (axis + 2) % 3
    V = np.zeros((4, 3), np.float32)
    V[:, u], V[:, v] = [0, 2, 2, 0], [0, 0, 2, 2]
    F = np.array([[0, 1, 2], [0, 2, 3]], np.int32)
    if flip:
        F = F[:, ::-1].copy()
    spec = synth.SceneSpec([synth.MeshSpec(V, F, None, None, np.full(3, 0.5, np.float32))], [], [synth.default_camera(4, 4)])
    a, b = np.meshgrid(np.arange(17) / 8.0, np.arange(17) / 8.0)
    rays = []
    for du, dv in ((0.0, 0.0), (0.25, 0.0), (0.0, -0.25), (0.25, 0.25), (-0.25, 0.5)):
        r = np.zeros((a.size, 6), np.float32)
        r[:, 3 + axis], r[:, 3 + u], r[:, 3 + v] = sign, du, dv
        r[:, axis], r[:, u], r[:, v] = -2.0 * sign, a.ravel() - 2.0 * du, b.ravel() - 2.0 * dv
        rays.append(r)
    rays = np.concatenate(rays)
    tri, bary, t = orc.intersect(spec, rays, use_bvh=False)
    zero = (tri >= 0)[:, None] & (bary == 0)
    assert zero.sum() > 100
    scene, _ = to_torch_scene(spec)
    for mode in (0, 1, 2):
        g_tri, g_bary, g_t = gpu_intersect(scene, rays, mode)
        np.testing.assert_array_equal(g_tri, tri)
        hit = tri >= 0
        np.testing.assert_array_equal(g_bary[hit].view(np.int32), bary[hit].view(np.int32))
        np.testing.assert_array_equal(g_t[hit].view(np.int32), t[hit].view(np.int32))
