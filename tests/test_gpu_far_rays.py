"""Rays whose origins lie far outside the scene, and rays of very long or short direction vectors:
the traversal's box tests must not cull a triangle that brute force hits (bit for bit)."""
import ctypes as C

import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import _lib as L
from torch_psdr_b200 import synth
from test_gpu_parity import _stream

pytestmark = pytest.mark.gpu


def _scene(kind, scale):
    rng = np.random.default_rng(0)
    if kind == "sphere":
        V, F = synth.icosphere(4)
        V = synth.radial_noise(V, 0.02, 2)
    else:  # flat boxes: axis-aligned quads
        c, s = rng.uniform(0, 1, (1000, 1, 3)), 0.016
        k = np.arange(1000) % 3
        u, w = np.eye(3)[(k + 1) % 3][:, None] * s, np.eye(3)[(k + 2) % 3][:, None] * s
        V = np.concatenate([c - u - w, c + u - w, c + u + w, c - u + w], 1).reshape(-1, 3)
        q = 4 * np.arange(1000)[:, None]
        F = np.concatenate([q + [0, 1, 2], q + [0, 2, 3]])
    V = torch.as_tensor(V * scale, dtype=torch.float32, device="cuda")
    F = torch.as_tensor(F, dtype=torch.int32, device="cuda")
    mesh = dr.Mesh(V, None, F, None, dr.DiffuseMaterial(torch.full((3,), 0.5, device="cuda")))
    return dr.Scene([], [mesh], []), V.double(), F.long()


def _hits(scene, rays, mode):
    n = rays.shape[0]
    tri = torch.empty(n, dtype=torch.int32, device="cuda")
    bary, t = torch.empty((n, 2), device="cuda"), torch.empty(n, device="cuda")
    L.check(L.load().psdr_intersect(scene.handle, rays.data_ptr(), n, tri.data_ptr(), bary.data_ptr(), t.data_ptr(), mode,
                                    C.c_void_p(_stream().value)), "intersect")
    return tri, bary, t


@pytest.mark.parametrize("kind", ["sphere", "quads"])
@pytest.mark.parametrize("distance,length,scale", [(10.0, 1.0, 1.0), (100.0, 1.0, 1.0), (1000.0, 1.0, 1.0),
                                                   (2.0, 2.0 ** -40, 1.0), (2.0, 2.0 ** 60, 1.0),
                                                   (2.0, 1.9 * 2.0 ** 126, 1024.0)])
def test_hits_equal_brute_force(cuda, kind, distance, length, scale):
    scene, V, F = _scene(kind, scale)
    gen = torch.Generator(device="cuda").manual_seed(1)
    n = 1 << 17
    f = F[torch.randint(0, F.shape[0], (n,), generator=gen, device="cuda")]
    # targets inside triangles, on edges and at vertices
    w = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    w = w * (torch.rand((n, 3), generator=gen, device="cuda") > 0.5) + 1e-12
    target = (V[f] * (w / w.sum(1, keepdim=True))[:, :, None]).sum(1)
    u = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    u[: n // 4, 0] *= 1e-3  # nearly in an axis plane
    u /= u.norm(dim=1, keepdim=True)
    rays = torch.empty((n, 8), device="cuda")
    rays[:, :3] = target + u * distance * scale
    d = target - rays[:, :3].double()
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True) * length
    rays[:, 3], rays[:, 7] = 0.0, float("inf")
    brute = _hits(scene, rays, 1)
    assert (brute[0] >= 0).float().mean() > 0.5
    for mode in (0, 2):
        for got, want in zip(_hits(scene, rays, mode), brute):
            assert torch.equal(got, want)
