"""The geometry build at the sizes where its kernels change path: warp and 32-group ends of
the node-box levels, the 2048-key sort tile (683 triangles are 2049 half-edges), the 32- and
64-bit half-edge keys (65,536 vertices) and the hand-over of subtrees to warps. Hits against
brute force bit for bit, edges against a host grouping of the half-edges, after a full build
and after a refit."""
import ctypes as C

import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import _lib as L
from torch_psdr_b200 import synth
from helpers import to_torch_scene
from test_gpu_parity import _stream, gpu_intersect

pytestmark = pytest.mark.gpu

GREY = np.array([0.5, 0.5, 0.5], np.float32)


def _soup(n, rng):
    """n small disjoint triangles in the unit cube (3 n vertices)."""
    c = rng.uniform(0, 1, (n, 1, 3))
    V = (c + rng.normal(0, 0.3 / max(1.0, n) ** (1 / 3), (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    return V, np.arange(3 * n, dtype=np.int32).reshape(n, 3)


def _strip(n, rng):
    """n triangles of a bumpy strip, neighbours sharing an edge."""
    k = np.arange(n + 2)
    V = np.stack([k / n, (k % 2) * 0.1, 0.05 * rng.normal(size=n + 2)], -1).astype(np.float32)
    f = np.arange(n)
    return V, np.stack([f, f + 1 + f % 2, f + 2 - f % 2], -1).astype(np.int32)


def _edges(scene, cap):
    v01 = torch.empty((cap, 2), dtype=torch.int32, device="cuda")
    geo = torch.empty((cap, 16), dtype=torch.float32, device="cuda")
    n = C.c_int64()
    L.check(L.load().psdr_scene_edges(scene.handle, v01.data_ptr(), geo.data_ptr(), cap, C.byref(n), _stream()), "edges")
    return v01[:n.value].cpu().numpy(), geo[:n.value].cpu().numpy()


@pytest.mark.parametrize("kind,n", [("soup", 1), ("soup", 2), ("strip", 2), ("soup", 3), ("strip", 31), ("strip", 32),
                                    ("strip", 33), ("soup", 682), ("strip", 683), ("strip", 1025), ("soup", 1365),
                                    ("strip", 5000), ("soup", 21845), ("soup", 21846), ("strip", 70000)])
def test_build_and_refit(cuda, kind, n):
    rng = np.random.default_rng(n)
    V, F = (_soup if kind == "soup" else _strip)(n, rng)
    spec = synth.SceneSpec([synth.MeshSpec(V, F, None, None, GREY)], [], [synth.default_camera(4, 4)])
    scene, _ = to_torch_scene(spec)
    target = V[F[rng.integers(0, n, 512)]].mean(1) + rng.normal(0, 0.01, (512, 3))
    o = rng.uniform(-1, 2, (512, 3))
    rays = np.concatenate([o, (target - o) / np.linalg.norm(target - o, axis=1, keepdims=True)], 1).astype(np.float32)
    for step in ("build", "refit"):
        if step == "refit":
            V = (V * np.float32(1.1) + np.float32(0.02)).astype(np.float32)
            scene.meshes[0].set_vertices(torch.tensor(V, device="cuda"))
            scene.update(refit=True)
        brute = gpu_intersect(scene, rays, 1)
        for mode in (0, 2):
            for got, want in zip(gpu_intersect(scene, rays, mode), brute):
                np.testing.assert_array_equal(got, want, err_msg=f"{step}, mode {mode}")
        # edges: the (min, max) vertex pairs in order, lengths exactly rounded from the vertices
        he = np.sort(np.concatenate([F[:, [0, 1]], F[:, [1, 2]], F[:, [2, 0]]]), axis=1)
        want = np.unique(he, axis=0)
        v01, geo = _edges(scene, 3 * n)
        np.testing.assert_array_equal(v01, want)
        length = np.linalg.norm(V[want[:, 0]].astype(np.float64) - V[want[:, 1]], axis=1)
        # three squares, two sums and a root in 32 bits: within 4 ulp
        np.testing.assert_allclose(geo[:, 15], length, rtol=4 * 2.0 ** -24)


def test_kept_tree_renders_as_a_new_one(cuda):
    """Refits after moves that change every box, on a scene with several objects."""
    spec = synth.large_scene(n_spheres=3, level=3, tex_hw=8, height=24, width=20)
    scene, _ = to_torch_scene(spec)
    integ = dr.PathIntegrator(spp_interior=4, max_bounce=3)
    for k in range(2):
        for m, s in zip(scene.meshes[:3], spec.meshes):
            s.vertices = (s.vertices * np.float32(0.9) + np.float32(0.1 * k)).astype(np.float32)
            m.set_vertices(torch.tensor(s.vertices, device="cuda"))
        scene.update(refit=True)
        fresh, _ = to_torch_scene(spec)
        assert torch.equal(integ.renderC(scene)[0], integ.renderC(fresh)[0])


def test_index_bounds(cuda):
    """psdr_index_bounds over more buffers than one launch takes, empty ones and both ends of
    the 32-bit range among them."""
    rng = np.random.default_rng(0)
    bufs = [rng.integers(-2 ** 31, 2 ** 31, size=n, dtype=np.int64).astype(np.int32)
            for n in (1, 31, 257, 0, 100000) + (3,) * 35]
    bufs.append(np.array([2 ** 31 - 1, -2 ** 31, 0], np.int32))
    dev = [torch.tensor(b, device="cuda") for b in bufs]
    n = len(bufs)
    out = (C.c_int32 * (2 * n))()
    L.check(L.load().psdr_index_bounds((C.c_void_p * n)(*[t.data_ptr() for t in dev]),
                                       (C.c_int64 * n)(*[b.size for b in bufs]), n, out, _stream()), "bounds")
    for i, b in enumerate(bufs):
        want = (b.min(), b.max()) if b.size else (2 ** 31 - 1, -2 ** 31)
        assert (out[2 * i], out[2 * i + 1]) == want, i
