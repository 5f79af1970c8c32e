"""Forwards whose replay records are not kept give the gradients of those whose records are:
graphs beyond the memory limit, scenes made under inference mode, and camera gradients."""
import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import api, synth
from helpers import to_torch_scene

pytestmark = pytest.mark.gpu

KINDS = {"verts", "tex", "emit", "light_verts", "cam"}


def _spec(k=0, size=128):
    spec = synth.sphere_scene(level=2, tex_hw=9, noise_sigma=0.03, height=size, width=size)
    spec.cameras[0].look_from = spec.cameras[0].look_from + np.float32(0.1 * k)
    return spec


def _integ(records, spp=32, **kw):
    return dr.PathIntegrator(batch_records=records, spp_interior=spp, max_bounce=3, estimator="unbiased",
                             primary_edge_hypercube_resolution=300, secondary_edge_hypercube_resolution=[100, 2, 2], **kw)


def _loss(img):
    w = torch.as_tensor(np.random.default_rng(1).normal(size=tuple(img.shape)), dtype=torch.float32, device="cuda")
    return (img * w).sum()


def _equal(a, b):
    got = {k: t.grad for k, t in a.items() if t is not None and t.grad is not None}
    assert len(got) >= 5
    for k, g in got.items():
        assert torch.equal(g, b[k].grad), k


def test_graphs_beyond_the_limit_retrace(cuda, monkeypatch):
    """Three losses before one backward; the records of one (138 MB) fit the quarter."""
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (700 << 20, 0))
    none = {k: {"all": {"current": 0}} for k in ("reserved_bytes", "allocated_bytes")}
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda *a: none)
    dev = torch.device("cuda", torch.cuda.current_device())
    before, out = api._Records.held(dev), []
    for records in (0, -1):
        integ = _integ(records)
        built = [to_torch_scene(_spec(k), requires_grad=KINDS) for k in range(3)]
        total = sum(_loss(integ.renderD(scene)[0]) for scene, _ in built)
        held = api._Records.held(dev) - before
        assert (100 << 20) < held < (200 << 20) if records == 0 else held == 0
        total.backward()
        out.append([T for _, T in built])
    assert api._Records.held(dev) == before
    for a, b in zip(*out):
        _equal(a, b)


def test_scene_made_under_inference_mode(cuda):
    with torch.inference_mode():
        made = to_torch_scene(_spec(size=24))[0]
    T = {}
    out = []
    for inside in (True, False):
        spec = _spec(size=24)
        _, T = to_torch_scene(spec, requires_grad=KINDS)
        mesh = [(T[f"verts{i}"], T[f"tex{i}"]) for i in range(len(spec.meshes))]
        with torch.inference_mode(inside):
            meshes = [dr.Mesh(v, None, torch.as_tensor(m.faces, dtype=torch.int32, device="cuda"), None,
                              dr.DiffuseMaterial(t)) for (v, t), m in zip(mesh, spec.meshes)]
            light = dr.AreaLight(T["lverts0"], torch.as_tensor(spec.lights[0].faces, dtype=torch.int32, device="cuda"),
                                 T["emit0"])
            scene = dr.Scene(made.cameras, meshes, [light])
        img = _integ(0, spp=4).renderD(scene)[0]
        _loss(img).backward()
        out.append((img.detach(), [t.grad for t in T.values() if t is not None and t.grad is not None]))
    assert torch.equal(out[0][0], out[1][0]) and len(out[0][1]) >= 4
    for a, b in zip(out[0][1], out[1][1]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("estimator", ["reference", "unbiased"])
def test_camera_gradients_from_kept_records(cuda, estimator):
    """The camera's origin and, for the unbiased estimator, its lens (look_at, up, fov)."""
    out = []
    for records in (1, -1):
        spec = _spec(size=24)
        scene, _ = to_torch_scene(spec)
        c = spec.cameras[0]
        par = [torch.tensor(np.atleast_1d(x), dtype=torch.float32, device="cuda", requires_grad=True)
               for x in (c.look_from, c.look_at, c.up, c.vfov)]
        scene = dr.Scene([dr.PerspectiveCamera(*par, 24, 24)], scene.meshes, scene.lights)
        integ = dr.PathIntegrator(batch_records=records, spp_interior=9, max_bounce=3, estimator=estimator)
        _loss(integ.renderD(scene)[0]).backward()
        out.append([p.grad for p in par])
    assert all(g.any() for g in out[0][:1 if estimator == "reference" else 4])
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_records_give_way_to_the_workspace(cuda):
    """Memory for the records or for the render's workspace, not for both: the records go (unless
    the library still keeps that much from earlier objects), and the backward re-traces."""
    scene, T = to_torch_scene(_spec(), requires_grad=KINDS)
    want_scene, want = to_torch_scene(_spec(), requires_grad=KINDS)
    img = _integ(-1).renderD(want_scene)[0]
    _loss(img).backward()
    integ = _integ(1)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # records of 138 MB; the workspace takes 160 MB
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (260 << 20), dtype=torch.uint8, device="cuda")
    got = integ.renderD(scene)[0]
    del hog
    _loss(got).backward()
    assert torch.equal(img.detach(), got.detach())
    _equal(want, T)
