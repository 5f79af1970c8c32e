"""Jobs of several automatic tiles (2^20 to 2^22 paths, by lanes, records, memory and what the
workspace holds): the images and every gradient are bitwise the same for all of them, and for
tiles that the caller sets."""
import ctypes as C

import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import _lib as L
from torch_psdr_b200 import synth
from helpers import to_torch_scene

pytestmark = pytest.mark.gpu

KINDS = {"verts", "tex", "light_verts", "emit", "cam"}


def _step(spec, batch, spp, **kw):
    scene, T = to_torch_scene(spec, requires_grad=KINDS)
    integ = dr.PathIntegrator(spp_interior=spp, max_bounce=2, spp_primary_edge=1, spp_secondary_edge=1,
                              enable_light_visable=True, primary_edge_hypercube_resolution=500,
                              secondary_edge_hypercube_resolution=[100, 3, 3], **kw)
    imgs = dr.BatchRender(integ, [scene]).renderD() if batch else integ.renderD(scene)
    gs = [torch.as_tensor(np.random.default_rng(k).normal(size=tuple(i.shape)), dtype=torch.float32, device="cuda")
          for k, i in enumerate(imgs)]
    torch.autograd.backward(imgs, gs)
    return {**{f"image{k}": i.detach().clone() for k, i in enumerate(imgs)},
            **{k: t.grad.clone() for k, t in T.items() if t is not None and t.grad is not None}}


@pytest.mark.parametrize("estimator", ["reference", "unbiased"])
@pytest.mark.parametrize("spp", [32, 37])
def test_tile_choice_changes_nothing(cuda, estimator, spp):
    spec = synth.sphere_scene(level=3, tex_hw=65, noise_sigma=0.02, height=500, width=490)
    c = spec.cameras[0]
    # views of 245,000 and 10,201 pixels: 8.2 M and 9.4 M paths, an odd number of them in all
    spec.cameras.append(synth.CameraSpec(np.array([1.5, 0.5, 3.5], np.float32), c.look_at, c.up, c.vfov, 101, 101))
    want = _step(spec, False, spp, estimator=estimator, batch_records=-1, tile_paths=1 << 20)
    assert len(want) >= 7
    for batch, kw in ((False, dict(batch_records=-1)), (False, dict(batch_records=1)),
                      (False, dict(tile_paths=1 << 18)), (True, dict(batch_lanes=1, batch_records=-1)),
                      (True, dict(batch_lanes=4, batch_records=1)), (True, dict(batch_lanes=8, batch_records=-1))):
        got = _step(spec, batch, spp, estimator=estimator, **kw)
        assert want.keys() == got.keys()
        for k in want:
            assert want[k].any(), k
            assert torch.equal(want[k], got[k]), (batch, kw, k)


def test_workspace_history_changes_nothing(cuda):
    """A workspace that a larger job has grown, and one that has not."""
    big = synth.sphere_scene(level=2, tex_hw=9, height=512, width=512)
    small = synth.sphere_scene(level=3, tex_hw=9, noise_sigma=0.02, height=300, width=301)
    out = []
    for grown in (False, True):
        scene, T = to_torch_scene(small, requires_grad=KINDS)
        integ = dr.PathIntegrator(spp_interior=17, max_bounce=2, batch_records=-1)
        if grown:
            integ.renderC(to_torch_scene(big)[0])
        img = integ.renderD(scene)[0]
        img.backward(torch.as_tensor(np.random.default_rng(0).normal(size=(300, 301, 3)), dtype=torch.float32, device="cuda"))
        out.append([img.detach()] + [t.grad for t in T.values() if t is not None and t.grad is not None])
    for a, b in zip(*out):
        assert torch.equal(a, b)


def _trace_launches(run):
    lib = L.load()
    out, ms = (C.c_int64 * 3)(), C.c_double()
    L.check(lib.psdr_profile_enable(1), "enable")
    L.check(lib.psdr_profile_reset(), "reset")
    try:
        run()
        torch.cuda.synchronize()
        L.check(lib.psdr_profile_read(out, C.byref(ms)), "read")
    finally:
        lib.psdr_profile_enable(0)
    return out[1]


@pytest.mark.parametrize("spp", [32, 37])
def test_whole_groups_cut_no_extra_tile(cuda, spp):
    """One tile for a job that fits it, and one per lane for a batch, at any samples per pixel."""
    spec = synth.sphere_scene(level=1, tex_hw=9, height=170, width=171)
    scene, _ = to_torch_scene(spec)
    kw = dict(spp_interior=spp, max_bounce=2)
    assert _trace_launches(lambda: dr.PathIntegrator(**kw).renderC(scene)) == 2
    spec.cameras[0].height, spec.cameras[0].width = 499, 491
    scene, _ = to_torch_scene(spec)
    for lanes in (2, 4, 7):
        batch = dr.BatchRender(dr.PathIntegrator(batch_lanes=lanes, **kw), [scene], differentiable=False)
        tiles = max(lanes, -(-499 * 491 * spp // (1 << 21)))
        assert _trace_launches(batch.forward) == 2 * tiles, lanes
