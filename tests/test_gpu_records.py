"""renderD keeps the paths' replay records for its backward: the gradients are bitwise those of
the backward that re-traces the paths (batch_records = -1), which is also what a backward
falls back to when the scene, a texture or a camera changed in between, and on a second
backward through the same graph."""
import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import synth
from helpers import to_torch_scene

pytestmark = pytest.mark.gpu

KINDS = {"verts", "tex", "emit", "light_verts"}


def _spec(rough=False, ortho=False, views=1):
    spec = synth.sphere_scene(level=2, tex_hw=9, noise_sigma=0.03, height=19, width=23)
    if rough:
        spec.meshes[0].roughness = np.full(1, 0.5, np.float32)
    spec.cameras = [synth.CameraSpec(np.array([0.4 * k, 0.5, 4], np.float32), np.zeros(3, np.float32),
                                     np.array([0, 1, 0], np.float32), 3.0 if ortho else 0.8, 19 + 4 * k, 23 - 2 * k,
                                     1 if ortho else 0) for k in range(views)]
    return spec


def _run(spec, records, between=None, twice=False, **kw):
    scene, T = to_torch_scene(spec, requires_grad=KINDS)
    integ = dr.PathIntegrator(batch_records=records, primary_edge_hypercube_resolution=300,
                              secondary_edge_hypercube_resolution=[100, 2, 2], **kw)
    imgs = integ.renderD(scene)
    if between is not None:
        between(scene)
    g = [torch.tensor(np.random.default_rng(k).normal(size=tuple(i.shape)), dtype=torch.float32, device="cuda")
         for k, i in enumerate(imgs)]
    for _ in range(2 if twice else 1):
        torch.autograd.backward(imgs, g, retain_graph=twice)
    return [i.detach() for i in imgs], {k: t.grad for k, t in T.items() if t is not None and t.grad is not None}


def _same(a, b):
    assert all(torch.equal(x, y) for x, y in zip(a[0], b[0]))
    assert a[1].keys() == b[1].keys()
    for k in a[1]:
        assert torch.equal(a[1][k], b[1][k]), k


@pytest.mark.parametrize("estimator", ["reference", "unbiased"])
@pytest.mark.parametrize("case", [dict(), dict(rough=True), dict(ortho=True), dict(views=3)])
@pytest.mark.parametrize("kw", [dict(spp_interior=1, max_bounce=1), dict(spp_interior=5, max_bounce=4),
                                dict(spp_interior=8, max_bounce=2, mis_light_samples=2, mis_bsdf_samples=0, tile_paths=1024,
                                     enable_light_visable=True)])
def test_records_give_the_replayed_gradients(cuda, estimator, case, kw):
    spec = _spec(**case)
    _same(_run(spec, 0, estimator=estimator, **kw), _run(spec, -1, estimator=estimator, **kw))


def _move(scene):
    scene.meshes[0].set_vertices(scene.meshes[0].v * 1.05)
    scene.update()


def _repaint(scene):
    scene.meshes[0].material.texture.data.mul_(0.5)


def _turn(scene):
    with torch.no_grad():
        scene.cameras[0].look_from.add_(torch.tensor([0.1, 0.0, 0.0], device="cuda"))


@pytest.mark.parametrize("between", [_move, _repaint, _turn])
def test_changes_in_between_are_seen(cuda, between):
    kw = dict(spp_interior=4, max_bounce=3, gradient_terms=1)
    _same(_run(_spec(), 0, between, **kw), _run(_spec(), -1, between, **kw))


def test_second_backward(cuda):
    kw = dict(spp_interior=4, max_bounce=3)
    _same(_run(_spec(), 0, twice=True, **kw), _run(_spec(), -1, twice=True, **kw))
