"""Large tiles make the light test of MIS BSDF-sample rays where they are sampled and list
the rays that need a traversal; small tiles make it as the ray is traversed. A job cut into
small tiles must render the same bits and the same gradients up to the partial sums that
warps keep in fp32 (texel and emission gradients of a tile's consecutive paths)."""
import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import synth
from helpers import rel_l2, to_torch_scene

pytestmark = pytest.mark.gpu

KW = dict(spp_interior=64, max_bounce=3, gradient_terms=1)


def _spec(light, level=2, size=(97, 91)):
    spec = synth.sphere_scene(level=level, tex_hw=9, noise_sigma=0.05, height=size[0], width=size[1])
    if light == "fine":  # more triangles than the light test takes
        V, F = synth.icosphere(1, 0.7)
        spec.lights[0].vertices = (V + np.array([0.0, 3.0, 0.0])).astype(np.float32)
        spec.lights[0].faces = F
    elif light == "two":
        l = spec.lights[0]
        spec.lights.append(synth.LightSpec(l.vertices - np.array([1.0, 0.5, 1.0], np.float32), l.faces, 0.5 * l.emit))
    return spec


def _run(specs, tile, batch, **kw):
    made = [to_torch_scene(s, requires_grad={"verts", "tex", "emit"}) for s in specs]
    it = dr.PathIntegrator(tile_paths=tile, **{**KW, **kw})
    if batch:
        imgs = dr.BatchRender(it, [m[0] for m in made]).renderD()
    else:
        imgs = [im for m in made for im in it.renderD(m[0])]
    rng = np.random.default_rng(3)
    torch.autograd.backward(imgs, [torch.as_tensor(rng.normal(size=tuple(i.shape)), dtype=torch.float32, device="cuda")
                                   for i in imgs])
    return [i.detach().clone() for i in imgs], [t.grad.cpu().numpy() for _, T in made for t in T.values()
                                                if t is not None and t.grad is not None]


def _same(a, b):
    assert len(a[0]) == len(b[0]) and len(a[1]) == len(b[1]) > 2
    for x, y in zip(a[0], b[0]):
        assert torch.equal(x, y), (x - y).abs().max()
    for x, y in zip(a[1], b[1]):
        # the same fp32 terms in another grouping
        assert np.array_equal(x, y) or rel_l2(x, y) < 2e-5, rel_l2(x, y)


# 97 x 91 x 64 = 564928 paths: a tile above the line of 2^19 and, cut at 2^18, two and a bit below
@pytest.mark.parametrize("light,nl,nb", [("lamp", 1, 1), ("lamp", 0, 1), ("lamp", 2, 3), ("lamp", 1, 0),
                                         ("fine", 1, 1), ("two", 1, 2)])
def test_listed_rays_match_small_tiles(cuda, light, nl, nb):
    kw = dict(mis_light_samples=nl, mis_bsdf_samples=nb)
    _same(_run([_spec(light)], 1 << 20, False, **kw), _run([_spec(light)], 1 << 18, False, **kw))


def test_most_samples(cuda):
    spec = _spec("lamp", level=1, size=(725, 726))
    kw = dict(mis_bsdf_samples=16, spp_interior=1, max_bounce=1)
    _same(_run([spec], 1 << 20, False, **kw), _run([spec], 1 << 18, False, **kw))


def test_several_scenes_in_a_tile(cuda):
    specs = [_spec("lamp", 2), _spec("two", 1, (64, 80))]
    _same(_run(specs, 1 << 20, True), _run(specs, 1 << 18, False))
