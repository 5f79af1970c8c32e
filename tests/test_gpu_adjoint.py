"""The interior adjoint of DiffuseMaterial scenes works on its path vertices and light hits
from per-warp lists. The kernel for material scenes walks each path on its own, and a
DiffuseBsdfMaterial of roughness 0 is the same material: both must give the same gradients,
at depths, sample counts and image sizes that leave lists empty, part-filled and full."""
import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import synth
from helpers import rel_l2, to_torch_scene

pytestmark = pytest.mark.gpu

KINDS = {"verts", "tex", "emit", "light_verts"}


def _grads(rough, size, kw):
    spec = synth.sphere_scene(level=2, tex_hw=9, noise_sigma=0.05, height=size[0], width=size[1])
    if rough:
        for m in spec.meshes:
            m.roughness = np.zeros(1, np.float32)
    scene, T = to_torch_scene(spec, requires_grad=KINDS)
    img = dr.PathIntegrator(gradient_terms=1, **kw).renderD(scene)[0]
    w = np.random.default_rng(1).normal(size=tuple(img.shape))
    img.backward(torch.tensor(w, dtype=torch.float32, device="cuda"))
    return img.detach(), {k: t.grad.cpu().numpy() for k, t in T.items() if t is not None and t.grad is not None}


@pytest.mark.parametrize("estimator", ["reference", "unbiased"])
@pytest.mark.parametrize("size,spp,depth,nl,nb", [((1, 1), 1, 1, 1, 1), ((3, 5), 1, 2, 1, 0), ((7, 9), 3, 1, 0, 1),
                                                  ((33, 31), 32, 3, 1, 1), ((40, 24), 5, 6, 2, 3),
                                                  ((16, 16), 16, 16, 0, 16)])
def test_list_adjoint_matches_path_walk(cuda, estimator, size, spp, depth, nl, nb):
    kw = dict(estimator=estimator, spp_interior=spp, max_bounce=depth, mis_light_samples=nl, mis_bsdf_samples=nb,
              enable_light_visable=True)
    a_img, a = _grads(False, size, kw)
    b_img, b = _grads(True, size, kw)
    # the images agree to the rounding of the two kernels' material code
    np.testing.assert_allclose(a_img.cpu(), b_img.cpu(), rtol=1e-5, atol=1e-6)
    assert a.keys() == b.keys()
    for k in a:
        if not np.any(b[k]):
            assert not np.any(a[k]), k
            continue
        # sums of the same fp32 terms in another grouping: about sqrt(terms) 2^-24 of their size,
        # and terms of both signs cancel to about a tenth of it
        assert rel_l2(a[k], b[k]) < 2e-5, (k, rel_l2(a[k], b[k]))


@pytest.mark.parametrize("estimator", ["reference", "unbiased"])
@pytest.mark.parametrize("size,spp,depth,nl,nb", [((1, 1), 1, 1, 1, 1), ((7, 9), 3, 1, 0, 1), ((33, 31), 32, 3, 1, 1),
                                                  ((40, 24), 5, 6, 2, 3)])
@pytest.mark.parametrize("batch", [False, True])
def test_other_gradients_do_not_depend_on_vertex_gradients(cuda, estimator, size, spp, depth, nl, nb, batch):
    """The kernel without vertex gradients forms the same texel, emission and camera adjoints."""
    spec = synth.sphere_scene(level=2, tex_hw=9, noise_sigma=0.05, height=size[0], width=size[1])
    d_image = torch.as_tensor(np.random.default_rng(1).normal(size=size + (3,)), dtype=torch.float32, device="cuda")
    out = []
    for kinds in ({"tex", "emit", "cam"}, {"tex", "emit", "cam", "verts", "light_verts"}):
        scene, T = to_torch_scene(spec, requires_grad=kinds)
        it = dr.PathIntegrator(gradient_terms=1, estimator=estimator, spp_interior=spp, max_bounce=depth,
                               mis_light_samples=nl, mis_bsdf_samples=nb, enable_light_visable=True)
        img = dr.BatchRender(it, [scene]).renderD()[0] if batch else it.renderD(scene)[0]
        img.backward(d_image)
        out.append((img.detach().clone(), {k: t.grad.clone() for k, t in T.items() if k.startswith(("tex", "emit", "cam"))
                                           and t is not None and t.grad is not None}))
    assert torch.equal(out[0][0], out[1][0])
    assert out[0][1] and out[0][1].keys() == out[1][1].keys()
    for k, a in out[0][1].items():
        if torch.equal(a, out[1][1][k]):
            continue
        # the same fp32 terms up to the rounding of differently contracted products, summed in
        # fixed point
        assert rel_l2(a.cpu().numpy(), out[1][1][k].cpu().numpy()) < 1e-6, k
