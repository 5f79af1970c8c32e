"""Preprocess rounds of the shadow-boundary guide run several to a launch, each drawing from its
own place in its cells' sampler streams and adding its masses in order. Against the oracle,
which runs them one after another, at round counts below, at and beyond one launch's share
(8 rounds; the unbiased estimator runs four per requested round), and at cell counts that
leave the launch's queue part-filled."""
import numpy as np
import pytest
import torch

import orc
import torch_psdr_b200 as dr
from helpers import gradient_case, to_torch_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounds,cells", [(1, [40, 2, 2]), (2, [7, 3, 1]), (3, [40, 2, 2]), (5, [1, 1, 1])])
def test_guide_rounds_match_oracle(cuda, rounds, cells):
    spec, mesh = gradient_case("shadow", 33, 33)
    kw = dict(spp_interior=1, spp_secondary_edge=4, max_bounce=2, secondary_edge_hypercube_resolution=cells,
              secondary_edge_preprocess_rounds=rounds)
    g = np.random.default_rng(2).normal(size=(33, 33, 3))
    nv = sum(m.vertices.shape[0] for m in spec.meshes) + sum(l.vertices.shape[0] for l in spec.lights)
    seeds = np.zeros((nv, 3, 8))
    n0 = spec.meshes[mesh].vertices.shape[0]
    seeds[:n0] = np.random.default_rng(3).normal(size=(n0, 3, 8))
    want = orc.grad_dir(spec, [g], which=4, mode=1, seed_verts=seeds, **kw)
    scene, T = to_torch_scene(spec, requires_grad={"verts"})
    img = dr.PathIntegrator(estimator="unbiased", gradient_terms=4, **kw).renderD(scene)[0]
    img.backward(torch.tensor(g, dtype=torch.float32, device="cuda"))
    got = np.einsum("vk,vkd->d", T[f"verts{mesh}"].grad.double().cpu().numpy(), seeds[:n0])
    # a guide built from other samples, or a round left out, moves the samples' cells and with
    # them the estimate by tens of percent; the same samples differ by 32-bit rounding only
    np.testing.assert_allclose(got, want, atol=2e-3 * np.abs(want).max())
