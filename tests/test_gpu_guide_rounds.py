"""Many preprocess rounds of the shadow-boundary guide: each round finds its place in the cells'
sampler streams without stepping through the earlier rounds' draws."""
import numpy as np
import pytest
import torch

import orc
import torch_psdr_b200 as dr
from helpers import gradient_case, to_torch_scene

pytestmark = pytest.mark.gpu


def test_many_rounds_match_oracle(cuda):
    """As the guide tests at few rounds: the same samples, or an estimate that is tens of percent off."""
    spec, mesh = gradient_case("shadow", 33, 33)
    kw = dict(spp_interior=1, spp_secondary_edge=4, max_bounce=2, secondary_edge_hypercube_resolution=[20, 2, 2],
              secondary_edge_preprocess_rounds=37)
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
    np.testing.assert_allclose(got, want, atol=2e-3 * np.abs(want).max())


def test_time_is_linear_in_the_rounds(cuda):
    spec, _ = gradient_case("shadow", 33, 33)

    def ms(rounds):
        integ = dr.PathIntegrator(estimator="unbiased", gradient_terms=4, spp_interior=1, spp_secondary_edge=1,
                                  max_bounce=2, secondary_edge_hypercube_resolution=[2000, 4, 4],
                                  secondary_edge_preprocess_rounds=rounds)
        best = np.inf
        for _ in range(4):
            img = integ.renderD(to_torch_scene(spec, requires_grad={"verts"})[0])[0]
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            img.backward(torch.ones_like(img))
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]))
        return best

    few, many = ms(64), ms(1024)
    print(f"64 rounds {few:.2f} ms, 1024 rounds {many:.2f} ms")
    # 16 times the rounds; stepping through the draws would make it some hundred times the steps
    assert many < 24 * few
