"""Explicit gradient_terms masks over environment lights with DiffuseMaterial meshes only: the
BRDF-jump bit (16) adds nothing without a DiffuseBsdfMaterial mesh, also where the job has many
more paths (its samples) than any other boundary term has samples."""
import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from helpers import to_torch_scene
from test_gpu_envlight import compact_env_spec

pytestmark = pytest.mark.gpu


def _grads(spec, terms, batch, records=0):
    scene, T = to_torch_scene(spec, requires_grad={"verts", "tex", "env", "cam"})
    it = dr.PathIntegrator(estimator="unbiased", gradient_terms=terms, spp_interior=64, max_bounce=2,
                           batch_records=records, primary_edge_hypercube_resolution=100,
                           secondary_edge_hypercube_resolution=[20, 2, 2])
    img = (dr.BatchRender(it, [scene]).renderD() if batch else it.renderD(scene))[0]
    img.backward(torch.as_tensor(np.random.default_rng(3).normal(size=tuple(img.shape)), dtype=torch.float32, device="cuda"))
    return {k: t.grad for k, t in T.items() if t is not None and t.grad is not None}


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("terms", [1, 111])
def test_jump_bit_without_rough_meshes_adds_nothing(cuda, kind, batch, terms):
    spec = compact_env_spec(kind, height=33, width=31)
    want, got = _grads(spec, terms, batch), _grads(spec, terms | 16, batch)
    assert len(want) >= 4 and want.keys() == got.keys()
    for k in want:
        assert torch.equal(want[k], got[k]), k


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("batch", [False, True])
def test_jump_bit_alone_gives_zeros(cuda, kind, batch):
    got = _grads(compact_env_spec(kind, height=33, width=31), 16, batch)
    assert len(got) >= 4 and not any(t.any() for t in got.values())


@pytest.mark.parametrize("kind", [1, 2])
def test_kept_records_over_an_environment_light(cuda, kind):
    spec = compact_env_spec(kind, height=33, width=31)
    kept, replayed = _grads(spec, 127, False), _grads(spec, 127, False, records=-1)
    for k in kept:
        assert torch.equal(kept[k], replayed[k]), k
