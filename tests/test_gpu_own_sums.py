"""The sums that a thread keeps of its own contributions to one gradient (light vertices and
emission of a scene's first lights, camera origin and lens) are exact: with whole 32-path groups
per tile no gradient depends on the tile, several lights or scenes in a job give what the
scattered accumulation gives, and contributions beyond a thread's range go to the accumulators."""
import numpy as np
import pytest
import torch

import orc
import torch_psdr_b200 as dr
from torch_psdr_b200 import synth
from helpers import to_torch_scene

pytestmark = pytest.mark.gpu

KINDS = {"verts", "tex", "light_verts", "emit", "cam"}
KW = dict(spp_interior=16, spp_primary_edge=2, spp_secondary_edge=2, max_bounce=3, enable_light_visable=True,
          primary_edge_hypercube_resolution=300, secondary_edge_hypercube_resolution=[100, 2, 2])


def _spec(lights=1, fan=0, size=64, rough=False):
    """A noisy sphere over the ground under `lights` small lights, the first with `fan` vertices
    (0: the four of a square)."""
    spec = synth.sphere_scene(level=2, tex_hw=9, noise_sigma=0.03, height=size, width=size)
    if rough:
        spec.meshes[0].roughness = np.full(1, 0.5, np.float32)
    spec.lights = []
    for j in range(lights):
        V, F = synth.quad((1.1 * j - 2.0, 0.3 * j), 0.4, 3.0 - 0.1 * j, facing_down=True)
        spec.lights.append(synth.LightSpec(V, F, np.array([20, 10 + j, 5 * j + 1], np.float32)))
    if fan:
        a = np.linspace(0, 2 * np.pi, fan - 1, endpoint=False)
        V = np.concatenate([np.array([[0, 3, 0]]), np.stack([0.5 * np.cos(a), 3 + 0 * a, 0.5 * np.sin(a)], 1)])
        k = np.arange(1, fan)
        F = np.stack([0 * k, k, k % (fan - 1) + 1], 1)
        spec.lights[0] = synth.LightSpec(V.astype(np.float32), F.astype(np.int32), spec.lights[0].emit)
    return spec


def _grads(spec, scale=1.0, lens=False, **kw):
    scene, T = to_torch_scene(spec, requires_grad=KINDS)
    if lens:
        c = spec.cameras[0]
        T = {n: torch.tensor(np.atleast_1d(getattr(c, n)), dtype=torch.float32, device="cuda", requires_grad=True)
             for n in ("look_from", "look_at", "up", "vfov")}
        scene = dr.Scene([dr.PerspectiveCamera(*T.values(), c.height, c.width)], scene.meshes, scene.lights)
    img = dr.PathIntegrator(**dict(KW, **kw)).renderD(scene)[0]
    g = np.random.default_rng(7).normal(size=tuple(img.shape)) * scale
    img.backward(torch.tensor(g, dtype=torch.float32, device="cuda"))
    return {k: v.grad.cpu().numpy() for k, v in T.items() if v is not None and v.grad is not None}


@pytest.mark.parametrize("estimator", ["reference", "unbiased"])
@pytest.mark.parametrize("case", [dict(), dict(lights=6), dict(fan=12), dict(rough=True, lights=2)])
def test_tiles_give_bitwise_equal_gradients(cuda, estimator, case):
    spec = _spec(size=256, **case)  # 2^20 paths: some fourteen to a thread in one tile
    want = _grads(spec, estimator=estimator)
    assert len(want) >= 5
    for records, tile in ((0, 1 << 14), (-1, 1 << 18)):
        got = _grads(spec, estimator=estimator, tile_paths=tile, batch_records=records)
        for k in want:
            assert want[k].any(), k
            assert np.array_equal(want[k], got[k]), (tile, k)


def test_tiles_give_bitwise_equal_lens_gradients(cuda):
    want, got = (_grads(_spec(size=256), lens=True, estimator="unbiased", tile_paths=t) for t in (0, 1 << 14))
    for k in want:
        assert want[k].any() and np.array_equal(want[k], got[k]), k


@pytest.mark.parametrize("estimator", ["reference", "unbiased"])
def test_scenes_of_a_batch_give_the_plain_gradients(cuda, estimator):
    """Three scenes of one, six and one lights; every view holds whole groups of 32 paths, so
    the batch sums the same terms as three plain steps."""
    specs = [_spec(size=128), _spec(lights=6, size=160), _spec(fan=12, size=192)]
    plain, Ts, scenes = [_grads(s, estimator=estimator) for s in specs], [], []
    for s in specs:
        scene, T = to_torch_scene(s, requires_grad=KINDS)
        scenes.append(scene)
        Ts.append(T)
    imgs = dr.BatchRender(dr.PathIntegrator(estimator=estimator, **KW), scenes).renderD()
    gs = [torch.tensor(np.random.default_rng(7).normal(size=tuple(i.shape)), dtype=torch.float32, device="cuda")
          for i in imgs]
    torch.autograd.backward(imgs, gs)
    for p, T in zip(plain, Ts):
        for k, g in p.items():
            assert np.array_equal(T[k].grad.cpu().numpy(), g), k


def test_emission_of_many_lights_matches_oracle(cuda):
    spec = _spec(lights=6, size=33)
    kw = dict(spp_interior=8, max_bounce=3, enable_light_visable=True)
    g = np.random.default_rng(7).normal(size=(33, 33, 3))
    got = _grads(spec, gradient_terms=1, **kw)
    seeds = np.random.default_rng(5).normal(size=(6, 3, 8))
    want = orc.grad_dir(spec, [g], which=1, seed_emit=seeds, **kw)
    dirs = sum(np.einsum("c,cd->d", got[f"emit{j}"].astype(np.float64), seeds[j]) for j in range(6))
    # the bound of the emission parity tests: rounding of 32-bit path terms
    np.testing.assert_allclose(dirs, want, atol=1e-4 * np.abs(want).max())


@pytest.mark.parametrize("estimator", ["reference", "unbiased"])
def test_large_contributions(cuda, estimator):
    """A loss scaled by a power of two scales every term exactly; its terms and sums pass a
    thread's range of 512."""
    want = _grads(_spec(), estimator=estimator)
    for e in (12, 24):
        got = _grads(_spec(), scale=2.0 ** e, estimator=estimator)
        for k in want:
            # (each term is rounded to 2^-52 before the scale and after it)
            np.testing.assert_allclose(got[k] * 2.0 ** -e, want[k], rtol=3e-7, atol=1e-9 * np.abs(want[k]).max())
