"""Performance cases: the work that a user of torch_psdr_b200 has it do.

Every case is one pass through the public entry points on a synthetic scene of noisy
textured spheres over a ground quad under a square light (the scenes of
torch_psdr_b200.synth): plain renders (PathIntegrator.renderC), optimisation steps (a new
Scene, renderD, an L2 loss and its backward) and batched steps (BatchRender: persistent
scenes whose vertices are replaced, both directions replayed from CUDA graphs).

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a
program holds before the call, run() is one pass and exact() the same outputs in 64 bits
where plain torch arithmetic can give them (images and texture gradients of the simplest
scenes: the path estimator with the renderer's sample streams, every ray tested against
every triangle).

Fields of a case:
  mode        "render" (new Scene + renderC), "refit" / "update" (new vertices into a
              persistent Scene, psdr_scene_refit / full rebuild, renderC), "step" (new Scene,
              renderD, loss, backward) or "batch" (BatchRender step)
  spheres     number of spheres; one sits at the origin, more are spread over a 10^3 box
  freq        geodesic frequency of each sphere (20 freq^2 triangles)
  tex         texture size; 0 gives the spheres one colour each
  height, width, views, spp, depth, nl, nb   image size, cameras, samples, bounces, light and
              BSDF samples per vertex
  scenes      "batch" only: 3 assigns the views to three scenes of freq, 3 freq and 6 freq
  estimator   "reference" or "unbiased"; edge_spp samples of the boundary terms; terms the
              gradient_terms mask (0: all that apply)
  grads       the tensors that require grad: v vertices, t textures, e emission, l light
              vertices, c camera, r roughness, n normal map, p environment light
  material    "diffuse" or "rough" (DiffuseBsdfMaterial with roughness and normal map)
  light       "area", "env" (area + EnvLight) or "sh9" (area + SH9Light)
  ortho       orthographic cameras; visible: lights seen by the camera
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import synth

_BASE = dict(mode="render", spheres=1, freq=8, tex=256, height=128, width=128, views=1, spp=16, depth=3, nl=1, nb=1,
             scenes=1, estimator="reference", edge_spp=1, terms=0, grads="", material="diffuse", light="area",
             ortho=False, visible=False, noise=0.0)


def _case(name=None, **kw):
    c = dict(_BASE, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a preview thumbnail, as an interactive viewer or a unit test renders: launches and latency
        _case("thumbnail_render", freq=4, tex=16, height=32, width=32, spp=4),
        # the plain forward workload of the benchmark suite: 1,284 triangles, 128^2, 16 spp
        _case("plain_render", freq=8, height=128, width=128, spp=16),
        # a ragged image of several objects, more bounces and light samples than the defaults
        _case("ragged_render", spheres=5, freq=11, tex=50, height=97, width=61, spp=7, depth=5, nl=2, nb=3, noise=0.02,
              visible=True),
        # a frame of an animation: moved vertices, the tree's boxes refitted, one render
        _case("refit_render", mode="refit", freq=32, height=256, width=256, spp=16, noise=0.02),
        # a frame of the large scene (16 level-6 spheres, 1.31 M triangles): rebuild and render
        _case("large_render", mode="update", spheres=16, freq=64, tex=512, height=1024, width=1024, spp=16, depth=5,
              noise=0.02),
        # texture optimisation: 256^2, 64 spp, interior term
        _case("texture_step", mode="step", freq=8, height=256, width=256, spp=64, terms=1, grads="t"),
        # the reference estimator with everything differentiable (vertices, texture, light, camera)
        _case("reference_step", mode="step", freq=32, height=250, width=250, spp=16, grads="vtelc", noise=0.02),
        # rough material with normal map under an environment map, unbiased estimator
        _case("material_step", mode="step", freq=8, tex=64, height=129, width=129, spp=16, estimator="unbiased",
              grads="vtrnp", material="rough", light="env", noise=0.02),
        # the geometry-gradient workload: 20,484 triangles, 512^2, 32 spp, unbiased estimator
        _case("geometry_step", mode="step", freq=32, height=512, width=512, spp=32, estimator="unbiased", edge_spp=4,
              grads="v", noise=0.02),
        _case("geometry_batch", mode="batch", freq=32, height=512, width=512, spp=32, estimator="unbiased", edge_spp=4,
              grads="v", noise=0.02),
        # uneven views of scenes of 5k, 50k and 200k triangles in one batch
        _case("multiview_batch", mode="batch", freq=16, tex=256, height=512, width=512, views=9, spp=16, depth=4,
              scenes=3, estimator="unbiased", grads="vt", noise=0.02),
        # the large workload: 1.31 M triangles, 1024^2, depth 5, vertex and texture gradients
        _case("large_batch", mode="batch", spheres=16, freq=64, tex=512, height=1024, width=1024, spp=32, depth=5,
              estimator="unbiased", edge_spp=4, grads="vt", noise=0.02),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    mode = rng.choice(["render", "render", "refit", "update", "step", "step", "step", "batch", "batch"])
    c = _case(mode=mode, spheres=rng.choice([1, 1, 1, 2, 7, 16]), tex=rng.choice([0, 16, 64, 100, 256, 512]),
              height=log_int(24, 640), width=log_int(24, 640), depth=rng.choice([1, 2, 3, 3, 4, 5, 6]),
              noise=rng.choice([0.0, 0.02, 0.02]), visible=rng.random() < 0.2)
    c["freq"] = log_int(2, 100 if c["spheres"] == 1 else 48)
    c["spp"] = min(log_int(1, 128), max(1, 6_000_000 // (c["height"] * c["width"])))
    c["nl"], c["nb"] = rng.choice([(1, 1), (1, 1), (1, 1), (1, 0), (0, 1), (2, 1), (1, 2), (3, 2)])
    c["ortho"] = rng.random() < 0.1
    if rng.random() < 0.25:
        c["material"] = "rough"
    c["light"] = rng.choice(["area", "area", "area", "area", "env", "sh9"])
    if mode in ("step", "batch"):
        c["estimator"] = rng.choice(["reference", "unbiased", "unbiased"])
        c["edge_spp"] = rng.choice([1, 2, 4])
        c["grads"] = rng.choice(["v", "t", "vt", "vte", "vtelc"])
        if c["grads"] == "t":
            c["terms"] = 1
        if c["material"] == "rough" and c["spheres"] <= 7 and rng.random() < 0.5:
            c["grads"] += "rn"
        if c["light"] != "area" and rng.random() < 0.5:
            c["grads"] += "p"
        c["views"] = rng.choice([1, 1, 2, 5])
        if mode == "batch" and c["freq"] <= 16 and c["spheres"] <= 2:
            c["scenes"] = rng.choice([1, 3])
            c["views"] = max(c["views"], c["scenes"])
        c["spp"] = max(1, c["spp"] // c["views"])
    return c


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=16)
def _sphere(freq):
    """Vertices, faces and uvs of a geodesic sphere (fixed for every seed)."""
    V, F = synth.geodesic_sphere(freq)
    uvs, uvi = synth.spherical_uv(V, F)
    return V, F, uvs, uvi


def _gpu(a, dtype=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a)).to("cuda", dtype)


def _rand(gen, *shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(*shape, generator=gen, device="cuda")


def _inputs(case, seed, freq):
    """Tensors of one scene: meshes, light, environment parameters."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + freq)
    V, F, uvs, uvi = _sphere(freq)
    n = case["spheres"]
    centres = np.random.default_rng(4).uniform(-5.0, 5.0, size=(n, 3)) if n > 1 else np.zeros((1, 3))
    base, faces, uv, uvidx = _gpu(V), _gpu(F, torch.int32), _gpu(uvs), _gpu(uvi, torch.int32)
    meshes = []
    for k in range(n):
        v = base
        if case["noise"]:
            v = v * (1.0 + case["noise"] * torch.randn(v.shape[0], 1, generator=gen, device="cuda"))
        v = (v + _gpu(centres[k]) + 0.01 * _rand(gen, 3, lo=-1.0)).contiguous()
        t = case["tex"]
        m = {"v": v, "f": faces, "uv": uv if t else None, "uvi": uvidx if t else None,
             "t": _rand(gen, t, t, 3, lo=0.2, hi=0.8) if t else _rand(gen, 3, lo=0.2, hi=0.8)}
        if case["material"] == "rough":
            m["r"] = _rand(gen, t, t, 1, lo=0.1, hi=0.9) if t else _rand(gen, 1, lo=0.1, hi=0.9)
            tilt = _rand(gen, *((t, t) if t else ()), 3, lo=-0.08, hi=0.08)
            m["n"] = torch.tensor([0.5, 0.5, 0.92], device="cuda") + tilt
        meshes.append(m)
    wide = n > 1
    gV, gF = synth.quad((0.0, 0.0), 40.0 if wide else 10.0, -6.5 if wide else -1.0, facing_down=False)
    meshes.append({"v": _gpu(gV), "f": _gpu(gF, torch.int32), "uv": None, "uvi": None,
                   "t": torch.full((3,), 0.5, device="cuda")})
    lV, lF = synth.quad((0.0, 0.0), 4.0 if wide else 1.0, 7.0 if wide else 3.0, facing_down=True)
    light = {"v": _gpu(lV), "f": _gpu(lF, torch.int32), "e": torch.full((3,), 20.0, device="cuda")}
    env = None
    if case["light"] == "env":
        env = _rand(gen, 48, 64, 3, lo=0.1, hi=0.6)
    elif case["light"] == "sh9":
        env = _rand(gen, 9, 3, lo=-0.05, hi=0.05)
        env[0] = 0.8
    return {"meshes": meshes, "light": light, "env": env}


def _view_sizes(case):
    """(height, width) of every view; several views are uneven, from a quarter of the size up."""
    if case["views"] == 1:
        return [(case["height"], case["width"])]
    rng = np.random.default_rng(3)
    f = rng.uniform(0.25, 1.0, size=(case["views"], 2))
    return [(max(8, int(case["height"] * a)), max(8, int(case["width"] * b))) for a, b in f]


def _camera_params(case):
    """(look_from, look_at, up, fov or view width) of every view as float32 tensors."""
    wide = case["spheres"] > 1
    if case["views"] == 1:
        eyes = [np.array([0, 4, 20] if wide else [0, 0.5, 4], np.float32)]
    else:
        d = np.random.default_rng(5).normal(size=(case["views"], 3))
        d[:, 1] = np.abs(d[:, 1]) * 0.6 + 0.1
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        eyes = list((d * (20.0 if wide else 4.0)).astype(np.float32))
    lens = (14.0 if wide else 3.0) if case["ortho"] else math.pi / 4
    return [(_gpu(e), _gpu([0.0, 0.0, 0.0]), _gpu([0.0, 1.0, 0.0]), _gpu([lens])) for e in eyes]


def _targets(case, seed):
    """Smooth target images of the L2 loss, shifted by the seed."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 104729 + 1)
    out = []
    for h, w in _view_sizes(case):
        ph = _rand(gen, 3, hi=2 * math.pi)
        y = torch.linspace(0, 3.0, h, device="cuda")[:, None, None]
        x = torch.linspace(0, 2.0, w, device="cuda")[None, :, None]
        out.append((0.4 + 0.25 * torch.sin(x + 2.0 * y + ph)).contiguous())
    return out


def _leaf(t, on):
    return t.detach().requires_grad_() if on else t


def _scene(case, data, cams, on):
    """A Scene over the input tensors; `on` names the kinds that require grad. Returns the
    scene and the leaves {name: tensor}."""
    leaves, meshes = {}, []

    def leaf(t, kind, name):
        t = _leaf(t, kind in on)
        if kind in on:
            leaves[name] = t
        return t

    for k, m in enumerate(data["meshes"]):
        ground = k == len(data["meshes"]) - 1
        own = "" if ground else on
        v = leaf(m["v"], "v", f"v{k}") if own else m["v"]
        t = leaf(m["t"], "t", f"t{k}") if own else m["t"]
        if "r" in m:
            mat = dr.DiffuseBsdfMaterial(t, leaf(m["r"], "r", f"r{k}"), leaf(m["n"], "n", f"n{k}"))
        else:
            mat = dr.DiffuseMaterial(t)
        meshes.append(dr.Mesh(v, m["uv"], m["f"], m["uvi"], mat))
    li = data["light"]
    lights = [dr.AreaLight(leaf(li["v"], "l", "lv"), li["f"], leaf(li["e"], "e", "e"))]
    if case["light"] == "env":
        lights.append(dr.EnvLight(dr.Texture(leaf(data["env"], "p", "p"))))
    elif case["light"] == "sh9":
        lights.append(dr.SH9Light(leaf(data["env"], "p", "p")))
    cls = dr.OrthographicCamera if case["ortho"] else dr.PerspectiveCamera
    views = []
    for k, (eye, at, up, lens, h, w) in cams:
        views.append(cls(leaf(eye, "c", f"c{k}"), at, up, lens, h, w))
    return dr.Scene(views, meshes, lights), leaves


def prepare(case, seed):
    # scenes of one batch: frequencies f, 3 f and 6 f (5k, 50k and 200k triangles for f = 16)
    freqs = [case["freq"] * k for k in ((1, 3, 6) if case["scenes"] == 3 else (1,))]
    data = [_inputs(case, seed, f) for f in freqs]
    cams = [(k, p + s) for k, (p, s) in enumerate(zip(_camera_params(case), _view_sizes(case)))]
    integ = dr.PathIntegrator(spp_interior=case["spp"], max_bounce=case["depth"], mis_light_samples=case["nl"],
                              mis_bsdf_samples=case["nb"], enable_light_visable=case["visible"],
                              spp_primary_edge=case["edge_spp"], spp_secondary_edge=case["edge_spp"],
                              estimator=case["estimator"], gradient_terms=case["terms"])
    st = {"case": case, "data": data, "cams": cams, "integ": integ}
    if case["mode"] in ("step", "batch"):
        st["targets"] = _targets(case, seed)
    if case["mode"] in ("refit", "update"):
        st["scene"], _ = _scene(case, data[0], cams, "")
        # the frame's vertices: the spheres as they were built, shrunk by a thousandth
        st["moved"] = [m["v"] * 0.999 for m in data[0]["meshes"][:-1]]
    if case["mode"] == "batch":
        n = len(data)
        built = [_scene(case, d, cams[i::n], case["grads"]) for i, d in enumerate(data)]
        st["scenes"] = [b[0] for b in built]
        st["leaves"] = [b[1] for b in built]
        st["targets"] = [t for i in range(n) for t in st["targets"][i::n]]  # in the scenes' order
        st["batch"] = dr.BatchRender(integ, st["scenes"])
    return st


def _loss(images, targets):
    return sum(((i - t) ** 2).sum() for i, t in zip(images, targets))


def run(st):
    case, integ = st["case"], st["integ"]
    mode = case["mode"]
    if mode == "render":
        scene, _ = _scene(case, st["data"][0], st["cams"], "")
        return {"images": integ.renderC(scene)}
    if mode in ("refit", "update"):
        for m, v in zip(st["scene"].meshes, st["moved"]):
            m.set_vertices(v)
        st["scene"].update(refit=mode == "refit")
        return {"images": integ.renderC(st["scene"])}
    if mode == "step":
        scene, leaves = _scene(case, st["data"][0], st["cams"], case["grads"])
        images = integ.renderD(scene)
        _loss(images, st["targets"]).backward()
        return {"images": [i.detach() for i in images], "grads": {k: t.grad for k, t in leaves.items()}}
    # batch: new vertex tensors into the persistent scenes, one step
    for scene, leaves, d in zip(st["scenes"], st["leaves"], st["data"]):
        for k, (m, src) in enumerate(zip(scene.meshes, d["meshes"])):
            if f"v{k}" in leaves:
                leaves[f"v{k}"] = _leaf(src["v"], True)
                m.set_vertices(leaves[f"v{k}"])
        for t in leaves.values():
            t.grad = None
    images = st["batch"].renderD()
    _loss(images, st["targets"]).backward()
    return {"images": [i.detach() for i in images],
            "grads": [{k: t.grad for k, t in leaves.items()} for leaves in st["leaves"]]}


def work(case):
    """Input tensors read once, images and gradients written once; operations of the rays a
    path takes when it stays in the scene to the last bounce: a ray walks about log4 of the
    triangle count in nodes of four boxes (6 multiply-adds each) and tests two triangles of
    about 60 operations; about 200 operations of shading per vertex. A backward pass shades
    every vertex again and propagates its adjoint (three times the shading) and traces its
    boundary samples (two rays each, then a path)."""
    freqs = [case["freq"] * k for k in ((1, 3, 6) if case["scenes"] == 3 else (1,))]
    tris = sum(case["spheres"] * 20 * f * f + 4 for f in freqs)
    texels = len(freqs) * case["spheres"] * (case["tex"] ** 2 if case["tex"] else 1)
    pixels = sum(h * w for h, w in _view_sizes(case))
    nbytes = tris * (12 + (12 + 24 if case["tex"] else 0)) + tris // 2 * 12 + texels * 12 + pixels * 12
    ray = max(1.0, math.log(tris) / math.log(4.0)) * 4 * 12 + 120
    per_vertex = 200
    rays = case["depth"] * (case["nl"] + case["nb"] + 1)
    path = rays * ray + case["depth"] * per_vertex
    flops = pixels * case["spp"] * path
    if case["mode"] in ("step", "batch"):
        nbytes += pixels * 12 + (tris // 2 * 12 if "v" in case["grads"] else 0) + (texels * 12 if "t" in case["grads"] else 0)
        flops += pixels * case["spp"] * case["depth"] * 4 * per_vertex
        if case["terms"] != 1:
            kinds = 4 if case["estimator"] == "unbiased" else 2
            flops += kinds * pixels * case["edge_spp"] * (2 * ray + path)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- 64-bit values
def _u32(x):
    return x & 0xFFFFFFFF


class _Pcg32:
    """The renderer's sample streams: PCG32 (O'Neill 2014) seeded through four rounds of TEA,
    stream i from (i + the default state, i); 64-bit words in wrapping int64."""
    MULT, STATE = 0x5851F42D4C957F2D, 0x853C49E6748FEA9B - (1 << 64)

    def __init__(self, n):
        i = torch.arange(n, device="cuda", dtype=torch.int64)
        a, b = _u32(i + self.STATE), _u32(i)
        init, seq = self._tea(a, b), self._tea(b, a)
        self.inc = (seq << 1) | 1
        self.state = torch.zeros_like(i)
        self._next(i)
        self.state = self.state + init
        self._next(i)

    @staticmethod
    def _tea(v0, v1):
        s = 0
        for _ in range(4):
            s = (s + 0x9E3779B9) & 0xFFFFFFFF
            v0 = _u32(v0 + ((_u32(v1 << 4) + 0xA341316C) ^ (v1 + s) ^ ((v1 >> 5) + 0xC8013EA4)))
            v1 = _u32(v1 + ((_u32(v0 << 4) + 0xAD90777D) ^ (v0 + s) ^ ((v0 >> 5) + 0x7E95761E)))
        return v0 | (v1 << 32)

    def _next(self, rows):
        old = self.state[rows]
        self.state[rows] = old * self.MULT + self.inc[rows]
        lsr = lambda x, k: (x >> k) & ((1 << (64 - k)) - 1)  # noqa: E731
        xs = _u32(lsr(lsr(old, 18) ^ old, 27))
        rot = lsr(old, 59)
        return _u32((xs >> rot) | (xs << ((32 - rot) & 31)))

    def uniform(self, rows):
        return (self._next(rows) >> 9).double() * 2.0 ** -23


class _Exact:
    """The forward estimator in 64 bits on diffuse meshes and one square area light, one light
    and one BSDF sample, perspective camera."""

    def __init__(self, data):
        P, uv, obj = [], [], []
        parts = data["meshes"] + [data["light"]]
        for k, m in enumerate(parts):
            f = m["f"].long()
            P.append(m["v"].double()[f])
            if m.get("uv") is not None:
                uv.append(m["uv"].double()[m["uvi"].long()])
            else:
                uv.append(torch.tensor([[0, 0], [0, 1], [1, 0]], dtype=torch.float64, device="cuda").expand(len(f), 3, 2))
            obj.append(torch.full((len(f),), k, device="cuda"))
        self.groups = [len(p) for p in P]
        self.P, self.uv, self.obj = torch.cat(P), torch.cat(uv), torch.cat(obj)
        c, b = self.P[:, 1] - self.P[:, 0], self.P[:, 0] - self.P[:, 2]
        cr = torch.linalg.cross(c, b)
        self.area = 0.5 * cr.norm(dim=1)
        self.N = cr / cr.norm(dim=1, keepdim=True)
        du1, du2 = self.uv[:, 1, 1] - self.uv[:, 0, 1], self.uv[:, 2, 1] - self.uv[:, 0, 1]
        t = c * du2[:, None] + b * du1[:, None]
        self.T = t / t.norm(dim=1, keepdim=True)
        self.light = len(parts) - 1
        self.lt = torch.nonzero(self.obj == self.light)[:, 0]
        self.emit = data["light"]["e"].double()
        self.larea = self.area[self.lt].sum()
        self.tex = [m["t"].double() for m in data["meshes"]]

    def closest(self, o, d):
        """Closest hit beyond 1e-3: (triangle or -1, b1, b2)."""
        n = len(o)
        best = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
        tri = torch.full((n,), -1, device="cuda")
        b1, b2 = torch.zeros_like(best), torch.zeros_like(best)
        first = 0
        for cnt in self.groups:
            P = self.P[first:first + cnt]
            mid = 0.5 * (P.amin((0, 1)) + P.amax((0, 1)))
            rad = (P - mid).norm(dim=2).max() * (1 + 1e-9)
            m = o - mid
            perp = m.square().sum(1) - (m * d).sum(1) ** 2 / d.square().sum(1)
            rows = torch.nonzero(perp <= rad ** 2)[:, 0]
            e1, e2 = P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]
            nrm = torch.linalg.cross(e1, e2)
            off = (nrm * P[:, 0]).sum(1)
            # b1, b2 as inner products of the ray's (d, o x d) with per-triangle 6-vectors
            k1 = torch.cat([-torch.linalg.cross(P[:, 0], e2), -e2], 1)
            k2 = torch.cat([torch.linalg.cross(P[:, 0], e1), e1], 1)
            step = max(1, (1 << 26) // cnt)
            for s in range(0, len(rows), step):
                r = rows[s:s + step]
                oo, dd = o[r], d[r]
                den = dd @ nrm.T
                t = (off - oo @ nrm.T) / den
                pl = torch.cat([dd, torch.linalg.cross(oo, dd)], 1)
                u, v = (pl @ k1.T) / den, (pl @ k2.T) / den
                t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-3), t, math.inf)
                tb, kb = t.min(1)
                near = tb < best[r]
                rr, kk = r[near], kb[near]
                best[rr], tri[rr] = tb[near], kk + first
                b1[rr], b2[rr] = u[near, kk], v[near, kk]
            first += cnt
        return tri, b1, b2

    def surface(self, tri, b1, b2, org):
        P = self.P[tri]
        p = P[:, 0] + b1[:, None] * (P[:, 1] - P[:, 0]) + b2[:, None] * (P[:, 2] - P[:, 0])
        U = self.uv[tri]
        uv = U[:, 0] + b1[:, None] * (U[:, 1] - U[:, 0]) + b2[:, None] * (U[:, 2] - U[:, 0])
        sgn = torch.where(((org - p) * self.N[tri]).sum(1) > 0, 1.0, -1.0).double()[:, None]
        return {"p": p, "n": self.N[tri] * sgn, "t": self.T[tri] * sgn, "uv": uv, "obj": self.obj[tri],
                "sqd": (p - org).square().sum(1)}

    def albedo(self, s):
        out = torch.zeros_like(s["p"])
        for k, tx in enumerate(self.tex):
            rows = torch.nonzero(s["obj"] == k)[:, 0]
            if tx.dim() == 1:
                val = tx.expand(len(rows), 3)
            else:
                h, w = tx.shape[:2]
                u = (s["uv"][rows, 0] * w - 0.5).clamp(-1, w).round().long().clamp(0, w - 1)
                v = (s["uv"][rows, 1] * h - 0.5).clamp(-1, h).round().long().clamp(0, h - 1)
                val = tx[h - 1 - v, u]
            out = out.index_put((rows,), val)
        return out

    def render(self, cam, spp, depth):
        eye, at, up, fov, H, W = cam
        eye, at, up = eye.double(), at.double(), up.double()
        back = eye - at
        back = back / back.norm()
        right = torch.linalg.cross(up / up.norm(), back)
        nup = torch.linalg.cross(back, right)
        n = H * W * spp
        rng = _Pcg32(n)
        every = torch.arange(n, device="cuda")
        jx, jy = rng.uniform(every), rng.uniform(every)
        pix = every // spp
        tan = math.tan(float(fov[0]) / 2)
        cx = ((pix % W + jx) * 2 / W - 1) * tan
        cy = (1 - (pix // W + jy) * 2 / H) * tan
        d = cx[:, None] * right + cy[:, None] * nup - back
        d = d / d.norm(dim=1, keepdim=True)
        L = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        ids, org, T = every, eye.expand(n, 3), torch.ones(n, 3, dtype=torch.float64, device="cuda")
        hit = self.closest(org, d)
        for k in range(depth):
            keep = hit[0] >= 0
            keep[keep.clone()] = self.obj[hit[0][keep]] != self.light
            ids, org, T = ids[keep], org[keep], T[keep]
            x = self.surface(*(h[keep] for h in hit), org)
            f = self.albedo(x) / math.pi
            C = torch.zeros_like(T)
            # light sample
            rx, ry = rng.uniform(ids), rng.uniform(ids)
            pick = (rx > self.area[self.lt[0]] / self.larea).long()
            rx = (rx - pick * (self.area[self.lt[0]] / self.larea)) / (self.area[self.lt[pick]] / self.larea)
            sq = ry.sqrt()
            Q = self.P[self.lt[pick]]
            y = Q[:, 0] + (Q[:, 1] - Q[:, 0]) * (rx * sq)[:, None] + (Q[:, 2] - Q[:, 0]) * (1 - sq)[:, None]
            w = y - x["p"]
            w = w / w.norm(dim=1, keepdim=True)
            C = C + self._light(x, w, f, 1.0 / self.larea, target=y)
            # BSDF sample
            w, ct = self._cosine(x, rng, ids)
            C = C + self._light(x, w, f, ct / math.pi)
            L = L.index_add(0, ids, T * C)
            if k == depth - 1:
                break
            w, ct = self._cosine(x, rng, ids)
            hit, org, T = self.closest(x["p"], w), x["p"], T * f * math.pi * ((x["n"] * w).sum(1) / ct)[:, None]
        return L.reshape(H * W, spp, 3).mean(1).reshape(H, W, 3)

    def _cosine(self, x, rng, ids):
        ru, rv = rng.uniform(ids), rng.uniform(ids)
        ct, st, ph = ru.sqrt(), (1 - ru).sqrt(), 2 * math.pi * rv
        w = (x["t"] * (ph.cos() * st)[:, None] + torch.linalg.cross(x["n"], x["t"]) * (ph.sin() * st)[:, None] +
             x["n"] * ct[:, None])
        return w / w.norm(dim=1, keepdim=True), ct

    def _light(self, x, w, f, pdf, target=None):
        """MIS-weighted (power heuristic) contribution of a light (target) or BSDF sample."""
        out = torch.zeros_like(x["p"])
        tri, b1, b2 = self.closest(x["p"], w)
        ok = tri >= 0
        ok[ok.clone()] = self.obj[tri[ok]] == self.light
        q = self.surface(tri[ok], b1[ok], b2[ok], x["p"][ok])
        if target is not None:
            near = (q["p"] - target[ok]).square().sum(1) < 1e-5
            rows = torch.nonzero(ok)[:, 0][near]
            q = {k: v[near] for k, v in q.items()}
        else:
            rows = torch.nonzero(ok)[:, 0]
        ww, n = w[rows], x["n"][rows]
        cosx = (n * ww).sum(1)
        tmp = -(q["n"] * ww).sum(1) / q["sqd"]
        if target is not None:
            pl = torch.as_tensor(pdf)
            pb = cosx / math.pi * tmp
            val = cosx * tmp / pl * pl ** 2 / (pl ** 2 + pb ** 2)
        else:
            pb = pdf[rows] * tmp
            pl = 1.0 / self.larea
            val = cosx * tmp / pb * pb ** 2 / (pb ** 2 + pl ** 2)
        return out.index_add(0, rows, self.emit * f[rows] * val[:, None])


def exact(case, seed):
    simple = (case["spheres"] == 1 and case["views"] == 1 and (case["nl"], case["nb"]) == (1, 1) and
              case["material"] == "diffuse" and case["light"] == "area" and not case["ortho"] and not case["visible"] and
              case["mode"] in ("render", "refit", "update", "step"))
    tests = case["height"] * case["width"] * case["spp"] * (1 + 3 * case["depth"]) * 20 * case["freq"] ** 2
    if not simple or tests > 1e11:
        return None
    data = _inputs(case, seed, case["freq"])
    if case["mode"] in ("refit", "update"):
        for m in data["meshes"][:-1]:
            m["v"] = m["v"] * 0.999
    tex = data["meshes"][0]["t"] = data["meshes"][0]["t"].double().requires_grad_("t" in case["grads"])
    image = _Exact(data).render(_camera_params(case)[0] + _view_sizes(case)[0], case["spp"], case["depth"])
    if case["mode"] != "step":
        return {"images": [image]}
    grads = {}
    if "t" in case["grads"] and case["material"] == "diffuse":
        _loss([image], [t.double() for t in _targets(case, seed)]).backward()
        grads = {"t0": tex.grad}
    return {"images": [image.detach()], "grads": grads}
