"""PyTorch API of the B200 path tracer: a drop-in for torch_psdr's Python surface.

Mirrors src/python/torch_psdr.py (class names, constructor arguments, asserts and
the renderC / renderD contract). Tensors are borrowed as CUDA buffers and handed to
the native library through the C ABI; the only PyTorch machinery is the
torch.autograd.Function below, whose forward calls psdr_render_fwd and whose backward
calls psdr_render_bwd (the path-replay adjoint).
"""
from __future__ import annotations

import ctypes as C
import json
import os
import threading
import weakref
from typing import List, Optional, Union

import numpy as np
import torch
from torch import Tensor

from . import _lib as L
from . import synth


def _dev_tensor(t: Tensor, dtype) -> Tensor:
    if not isinstance(t, Tensor):
        t = torch.as_tensor(t)
    if not t.is_cuda:
        raise ValueError("torch_psdr_b200 renders on the GPU: tensors must be CUDA tensors")
    return t.detach().to(dtype=dtype, copy=True, memory_format=torch.contiguous_format)


def check_indices(idx: Tensor, n: int, what: str) -> None:
    """Every entry of the index buffer idx must lie in [0, n): the native kernels gather
    vertices and uvs through these buffers without bounds checks (as the reference's
    gathers do), so an out-of-range index would read outside the buffer. One device
    reduction and one host read; empty buffers are left to the library's own check."""
    if idx.numel() == 0:
        return
    lo, hi = torch.stack([idx.min(), idx.max()]).tolist()
    if lo < 0 or hi >= n:
        raise ValueError(f"{what} must lie in [0, {n}): found values in [{lo}, {hi}]")


def _check_index_buffers(jobs) -> None:
    """check_indices for the (int32 CUDA tensor, bound, name) triples of one object, with one
    kernel and one host read for all of them, on the GPU that holds them (which need not be
    the current one)."""
    jobs = [j for j in jobs if j[0].numel()]
    n = len(jobs)
    if n == 0:
        return
    dev = jobs[0][0].device
    if n > 1 and any(j[0].device != dev for j in jobs):
        for d in dict.fromkeys(j[0].device for j in jobs):
            _check_index_buffers([j for j in jobs if j[0].device == d])
        return
    if dev.index != torch.cuda.current_device():  # (entering a device takes 10 us, as long as the kernel)
        with torch.cuda.device(dev):
            _check_index_buffers(jobs)
        return
    ptrs = (C.c_void_p * n)(*[t.data_ptr() for t, _, _ in jobs])
    counts = (C.c_int64 * n)(*[t.numel() for t, _, _ in jobs])
    out = (C.c_int32 * (2 * n))()
    L.check(L.load().psdr_index_bounds(ptrs, counts, n, out, _stream()), "psdr_index_bounds")
    for i, (_, bound, what) in enumerate(jobs):
        if out[2 * i] < 0 or out[2 * i + 1] >= bound:
            raise ValueError(f"{what} must lie in [0, {bound}): found values in [{out[2 * i]}, {out[2 * i + 1]}]")


def _native(call, what: str) -> None:
    """A native call that may allocate. Memory that torch keeps from freed tensors is out of the
    library's reach: when the library runs out, torch gives its cache back and the call is
    made once more (a call that failed has changed nothing)."""
    try:
        return L.check(call(), what)
    except L.PsdrOutOfMemory:
        pass
    torch.cuda.empty_cache()
    L.check(call(), what)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _host_lists(tensors) -> list:
    """The tensors' values as lists of floats, with one host read when they are float32 tensors
    on one GPU (each read waits for the stream)."""
    flat = [t.detach().reshape(-1) for t in tensors]
    if len(flat) > 1 and all(f.is_cuda and f.dtype == torch.float32 and f.device == flat[0].device for f in flat):
        values, out = torch.cat(flat).tolist(), []
        for f in flat:
            out.append(values[:f.numel()])
            values = values[f.numel():]
        return out
    return [f.float().cpu().tolist() for f in flat]


class VarContex:
    """Collects the tensors that require grad, in the order torch_psdr.py:84-103 does."""

    def __init__(self):
        self.torch_vars: List[Tensor] = []

    def append_variable(self, torch_var: Tensor):
        if isinstance(torch_var, Tensor) and torch_var.requires_grad:
            self.torch_vars.append(torch_var)

    def merge_variables(self, torch_vars):
        for t in torch_vars:
            if t.requires_grad:
                self.torch_vars.append(t)

    def get_variables(self):
        return self.torch_vars


class BaseCamera(VarContex):
    """Base class of PerspectiveCamera and OrthographicCamera (torch_psdr.py:106-110)."""

    def _desc(self):
        return _camera_descs([self])[0]


def _camera_descs(cams):
    """Descriptors of the cameras (their parameters are read from the GPU in one go)."""
    values = iter(_host_lists([t for c in cams for t in (c.look_from, c.look_at, c.up, c.vfov)]))
    out = (L.CameraDesc * len(cams))()
    for d, c in zip(out, cams):
        d.type = L.CAM_ORTHOGRAPHIC if isinstance(c, OrthographicCamera) else L.CAM_PERSPECTIVE
        d.look_from = (C.c_float * 3)(*next(values))
        d.look_at = (C.c_float * 3)(*next(values))
        d.up = (C.c_float * 3)(*next(values))
        d.fov = next(values)[0]
        d.height, d.width = c.height, c.width
    return out


class PerspectiveCamera(BaseCamera):
    def __init__(self, look_from: Tensor, look_at: Tensor, up: Tensor, vfov: Tensor, height: int, width: int):
        """Pinhole camera (torch_psdr.py:113-158; camera.h:208-277).

        Args:
            look_from: (3,) camera position.  look_at: (3,) target.  up: (3,) up vector.
            vfov: (1,) vertical field of view in radians.  height, width: image size.
        """
        super().__init__()
        assert look_from.size() == (3,)
        assert look_at.size() == (3,)
        assert up.size() == (3,)
        assert vfov.size() == (1,)
        assert height > 0 and width > 0
        self.look_from, self.look_at, self.up, self.vfov = look_from, look_at, up, vfov
        for t in (look_from, look_at, up, vfov):
            self.append_variable(t)
        self.height = int(height)
        self.width = int(width)


Camera = PerspectiveCamera  # example/optimize_texture.py:76 uses dr.Camera


class OrthographicCamera(BaseCamera):
    def __init__(self, look_from, look_at, up, view_width, height: int, width: int):
        """Orthographic camera (torch_psdr.py:161-206; camera.h:279-353): parallel rays
        along the view direction from a view box view_width wide and view_width * height /
        width high."""
        super().__init__()
        assert look_from.size() == (3,)
        assert look_at.size() == (3,)
        assert up.size() == (3,)
        assert view_width.size() == (1,)
        assert height > 0 and width > 0
        self.look_from, self.look_at, self.up, self.view_width = look_from, look_at, up, view_width
        self.vfov = view_width  # the lens parameter slot shared with PerspectiveCamera
        for t in (look_from, look_at, up, view_width):
            self.append_variable(t)
        self.height = int(height)
        self.width = int(width)


class Texture(VarContex):
    def __init__(self, tex: Tensor):
        """Constant (1,)/(3,) or image (H,W,1)/(H,W,3) texture (torch_psdr.py:209-269).

        The image keeps the caller's row order; the library applies the row flip of
        torch_psdr.py:250 when it indexes (nearest texel, texture.h:65-74).
        """
        super().__init__()
        tex_type = None
        size = tuple(tex.size())
        if tex.dim() == 1:
            if size == (1,):
                tex_type = "Constant1f"
            elif size == (3,):
                tex_type = "Constant3f"
        elif tex.dim() == 2:
            # torch_psdr.py:232-234 tests `tex_type == "UV1f"` (a comparison, not an
            # assignment), so a (H, W) texture fails its assert; kept as is.
            pass
        elif tex.dim() == 3:
            if size[-1] == 1:
                tex_type = "UV1f"
            elif size[-1] == 3:
                tex_type = "UV3f"
        assert tex_type is not None
        self.tex_type = tex_type
        self.tensor = tex
        self.append_variable(tex)
        self.data = _dev_tensor(tex, torch.float32)

    def _desc(self):
        d = L.TextureDesc()
        if self.tex_type.startswith("Constant"):
            d.kind = L.TEX_CONSTANT
            d.channels = 1 if self.tex_type == "Constant1f" else 3
            d.height = d.width = 1
        else:
            d.kind = L.TEX_UV
            d.height, d.width = int(self.data.shape[0]), int(self.data.shape[1])
            d.channels = int(self.data.shape[2])
        d.data = self.data.data_ptr()
        return d


class Material(VarContex):
    """Base class of the materials (torch_psdr.py:272-277)."""


class DiffuseMaterial(Material):
    def __init__(self, tex: Union[Tensor, Texture]):
        """Lambertian reflectance (torch_psdr.py:280-295; diffuse_material.cc:3-45)."""
        super().__init__()
        if isinstance(tex, Tensor):
            tex = Texture(tex)
        assert tex.tex_type == "Constant3f" or tex.tex_type == "UV3f"
        self.texture = tex
        self.roughness = None
        self.normal = None
        self.merge_variables(tex.get_variables())
        self.mat_type = L.MAT_DIFFUSE


class DiffuseBsdfMaterial(Material):
    def __init__(self, color, roughness, normal=None):
        """Lambertian / Oren-Nayar diffuse reflection (torch_psdr.py:298-335;
        diffuse_bsdf.cc:3-88): color (3,) or (H,W,3), roughness (1,) or (H,W,1) (0 is
        Lambertian), normal (3,) or (H,W,3) shading normals in the (tangent,
        normal x tangent, normal) frame, 0.5 + n/2 per channel; None = geometric normal."""
        super().__init__()
        if isinstance(color, Tensor):
            color = Texture(color)
        if isinstance(roughness, Tensor):
            roughness = Texture(roughness)
        if isinstance(normal, Tensor):
            normal = Texture(normal)
        assert color.tex_type == "Constant3f" or color.tex_type == "UV3f"
        assert roughness.tex_type == "Constant1f" or roughness.tex_type == "UV1f"
        assert normal is None or normal.tex_type == "Constant3f" or normal.tex_type == "UV3f"
        self.texture = color
        self.roughness = roughness
        self.normal = normal
        self.merge_variables(color.get_variables())
        self.merge_variables(roughness.get_variables())
        if normal is not None:
            self.merge_variables(normal.get_variables())
        self.mat_type = L.MAT_DIFFUSE_BSDF


class PrincipledMaterial(Material):
    pass


class Mesh(VarContex):
    def __init__(self, vertices: Tensor, uvs, face_indices: Tensor, uv_indices, material: Material):
        """Triangle mesh with its material (torch_psdr.py:343-379; mesh.cc:5-95)."""
        super().__init__()
        assert vertices.dim() == 2 and vertices.size(-1) == 3
        assert uvs is None or (uvs.dim() == 2 and uvs.size(-1) == 2)
        assert face_indices.dim() == 2 and face_indices.size(-1) == 3
        assert uv_indices is None or (uv_indices.dim() == 2 and uv_indices.size(-1) == 3)
        assert uvs is None or uv_indices is None or uv_indices.size(0) == face_indices.size(0)
        self.vertices = vertices
        self.v = _dev_tensor(vertices, torch.float32)
        self.f = _dev_tensor(face_indices, torch.int32)
        no_uvs = uvs is None or uv_indices is None
        self.uv = None if no_uvs else _dev_tensor(uvs, torch.float32)
        self.uvi = None if no_uvs else _dev_tensor(uv_indices, torch.int32)
        _check_index_buffers([(self.f, self.v.shape[0], "face_indices")] +
                             ([] if no_uvs else [(self.uvi, self.uv.shape[0], "uv_indices")]))
        self.material = material
        self.append_variable(vertices)
        self.merge_variables(material.get_variables())

    def set_vertices(self, vertices: Tensor):
        """Copy new vertex positions (same count) into the buffer the native scene reads
        when it rebuilds (psdr_scene_update, or the forward graph of a BatchRender); the
        given tensor becomes the one that receives the vertex gradient."""
        assert tuple(vertices.shape) == tuple(self.v.shape)
        self.v.copy_(vertices.detach())
        self.vertices = vertices

    def get_variables(self):
        out = [self.vertices] if self.vertices.requires_grad else []
        return out + self.material.get_variables()

    def _desc(self):
        d = L.MeshDesc()
        d.vertices, d.num_vertices = self.v.data_ptr(), int(self.v.shape[0])
        d.faces, d.num_faces = self.f.data_ptr(), int(self.f.shape[0])
        if self.uv is not None:
            d.uvs, d.num_uvs, d.uv_indices = self.uv.data_ptr(), int(self.uv.shape[0]), self.uvi.data_ptr()
        d.material = self.material.mat_type
        d.color = self.material.texture._desc()
        none = L.TextureDesc(L.TEX_NONE, 0, 0, 0, None)
        d.roughness = self.material.roughness._desc() if self.material.roughness is not None else none
        d.normal = self.material.normal._desc() if self.material.normal is not None else none
        return d


class Light(VarContex):
    """Base class of the lights (torch_psdr.py:382-385)."""


class AreaLight(Light):
    def __init__(self, vertices: Tensor, face_indices: Tensor, emit: Tensor):
        """Triangle-mesh emitter with constant radiance (torch_psdr.py:388-414; emitter.cc:4-92)."""
        super().__init__()
        assert vertices.dim() == 2 and vertices.size(-1) == 3
        assert face_indices.dim() == 2 and face_indices.size(-1) == 3
        assert emit.dim() == 1 and emit.size(0) == 3
        self.vertices, self.emit = vertices, emit
        self.v = _dev_tensor(vertices, torch.float32)
        self.f = _dev_tensor(face_indices, torch.int32)
        _check_index_buffers([(self.f, self.v.shape[0], "face_indices")])
        self.append_variable(vertices)
        self.append_variable(emit)

    def _desc(self, emit=None):
        d = L.AreaLightDesc()
        d.vertices, d.num_vertices = self.v.data_ptr(), int(self.v.shape[0])
        d.faces, d.num_faces = self.f.data_ptr(), int(self.f.shape[0])
        d.emit = (C.c_float * 3)(*(emit if emit is not None else _host_lists([self.emit])[0]))
        return d


class EnvLight(Light):
    def __init__(self, cube_map: Texture):
        """Cube-map environment light (torch_psdr.py:417-430; emitter.cc:94-141): an
        emissive box around the scene, 1000 times its size (scene.cc:31-49), showing the
        cube map laid out as a 4 x 3 cross."""
        super().__init__()
        assert cube_map.tex_type == "UV3f"
        self.cube_map = cube_map
        self.merge_variables(cube_map.get_variables())
        self.vertices = self.v = self.emit = None
        self.params, self.params_data = cube_map.tensor, cube_map.data

    def _desc(self, _, box):
        d = L.AreaLightDesc()
        d.type = L.LIGHT_ENV
        d.cube_map = self.cube_map._desc()
        d.box_min, d.box_max = (C.c_float * 3)(*map(float, box[0])), (C.c_float * 3)(*map(float, box[1]))
        return d


class SH9Light(Light):
    def __init__(self, sh9_coeff: Tensor):
        """Second-order spherical-harmonics light (torch_psdr.py:433-447;
        emitter.cc:206-283): the same box as EnvLight, emitting sum_k c_k Y_k(wi) of the
        incoming direction wi at its hit point. sh9_coeff: (9, 3)."""
        super().__init__()
        assert sh9_coeff.size() == (9, 3)
        self.sh9_coeff = sh9_coeff
        self.append_variable(sh9_coeff)
        self.vertices = self.v = self.emit = None
        self.params = sh9_coeff
        self.params_data = torch.zeros((9, 3), dtype=torch.float32, device="cuda")

    def _desc(self, sh9, box):
        d = L.AreaLightDesc()
        d.type = L.LIGHT_SH9
        d.sh9 = (C.c_float * 27)(*sh9)
        d.box_min, d.box_max = (C.c_float * 3)(*map(float, box[0])), (C.c_float * 3)(*map(float, box[1]))
        return d


def _is_env(light):
    return isinstance(light, (EnvLight, SH9Light))


class Scene(VarContex):
    def __init__(self, cameras: List[BaseCamera], meshes: List[Mesh], lights: List[Light]):
        """Cameras, meshes and lights (torch_psdr.py:450-474). Builds the native scene
        (triangle records, edge list, sampling CDFs, LBVH) on the current stream."""
        super().__init__()
        self.cameras = list(cameras)
        self.meshes = list(meshes)
        # scene.cc:15-53: one environment light, appended after the other lights around the
        # box of the camera positions and mesh vertices (self.lights keeps that order)
        env = [lt for lt in lights if _is_env(lt)]
        assert len(env) <= 1, "only support no more than one env_light"
        self.lights = [lt for lt in lights if not _is_env(lt)] + env
        # light radiances and coefficients, and for an environment light the camera positions and
        # the meshes' boxes (minima and maxima taken on the GPU), in one host read
        par = [lt.sh9_coeff if isinstance(lt, SH9Light) else lt.emit for lt in self.lights
               if not isinstance(lt, EnvLight)]
        ext = []
        if env:
            ext = [c.look_from for c in self.cameras] + [e for m in self.meshes for e in (m.v.amin(0), m.v.amax(0))]
        values = _host_lists(par + ext)
        box = None
        if env:
            pts = np.array(values[len(par):], np.float32)
            box = synth.env_box(pts[:len(self.cameras)], [pts[len(self.cameras):]])
        values = iter(values[:len(par)])
        lib = L.load()
        md = (L.MeshDesc * max(1, len(self.meshes)))(*[m._desc() for m in self.meshes])
        ld = (L.AreaLightDesc * max(1, len(self.lights)))(*[
            lt._desc(None, box) if isinstance(lt, EnvLight) else
            lt._desc(next(values), box) if isinstance(lt, SH9Light) else lt._desc(next(values)) for lt in self.lights])
        desc = L.SceneDesc(md, len(self.meshes), ld, len(self.lights))
        handle = C.c_void_p()
        _native(lambda: lib.psdr_scene_create(C.byref(desc), _stream(), C.byref(handle)), "psdr_scene_create")
        self._handle = handle
        self._lib = lib
        self._builds = 0  # rebuilds since creation

    def _stamp(self):
        """Changes whenever the native scene, or a buffer it reads while rendering, does; None when
        that cannot be told (buffers made under inference mode track no versions)."""
        tex = [t.data for m in self.meshes for t in (m.material.texture, m.material.roughness, m.material.normal)
               if t is not None]
        tex += [lt.cube_map.data for lt in self.lights if isinstance(lt, EnvLight)]
        tex += [o.v for o in self.meshes + self.lights if o.v is not None]
        if any(t.is_inference() for t in tex):
            return None
        return self._builds, tuple((t.data_ptr(), t._version) for t in tex)

    @property
    def handle(self):
        return self._handle

    def get_variables(self):
        """Tensors requiring grad, cameras then meshes then lights (torch_psdr.py:469-471)."""
        out = []
        for part in self.cameras + self.meshes + self.lights:
            out += [t for t in part.get_variables() if t.requires_grad]
        return out

    def info(self):
        out = (C.c_int64 * 6)()
        L.check(self._lib.psdr_scene_info(self._handle, out), "psdr_scene_info")
        return dict(zip(["triangles", "vertices", "edges", "bvh_nodes", "lights", "objects"], list(out)))

    def update(self, refit: bool = False):
        """Rebuild triangle records, edges, CDFs and the BVH after Mesh.set_vertices.
        refit=True keeps the BVH's tree and recomputes only its boxes (same hits; for small
        vertex moves between full rebuilds)."""
        self._builds += 1
        if refit:
            L.check(self._lib.psdr_scene_refit(self._handle, _stream()), "psdr_scene_refit")
        else:
            L.check(self._lib.psdr_scene_update(self._handle, _stream()), "psdr_scene_update")

    def _camera_descs(self):
        return _camera_descs(self.cameras)

    def __del__(self):
        h = getattr(self, "_handle", None)
        if h is not None and h.value:
            try:
                self._lib.psdr_scene_destroy(h)
            except Exception:
                pass
            self._handle = None


class _RenderD(torch.autograd.Function):
    """Replaces Wrap2torch (torch_psdr.py:29-72): forward renders, backward runs the
    path-replay adjoint and returns the gradient of every input tensor. The forward keeps
    the paths' replay records for the backward when they fit (_Records)."""

    @staticmethod
    def forward(ctx, integrator, scene, keep, *torch_vars):
        cams = scene._camera_descs()
        ctx.records = integrator._new_records(scene, cams) if keep else None
        imgs = None
        try:
            imgs = integrator._render(scene, cams, ctx.records)
        except L.PsdrOutOfMemory:
            if ctx.records is None:
                raise
            ctx.records = None
        if imgs is None:  # the records took the memory that the render needs
            imgs = integrator._render(scene, cams)
        ctx.integrator = integrator
        ctx.scene = scene
        ctx.n_vars = len(torch_vars)
        ctx.vars = torch_vars
        return tuple(imgs)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, *grads):
        grads = [g if g is not None else None for g in grads]
        records, ctx.records = ctx.records, None  # a second backward re-traces the paths
        out = None
        try:
            out = ctx.integrator._backward(ctx.scene, grads, ctx.vars, records)
        except L.PsdrOutOfMemory:
            if records is None:
                raise
            records = None
        if out is None:
            out = ctx.integrator._backward(ctx.scene, grads, ctx.vars)
        return (None, None, None) + tuple(out)


class _Records:
    """Replay records of one renderD forward: the device memory (a tensor, so it goes back to
    torch's allocator with the autograd graph) and what they were made from. The backward
    uses them only when the scene, cameras and configuration are still the same; otherwise
    it re-traces the paths, as it does without records."""

    _alive = weakref.WeakSet()
    _lock = threading.Lock()

    def __init__(self, data, stamp):
        self.data, self.stamp = data, stamp
        self.stream = torch.cuda.current_stream()
        with _Records._lock:
            _Records._alive.add(self)

    @staticmethod
    def held(device) -> int:
        """Bytes of the records on a GPU that autograd graphs hold now."""
        if not _Records._alive:
            return 0
        with _Records._lock:
            return sum(r.data.numel() for r in _Records._alive if r.data.device == device)

    def pointer(self, stamp):
        """Address for a backward with this stamp; None: re-trace."""
        if stamp != self.stamp:
            return None
        cur = torch.cuda.current_stream()
        if cur != self.stream:
            self.data.record_stream(cur)
        return self.data.data_ptr()


def _grad_buf(param, internal, new=torch.zeros_like):
    """Gradient buffer shaped like `internal` (zeroed unless `new` says otherwise), or None
    when `param` does not require grad."""
    if isinstance(param, Tensor) and param.requires_grad:
        return new(internal)
    return None


def _tex_grad(tex, new=torch.zeros_like):
    """Gradient buffer of an optional Texture (None when absent or not requiring grad)."""
    return None if tex is None else _grad_buf(tex.tensor, tex.data, new)


def _ptrs(bufs):
    """ctypes pointer array of optional tensors (at least one entry)."""
    P = C.c_void_p
    return (P * max(1, len(bufs)))(*[None if t is None else t.data_ptr() for t in bufs])


def _wants(t) -> bool:
    return isinstance(t, Tensor) and t.requires_grad


def _lens_buf(cam, unbiased: bool):
    """(10,) camera-lens gradient buffer (look_from through the basis, look_at, up, fov), or
    None when no camera parameter that enters the basis or the projection requires grad.
    With the unbiased estimator look_from needs it too: moving look_from with look_at fixed
    turns the camera. Orthographic cameras have no lens gradient: their look_at, up and
    view_width gradients are refused rather than returned as zeros."""
    lens_params = (cam.look_at, cam.up, cam.vfov)
    if isinstance(cam, OrthographicCamera):
        if any(_wants(t) for t in lens_params):
            raise NotImplementedError("gradients of an OrthographicCamera's look_at, up and view_width are not "
                                      "implemented; only look_from (with the camera's basis held fixed)")
        return None
    if any(_wants(t) for t in lens_params) or (unbiased and _wants(cam.look_from)):
        return torch.zeros(10, dtype=torch.float32, device="cuda")
    return None


def _add_camera_grads(add, cam, origin_g, lens_g):
    """Map a camera's origin gradient (basis fixed) and its lens gradient onto its tensors."""
    if lens_g is None:
        add(cam.look_from, origin_g)
        return
    add(cam.look_from, origin_g + lens_g[0:3])
    add(cam.look_at, lens_g[3:6])
    add(cam.up, lens_g[6:9])
    add(cam.vfov, lens_g[9:10])


class PathIntegrator:
    def __init__(self, enable_light_visable: bool = False, n_pass: int = 1, spp_interior: int = 1,
                 max_bounce: int = 3, mis_light_samples: int = 1, mis_bsdf_samples: int = 1,
                 spp_primary_edge: int = 1, spp_secondary_edge: int = 1, primary_edge_preprocess_rounds: int = 1,
                 secondary_edge_preprocess_rounds: int = 1, primary_edge_hypercube_resolution: int = 10000,
                 secondary_edge_hypercube_resolution: List[int] = [10000, 6, 6], estimator: str = "reference",
                 seed: int = 0, tile_paths: int = 0, gradient_terms: int = 0,
                 spp_pixel_boundary: Optional[int] = None, trace_queue: int = 0, batch_lanes: int = 0,
                 batch_records: int = 0):
        """Path-space differentiable integrator (torch_psdr.py:477-536; path_integrator.h:8-21).

        B200 extensions: estimator ("reference" reproduces renderD exactly; "unbiased"
        is the derivative of the rendered image: material-form interior term plus
        pixel-border, silhouette and shadow-boundary terms), seed (0 = the reference's
        sample streams), tile_paths (wavefront tile, 0 = automatic), gradient_terms
        (bitmask: 1 interior, 2 primary edges, 4 direct edges, 8 pixel borders, 16
        DiffuseBsdfMaterial BRDF jumps, 32 interpenetration creases, 64 indirect shadow
        boundaries; 0 = all that apply: bits 8-64 with the unbiased estimator only, bit 16
        when a DiffuseBsdfMaterial mesh is in the scene),
        spp_pixel_boundary (unbiased: samples per unit pixel-border segment; default
        spp_primary_edge), trace_queue (rays each SM traverses concurrently, in units of
        128; 0 = 8, the autotuner picks it), batch_lanes (BatchRender only: concurrent
        streams, each with its own workspace, over which a batch spreads its forward tiles
        and its backward's interior tiles and per-view boundary terms; 1..8, 0 = 4; the
        gradients do not depend on it), batch_records (renderD and BatchRender: the forward keeps
        every interior path's replay record and the backward runs the adjoint from them
        instead of re-tracing; 0 = when they fit in a quarter of the free device memory
        (renderD: together with those of every other image whose graph is still alive; an
        image kept without a backward holds its records), 1 = always, -1 = never; the
        gradients do not depend on it).
        """
        assert n_pass > 0
        assert spp_interior > 0
        assert spp_primary_edge > 0
        assert spp_secondary_edge > 0
        assert max_bounce > 0
        assert mis_light_samples >= 0
        assert mis_bsdf_samples >= 0
        assert primary_edge_preprocess_rounds > 0
        assert secondary_edge_preprocess_rounds > 0
        assert primary_edge_hypercube_resolution > 0
        assert len(secondary_edge_hypercube_resolution) == 3
        for reso in secondary_edge_hypercube_resolution:
            assert reso > 0
        assert estimator in ("reference", "unbiased")
        cfg = L.Config()
        cfg.n_pass = n_pass
        cfg.spp_interior = spp_interior
        cfg.enable_light_visable = int(bool(enable_light_visable))
        cfg.spp_primary_edge = spp_primary_edge
        cfg.spp_secondary_edge = spp_secondary_edge
        cfg.max_bounce = max_bounce
        cfg.mis_light_samples = mis_light_samples
        cfg.mis_bsdf_samples = mis_bsdf_samples
        cfg.primary_edge_preprocess_rounds = primary_edge_preprocess_rounds
        cfg.secondary_edge_preprocess_rounds = secondary_edge_preprocess_rounds
        cfg.primary_edge_hypercube_resolution = primary_edge_hypercube_resolution
        cfg.secondary_edge_hypercube_resolution = (C.c_int32 * 3)(*secondary_edge_hypercube_resolution)
        cfg.estimator = L.EST_REFERENCE if estimator == "reference" else L.EST_UNBIASED
        cfg.tile_paths = tile_paths
        cfg.terms = gradient_terms
        cfg.spp_pixel_boundary = spp_primary_edge if spp_pixel_boundary is None else spp_pixel_boundary
        assert cfg.spp_pixel_boundary >= 0
        cfg.seed = seed
        assert 0 <= trace_queue <= 8
        cfg.trace_queue = trace_queue
        assert 0 <= batch_lanes <= 8
        cfg.batch_lanes = batch_lanes
        assert batch_records in (-1, 0, 1)
        cfg.batch_records = batch_records
        self.cfg = cfg
        self._lib = L.load()
        self._ws = None
        self._records_granted = 0  # bytes of replay records, all graphs' together, that fitted before

    def _workspace(self):
        if self._ws is None:
            h = C.c_void_p()
            L.check(self._lib.psdr_workspace_create(C.byref(h)), "psdr_workspace_create")
            self._ws = h
        return self._ws

    def __del__(self):
        if getattr(self, "_ws", None) is not None:
            try:
                self._lib.psdr_workspace_destroy(self._ws)
            except Exception:
                pass

    def _render(self, scene: Scene, cams=None, records=None) -> List[Tensor]:
        imgs = [torch.empty((c.height, c.width, 3), dtype=torch.float32, device="cuda") for c in scene.cameras]
        ptrs = (C.c_void_p * len(imgs))(*[i.data_ptr() for i in imgs])
        cams = scene._camera_descs() if cams is None else cams
        rec = None if records is None else records.data.data_ptr()
        _native(lambda: self._lib.psdr_render_fwd_records(scene.handle, self._workspace(), cams, len(imgs),
                                                          C.byref(self.cfg), ptrs, rec, _stream()), "psdr_render_fwd")
        return imgs

    def _stamp(self, scene: Scene, cams):
        own = scene._stamp()
        return None if own is None else (bytes(cams), bytes(self.cfg), own)

    def _new_records(self, scene: Scene, cams):
        """Memory for the replay records of a renderD forward, or None when they are not wanted
        (batch_records = -1, no interior term), could not be checked against the scene of the
        backward, or take more than a quarter of the free memory."""
        if self.cfg.batch_records < 0 or (self.cfg.terms and not self.cfg.terms & 1):
            return None
        stamp = self._stamp(scene, cams)
        if stamp is None:
            return None
        n = C.c_int64()
        L.check(self._lib.psdr_records_bytes(cams, len(cams), C.byref(self.cfg), C.byref(n)), "psdr_records_bytes")
        n = int(n.value)
        # All graphs' records together may take a quarter of the memory there would be without
        # them. The query takes 0.1 to 0.3 ms: it is left out up to 64 MB in all and for totals
        # granted before (should the memory have gone elsewhere since, _RenderD drops the records).
        dev = torch.device("cuda", torch.cuda.current_device())
        total = _Records.held(dev) + n
        if self.cfg.batch_records == 0 and total > max(64 << 20, self._records_granted):
            stats = torch.cuda.memory_stats_as_nested_dict(dev)
            cached = stats["reserved_bytes"]["all"]["current"] - stats["allocated_bytes"]["all"]["current"]
            if total > (torch.cuda.mem_get_info(dev)[0] + cached + total - n) // 4:
                return None
        try:
            data = torch.empty(n, dtype=torch.uint8, device=dev)
        except torch.OutOfMemoryError:
            self._records_granted = 0
            return None
        if self.cfg.batch_records == 0:
            self._records_granted = max(total, self._records_granted)
        return _Records(data, stamp)

    def autotune(self, scene: Scene, cache: Optional[str] = None) -> dict:
        """Pick the wavefront tile size and the scene's BVH leaf size by timing forward
        renders of the scene's cameras (psdr_autotune); the integrator keeps the tile
        size (0: the automatic one was fastest, and stays), the scene keeps the leaf size.
        Extension: the reference has no tuner.

        cache: path of a JSON file of earlier results, keyed by the GPU (name, SM count)
        and the job's shape (triangles, view sizes, spp, depth, light and BSDF samples,
        estimator). A hit applies the stored sizes without timing (and returns them with
        "cached": True); a miss tunes and adds its result to the file."""
        key = self._tune_key(scene) if cache else None
        if key is not None and os.path.exists(cache):
            with open(cache) as f:
                entry = json.load(f).get(key)
            if entry is not None:
                self._apply_tuning(scene, entry)
                return dict(entry, cached=True)
        entry = self._autotune_native(scene)
        if key is not None:
            table = {}
            if os.path.exists(cache):
                with open(cache) as f:
                    table = json.load(f)
            table[key] = entry
            tmp = cache + ".tmp"
            with open(tmp, "w") as f:
                json.dump(table, f, indent=1, sort_keys=True)
            os.replace(tmp, cache)
        return entry

    def _autotune_native(self, scene: Scene) -> dict:
        leaf = C.c_int32()
        ms = C.c_float()
        cams = scene._camera_descs()
        scene._builds += 1
        L.check(self._lib.psdr_autotune(scene.handle, self._workspace(), cams, len(cams), C.byref(self.cfg),
                                        C.byref(leaf), C.byref(ms), _stream()), "psdr_autotune")
        return {"tile_paths": int(self.cfg.tile_paths), "leaf_size": int(leaf.value),
                "trace_queue": int(self.cfg.trace_queue), "forward_ms": float(ms.value)}

    def _apply_tuning(self, scene: Scene, entry: dict) -> None:
        self.cfg.tile_paths = int(entry["tile_paths"])
        self.cfg.trace_queue = int(entry.get("trace_queue", 0))
        scene._builds += 1
        L.check(self._lib.psdr_scene_set_leaf_size(scene.handle, int(entry["leaf_size"]), _stream()),
                "psdr_scene_set_leaf_size")

    @staticmethod
    def _gpu_id() -> dict:
        p = torch.cuda.get_device_properties(torch.cuda.current_device())
        return {"gpu": p.name, "sms": int(p.multi_processor_count)}

    def _tune_key(self, scene: Scene) -> str:
        c = self.cfg
        tris = sum(int(m.f.shape[0]) for m in scene.meshes) + sum(
            int(lt.f.shape[0]) for lt in scene.lights if getattr(lt, "f", None) is not None)
        shape = dict(self._gpu_id(), tris=tris, views=[[int(v.height), int(v.width)] for v in scene.cameras],
                     spp=int(c.spp_interior), depth=int(c.max_bounce), nl=int(c.mis_light_samples),
                     nb=int(c.mis_bsdf_samples), estimator=int(c.estimator))
        return json.dumps(shape, sort_keys=True)

    def render_samples(self, scene: Scene, camera_index: int = 0) -> Tensor:
        """Per-sample interior radiance (H*W*spp, 3) of one camera (the values the film averages)."""
        c = scene.cameras[camera_index]
        out = torch.empty((c.height * c.width * self.cfg.spp_interior, 3), dtype=torch.float32, device="cuda")
        cams = scene._camera_descs()
        L.check(self._lib.psdr_render_samples(scene.handle, self._workspace(), C.byref(cams[camera_index]),
                                              C.byref(self.cfg), out.data_ptr(), _stream()), "psdr_render_samples")
        return out

    def _backward(self, scene: Scene, grads, torch_vars, records=None):
        dev = "cuda"
        dimgs = []
        for g, c in zip(grads, scene.cameras):
            if g is None:
                g = torch.zeros((c.height, c.width, 3), dtype=torch.float32, device=dev)
            dimgs.append(g.detach().float().contiguous())
        nm, nl = len(scene.meshes), len(scene.lights)
        # vertex gradients only for the meshes/lights whose vertices require grad (the
        # library then skips the others' scatters)
        # (the buffers are written in full: none needs to be cleared first)
        new = torch.empty_like
        vert_g = [_grad_buf(m.vertices, m.v, new) for m in scene.meshes] + [_grad_buf(lt.vertices, lt.v, new)
                                                                             for lt in scene.lights]
        tex_g = [_grad_buf(m.material.texture.tensor, m.material.texture.data, new) for m in scene.meshes]
        rough_g = [_tex_grad(m.material.roughness, new) for m in scene.meshes]
        nrm_g = [_tex_grad(m.material.normal, new) for m in scene.meshes]
        emit_g = list(torch.empty((nl, 3), dtype=torch.float32, device=dev))
        light_g = [_grad_buf(lt.params, lt.params_data, new) if _is_env(lt) else None for lt in scene.lights]
        cam_g = list(torch.empty((len(scene.cameras), 3), dtype=torch.float32, device=dev))
        unb = self.cfg.estimator == L.EST_UNBIASED
        lens_g = [_lens_buf(c, unb) for c in scene.cameras]
        P = C.c_void_p
        vp = (P * (nm + nl))(*[None if t is None else t.data_ptr() for t in vert_g])
        tp = (P * max(1, nm))(*[None if t is None else t.data_ptr() for t in tex_g])
        ep = (P * max(1, nl))(*[t.data_ptr() for t in emit_g])
        cp = (P * len(cam_g))(*[t.data_ptr() for t in cam_g])
        tg = L.GradTargets(vp, tp, ep, cp, 0, _ptrs(rough_g), _ptrs(nrm_g), _ptrs(light_g), _ptrs(lens_g))
        dp = (P * len(dimgs))(*[d.data_ptr() for d in dimgs])
        cams = scene._camera_descs()
        rec = None if records is None else records.pointer(self._stamp(scene, cams))
        _native(lambda: self._lib.psdr_render_bwd_records(scene.handle, self._workspace(), cams, len(dimgs),
                                                          C.byref(self.cfg), dp, C.byref(tg), rec, _stream()),
                "psdr_render_bwd")
        # map the accumulators onto the input tensors (a tensor may play several roles)
        acc = {}

        def add(t, g):
            if t is None or not isinstance(t, Tensor) or not t.requires_grad:
                return
            g = g.reshape(t.shape).to(t.dtype)
            key = id(t)
            acc[key] = g if key not in acc else acc[key] + g

        for i, m in enumerate(scene.meshes):
            add(m.vertices, vert_g[i])
            add(m.material.texture.tensor, tex_g[i])
            if rough_g[i] is not None:
                add(m.material.roughness.tensor, rough_g[i])
            if nrm_g[i] is not None:
                add(m.material.normal.tensor, nrm_g[i])
        for j, lt in enumerate(scene.lights):
            add(lt.vertices, vert_g[nm + j])
            add(lt.emit, emit_g[j])
            if light_g[j] is not None:
                add(lt.params, light_g[j])
        for k, c in enumerate(scene.cameras):
            _add_camera_grads(add, c, cam_g[k], lens_g[k])
        return [acc[id(t)] if id(t) in acc else torch.zeros_like(t) for t in torch_vars]

    def renderC(self, scene: Scene) -> List[Tensor]:
        """Plain render (path_integrator.cc:408-410): one (H, W, 3) image per camera."""
        with torch.no_grad():
            return self._render(scene)

    def renderD(self, scene: Scene) -> List[Tensor]:
        """Differentiable render (torch_psdr.py:547-556): images requiring grad; their
        backward runs the path-replay adjoint with both edge-sampling terms."""
        torch_vars = scene.get_variables()
        if not torch_vars:
            return self._render(scene)
        for c in scene.cameras:  # refuse unsupported camera gradients before rendering
            _lens_buf(c, self.cfg.estimator == L.EST_UNBIASED)
        imgs = _RenderD.apply(self, scene, torch.is_grad_enabled(), *torch_vars)
        return list(imgs)


class BatchRender:
    """All cameras of one or more scenes rendered as one work list from CUDA graphs.

    The forward graph rebuilds every scene's geometry from its meshes' vertex buffers
    (update them in place with `Mesh.set_vertices`) and renders every camera; the
    backward graph runs the path-replay adjoint and every boundary term of the
    integrator's estimator for all views. Images, image gradients and gradient buffers
    are allocated once and bound to the graphs; vertex gradients are kept for the
    meshes and lights whose vertices require grad when the batch is created (keep
    that when swapping buffers with `Mesh.set_vertices`). Extension: the reference has
    no batching.

    Inside each graph the job's independent parts (the forward's tiles; the backward's
    interior tiles and every boundary term of every view) run on the integrator's
    `batch_lanes` concurrent streams, each with its own workspace, and with
    `batch_records` the forward keeps every interior path's replay record so that the
    backward runs the adjoint without re-tracing. Neither changes a bit of the images or
    gradients. Against `PathIntegrator.renderD` of each scene alone the images are equal
    and the gradients agree to float rounding (the batch packs all scenes' paths into
    shared tiles, which changes the per-thread sums of the light and camera gradients).
    The memory cost is one workspace per lane plus, with kept records,
    16 B x (1 + D R + 2 D) + 8 B per path (D = max_bounce, R = light + BSDF samples + 1).
    """

    def __init__(self, integrator: PathIntegrator, scenes: List[Scene], differentiable: bool = True):
        self.integrator = integrator
        self.scenes = list(scenes)
        self.lib = L.load()
        self.stream = torch.cuda.Stream()
        dev = "cuda"
        cams, cam_scene = [], []
        for si, sc in enumerate(self.scenes):
            for c in sc.cameras:
                cams.append(c)
                cam_scene.append(si)
        self.cams = cams
        self.images = [torch.zeros((c.height, c.width, 3), dtype=torch.float32, device=dev) for c in cams]
        self.d_images = [torch.zeros_like(i) for i in self.images] if differentiable else None
        P = C.c_void_p
        self._keep = []
        targets = []
        self.grads = []
        cam_g = [torch.zeros(3, dtype=torch.float32, device=dev) for _ in cams]
        cp = (P * len(cam_g))(*[t.data_ptr() for t in cam_g])
        self.cam_grads = cam_g
        unb = integrator.cfg.estimator == L.EST_UNBIASED
        self.lens_grads = [_lens_buf(c, unb) for c in cams] if differentiable else [None] * len(cams)
        lp_cam = _ptrs(self.lens_grads)
        for sc in self.scenes:
            vg = [_grad_buf(m.vertices, m.v) for m in sc.meshes] + [_grad_buf(lt.vertices, lt.v)
                                                                    for lt in sc.lights]
            tg = [_grad_buf(m.material.texture.tensor, m.material.texture.data) for m in sc.meshes]
            eg = [torch.zeros(3, dtype=torch.float32, device=dev) for _ in sc.lights]
            rg = [_tex_grad(m.material.roughness) for m in sc.meshes]
            ng = [_tex_grad(m.material.normal) for m in sc.meshes]
            lg = [_grad_buf(lt.params, lt.params_data) if _is_env(lt) else None for lt in sc.lights]
            self.grads.append((vg, tg, eg, rg, ng, lg))
            vp, tp, ep, rp, npp, lp = _ptrs(vg), _ptrs(tg), _ptrs(eg), _ptrs(rg), _ptrs(ng), _ptrs(lg)
            self._keep += [vp, tp, ep, rp, npp, lp]
            targets.append(L.GradTargets(vp, tp, ep, cp, 0, rp, npp, lp, lp_cam))
        self._keep += [cp, lp_cam]
        tgt = (L.GradTargets * len(targets))(*targets)
        sh = (P * len(self.scenes))(*[s.handle for s in self.scenes])
        cd = _camera_descs(cams)
        csc = (C.c_int32 * len(cams))(*cam_scene)
        ip = (P * len(cams))(*[t.data_ptr() for t in self.images])
        dp = (P * len(cams))(*[t.data_ptr() for t in self.d_images]) if differentiable else None
        self._keep += [tgt, sh, cd, csc, ip, dp]
        h = C.c_void_p()
        torch.cuda.synchronize()
        _native(lambda: self.lib.psdr_batch_create(sh, len(self.scenes), cd, csc, len(cams), C.byref(integrator.cfg), ip,
                                                   dp, tgt, C.byref(h)), "psdr_batch_create")
        self._handle = h

    def forward(self) -> List[Tensor]:
        """Rebuild geometry and render every camera (returns the bound image buffers)."""
        cur = torch.cuda.current_stream()
        self.stream.wait_stream(cur)
        for sc in self.scenes:
            sc._builds += 1  # the graph rebuilds every scene
        L.check(self.lib.psdr_batch_forward(self._handle, C.c_void_p(self.stream.cuda_stream)), "psdr_batch_forward")
        cur.wait_stream(self.stream)
        return self.images

    def backward(self, d_images: List[Tensor]):
        """Run the adjoint for dLoss/dImage of every camera; fills the bound gradient buffers."""
        for dst, g in zip(self.d_images, d_images):
            if g is None:
                dst.zero_()
            else:
                dst.copy_(g)
        cur = torch.cuda.current_stream()
        self.stream.wait_stream(cur)
        L.check(self.lib.psdr_batch_backward(self._handle, C.c_void_p(self.stream.cuda_stream)),
                "psdr_batch_backward")
        cur.wait_stream(self.stream)

    def renderD(self) -> List[Tensor]:
        """Differentiable batched render: images whose backward fills .grad of the
        scenes' input tensors, like PathIntegrator.renderD."""
        torch_vars = []
        for sc in self.scenes:
            torch_vars += sc.get_variables()
        return list(_BatchRenderD.apply(self, *torch_vars))

    def _map_grads(self, torch_vars):
        acc = {}

        def add(t, g):
            if t is None or not isinstance(t, Tensor) or not t.requires_grad:
                return
            g = g.reshape(t.shape).to(t.dtype)
            acc[id(t)] = g if id(t) not in acc else acc[id(t)] + g

        k = 0
        for sc, (vg, tg, eg, rg, ng, lg) in zip(self.scenes, self.grads):
            nm = len(sc.meshes)
            for i, m in enumerate(sc.meshes):
                add(m.vertices, vg[i])
                add(m.material.texture.tensor, tg[i])
                if rg[i] is not None:
                    add(m.material.roughness.tensor, rg[i])
                if ng[i] is not None:
                    add(m.material.normal.tensor, ng[i])
            for j, lt in enumerate(sc.lights):
                add(lt.vertices, vg[nm + j])
                add(lt.emit, eg[j])
                if lg[j] is not None:
                    add(lt.params, lg[j])
            for c in sc.cameras:
                _add_camera_grads(add, c, self.cam_grads[k], self.lens_grads[k])
                k += 1
        return [acc[id(t)] if id(t) in acc else torch.zeros_like(t) for t in torch_vars]

    def __del__(self):
        h = getattr(self, "_handle", None)
        if h is not None and h.value:
            try:
                torch.cuda.synchronize()
                self.lib.psdr_batch_destroy(h)
            except Exception:
                pass
            self._handle = None


class _BatchRenderD(torch.autograd.Function):
    @staticmethod
    def forward(ctx, batch, *torch_vars):
        imgs = batch.forward()
        ctx.batch = batch
        ctx.vars = torch_vars
        return tuple(i.clone() for i in imgs)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, *grads):
        ctx.batch.backward(list(grads))
        return (None,) + tuple(ctx.batch._map_grads(ctx.vars))
