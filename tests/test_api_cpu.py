"""Host side of the Python API that needs no GPU: fakes stand in for CUDA tensors and the
native library."""
import contextlib
import types

import pytest
import torch

from torch_psdr_b200 import api


class _OnGpu:
    """A CUDA index tensor of another GPU, as far as the index check looks at it."""

    def __init__(self, values, index):
        self.values, self.device = values, torch.device("cuda", index)

    def numel(self):
        return len(self.values)

    def data_ptr(self):
        return id(self)


def _fake_cuda(monkeypatch, tensors):
    """Native index bounds of the fakes, noting the current device of every call."""
    by_ptr, current, calls = {t.data_ptr(): t for t in tensors}, [torch.device("cuda", 0)], []

    @contextlib.contextmanager
    def device(d):
        current.append(torch.device(d))
        yield
        current.pop()

    def bounds(ptrs, counts, n, out, stream):
        for i in range(n):
            t = by_ptr[ptrs[i]]
            assert counts[i] == t.numel()
            calls.append((t.device, current[-1], stream))
            out[2 * i], out[2 * i + 1] = min(t.values), max(t.values)
        return 0

    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(api, "_stream", lambda: current[-1].index)
    monkeypatch.setattr(api.L, "load", lambda: types.SimpleNamespace(psdr_index_bounds=bounds))
    return calls


def test_index_check_runs_on_the_gpu_of_the_buffers(monkeypatch):
    """Faces and uvs on GPU 1 (and one buffer on GPU 2) while GPU 0 is current."""
    f, u, w, none = _OnGpu([0, 2, 1], 1), _OnGpu([3, 0], 1), _OnGpu([5], 2), _OnGpu([], 1)
    calls = _fake_cuda(monkeypatch, [f, u, w, none])
    api._check_index_buffers([(f, 3, "face_indices"), (none, 0, "empty"), (w, 6, "other"), (u, 4, "uv_indices")])
    assert len(calls) == 3 and all(of == on and stream == on.index for of, on, stream in calls)
    with pytest.raises(ValueError, match=r"uv_indices must lie in \[0, 3\): found values in \[0, 3\]"):
        api._check_index_buffers([(f, 3, "face_indices"), (u, 3, "uv_indices")])


def _scene_of(buffers):
    """A Scene without its native part, over these internal texture buffers."""
    scene = api.Scene.__new__(api.Scene)
    mat = [types.SimpleNamespace(texture=types.SimpleNamespace(data=b), roughness=None, normal=None) for b in buffers]
    scene.meshes = [types.SimpleNamespace(material=m, v=m.texture.data) for m in mat]
    scene.lights, scene._builds = [], 0
    return scene


def test_scene_made_under_inference_mode_has_no_stamp():
    """Its buffers track no versions: renderD re-traces the paths instead of keeping records."""
    src = torch.ones(3)
    with torch.inference_mode():
        inside = src.detach().to(copy=True)
    outside = src.detach().to(copy=True)
    assert _scene_of([outside, inside])._stamp() is None
    integ = api.PathIntegrator.__new__(api.PathIntegrator)
    integ.cfg = api.L.Config()
    assert integ._new_records(_scene_of([inside]), (api.L.CameraDesc * 1)()) is None
    stamp = _scene_of([outside])._stamp()
    outside.mul_(2.0)
    assert stamp is not None and _scene_of([outside])._stamp() != stamp
