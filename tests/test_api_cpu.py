"""Host side of the Python API that needs no GPU: fakes stand in for CUDA tensors and the
native library."""
import contextlib
import types
import weakref

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
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current[-1].index)
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


class _Memory:
    """A GPU's memory as _new_records sees it: free bytes outside torch's cache, the cache, and
    the tensors allocated from it (kept by the records that hold them)."""

    def __init__(self, monkeypatch, free):
        self.free, self.reserved, self.tensors, self.queries = free, 0, weakref.WeakSet(), 0
        monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
        monkeypatch.setattr(torch.cuda, "current_stream", lambda: "stream")
        monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda d=None: {
            k: {"all": {"current": v}} for k, v in (("reserved_bytes", self.reserved), ("allocated_bytes", self.allocated()))})
        monkeypatch.setattr(torch.cuda, "mem_get_info", self.query)
        monkeypatch.setattr(torch, "empty", self.empty)

    def allocated(self):
        return sum(t.numel() for t in self.tensors)

    def query(self, d=None):
        self.queries += 1
        return self.free, 0

    def empty(self, n, dtype=None, device=None):
        grow = max(0, self.allocated() + n - self.reserved)
        if grow > self.free:
            raise torch.OutOfMemoryError()
        self.free -= grow
        self.reserved += grow
        t = _OnGpu([], 0)
        t.numel = lambda: n
        self.tensors.add(t)
        return t


@pytest.mark.parametrize("size", [1 << 30, 40 << 20])
def test_records_of_all_graphs_share_one_limit(monkeypatch, size):
    """Graphs kept alive, whichever integrator made them: together their records take at most a
    quarter of the memory, and a graph that would go beyond it re-traces its paths."""
    mem = _Memory(monkeypatch, 16 << 30)
    monkeypatch.setattr(api.PathIntegrator, "_stamp", lambda *a: "stamp")

    def records_bytes(cams, n, cfg, out):
        out._obj.value = size
        return 0

    def integrator():
        it = api.PathIntegrator.__new__(api.PathIntegrator)
        it.cfg, it._records_granted = api.L.Config(), 0
        it._lib = types.SimpleNamespace(psdr_records_bytes=records_bytes)
        return it

    first, second = integrator(), integrator()
    kept = []
    for k in range(150):
        kept.append((first if k % 2 else second)._new_records(None, [None]))
    held = [r for r in kept if r is not None]
    assert len(held) == (4 << 30) // size and mem.allocated() <= 4 << 30
    # with the graphs gone, the next ones take the cache's memory, without asking again
    mem.queries = 0
    del kept, held
    free = mem.free
    for _ in range(5):
        assert first._new_records(None, [None]) is not None
    assert mem.free == free and mem.queries == 0


def _graph(monkeypatch, limit):
    """renderD over fakes: forwards and backwards run out of memory while records are held and
    `limit` (the calls that may fail) is not used up. Returns the integrator and its calls."""
    calls = []

    class Integ:
        def _new_records(self, scene, cams):
            return api._Records(_OnGpu([], 0), "stamp")

        def _render(self, scene, cams=None, records=None):
            calls.append(("fwd", records is not None))
            if records is not None and "fwd" in limit:
                raise api.L.PsdrOutOfMemory("fwd")
            return [torch.ones(2)]

        def _backward(self, scene, grads, torch_vars, records=None):
            calls.append(("bwd", records is not None))
            if records is not None and "bwd" in limit:
                raise api.L.PsdrOutOfMemory("bwd")
            return [torch.full((2,), 3.0) for _ in torch_vars]

    monkeypatch.setattr(torch.cuda, "current_stream", lambda: "stream")
    scene = types.SimpleNamespace(_camera_descs=lambda: "cams")
    return Integ(), scene, calls


@pytest.mark.parametrize("limit,want", [
    ((), [("fwd", True), ("bwd", True)]),
    (("fwd",), [("fwd", True), ("fwd", False), ("bwd", False)]),
    (("bwd",), [("fwd", True), ("bwd", True), ("bwd", False)])])
def test_records_are_dropped_when_the_library_runs_out_of_memory(monkeypatch, limit, want):
    integ, scene, calls = _graph(monkeypatch, limit)
    before = len(api._Records._alive)
    x = torch.zeros(2, requires_grad=True)
    (img,) = api._RenderD.apply(integ, scene, True, x)
    assert len(api._Records._alive) == before + (limit != ("fwd",))
    img.sum().backward()
    assert calls == want and torch.equal(x.grad, torch.full((2,), 3.0))
    assert len(api._Records._alive) == before


def test_native_calls_get_torchs_cache_back(monkeypatch):
    """An out-of-memory status empties torch's cache and repeats the call once."""
    empties = []
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: empties.append(1))
    status = [api.L.PSDR_ERR_OOM, 0]
    api._native(lambda: status.pop(0), "call")
    assert empties == [1] and not status
    with pytest.raises(api.L.PsdrOutOfMemory):
        api._native(lambda: api.L.PSDR_ERR_OOM, "call")
    with pytest.raises(ValueError):
        api._native(lambda: api.L.PSDR_ERR_INVALID_ARG, "call")
    assert empties == [1, 1]
