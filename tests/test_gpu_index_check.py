"""The index check of meshes, lights and scenes: several at a time from several threads, many
buffers in one scene, and its cost in a program that has nothing else of the library alive."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import api, synth

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_threads_get_their_own_bounds(cuda):
    """More threads than the library keeps result slots, each with its own stream and bounds."""
    wrong = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            bufs = [torch.randint(k, 1000 + k, (n,), dtype=torch.int32, device="cuda") for n in (1, 33, 70000)]
            ends = [(int(b.min()), int(b.max())) for b in bufs]
            for _ in range(20):
                api._check_index_buffers([(b, hi + 1, "ok") for b, (lo, hi) in zip(bufs, ends)])
                for i, (lo, hi) in enumerate(ends):
                    try:
                        api._check_index_buffers([(b, hi if q == i else e + 1, f"b{q}")
                                                  for q, (b, (_, e)) in enumerate(zip(bufs, ends))])
                        wrong.append((k, i))
                    except ValueError as err:
                        if f"found values in [{lo}, {hi}]" not in str(err):
                            wrong.append((k, i, str(err)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(24)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]


@pytest.mark.parametrize("n,bad", [(31, None), (32, 31), (33, 32), (70, 64), (256, 255), (257, 255), (300, None)])
def test_scene_of_many_meshes(cuda, n, bad):
    """More index buffers than one launch checks; an index out of range in the last of them."""
    V, F = synth.quad((0.0, 0.0), 1.0, 0.0, facing_down=False)
    v, f = torch.as_tensor(V, device="cuda"), torch.as_tensor(F, dtype=torch.int32, device="cuda")
    meshes = [dr.Mesh(v, None, f, None, dr.DiffuseMaterial(torch.full((3,), 0.5, device="cuda"))) for _ in range(n)]
    lV, lF = synth.quad((0.0, 0.0), 1.0, 3.0, facing_down=True)
    light = dr.AreaLight(torch.as_tensor(lV, device="cuda"), torch.as_tensor(lF, dtype=torch.int32, device="cuda"),
                         torch.ones(3, device="cuda"))
    if bad is None:
        assert dr.Scene([], meshes, [light]).handle
        return
    meshes[bad].f = meshes[bad].f.clone()
    meshes[bad].f[0, 0] = 4
    with pytest.raises(ValueError, match=rf"mesh {bad} face"):
        dr.Scene([], meshes, [light])


COST = """
import time, torch, torch_psdr_b200 as dr
from torch_psdr_b200 import synth
V, F = synth.quad((0.0, 0.0), 1.0, 0.0, facing_down=True)
v, f = torch.as_tensor(V, device="cuda"), torch.as_tensor(F, dtype=torch.int32, device="cuda")
def cost():
    ts = []
    for _ in range(60):
        t = time.perf_counter()
        dr.AreaLight(v, f, torch.ones(3))
        ts.append(time.perf_counter() - t)
    return sorted(ts)[30]
cost()
alone = cost()
scene = dr.Scene([], [], [dr.AreaLight(v, f, torch.ones(3))])
print(alone, cost())
"""


def test_cost_without_other_objects(cuda):
    """A light made while nothing of the library is alive costs what it does beside a scene (a
    temporary allocation took ten times as long)."""
    out = subprocess.run([sys.executable, "-c", COST], cwd=ROOT, check=True, capture_output=True, text=True, timeout=300)
    alone, beside = map(float, out.stdout.split())
    assert alone < 3 * beside, (alone, beside)
