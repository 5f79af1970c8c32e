"""Tuning a job whose automatic tile is larger than the fixed sizes the tuner tries: the automatic
tile is tried too, and kept as automatic when it is the fastest (a tuned render of 8.4 M paths
took 9 % longer than an untuned one while the tuner stopped at 2^21)."""
import ctypes as C

import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import _lib as L
from torch_psdr_b200 import synth
from helpers import to_torch_scene

pytestmark = pytest.mark.gpu


# 2^23 paths: 32, 16, 8 and 4 tiles of the fixed sizes and 2 automatic ones; 2^20: the fixed sizes
@pytest.mark.parametrize("size,tiles", [(1024, 32 + 16 + 8 + 4 + 2), (362, 4 + 2 + 1 + 1)])
def test_automatic_tile_is_a_candidate(cuda, size, tiles):
    """Counted by the traversal launches of the tuner's renders: three of each combination of
    tile, three leaf sizes and three queue depths."""
    depth, lib = 3, L.load()
    scene, _ = to_torch_scene(synth.sphere_scene(level=4, tex_hw=64, noise_sigma=0.02, height=size, width=size))
    kw = dict(spp_interior=8, max_bounce=depth)
    before = dr.PathIntegrator(**kw).renderC(scene)[0]
    integ = dr.PathIntegrator(**kw)
    out, ms = (C.c_int64 * 3)(), C.c_double()
    L.check(lib.psdr_profile_enable(1), "enable")
    L.check(lib.psdr_profile_reset(), "reset")
    try:
        info = integ.autotune(scene)
        torch.cuda.synchronize()
        L.check(lib.psdr_profile_read(out, C.byref(ms)), "read")
    finally:
        lib.psdr_profile_enable(0)
    assert out[1] == 3 * 3 * 3 * depth * tiles
    assert info["tile_paths"] in (0, 1 << 18, 1 << 19, 1 << 20, 1 << 21) and (size > 362 or info["tile_paths"])
    assert torch.equal(before, integ.renderC(scene)[0])
    integ.renderD(scene)
    dr.BatchRender(integ, [scene], differentiable=False).forward()
