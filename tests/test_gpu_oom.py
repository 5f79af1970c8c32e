"""A workspace whose growth failed for want of memory: the call returns the error, and later calls
on the same workspace work, at the sizes it had and at the sizes that failed."""
import numpy as np
import pytest
import torch

import torch_psdr_b200 as dr
from torch_psdr_b200 import _lib as L
from torch_psdr_b200 import synth
from helpers import to_torch_scene

pytestmark = pytest.mark.gpu

KW = dict(spp_interior=4, max_bounce=2, estimator="unbiased", primary_edge_hypercube_resolution=100,
          secondary_edge_hypercube_resolution=[20, 2, 2])


def _step(integ, spec):
    scene, T = to_torch_scene(spec, requires_grad={"verts", "tex", "emit"})
    img = integ.renderD(scene)[0]
    img.backward(torch.as_tensor(np.random.default_rng(0).normal(size=tuple(img.shape)), dtype=torch.float32, device="cuda"))
    return [img.detach()] + [t.grad for t in T.values() if t is not None and t.grad is not None]


@pytest.mark.parametrize("first", [False, True])
def test_workspace_after_a_failed_growth(cuda, first):
    spec = synth.sphere_scene(level=1, tex_hw=9, height=48, width=40)
    want = _step(dr.PathIntegrator(**KW), spec)
    integ = dr.PathIntegrator(batch_records=-1, **KW)
    if not first:
        _step(integ, spec)
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    integ.cfg.tile_paths = 1 << 23  # 2.4 GB and more for the backward
    with pytest.raises(L.PsdrError, match="memory"):
        _step(integ, spec)
    # a smaller tile, and the failed one once there is memory
    integ.cfg.tile_paths = 1 << 16
    for a, b in zip(want, _step(integ, spec)):
        assert torch.equal(a, b)
    del hog
    torch.cuda.empty_cache()
    integ.cfg.tile_paths = 1 << 23
    for a, b in zip(want, _step(integ, spec)):
        assert torch.equal(a, b)
