"""Launch shapes at the ends of what the calls accept: block sizes up to the
largest, on meshes whose walks may need more stack entries than a block's share
of shared memory, in every mode and under stream capture. Hits are compared bit
for bit with the C restatement's walk of the binary tree."""
import numpy as np
import pytest
import torch

import photorealisticrender4610_b200 as prr
from photorealisticrender4610_b200 import scenes

pytestmark = pytest.mark.gpu


def equal(got, want):
    hid, t = want[:2]
    assert np.array_equal(got[0].cpu().numpy(), hid)
    assert np.array_equal(got[1].cpu().numpy().view(np.uint32), t.view(np.uint32))


# 1,280 rays per SM (189,440) is where the default mode changes kernels
@pytest.mark.parametrize("block", [32, 512, 640, 672, 1024])
@pytest.mark.parametrize("rays", [1, 3_000, 189_440, 189_441, 400_000])
def test_default_mode_block_sizes(port, cuda, block, rays):
    v, o, d = scenes.query_set(3_000, rays, seed=9)
    s = prr.Scene.single_mesh(v)
    got = s.mesh_intersect(0, torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda),
                           config={"block_size": block})
    equal(got, port.mesh(v).intersect(o, d))
