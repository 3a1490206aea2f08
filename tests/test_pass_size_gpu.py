"""How much a wavefront render traces and holds at once by default."""
import pytest
import torch

import photorealisticrender4610_b200 as prr
from photorealisticrender4610_b200 import scenes

pytestmark = pytest.mark.gpu


def launches(s):
    return s.stats()["last_render_launches"]


def test_adaptive_passes_do_not_grow_with_the_budget(cuda):
    """A pass traces all its samples, wanted or not: 256 x 128 x 1024 samples
    are 33.5M paths, which fixed sampling takes in one pass (of 32M = 2^25) and
    adaptive sampling in four."""
    s = prr.Scene.from_desc(scenes.cornell_box(256, 128))
    s.render(1024, 2, mode="wavefront")
    # generate + film + 13 per bounce (two, and one past the last), resolve
    assert launches(s) == 2 + 13 * 3 + 1
    s.render(1024, 2, mode="wavefront", min_spp=1, threshold=1e9)
    assert launches(s) == 4 * (6 + 13 * 3) + 2


@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("threshold", [1e9, 0.5])
@pytest.mark.parametrize("per_pass", [4, 85, 86, 256])
def test_passes_after_the_last_pixel_stopped(cuda, ordered, threshold, per_pass):
    """Passes, and bounces of a pass, without paths: image and sample counts are
    the plain adaptive renderer's. (From 128 tiles of 4,096 paths on, 85.3
    samples of 96x64, partitions look for that.)"""
    s = prr.Scene.from_desc(scenes.cornell_box(96, 64))
    s.set_wavefront(paths_per_pass=96 * 64 * per_pass, stack_smem=8, ordered=ordered)
    spp = 4 * per_pass
    got, n = s.render(spp, 12, mode="wavefront", min_spp=1, threshold=threshold)
    want, m = s.render(spp, 12, mode="plain", min_spp=1, threshold=threshold)
    assert torch.equal(n, m) and torch.equal(got, want)


def test_default_pass_leaves_memory_to_others(cuda):
    """With 24 GB free a frame of 33.5M paths (10.7 GB of path state) is split:
    no more than a quarter of the free memory is taken, and the image stays."""
    s = prr.Scene.from_desc(scenes.cornell_box(1024, 1024))
    want = s.render(32, 2, mode="plain", slices=1)[0]
    torch.cuda.synchronize()
    ballast = []
    try:
        spare = torch.cuda.mem_get_info()[0] - (24 << 30)
        while spare > 0:
            ballast.append(torch.empty(min(spare, 16 << 30), dtype=torch.uint8, device=cuda))
            spare -= 16 << 30
        free = torch.cuda.mem_get_info()[0]
        got = s.render(32, 2, mode="wavefront")[0]
        torch.cuda.synchronize()
        taken = free - torch.cuda.mem_get_info()[0]
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert taken <= free / 4 + (64 << 20)  # and the image's own block
    assert launches(s) > 2 + 13 * 3 + 1
    assert torch.equal(got, want)
    again = s.render(32, 2, mode="wavefront")[0]
    assert torch.equal(again, want)
