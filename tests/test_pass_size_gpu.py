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
