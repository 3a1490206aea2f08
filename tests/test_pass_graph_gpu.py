"""A render of several passes replays one captured pass; the capture is used
again only for the same inputs."""
import pytest
import torch

import photorealisticrender4610_b200 as prr
from photorealisticrender4610_b200 import scenes

pytestmark = pytest.mark.gpu


def box(size=128):
    desc = scenes.cornell_box(size, size)
    s = prr.Scene.from_desc(desc)
    s.set_wavefront(paths_per_pass=size * size, stack_smem=8)  # a pass per sample
    return s


def both(s, **kw):
    got = s.render(4, 3, mode="wavefront", **kw)[0].clone()
    return got, s.render(4, 3, mode="plain", slices=1, **kw)[0]


def test_background_changed_between_renders(cuda):
    s = box()
    images = []
    for rgb in ((0.1, 0.2, 0.3), (0.9, 0.4, 0.2)):
        s.set_background(rgb)
        got, want = both(s)
        assert torch.equal(got, want)
        images.append(got)
    assert not torch.equal(images[0], images[1])


@pytest.mark.parametrize("first, second", [
    (dict(window=(0, 0, 128, 64), seed=64), dict(window=(0, 64, 128, 128), seed=0)),
    (dict(window=(0, 0, 128, 64), seed=1), dict(window=(0, 0, 128, 64), seed=2)),
    (dict(window=(0, 0, 64, 64), seed=1), dict(window=(64, 0, 128, 64), seed=1)),
    (dict(seed=1), dict(seed=1, sample_offset=1)),
    (dict(seed=1), dict(seed=1, indirect_clamp=0.25)),
])
def test_other_window_seed_or_samples(cuda, first, second):
    s = box()
    both(s, **first)
    got, want = both(s, **second)
    assert torch.equal(got, want)
