"""The plain renderer runs large windows of scenes with small meshes in blocks
whose warps keep step. The image is that of the same render in small windows,
which run in independent warps, bit for bit."""
import numpy as np
import pytest

import photorealisticrender4610_b200 as prr
from photorealisticrender4610_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [scenes.cornell_box,
                                  lambda w, h: scenes.caustics(w, h, level=2),
                                  lambda w, h: scenes.museum_like(w, h, level=1,
                                                                  env_size=(64, 32))])
@pytest.mark.parametrize("size", [(250, 130), (403, 77)])
def test_large_window_equals_small_ones(cuda, make, size):
    w, h = size
    s = prr.Scene.from_desc(make(w, h))
    whole, _ = s.render(8, 6, seed=5, mode="plain", slices=4)
    whole = whole.cpu().numpy()
    for y in range(0, h, 26):
        for x in range(0, w, 50):
            win = (x, y, min(x + 50, w), min(y + 26, h))
            part, _ = s.render(8, 6, seed=5, mode="plain", slices=4, window=win)
            assert np.array_equal(part.cpu().numpy().view(np.uint32),
                                  np.ascontiguousarray(whole[y:win[3], x:win[2]]).view(np.uint32))


@pytest.mark.parametrize("size, spp, slices", [((161, 121), 16, 16), ((161, 121), 17, 16),
                                               ((161, 121), 12, 6), ((161, 121), 66, 33),
                                               ((161, 121), 64, 64), ((321, 203), 6, 4),
                                               ((1, 4001), 32, 32), ((4001, 1), 32, 8)])
@pytest.mark.parametrize("small", [True, False])
def test_slices_side_by_side(cuda, size, spp, slices, small):
    """A pixel's slices share a warp: the image is the float32 sum, slice after
    slice, of the slices rendered alone, bit for bit."""
    w, h = size
    s = prr.Scene.from_desc(scenes.cornell_box(w, h) if small else
                            scenes.museum_like(w, h, level=3, env_size=(8, 4)))
    got, _ = s.render(spp, 3, seed=2, mode="plain", slices=slices)
    acc = None
    for k in range(slices):
        a, b = spp * k // slices, spp * (k + 1) // slices
        part = np.zeros((h, w, 3), np.float32)
        for n in range(a, b):
            one, _ = s.render(1, 3, seed=2, mode="plain", slices=1, sample_offset=n)
            part = part + one.cpu().numpy()
        acc = part if acc is None else acc + part
    want = acc / np.float32(spp)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("level", [1, 2])
def test_large_window_of_a_scene_with_deeper_meshes(cuda, level):
    """Enough blocks for meshes of 6 and 8 levels to keep step (32 slices)."""
    w, h = 330, 200
    s = prr.Scene.from_desc(scenes.museum_like(w, h, level=level, env_size=(64, 32)))
    whole, _ = s.render(32, 4, seed=5, mode="plain", slices=32)
    whole = whole.cpu().numpy()
    for y in range(0, h, 26):
        for x in range(0, w, 50):
            win = (x, y, min(x + 50, w), min(y + 26, h))
            part, _ = s.render(32, 4, seed=5, mode="plain", slices=32, window=win)
            assert np.array_equal(part.cpu().numpy().view(np.uint32),
                                  np.ascontiguousarray(whole[y:win[3], x:win[2]]).view(np.uint32))
