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
