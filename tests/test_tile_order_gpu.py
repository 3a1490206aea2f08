"""The wavefront orders a window's pixels in 8x4 tiles: at ragged windows its
film and spp map equal the plain renderer's, bit for bit and pixel for pixel,
and a served image equals them too."""
import numpy as np
import pytest
import torch

import photorealisticrender4610_b200 as prr
from photorealisticrender4610_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [(0, 0, 1, 1), (3, 2, 10, 5), (0, 0, 8, 4), (5, 1, 14, 6),
                                    (1, 7, 34, 13), (0, 0, 63, 1), (2, 0, 3, 41), (0, 0, 64, 48)])
def test_ragged_windows(cuda, window):
    s = prr.Scene.from_desc(scenes.cornell_box(64, 48))
    for kw in (dict(), dict(min_spp=1, threshold=0.2)):
        a, na = s.render(6, 4, seed=3, mode="plain", window=window, slices=1, **kw)
        b, nb = s.render(6, 4, seed=3, mode="wavefront", window=window, **kw)
        assert np.array_equal(a.cpu().numpy().view(np.uint32), b.cpu().numpy().view(np.uint32))
        assert torch.equal(na, nb)
    a, _ = s.render(6, 4, seed=3, mode="wavefront", window=window)
    srv = prr.Server()
    out = torch.empty_like(a)
    srv.wait(srv.submit(srv.add_scene(s), 6, 4, seed=3, window=window, out=out))
    assert np.array_equal(a.cpu().numpy().view(np.uint32), out.cpu().numpy().view(np.uint32))


@pytest.mark.parametrize("spp, paths", [(1, 0), (5, 0), (32, 0), (33, 0), (12, 3 * 37 * 21),
                                        (7, 1)])
def test_samples_of_a_pixel_in_a_row(cuda, spp, paths):
    """A pixel's samples are neighbouring paths, in one pass or several: the
    film is the plain renderer's, fixed and adaptive."""
    s = prr.Scene.from_desc(scenes.cornell_box(37, 21))
    s.set_wavefront(paths_per_pass=paths)
    for kw in (dict(), dict(min_spp=1, threshold=0.2)):
        a, na = s.render(spp, 4, seed=5, mode="plain", slices=1, **kw)
        b, nb = s.render(spp, 4, seed=5, mode="wavefront", **kw)
        assert np.array_equal(a.cpu().numpy().view(np.uint32), b.cpu().numpy().view(np.uint32))
        assert torch.equal(na, nb)
