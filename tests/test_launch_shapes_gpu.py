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


def captured(fn):
    """fn's outputs as a replayed CUDA graph leaves them."""
    fn()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = fn()
    for x in out:
        x.zero_()
    g.replay()
    torch.cuda.synchronize()
    return out


MODES = [{}, {"persistent": 1}, {"persistent": 2}, {"persistent": 3}]


@pytest.mark.parametrize("rays", [5_000, 200_000])
def test_largest_blocks_on_a_large_mesh(port, cuda, rays):
    """300,000 triangles: 21 entries for the binary walk's stack, about 30 for
    the four-wide one's, of which a block of 1,024 has shared memory for 28."""
    v, o, d = scenes.query_set(300_000, rays, seed=4)
    want = port.mesh(v).intersect(o, d)
    s = prr.Scene.single_mesh(v)
    to, td = torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda)
    for cfg in MODES:
        cfg = {**cfg, "block_size": 1024}
        equal(s.mesh_intersect(0, to, td, config=cfg), want)
        equal(captured(lambda: s.mesh_intersect(0, to, td, config=cfg)), want)


def spiral(base, n):
    """Triangles growing geometrically: a deep, one-sided tree."""
    x = base ** np.arange(n) * 1e-3
    v = np.zeros((n, 9))
    for a in range(3):
        v[:, 3 * a] = x * (1 + 0.01 * a)
        if a:
            v[:, 3 * a + a] = x * 0.01
    return v.astype(np.float32)


@pytest.mark.parametrize("base, n", [(1.5, 60), (1.4, 100), (1.3, 150), (1.2, 260), (1.15, 600)])
def test_stacks_beyond_shared_memory(cuda, base, n):
    """Trees of more levels than a block's share of shared memory holds, and
    rays that enter every box (a component without a bound on each axis but
    one): all modes and block sizes agree, captured or not."""
    verts = spiral(base, n)
    s = prr.Scene.single_mesh(verts)
    rng = np.random.default_rng(n)
    tri = verts.reshape(-1, 3, 3)[rng.integers(0, n, 4000)]
    target = (tri * rng.dirichlet([1, 1, 1], 4000)[:, :, None]).sum(1)
    o = np.where(rng.random((4000, 1)) < 0.5, -target, target * 0.5)
    d = target - o
    d = d / np.linalg.norm(d, axis=1, keepdims=True)
    d[::8] = [np.inf, np.nan, 1.0]
    to = torch.from_numpy(o.astype(np.float32)).to(cuda)
    td = torch.from_numpy(d.astype(np.float32)).to(cuda)
    tm = torch.full((4000,), np.inf, device=cuda)
    hid, t = s.mesh_intersect(0, to, td)
    want = (hid.cpu().numpy(), t.cpu().numpy())
    assert (want[0] >= 0).sum() > 200
    for cfg in MODES:
        for block in (32, 128, 256):
            cfg = {**cfg, "block_size": block}
            equal(s.mesh_intersect(0, to, td, config=cfg), want)
            equal(captured(lambda: s.mesh_intersect(0, to, td, config=cfg)), want)
    ob, prim, st = s.intersect(to, td)
    equal((prim, st), want)
    equal(captured(lambda: s.intersect(to, td)[1:]), want)
    for fn in (lambda: s.mesh_occluded(0, to, td, tm), lambda: s.intersectP(to, td, tm)):
        occ = fn().cpu().numpy() > 0
        assert np.array_equal(occ, want[0] >= 0)
        assert np.array_equal(captured(lambda: (fn(),))[0].cpu().numpy() > 0, occ)


def clutter(objects, size):
    """Many small meshes: a scene tree of 17 levels for 20,000."""
    rng = np.random.default_rng(1)
    desc = scenes.SceneDesc(width=size, height=size, name="clutter")
    m = desc.add_material(scenes.Material(scenes.DIFFUSE, (0.7, 0.6, 0.5), 0.6, 0.0))
    c = rng.uniform(0, 1, (objects, 1, 3))
    for tri in (c + rng.normal(0, 0.01, (objects, 6, 3))).astype(np.float32).reshape(-1, 2, 9):
        desc.objects.append(scenes.MeshObject(tri, m))
    desc.background = (0.3, 0.5, 0.8)
    desc.camera = scenes.Camera(eye=(2.2, 1.6, 2.4), target=(0.5, 0.5, 0.5), fovv=40, fovh=45)
    return desc


def test_wavefront_blocks_on_a_deep_scene_tree(cuda):
    """The scene level's entries alone exceed the 24 a block of 512 has shared
    memory for: they spill as the mesh level's do."""
    s = prr.Scene.from_desc(clutter(20_000, 64))
    assert s.stats()["tlas_depth"] >= 16
    want, spp = s.render(2, 4, mode="plain")
    for block, stack in ((512, 0), (512, 8), (512, 1), (256, 0), (64, 8)):
        s.set_wavefront(block_size=block, stack_smem=stack)
        got, n = s.render(2, 4, mode="wavefront")
        assert torch.equal(got, want) and torch.equal(n, spp), (block, stack)


# where the scene and any-hit queries change kernels (640 rays per SM), and
# where they begin to hand out rays from a counter (64 rays a warp: 2 x 75,776
# for the 4 resident blocks of the small batches' form, 2 x 151,552 for 8)
@pytest.mark.parametrize("rays", [75_777, 94_720, 94_721, 151_553, 303_104, 303_105, 340_993])
def test_scene_and_any_hit_batch_sizes(port, cuda, rays):
    v, o, d = scenes.query_set(400, rays, seed=2)
    tmax = np.linspace(0.05, 2, rays, dtype=np.float32)
    m = port.mesh(v)
    want = m.intersect(o, d)
    occ = np.asarray(m.occluded(o, d, tmax)) > 0
    s = prr.Scene.single_mesh(v)
    to, td, tm = (torch.from_numpy(a).to(cuda) for a in (o, d, tmax))
    ob, prim, t, geo = s.intersect(to, td, geo=True)
    equal((prim, t), want)
    hit = want[0] >= 0
    # coords as Triangle::finalize forms them: origin + direction * t
    coords = o + d * want[1][:, None]
    assert np.array_equal(geo.cpu().numpy()[hit, :3].view(np.uint32),
                          coords[hit].view(np.uint32))
    assert np.array_equal(s.mesh_occluded(0, to, td, tm).cpu().numpy() > 0, occ)
    assert np.array_equal(s.intersectP(to, td, tm).cpu().numpy() > 0, occ)
