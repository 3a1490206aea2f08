"""Closest hit and any hit over the four-wide mesh nodes against the C
restatement's walk of the binary tree, bit for bit, where the two could part:
tiny and ragged trees (empty slots), deep ones (not collapsed), boxes with
faces through the rays' origins, directions with zero, infinite and NaN
components; and at the batch sizes where the rays a warp holds change."""
import numpy as np
import pytest
import torch

import photorealisticrender4610_b200 as prr
from photorealisticrender4610_b200 import scenes

pytestmark = pytest.mark.gpu


def soup(n):
    return scenes.query_set(n, 1, seed=n, jitter=0.08)[0]


def lattice(n=7):
    """Unit quads on integer planes: box faces at small whole numbers."""
    g = np.arange(n, dtype=np.float32)
    tris = []
    for x in g:
        for y in g:
            a, b, c, d = (x, y, 0), (x + 1, y, 0), (x + 1, y + 1, 0), (x, y + 1, 0)
            tris += [a + b + c, a + c + d]
            tris += [tuple(p[k] for p in (a, b, c) for k in (2, 0, 1))]
    return np.array(tris, np.float32).reshape(-1, 9)


def spiral(base, n):
    """Triangles growing geometrically: a deep, one-sided tree."""
    x = base ** np.arange(n) * 1e-3
    v = np.zeros((n, 9))
    for a in range(3):
        v[:, 3 * a] = x * (1 + 0.01 * a)
        if a:
            v[:, 3 * a + a] = x * 0.01
    return v.astype(np.float32)


MESHES = {**{f"soup{n}": (lambda n=n: soup(n)) for n in (1, 2, 4, 5, 6, 9, 17, 33, 257, 5000)},
          "lattice": lattice, "deep": lambda: spiral(1.2, 260)}


def rays(verts, n, seed):
    rng = np.random.default_rng(seed)
    v = verts.reshape(-1, 3)
    lo, hi = v.min(0), v.max(0)
    o = (lo + (hi - lo) * rng.uniform(-0.5, 1.5, (n, 3))).astype(np.float32)
    tri = verts.reshape(-1, 3, 3)[rng.integers(0, len(verts), n)].astype(np.float64)
    b = rng.dirichlet([1, 1, 1], n)
    target = (tri * b[:, :, None]).sum(1)
    # half start about a triangle's size away from the triangle they aim at
    size = np.ptp(tri, axis=1).max(1, keepdims=True)
    near = (target + rng.normal(0, 2, (n, 3)) * size).astype(np.float32)
    o = np.where(rng.random((n, 1)) < 0.5, near, o)
    d = target - o
    d = (d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-20)).astype(np.float32)
    # a quarter: axis-parallel, or starting on a vertex's coordinate (a box face)
    k = np.arange(n)
    q = k % 8 == 0
    d[q, rng.integers(0, 3, n)[q]] = 0.0
    q = k % 8 == 1
    d[q] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, n)[q]] * np.where(k[q] % 16 == 1, 1, -1)[
        :, None]
    q = k % 8 < 3
    ax = rng.integers(0, 3, n)
    o[k[q], ax[q]] = v[rng.integers(0, len(v), n)[q], ax[q]]
    # and a few without meaning
    bad = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-42], np.float32)
    q = k % 32 == 31
    m = rng.random((n, 3)) < 0.6
    d = np.where(q[:, None] & m, bad[rng.integers(0, 6, (n, 3))], d)
    q = k % 64 == 63
    o = np.where(q[:, None] & ~m, bad[rng.integers(0, 6, (n, 3))], o)
    d[k % 128 == 127] = np.inf
    return o.astype(np.float32), d.astype(np.float32), rng.uniform(0, 2, n).astype(np.float32)


def bits(x):
    return np.ascontiguousarray(x).view(np.uint32)


@pytest.mark.parametrize("mesh", MESHES)
def test_quad_walk_equals_binary_walk(port, cuda, mesh):
    verts = MESHES[mesh]()
    o, d, tmax = rays(verts, 6000, 3)
    hid, t, _ = port.mesh(verts).intersect(o, d)
    occ = port.mesh(verts).occluded(o, d, tmax)
    s = prr.Scene.single_mesh(verts)
    to, td = torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda)
    for cfg in (None, {"persistent": 1}, {"persistent": 2}, {"persistent": 3}):
        h, tt = s.mesh_intersect(0, to, td, config=cfg)
        assert np.array_equal(h.cpu().numpy(), hid), cfg
        assert np.array_equal(bits(tt.cpu().numpy()), bits(t)), cfg
    got = s.mesh_occluded(0, to, td, torch.from_numpy(tmax).to(cuda))
    assert np.array_equal(got.cpu().numpy().astype(bool), np.asarray(occ).astype(bool))
    # the scene-level walks of the same single mesh
    ob, prim, st = s.intersect(to, td)
    assert np.array_equal(prim.cpu().numpy(), hid)
    assert np.array_equal(bits(st.cpu().numpy()), bits(t))
    got = s.intersectP(to, td, torch.from_numpy(tmax).to(cuda))
    assert np.array_equal(got.cpu().numpy().astype(bool), np.asarray(occ).astype(bool))


def walk(nodes, verts, o, d):
    """The binary walk (BVH.cpp:311-415) of one ray in numpy float32 scalars,
    with a stack of any depth: (triangle id, t)."""
    f = np.float32
    tri = verts.reshape(-1, 3, 3)
    inv = [f(1) / x if x != 0 else f(np.inf) for x in d]

    def slab(i):
        b = nodes["bounds"][i]
        lo, hi = f(0), f(np.inf)
        for k in range(3):
            p, q = (b[2 * k + 1], b[2 * k]) if d[k] < 0 else (b[2 * k], b[2 * k + 1])
            lo = np.fmax(lo, (p - o[k]) * inv[k])
            hi = np.fmin(hi, (q - o[k]) * inv[k])
        return lo if lo <= hi else f(np.inf)

    def hit(k):
        v0, e1, e2 = tri[k][0], tri[k][1] - tri[k][0], tri[k][2] - tri[k][0]
        cross = lambda a, b: (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],  # noqa: E731
                              a[0] * b[1] - a[1] * b[0])
        dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
        p, tv = cross(d, e2), o - v0
        det = dot(p, e1)
        r = f(1) / det
        u = dot(p, tv) * r
        q = cross(tv, e1)
        v, t = dot(q, d) * r, dot(q, e2) * r
        if abs(det) < f(1e-6) or u < 0 or v < 0 or u + v > 1 or t <= f(1e-3):
            return None
        return t

    best, bid, stack, i = f(np.inf), -1, [], 0
    while True:
        cnt = int(nodes["meta"][i]) & 0xFFFFFF
        nxt = None
        if cnt == 0:
            l, r = i + 1, int(nodes["first_child"][i])
            tl, tr = slab(l), slab(r)
            near, far = ((l, tl), (r, tr)) if tl <= tr else ((r, tr), (l, tl))
            if near[1] < best:
                nxt = near[0]
                if far[1] < best:
                    stack.append(far)
        else:
            first = int(nodes["first_child"][i])
            for k in nodes["ordered"][first:first + cnt]:
                t = hit(int(k))
                if t is not None and t < best:
                    best, bid = t, int(k)
        while nxt is None and stack:
            j, tj = stack.pop()
            if tj < best:
                nxt = j
        if nxt is None:
            return bid, best
        i = nxt


def test_tree_deeper_than_the_collapse_limit(cuda):
    """More levels than the mesh's four-wide form may need stack entries for
    (64): it keeps the binary shape. The C restatement, like the reference,
    stops at 64 levels, so the walk is restated here."""
    verts = spiral(1.15, 600)
    o, d, _ = rays(verts, 400, 3)
    s = prr.Scene.single_mesh(verts)
    assert s.stats()["blas_depth"] > 64
    nodes = s.export_nodes(0)
    with np.errstate(all="ignore"):
        want = [walk(nodes, verts, o[k], d[k]) for k in range(len(o))]
    ids = np.array([w[0] for w in want], np.int32)
    ts = np.array([w[1] for w in want], np.float32)
    assert (ids >= 0).sum() > 50
    for cfg in (None, {"persistent": 1}, {"persistent": 2}, {"persistent": 3}):
        h, t = s.mesh_intersect(0, torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda),
                                config=cfg)
        assert np.array_equal(h.cpu().numpy(), ids)
        assert np.array_equal(bits(t.cpu().numpy()), bits(ts))


@pytest.mark.parametrize("n", [1, 31, 33, 4_735, 4_737, 40_001, 94_720, 94_721, 189_441, 250_007])
def test_batch_sizes(port, cuda, n):
    verts = soup(300)
    o, d, tmax = rays(verts, n, n)
    hid, t, _ = port.mesh(verts).intersect(o, d)
    s = prr.Scene.single_mesh(verts)
    to, td = torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda)
    h, tt = s.mesh_intersect(0, to, td)
    assert np.array_equal(h.cpu().numpy(), hid)
    assert np.array_equal(bits(tt.cpu().numpy()), bits(t))
    ob, prim, st, geo = s.intersect(to, td, geo=True)
    assert np.array_equal(prim.cpu().numpy(), hid)
    assert np.array_equal(bits(st.cpu().numpy()), bits(t))


@pytest.mark.parametrize("n", [3_000, 250_007])
def test_captured_queries(port, cuda, n):
    """Under stream capture the queries allocate nothing and use fixed shares."""
    verts = soup(300)
    o, d, tmax = rays(verts, n, 5)
    hid, t, _ = port.mesh(verts).intersect(o, d)
    occ = port.mesh(verts).occluded(o, d, tmax)
    s = prr.Scene.single_mesh(verts)
    to, td = torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda)
    tm = torch.from_numpy(tmax).to(cuda)
    s.mesh_intersect(0, to, td)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        h, tt = s.mesh_intersect(0, to, td)
        oc = s.mesh_occluded(0, to, td, tm)
    for _ in range(2):
        h.zero_(), tt.zero_(), oc.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(h.cpu().numpy(), hid)
        assert np.array_equal(bits(tt.cpu().numpy()), bits(t))
        assert np.array_equal(oc.cpu().numpy().astype(bool), np.asarray(occ).astype(bool))
