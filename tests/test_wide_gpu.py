"""The walk over 8-wide nodes (wide.cuh) where it could part from the binary walk it stands for: the same
hits to the bit, ties in t among them, on every route a call can take - 8 lanes a ray (small
calls), one lane a ray (large ones), the wavefront's queues and the one-kernel path tracer. The binary
walk is reached through LRC_SORT_RAYS (a large batch of queries) and through a tree given as device
arrays (which is not collapsed)."""
import ctypes as C

import numpy as np
import pytest

import little_renderer_b200 as L
from little_renderer_b200 import render as R, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def own():
    return L.Context(0)


def tables():
    mask, tab = np.zeros(4096, np.uint16), np.zeros(2112, np.float32)
    L.lib().lrc_default_blue_noise(mask.ctypes.data)
    L.lib().lrc_default_bsdf_tables(tab.ctypes.data)
    return mask, tab


def made(s):
    """The queries' wide nodes made now (counting their walk makes them, else a few queries do)."""
    s.set_walk(2)
    s.trace_stats(np.zeros((1, 3), np.float32), np.ones((1, 3), np.float32))


def triangles(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "soup":
        return W.corners_to_quv(W.soup(n, seed))
    quv = np.zeros((n, 9), np.float32)
    quv[:, 0:3] = rng.random((n, 3), dtype=np.float32)
    quv[:, 3:9] = (rng.random((n, 6), dtype=np.float32) - 0.5) * 0.2
    if kind == "twice":                              # every triangle twice or more: all hits are ties
        quv = quv[rng.integers(0, max(1, n // 3), n)]
    if kind == "grid":                               # coplanar cells sharing edges, rays through their corners
        k = int(np.ceil(np.sqrt(n)))
        x, y = np.meshgrid(np.arange(k), np.arange(k))
        quv[:, 0], quv[:, 1], quv[:, 2] = x.reshape(-1)[:n] / np.float32(k), y.reshape(-1)[:n] / np.float32(k), 0.5
        quv[:, 3:9] = 0
        quv[:, 3], quv[:, 7] = 1.0 / k, 1.0 / k
    if kind == "far":                                # away from the origin, in another scale
        quv *= 300.0
        quv[:, 0:3] += 5000.0
    if kind == "wild":                               # boxes no grid holds: the binary walk answers
        quv[rng.integers(0, n), 3:6] = np.inf
        quv[rng.integers(0, n), 0:3] = np.nan
    return quv


def rays(kind, n, seed):
    o, d = W.rays_at_cube(n, seed)
    rng = np.random.default_rng(seed)
    if kind == "grid":
        o = rng.integers(0, 17, (n, 3)).astype(np.float32) / 16
        o[:, 2] = -1.0
        d = np.tile(np.array([0, 0, 1], np.float32), (n, 1))
    if kind == "far":
        o, d = (o * 300 + 5000).astype(np.float32), d
    d[: n // 50, rng.integers(0, 3)] = 0.0           # axis-parallel ones, of both zeros
    d[: n // 100] *= np.float32(-1)
    return np.ascontiguousarray(o), np.ascontiguousarray(d)


@pytest.mark.parametrize("kind", ["soup", "twice", "grid", "far", "wild"])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 100, 5000, 60_000])
@pytest.mark.parametrize("builder", [0, 1])
def test_queries_are_the_binary_walks(own, kind, n, builder):
    s = L.native.Scene(own)
    s.set_triangles(L.pack_tris(triangles(kind, n, 3)))
    s.build(builder, 30)
    made(s)
    m = 1 << 18                                      # (LRC_SORT_RAYS: the binary walk, from this many rays)
    o, d = rays(kind, m, 4)
    prim, t = np.zeros(m, np.int32), np.zeros(m, np.float32)
    own.check(own.L.lrc_scene_intersect(s.h, o.ctypes.data, d.ctypes.data, m, 0.0, 1e30, prim.ctypes.data, t.ctypes.data, 2))
    for k in (m, 16_385, 16_384, 1000, 1):           # one lane a ray, then 8
        p, tt = s.intersect(o[:k], d[:k])
        assert np.array_equal(p, prim[:k]) and np.array_equal(tt.view(np.uint32), t[:k].view(np.uint32))
    if kind == "wild":                               # (a triangle with an infinite edge is hit at a t that is no number)
        return
    tmax = np.where(prim >= 0, t, 3.0).astype(np.float32)
    tmax[::3] = np.nextafter(tmax[::3], np.float32(10))      # just past the hit: blocked
    want = (prim >= 0) & (tmax > t)
    for k in (m, 5000):
        assert np.array_equal(s.occluded(o[:k], d[:k], tmax[:k]).astype(bool), want[:k])
    s.close()


def as_given(own, sc, s, builder):
    """The scene again with the same tree given as device arrays (walked as it is)."""
    n = s.n + 1
    nodes, aux = np.zeros((2 * n - 1, 8), np.uint32), np.zeros(n, np.uint32)
    own.check(own.L.lrc_scene_tree(s.h, nodes.ctypes.data, aux.ctypes.data, 0))
    mask, tab = tables()
    b = R.world_scene(own, sc, builder, 30, mask, tab)
    dn, da = torch.from_numpy(nodes.view(np.int32)).cuda(), torch.from_numpy(aux.view(np.int32)).cuda()
    torch.cuda.synchronize()
    own.check(own.L.lrc_scene_set_tree(b.h, C.c_void_p(dn.data_ptr()), 2 * n - 1, C.c_void_p(da.data_ptr()), n,
                                       L.native.LRC_DEVICE))
    own.sync()
    return b


@pytest.mark.parametrize("builder", [0, 1])
@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("exact", [0, 1])
def test_images_are_the_binary_walks(own, builder, double, exact):
    """double: each shape's triangles once more with another material (every hit a tie)."""
    sc = W.box_scene(5, 3000, 72, 40)
    if double:
        sc["corners"] = np.concatenate([sc["corners"], sc["corners"]])
        sc["tri_mats"] = np.concatenate([sc["tri_mats"], np.roll(sc["tri_mats"], 7)])
    mask, tab = tables()
    s = R.world_scene(own, sc, builder, 30, mask, tab)
    b = as_given(own, sc, s, builder)
    p = L.native.trace_params(R.camera12(sc), 72, 40, 8, 1, 1, exact, 3)
    for spp in (1, 3, 8, 19):                        # 8 lanes a path, a pixel's samples in 1 to 16 of them
        want, r0 = b.trace(p, spp, flags=L.native.LRC_TRACE_MEGAKERNEL)
        got, r1 = s.trace(p, spp, flags=L.native.LRC_TRACE_MEGAKERNEL)
        assert np.array_equal(got, want) and r0 == r1
        for engine in (0, 1):
            img = torch.zeros(40, 72, 4, device="cuda")
            torch.cuda.synchronize()
            q = L.native.Batch(own)
            q.set_engine(engine)
            q.set_wavefront(1024)
            q.add(s, p, spp, img.data_ptr())
            q.run()
            own.sync()
            assert np.array_equal(img.cpu().numpy(), want)
            q.close()
    planes_s, planes_b = s.guide(p), b.guide(p)
    assert np.array_equal(planes_s, planes_b)
    if not exact:
        assert np.array_equal(s.trace_guided(p, 5, planes_s)[0], b.trace_guided(p, 5, planes_b)[0])
        assert np.array_equal(s.caustics(p, 3000, 9)[0], b.caustics(p, 3000, 9)[0])
        a, c = (x.trace_frame(p, p, 5, 1, pl, 32, 8) for x, pl in ((s, planes_s), (b, planes_b)))
        assert np.array_equal(a, c)
    s.close()
    b.close()


@pytest.mark.parametrize("leaf", [1, 3, 8, 9])
def test_given_trees_with_larger_leaves(own, leaf):
    """A tree given with leaves of several entries (up to a node's 8 slots; 9 stays binary): hits as the
    built tree's."""
    n = 700
    quv = triangles("plain", n, 8)
    s = L.native.Scene(own)
    s.set_triangles(L.pack_tris(quv))
    s.build(1, 30)
    o, d = rays("plain", 4000, 5)
    want = s.intersect(o, d)
    lo = np.minimum(np.minimum(quv[:, 0:3], quv[:, 0:3] + quv[:, 3:6]), quv[:, 0:3] + quv[:, 6:9]) - np.float32(1e-3)
    hi = np.maximum(np.maximum(quv[:, 0:3], quv[:, 0:3] + quv[:, 3:6]), quv[:, 0:3] + quv[:, 6:9]) + np.float32(1e-3)
    nodes, aux = [], []

    def make(ids):
        at = len(nodes)
        nodes.append(np.zeros(8, np.uint32))
        f = nodes[at].view(np.float32)
        f[0:3], f[4:7] = lo[ids].min(0), hi[ids].max(0)
        if len(ids) <= leaf:
            nodes[at][3], nodes[at][7] = len(aux), 0x80000000 | len(ids)
            aux.extend(ids.tolist())
        else:
            k = ids[np.argsort(quv[ids, at % 3], kind="stable")]
            a, b = make(k[: len(k) // 2]), make(k[len(k) // 2:])
            nodes[at][3], nodes[at][7] = a, b
        return at

    make(np.arange(n))
    s.set_tree(np.array(nodes), np.array(aux, np.uint32))
    made(s)
    got = s.intersect(o, d)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    s.close()
