"""What else may happen to a scene between the making of its wide nodes and a walk over them - builds and
moves in a caller's graph or a batch's, queries in one, other streams, boxes and rays that are no
numbers, trees deeper than a stack - against the binary walk (LRC_SORT_RAYS, the one-kernel path) or
a scene made anew."""
import ctypes as C

import numpy as np
import pytest

import little_renderer_b200 as L
from little_renderer_b200 import render as R, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEVICE = L.native.LRC_DEVICE


@pytest.fixture(scope="module")
def own():
    return L.Context(0)


def dev(a):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    torch.cuda.synchronize()
    return t


def soup(n, seed):
    return L.pack_tris(W.corners_to_quv(W.soup(n, seed)))


def made(s):
    """The queries' wide nodes made now (counting their walk makes them, else a few queries do)."""
    s.set_walk(2)
    s.trace_stats(np.zeros((1, 3), np.float32), np.ones((1, 3), np.float32))


def hits(own, tris, o, d):
    """The closest hits of a scene made anew."""
    s = L.native.Scene(own)
    s.set_triangles(tris)
    s.build(1, 30)
    out = s.intersect(o, d)
    s.close()
    return out


def captured(own, fn):
    """fn's calls as a graph of a caller's."""
    side = torch.cuda.Stream()
    own.set_stream(side.cuda_stream)
    g = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(g, stream=side):
            fn()
    finally:
        own.set_stream(None)
    return g


def replay(own, g):
    own.sync()
    g.replay()
    torch.cuda.synchronize()


def field(own, few=True, wild=None):
    """An instanced field: the scene, its dict and its records. few: meshes of some 25 triangles. wild: one
    triangle of each mesh has a coordinate of that value, the instances' boxes as they were."""
    sc = W.instanced_field(seed=3, n_instances=200, n_meshes=4, tri_range=(20, 30) if few else (200, 900),
                           width=72, height=40, sky_w=64, sky_h=32, spp=1, max_depth=6)
    records = W.instance_records(sc)
    if wild is not None:
        sc["meshes"] = [m.copy() for m in sc["meshes"]]
        for i, m in enumerate(sc["meshes"]):
            m[1 + i % 3, 0, i % 3] = wild
    s = L.native.Scene(own)
    g = sc["ground"]
    s.set_prims(W.make_quad(g["q"], g["u"], g["v"], g["material"]))
    s.set_light(-1)
    s.set_materials(W.material_records(sc["materials"]))
    s.build(1, 30)
    s.set_meshes([L.pack_tris(W.corners_to_quv(t), np.full(t.shape[0], m, np.int32))
                  for t, m in zip(sc["meshes"], sc["mesh_mats"])])
    s.set_instances(records)
    s.build_instances(0, 30)
    s.set_sky(sc["sky"])
    return s, sc, records


def wavefront(own, s, p, spp, **run):
    """The image by the wavefront engine (with a stepped run's flags: and its statistics)."""
    img = torch.zeros(p.height, p.width, 4, device="cuda")
    torch.cuda.synchronize()
    q = L.native.Batch(own)
    q.set_wavefront(1024)
    q.add(s, p, spp, img.data_ptr())
    q.run(**run)
    own.sync()
    stats = q.step_stats()
    q.close()
    return (img.cpu().numpy(), stats) if run else img.cpu().numpy()


def one_kernel(s, p, spp):
    return s.trace(p, spp, flags=L.native.LRC_TRACE_MEGAKERNEL)[0]


@pytest.mark.parametrize("m", [1000, 40_000])            # 8 lanes a ray, one
def test_captured_queries_see_the_next_build(own, m):
    n = 5000
    o, d = W.rays_at_cube(m, 2)
    s = L.native.Scene(own)
    s.set_triangles(soup(n, 5))
    s.build(1, 30)
    made(s)                                              # (the wide nodes are there when the graph is captured)
    ro, rd, far = dev(o), dev(d), torch.full((m,), 3.0, device="cuda")
    prim, t = torch.zeros(m, dtype=torch.int32, device="cuda"), torch.zeros(m, device="cuda")
    blocked = torch.zeros(m, dtype=torch.uint8, device="cuda")

    def queries():
        s.intersect_device(ro.data_ptr(), rd.data_ptr(), m, prim.data_ptr(), t.data_ptr())
        own.check(own.L.lrc_scene_occluded(s.h, *[C.c_void_p(x.data_ptr()) for x in (ro, rd, far)], m, 0.0,
                                           C.c_void_p(blocked.data_ptr()), DEVICE))

    g = captured(own, queries)
    for seed in (6, 7):
        s.set_triangles(soup(n, seed))
        s.build(1, 30)
        replay(own, g)
        want = hits(own, soup(n, seed), o, d)
        assert np.array_equal(prim.cpu().numpy(), want[0]) and np.array_equal(t.cpu().numpy(), want[1])
        assert np.array_equal(blocked.cpu().numpy().astype(bool), want[0] >= 0)
    s.close()


def test_captured_small_images_see_the_next_build(own):
    a = W.box_scene(5, 3000, 72, 40)
    other = (a["corners"] * np.float32([0.9, 1, 1])).astype(np.float32)
    s = R.world_scene(own, a, 1)
    p = L.native.trace_params(R.camera12(a), 72, 40, 8, 1, 1, 0, 3)
    first = s.trace(p, 2)[0]
    img, planes = torch.zeros(40, 72, 4, device="cuda"), torch.zeros(4, 40, 72, 4, device="cuda")
    torch.cuda.synchronize()

    def images():
        s.trace_device(p, 2, img.data_ptr())
        s.guide_device(p, planes.data_ptr())

    g = captured(own, images)
    s.set_triangles(L.pack_tris(W.corners_to_quv(other), a["tri_mats"]))
    s.build(1, 30)
    img.zero_()
    replay(own, g)
    got = img.cpu().numpy()
    assert np.array_equal(got, s.trace(p, 2)[0]) and not np.array_equal(got, first)
    assert np.array_equal(planes.cpu().numpy(), s.guide(p))
    s.close()


def test_captured_builds_are_seen_by_the_next_query(own):
    n, m = 5000, 40_000
    o, d = W.rays_at_cube(m, 2)
    s = L.native.Scene(own)
    tris = dev(soup(n, 5).view(np.int32))

    def build():
        s.set_triangles(None, tris.data_ptr(), n)
        s.build(1, 30)

    build()
    made(s)
    g = captured(own, build)
    for seed in (6, 7):
        tris.copy_(dev(soup(n, seed).view(np.int32)))
        torch.cuda.synchronize()
        replay(own, g)
        got, want = s.intersect(o, d), hits(own, soup(n, seed), o, d)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    s.close()


@pytest.mark.parametrize("mode", [0, 1])                 # refitted, rebuilt
def test_captured_moves_are_seen_by_the_next_image(own, mode):
    s, sc, records = field(own)
    p = L.native.trace_params(R.camera12(sc), 72, 40, 6, 1, 1, 0, 3)
    wavefront(own, s, p, 3)
    r = dev(records)

    def move():
        own.check(own.L.lrc_scene_move_instances(s.h, C.c_void_p(r.data_ptr()), records.shape[0], mode, DEVICE))

    move()
    g = captured(own, move)
    for _ in range(2):
        sc["xf"][:, 0, 3] += np.float32(1.5)
        r.copy_(dev(W.instance_records(sc)))
        torch.cuda.synchronize()
        replay(own, g)
        assert np.array_equal(wavefront(own, s, p, 3), one_kernel(s, p, 3))
    s.close()


@pytest.mark.parametrize("engine", [0, 1])
def test_replayed_builds_are_recorded(own, engine):
    """A batch's replayed build after a tree of another kind: given with larger leaves, or built by PLOC."""
    sc = W.box_scene(5, 3000, 72, 40)
    s = L.native.Scene(own)                              # (triangles alone: queries walk a copy of the tree)
    s.set_triangles(L.pack_tris(W.corners_to_quv(sc["corners"]), sc["tri_mats"]))
    s.set_materials(W.material_records(sc["materials"]))
    s.set_light(-1)
    s.build(0, 30)
    o, d = W.rays_at_cube(40_000, 4, centre=(278, 278, 278), scale=555.0)
    want = s.intersect(o, d)
    p = L.native.trace_params(R.camera12(sc), 72, 40, 8, 1, 1, 0, 3)
    image = s.trace(p, 2)[0]
    n = sc["corners"].shape[0]
    pairs = np.zeros((2 * n, 8), np.uint32), np.arange(n, dtype=np.uint32)
    box = pairs[0].view(np.float32)                      # (a list of leaves of 3 under one box)
    leaves = [(i, min(3, n - i)) for i in range(0, n, 3)]
    for k, (i, c) in enumerate(leaves[:-1]):
        for at in (2 * k, 2 * k + 1):
            box[at, 0:3], box[at, 4:7] = -1e4, 1e4
        pairs[0][2 * k][[3, 7]] = 2 * k + 1, 2 * k + 2
        pairs[0][2 * k + 1][[3, 7]] = i, 0x80000000 | c
    last = 2 * (len(leaves) - 1)
    box[last, 0:3], box[last, 4:7] = -1e4, 1e4
    pairs[0][last][[3, 7]] = leaves[-1][0], 0x80000000 | leaves[-1][1]
    img = torch.zeros(40, 72, 4, device="cuda")
    torch.cuda.synchronize()
    q = L.native.Batch(own)
    q.set_engine(engine)
    q.add(s, p, 2, img.data_ptr(), builder=0)
    run = lambda: q.run(build=True, graph=True, zero=True)
    for other in (lambda: s.build(1, 30), lambda: s.set_tree(pairs[0][: last + 1], pairs[1])):
        for _ in range(3):
            run()
        other()
        run()
        own.sync()
        assert q.info()["graph_used"] == 1
        got = s.intersect(o, d)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        assert np.array_equal(s.trace(p, 2)[0], image) and np.array_equal(img.cpu().numpy(), image)
    s.close()
    q.close()


@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("wild", [np.nan, np.inf, 1e19])
@pytest.mark.parametrize("exact", [0, 1])
def test_meshes_that_no_grid_holds(own, exact, wild, few):
    s, sc, _ = field(own, few, wild)
    p = L.native.trace_params(R.camera12(sc), 72, 40, 6, 1, 1, exact, 3)
    assert np.array_equal(wavefront(own, s, p, 5), one_kernel(s, p, 5))
    s.close()


def test_images_on_two_streams_at_once(own):
    """Large images (one batch of the context's traces them) queued on two streams, nothing between them."""
    jobs = []
    for seed, (w, h) in enumerate([(512, 512), (640, 400), (1100, 1000), (512, 512)]):
        sc = W.box_scene(5 + seed, 4000, w, h)
        s = R.world_scene(own, sc, 1)
        p = L.native.trace_params(R.camera12(sc), w, h, 8, 1, 1, 0, 3)
        jobs.append((s, p, one_kernel(s, p, 1), torch.zeros(h, w, 4, device="cuda")))
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        for _ in range(3):
            for k, (s, p, _, img) in enumerate(jobs):
                own.set_stream(streams[k % 2].cuda_stream)
                with torch.cuda.stream(streams[k % 2]):
                    img.zero_()
                s.trace_device(p, 1, img.data_ptr())
            torch.cuda.synchronize()
            for _, _, want, img in jobs:
                assert np.array_equal(img.cpu().numpy(), want)
    finally:
        own.set_stream(None)
    for s, *_ in jobs:
        s.close()


@pytest.mark.parametrize("w,h", [(64, 64), (200, 160), (512, 512)])   # each kind of route, captured on the one-kernel path
def test_images_in_a_callers_graph(own, w, h):
    sc = W.box_scene(5, 1000, w, h)
    s = R.world_scene(own, sc, 1)
    p = L.native.trace_params(R.camera12(sc), w, h, 8, 1, 1, 0, 3)
    planes = s.trace_frame(None, p, 0, 1, None, 0, 8)
    img, new = torch.zeros(h, w, 4, device="cuda"), torch.zeros(4, h, w, 4, device="cuda")
    torch.cuda.synchronize()

    def images():
        s.trace_device(p, 1, img.data_ptr())
        s.trace_frame_device(None, p, 0, 1, 0, new.data_ptr(), 0, 8)

    g = captured(own, images)
    replay(own, g)
    assert np.array_equal(img.cpu().numpy(), one_kernel(s, p, 1)) and np.array_equal(new.cpu().numpy(), planes)
    s.close()


def test_images_without_memory_for_the_wavefront():
    own = L.Context(0)                                   # (a context whose engine has no memory yet)
    w = h = 512
    sc = W.box_scene(5, 1000, w, h)
    s = R.world_scene(own, sc, 1)
    p = L.native.trace_params(R.camera12(sc), w, h, 8, 1, 1, 0, 3)
    want = one_kernel(s, p, 1)
    planes = s.guide(p)
    img, new = torch.zeros(h, w, 4, device="cuda"), torch.zeros(4, h, w, 4, device="cuda")
    torch.cuda.synchronize()
    s.trace_frame_device(None, p, 0, 1, 0, new.data_ptr(), 0, 8)
    own.sync()
    frame = new.cpu().numpy()
    other = L.Context(0)
    s2 = R.world_scene(other, sc, 1)
    s2.guide(p)
    torch.cuda.synchronize()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (24 << 20), dtype=torch.uint8, device="cuda")
    try:
        s2.trace_device(p, 1, img.data_ptr())
        new.zero_()
        torch.cuda.synchronize()
        s2.trace_frame_device(None, p, 0, 1, 0, new.data_ptr(), 0, 8)
        other.sync()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(img.cpu().numpy(), want) and np.array_equal(new.cpu().numpy(), frame)
    assert np.array_equal(frame[2:], planes[2:])
    for x in (s, s2, own, other):
        x.close()


def test_no_wide_nodes_where_none_are_walked(own):
    """Images between the warps' line and the wavefront's, the megakernel engine, caustics: they walk the
    binary nodes, and no memory goes to others."""
    n = 1_000_000
    sc = W.box_scene(5, n, 200, 160)
    s = R.world_scene(own, sc, 1)
    p = L.native.trace_params(R.camera12(sc), 200, 160, 8, 1, 1, 0, 3)
    img = torch.zeros(160, 200, 4, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    s.trace_device(p, 1, img.data_ptr())
    q = L.native.Batch(own)
    q.set_engine(0)
    q.add(s, p, 1, img.data_ptr(), builder=1)
    q.run(build=False)
    s.caustics(p, 1000, 3)
    own.sync()
    assert free - torch.cuda.mem_get_info()[0] < 48 * n  # (the wide nodes of a million shapes: 94 MB)
    q.close()
    s.close()


def odd_rays(m, seed):
    """Rays whose components are no numbers, infinite, all zero, very long or short, or far away: a 16th each."""
    o, d = W.rays_at_cube(m, seed)
    part = [slice(i * m // 16, (i + 1) * m // 16) for i in range(9)]
    o[part[0], seed % 3] = np.nan
    d[part[1], 1] = np.nan
    o[part[2], 0] = np.inf
    d[part[3], 2] = -np.inf
    d[part[4]] = 0.0
    d[part[5]] *= np.float32(1e30)
    d[part[6]] *= np.float32(1e19)
    d[part[7]] *= np.float32(1e-15)
    o[part[8]] *= np.float32(1e6)
    return o, d


def binary(own, s, o, d, tmin, tmax):
    m = o.shape[0]
    prim, t = np.zeros(m, np.int32), np.zeros(m, np.float32)
    own.check(own.L.lrc_scene_intersect(s.h, o.ctypes.data, d.ctypes.data, m, tmin, tmax, prim.ctypes.data, t.ctypes.data, 2))
    return prim, t


@pytest.mark.parametrize("tmin,tmax", [(0.0, 1e30), (0.0, np.inf), (0.0, np.nan), (-5.0, 2.5), (-4.0, -0.5), (2.0, 1.0),
                                       (np.nan, 1e30)])
def test_odd_rays(own, tmin, tmax):
    s = L.native.Scene(own)
    s.set_triangles(soup(5000, 3))
    s.build(1, 30)
    made(s)
    m = 1 << 18
    o, d = odd_rays(m, 4)
    want = binary(own, s, o, d, tmin, tmax)
    for idx in (slice(0, m), slice(0, m, 32)):           # one lane a ray, 8
        got = s.intersect(o[idx], d[idx], tmin, tmax)
        for g, w in zip(got, want):
            assert np.array_equal(g.view(np.uint32), w[idx].view(np.uint32))
    far = np.full(m, tmax, np.float32)
    arrays = [dev(x) for x in (o, d, far)]
    out = torch.zeros(m, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    replay(own, captured(own, lambda: own.check(own.L.lrc_scene_occluded(      # (in a capture: the binary walk)
        s.h, *[C.c_void_p(x.data_ptr()) for x in arrays], m, tmin, C.c_void_p(out.data_ptr()), DEVICE))))
    blocked = out.cpu().numpy()
    for idx in (slice(0, m), slice(0, m, 32)):
        assert np.array_equal(s.occluded(o[idx], d[idx], far[idx], tmin), blocked[idx])
    s.close()


@pytest.mark.parametrize("tmin,tmax", [(0.0, 1e30), (0.0, np.inf), (0.0, np.nan), (-900.0, 900.0), (-900.0, -0.5)])
def test_odd_rays_in_a_world_with_primitives(own, tmin, tmax):
    """Spheres and quads, some twice, beside triangles: the wide nodes against the tree given as device arrays."""
    rng = np.random.default_rng(4)
    prims = np.zeros((40, 24), np.float32)
    prims[:, 0:3], prims[:, 3] = rng.random((40, 3)) * 555, 40.0
    for i in range(0, 40, 4):
        prims[i] = W.make_quad(rng.random(3) * 555, rng.random(3) * 200, -rng.random(3) * 200, 0)
    prims[20:] = prims[:20]
    scenes = []
    for _ in range(2):
        s = L.native.Scene(own)
        s.set_triangles(L.pack_tris(W.corners_to_quv(W.soup(500, 3) * np.float32(555))))
        s.set_prims(prims)
        s.build(1, 30)
        scenes.append(s)
    n = 540
    nodes, aux = np.zeros((2 * n - 1, 8), np.uint32), np.zeros(n, np.uint32)
    own.check(own.L.lrc_scene_tree(scenes[0].h, nodes.ctypes.data, aux.ctypes.data, 0))
    dn, da = dev(nodes.view(np.int32)), dev(aux.view(np.int32))
    own.check(own.L.lrc_scene_set_tree(scenes[1].h, C.c_void_p(dn.data_ptr()), 2 * n - 1, C.c_void_p(da.data_ptr()), n, DEVICE))
    o, d = odd_rays(40_000, 4)
    o = (o * np.float32(555)).astype(np.float32)
    for _ in range(4):                                   # (a few queries make the wide nodes)
        got, want = (s.intersect(o, d, tmin, tmax) for s in scenes)
    for g, w in zip(got, want):
        assert np.array_equal(g.view(np.uint32), w.view(np.uint32))
    for s in scenes:
        s.close()


@pytest.mark.parametrize("away", [1.0, 100.0, 1000.0, 30_000.0])
@pytest.mark.parametrize("slivers", [False, True])
def test_hits_that_the_binary_boxes_round_away(own, slivers, away):
    """Rays from far beyond the boxes' padding, and triangles whose t is mostly rounding: the wide boxes
    let more of them through, the answer is the binary walk's, closest hits and any."""
    n, m = 20_000, 1 << 18
    quv = W.corners_to_quv(W.soup(n, 3))
    if slivers:
        quv[:, 6:9] = quv[:, 3:6] * np.float32(1.0001) + quv[:, 6:9] * np.float32(1e-5)
    s = L.native.Scene(own)
    s.set_triangles(L.pack_tris(quv))
    s.build(1, 30)
    made(s)
    rng = np.random.default_rng(2)
    o = rng.normal(size=(m, 3))
    o = 0.5 + 2.0 * away * o / np.linalg.norm(o, axis=1, keepdims=True)
    at = rng.integers(0, n, m)
    d = quv[at, 0:3] + (quv[at, 3:6] + quv[at, 6:9]) * rng.random((m, 1)) * 0.5 - o
    o, d = o.astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    want = binary(own, s, o, d, 0.0, 1e30)
    far = np.full(m, 1e30, np.float32)
    for idx in (slice(0, m), slice(0, m, 32)):
        got = s.intersect(o[idx], d[idx])
        assert np.array_equal(got[0], want[0][idx]) and np.array_equal(got[1], want[1][idx])
        assert np.array_equal(s.occluded(o[idx], d[idx], far[idx]).astype(bool), want[0][idx] >= 0)
    s.close()


@pytest.mark.parametrize("ties", [1, 2])
def test_trees_as_deep_as_the_queries_stack(own, ties):
    """80 levels, each one's leaf behind all that lies below it; the nearest triangle twice (the binary
    walk decides between the two)."""
    depth = 80
    n = depth + ties
    quv = np.tile(np.float32([-1, -1, 0, 4, 0, 0, 0, 4, 0]), (n, 1))
    quv[:, 2] = 100.0 - np.minimum(np.arange(n), depth)
    corners = np.stack([quv[:, 0:3], quv[:, 0:3] + quv[:, 3:6], quv[:, 0:3] + quv[:, 6:9]])
    lo, hi = corners.min(0) - np.float32(1e-3), corners.max(0) + np.float32(1e-3)
    nodes = np.zeros((2 * n - 1, 8), np.uint32)
    f = nodes.view(np.float32)
    for i in range(n):                                   # node 2 i: over the triangles from i on; 2 i + 1: leaf i
        f[2 * i, 0:3], f[2 * i, 4:7] = lo[i:].min(0), hi[i:].max(0)
        if i < n - 1:
            nodes[2 * i][[3, 7]] = 2 * i + 1, 2 * i + 2
            f[2 * i + 1, 0:3], f[2 * i + 1, 4:7] = lo[i], hi[i]
        nodes[min(2 * i + 1, 2 * n - 2)][[3, 7]] = i, 0x80000001
    s = L.native.Scene(own)
    s.set_triangles(L.pack_tris(quv))
    s.set_tree(nodes, np.arange(n, dtype=np.uint32))
    made(s)
    m = 1 << 18
    o, d = np.zeros((m, 3), np.float32), np.tile(np.float32([0, 0, 1]), (m, 1))
    want = binary(own, s, o, d, 0.0, 1e30)
    assert want[1][0] == 100.0 - depth
    for k in (100, 40_000):
        got = s.intersect(o[:k], d[:k])
        assert np.array_equal(got[0], want[0][:k]) and np.array_equal(got[1], want[1][:k])
        assert s.occluded(o[:k], d[:k], np.full(k, 200, np.float32)).all()
    s.close()


def test_sizes_in_turn_replay_their_graphs(own):
    sc = W.box_scene(5, 1000, 72, 40)
    s = R.world_scene(own, sc, 1)
    p = L.native.trace_params(R.camera12(sc), 72, 40, 8, 1, 1, 0, 3)
    want = one_kernel(s, p, 1)
    img = torch.zeros(40, 72, 4, device="cuda")
    torch.cuda.synchronize()
    q = L.native.Batch(own)
    q.set_wavefront(1 << 14)                             # (the largest first: its buffer holds the others)
    q.add(s, p, 1, img.data_ptr())
    for k in range(3):
        for slots in (1 << 14, 1 << 12, 1 << 13, 1 << 11):
            for variant in (9, 11):
                q.set_wavefront(slots, variant)
                q.run(zero=True)
                own.sync()
                assert np.array_equal(img.cpu().numpy(), want)
                assert k == 0 or q.info()["graph_used"] == 1
    q.close()
    s.close()


def test_the_counting_kernel_counts_the_walk_that_is_walked(own):
    """Its images are the plain one's; with instances it counts the wide walk (fewer and larger nodes than
    the binary walk of the same field, which a mesh without a grid has it take), and the binary walk's
    tests where that is walked."""
    counts = []
    for wild in (None, np.nan):
        s, sc, _ = field(own, False, wild)
        p = L.native.trace_params(R.camera12(sc), 72, 40, 6, 1, 1, 0, 3)
        img, stats = wavefront(own, s, p, 5, stepped=True, count=True)
        plain, _ = wavefront(own, s, p, 5, stepped=True)
        assert np.array_equal(img, plain)
        counts.append(stats["box_tests"] / stats["intersect_rays"])
        s.close()
    assert 0 < counts[0] < 0.9 * counts[1]
    sc = W.box_scene(5, 1000, 72, 40)
    p = L.native.trace_params(R.camera12(sc), 72, 40, 6, 1, 1, 0, 3)
    n = sc["corners"].shape[0] + 1
    for given in (False, True):
        s = R.world_scene(own, sc, 1)
        if given:                                        # (device arrays: walked as they are)
            nodes, aux = np.zeros((2 * n - 1, 8), np.uint32), np.zeros(n, np.uint32)
            own.check(own.L.lrc_scene_tree(s.h, nodes.ctypes.data, aux.ctypes.data, 0))
            dn, da = dev(nodes.view(np.int32)), dev(aux.view(np.int32))
            own.check(own.L.lrc_scene_set_tree(s.h, C.c_void_p(dn.data_ptr()), 2 * n - 1, C.c_void_p(da.data_ptr()), n, DEVICE))
        img, stats = wavefront(own, s, p, 5, stepped=True, count=True)
        assert np.array_equal(img, one_kernel(s, p, 5)) and stats["box_tests"] > 0 and stats["tri_tests"] > 0
        s.close()


@pytest.mark.parametrize("wild", [None, np.nan, np.inf])
def test_walk_statistics_of_trees_that_no_grid_holds(own, wild):
    quv = W.corners_to_quv(W.soup(5000, 3))
    if wild is not None:
        quv[7, 0] = wild
    s = L.native.Scene(own)
    s.set_triangles(L.pack_tris(quv))
    s.build(0, 30)
    o, d = W.rays_at_cube(3000, 2)
    binary = s.trace_stats(o, d)
    s.set_walk(2)
    wide = s.trace_stats(o, d)
    assert wide == binary if wild is not None else 0 < wide[0] < binary[0]
    s.close()


def test_nodes_are_made_when_the_queries_are_worth_them(own):
    """A few rays after a build walk the binary nodes (no wide ones are made, 94 MB of a million shapes), as more
    calls come, or many rays, the wide ones: the same answers."""
    n = 1_000_000
    o, d = W.rays_at_cube(1 << 20, 2)
    s = L.native.Scene(own)
    s.set_triangles(soup(n, 3))
    s.set_prims(W.make_quad([0, 0, 0.5], [1, 0, 0], [0, 1, 0], 0))
    s.build(1, 30)
    want = s.intersect(o, d)                             # (makes them)
    s.close()
    s = L.native.Scene(own)
    s.set_triangles(soup(n, 3))
    s.set_prims(W.make_quad([0, 0, 0.5], [1, 0, 0], [0, 1, 0], 0))
    s.build(1, 30)
    s.intersect(o[:1], d[:1])
    free = torch.cuda.mem_get_info()[0]
    taken = []
    for k in range(30):
        got = s.intersect(o[:1000], d[:1000])
        assert np.array_equal(got[0], want[0][:1000]) and np.array_equal(got[1], want[1][:1000])
        taken.append(free - torch.cuda.mem_get_info()[0] > 48 * n)
    assert not taken[0] and taken[-1]
    s.close()
