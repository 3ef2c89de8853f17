"""The two-level walk over wide nodes (the wavefront's, of scenes with instances) where it could part from
the binary one that the one-kernel path tracer takes: the same images to the bit, with instances that
coincide (every hit a tie), that lie in the world's triangles, with meshes of a few triangles,
mirrored, and after the instances moved. And the wide nodes' first use inside a graph's capture or before
another stream's."""
import numpy as np
import pytest

import little_renderer_b200 as L
from little_renderer_b200 import render as R, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def own():
    return L.Context(0)


def scene(own, kind, builder):
    few = kind == "few"
    sc = W.instanced_field(seed=3, n_instances=1 if kind == "one" else 200, n_meshes=4, tri_range=(20, 30) if few else (200, 900),
                           width=72, height=40, sky_w=64, sky_h=32, spp=1, max_depth=6)
    if few:
        sc["meshes"] = [m[: 1 + i] for i, m in enumerate(sc["meshes"])]
    if kind == "twice":                              # every instance once more, of another material's mesh
        sc["xf"] = np.concatenate([sc["xf"], sc["xf"]])
        sc["meshes"] = sc["meshes"] + sc["meshes"]
        sc["mesh_mats"] = sc["mesh_mats"] + [(m + 1) % 4 for m in sc["mesh_mats"]]
        sc["mesh_of"] = np.concatenate([sc["mesh_of"], sc["mesh_of"] + 4])
    if kind == "flat":                               # in the ground's plane: the world's hit at the same t counts
        sc["xf"][::2, 1, :] = 0.0
        sc["xf"][::2, 1, 1] = 1e-3
        sc["meshes"] = [np.concatenate([m, np.float32([[[-3, 0, -3], [3, 0, -3], [0, 0, 3]]])]).astype(np.float32)
                        for m in sc["meshes"]]
        sc["xf"][::4, :, :3] = np.eye(3, dtype=np.float32)
    if kind == "mirrored":
        sc["xf"][:, :, 0] *= np.float32(-1.5)
    mask, tab = np.zeros(4096, np.uint16), np.zeros(2112, np.float32)
    L.lib().lrc_default_blue_noise(mask.ctypes.data)
    L.lib().lrc_default_bsdf_tables(tab.ctypes.data)
    s = R.instanced_scene(own, sc, builder, blue_noise=mask, bsdf_tables=tab)
    return sc, s


def wavefront(own, s, p, spp):
    img = torch.zeros(40, 72, 4, device="cuda")
    torch.cuda.synchronize()
    q = L.native.Batch(own)
    q.set_engine(1)
    q.set_wavefront(1024)
    q.add(s, p, spp, img.data_ptr())
    q.run()
    own.sync()
    q.close()
    return img.cpu().numpy()


@pytest.mark.parametrize("builder", [0, 1])
@pytest.mark.parametrize("kind", ["field", "one", "few", "twice", "flat", "mirrored"])
def test_images_are_the_binary_walks(own, kind, builder):
    sc, s = scene(own, kind, builder)
    for exact in (0, 1):
        p = L.native.trace_params(R.camera12(sc), 72, 40, 6, 1, 1, exact, 3)
        want, _ = s.trace(p, 5, flags=L.native.LRC_TRACE_MEGAKERNEL)
        assert np.array_equal(wavefront(own, s, p, 5), want)
    # moved (refitted, then rebuilt): the top level's wide nodes follow
    sc["xf"][:, :, 3] += np.random.default_rng(1).uniform(-2, 2, sc["xf"][:, :, 3].shape).astype(np.float32)
    for mode in (0, 1):
        s.move_instances(W.instance_records(sc), mode)
        want, _ = s.trace(p, 3, flags=L.native.LRC_TRACE_MEGAKERNEL)
        assert np.array_equal(wavefront(own, s, p, 3), want)
        sc["xf"][:, 0, 3] += np.float32(1)
    s.close()


def test_first_use_in_a_capture_and_on_another_stream(own):
    n, m = 20_000, 40_000
    quv = W.corners_to_quv(W.soup(n, 5))
    o, d = W.rays_at_cube(m, 2)
    s = L.native.Scene(own)
    s.set_triangles(L.pack_tris(quv))
    s.build(1, 30)
    want = s.intersect(o, d)
    ro, rd = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    prim, t = torch.zeros(m, dtype=torch.int32, device="cuda"), torch.zeros(m, device="cuda")
    torch.cuda.synchronize()
    side, other = torch.cuda.Stream(), torch.cuda.Stream()

    def query(stream):
        own.check(own.L.lrc_set_stream(own.h, stream.cuda_stream))
        s.intersect_device(ro.data_ptr(), rd.data_ptr(), m, prim.data_ptr(), t.data_ptr())

    def same():
        torch.cuda.synchronize()
        ok = np.array_equal(prim.cpu().numpy(), want[0]) and np.array_equal(t.cpu().numpy(), want[1])
        prim.zero_()
        torch.cuda.synchronize()
        return ok

    try:
        for used in (False, True):                   # the capture's is the first query after the build, or not
            s.build(1, 30)
            own.sync()
            if used:
                for _ in range(4):                   # (a few queries make the wide nodes)
                    query(other)
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                query(side)
            g.replay()
            assert same()
            query(other)
            query(side)
            assert same()
            g.replay()
            assert same()
            del g
    finally:
        own.check(own.L.lrc_set_stream(own.h, None))
    s.close()


@pytest.mark.parametrize("world", ["box", "field"])
@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("w,h,spp,depth", [(384, 256, 1, 4), (383, 256, 1, 4), (96, 96, 16, 8), (95, 96, 16, 8), (104, 96, 16, 8),
                                           (103, 96, 16, 8), (104, 96, 40, 8), (512, 289, 1, 12), (512, 288, 1, 12),
                                           (512, 384, 1, 12), (512, 383, 1, 12), (320, 256, 3, 8), (256, 256, 16, 3)])
def test_images_at_the_wavefronts_line(own, world, exact, w, h, spp, depth):
    """lrc_trace on both sides of where it takes the wavefront engine: the one-kernel path's image."""
    if world == "field":
        sc, s = scene(own, "few", 1)
    else:
        sc = W.box_scene(5, 1000, w, h)
        mask, tab = np.zeros(4096, np.uint16), np.zeros(2112, np.float32)
        L.lib().lrc_default_blue_noise(mask.ctypes.data)
        L.lib().lrc_default_bsdf_tables(tab.ctypes.data)
        s = R.world_scene(own, sc, 1, 30, mask, tab)
    p = L.native.trace_params(R.camera12(sc), w, h, depth, 1, 1, exact, 3)
    want, rays = s.trace(p, spp, flags=L.native.LRC_TRACE_MEGAKERNEL)
    got, r = s.trace(p, spp)
    assert np.array_equal(got, want) and r == rays
    s.close()
