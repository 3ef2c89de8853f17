"""What a user of the backend has it do, as cases that can be timed: tree builds (a frame's top
level, a mesh), ray queries (a pick, a whole soup built and queried), path-traced images from the
smallest preview to a 720p one, an instanced field under a sky, a medium, a viewer's frame, the
denoiser, light-traced caustics and a batch of scenes built and traced in one run. Sizes are those
of bench.py's workloads, of the tests and of the reference's published measurements, or smaller
ones of the same kind so that a pass stays below a second."""
import math

import numpy as np
import torch

from little_renderer_b200 import native, render, workloads as W

DEV = "cuda"


def listed():
    return [
        # the top level over a field's instances, made again every frame (the smallest call: launches)
        {"name": "toplevel_4988", "kind": "build", "shape": "instances", "n": 4988, "builder": 0, "key_bits": 30},
        # a mesh of the size of the reference's published build, at its better builder
        {"name": "mesh_871k_ploc", "kind": "build", "shape": "surface", "n": 871_414, "builder": 1, "key_bits": 30},
        # picking / baking: a few rays against a resident tree
        {"name": "pick_16k", "kind": "query", "tris": 20_480, "rays": 16_384, "builder": 1, "key_bits": 30, "rebuild": 0},
        # new triangles each pass: build, then closest hits and shadow rays through the tree
        {"name": "soup_4m", "kind": "query", "tris": 1 << 22, "rays": 1 << 22, "builder": 1, "key_bits": 30, "rebuild": 1},
        # a preview image: the smallest trace call
        {"name": "preview_128", "kind": "image", "scene": "box", "tris": 4_000, "w": 128, "h": 128, "spp": 1, "depth": 8,
         "exact": 0},
        # one pass of the engine's view (1 sample a pixel, 640 x 640, the plain render's 20k triangles)
        {"name": "view_640", "kind": "image", "scene": "box", "tris": 20_492, "w": 640, "h": 640, "spp": 1, "depth": 8,
         "exact": 0},
        # a final image of a larger scene
        {"name": "image_720p", "kind": "image", "scene": "box", "tris": 200_000, "w": 1280, "h": 720, "spp": 8, "depth": 8,
         "exact": 0},
        # instanced meshes under a sampled sky
        {"name": "field_sky", "kind": "image", "scene": "field", "tris": 2000, "w": 640, "h": 360, "spp": 8, "depth": 12,
         "exact": 0},
        # a cloud in the box (delta and ratio tracking)
        {"name": "cloud_256", "kind": "image", "scene": "foggy", "tris": 5_132, "w": 256, "h": 256, "spp": 4, "depth": 8,
         "exact": 0},
        # a viewer's next frame: guide, temporal gradients, reprojection, 1 sample a pixel, denoised
        {"name": "frame_720p", "kind": "frame", "tris": 20_492, "w": 1280, "h": 720},
        # the denoiser alone on a full-HD image
        {"name": "denoise_1080p", "kind": "denoise", "w": 1920, "h": 1080, "passes": 5, "samples": 2},
        # scenes of uneven size built (LBVH, then PLOC) and traced in one captured run
        {"name": "batch_8", "kind": "batch", "scenes": 8, "spp": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "query", "image", "image", "image", "image", "frame", "denoise", "caustics",
                       "batch"])
    if kind == "build":
        shape = rng.choice(["instances", "surface", "soup"])
        return {"kind": kind, "shape": shape, "n": _log(rng, 1_000, 1_500_000), "builder": rng.randrange(2),
                "key_bits": rng.choice([30, 30, 63])}
    if kind == "query":
        return {"kind": kind, "tris": _log(rng, 2_000, 2_000_000), "rays": _log(rng, 1_000, 2_000_000),
                "builder": rng.randrange(2), "key_bits": rng.choice([30, 63]), "rebuild": rng.randrange(2)}
    if kind == "image":
        scene = rng.choice(["box", "box", "box", "textured", "field", "foggy"])
        w = _log(rng, 100, 1280)
        h = max(64, int(w * rng.choice([1.0, 0.5625, 0.75])))
        most = {"box": 7_000_000, "textured": 4_000_000, "field": 1_500_000, "foggy": 260_000}[scene]
        spp = max(1, min(_log(rng, 1, 16), most // (w * h)))
        if w * h > most:
            w, h = w // 3 + 1, h // 3 + 1
        tris = _log(rng, 1_000, 200_000) if scene == "box" else _log(rng, 50, 2_000) if scene == "field" else 5_132
        return {"kind": kind, "scene": scene, "tris": tris, "w": w, "h": h, "spp": spp, "depth": rng.choice([4, 8, 12]),
                "exact": 1 if rng.random() < 0.15 else 0}
    if kind == "frame":
        w = _log(rng, 320, 1280)
        return {"kind": kind, "tris": _log(rng, 1_000, 100_000), "w": w, "h": int(w * 0.5625) | 1}
    if kind == "denoise":
        w = _log(rng, 200, 1920)
        return {"kind": kind, "w": w, "h": int(w * rng.choice([0.5625, 1.0]) * 0.99), "passes": rng.randrange(3, 6),
                "samples": rng.choice([1, 2, 4, 16])}
    if kind == "caustics":
        return {"kind": kind, "photons": _log(rng, 20_000, 1_000_000), "w": rng.choice([256, 401, 640]), "exact": 0}
    return {"kind": "batch", "scenes": rng.randrange(2, 9), "spp": rng.choice([1, 4, 8])}


# ---- the context and the constants a program keeps ------------------------------------------------
_kept = {}


def _ctx():
    """One context on one stream for the whole program; its work goes to a torch stream, so that
    tensors made here and the library's kernels are ordered."""
    if "ctx" not in _kept:
        st = torch.cuda.Stream()
        ctx = native.Context(0)
        ctx.set_stream(st.cuda_stream)
        mask, tab = np.zeros(4096, np.uint16), np.zeros(2112, np.float32)
        ctx.L.lrc_default_blue_noise(mask.ctypes.data)
        ctx.L.lrc_default_bsdf_tables(tab.ctypes.data)
        _kept.update(ctx=ctx, stream=st, tables=(mask, tab))
    return _kept["ctx"], _kept["stream"]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


# ---- inputs ----------------------------------------------------------------------------------------
def _soup(n, seed, gen):
    """(n, 9) q, u, v: workloads.soup's distribution, made on the device."""
    cen = torch.rand(n, 3, generator=gen, device=DEV, dtype=torch.float64)
    sigma = 0.002 * n ** (-1.0 / 3.0)
    e = torch.randn(n, 2, 3, generator=gen, device=DEV, dtype=torch.float64) * sigma
    big = torch.rand(n, generator=gen, device=DEV) < 0.02
    e[big] *= 50.0
    a = cen - (e[:, 0] + e[:, 1]) / 3.0
    c = torch.stack([a, a + e[:, 0], a + e[:, 1]], 1).float()
    return torch.cat([c[:, 0], c[:, 1] - c[:, 0], c[:, 2] - c[:, 0]], 1).contiguous()


def _surface(n, gen):
    """(n, 9) q, u, v of small triangles over a bumpy sphere (a scanned mesh's distribution)."""
    d = torch.randn(n, 3, generator=gen, device=DEV, dtype=torch.float64)
    d /= d.norm(dim=1, keepdim=True)
    r = 1.0 + 0.15 * torch.sin(7 * d[:, :1]) * torch.cos(5 * d[:, 1:2]) + 0.05 * torch.sin(31 * d[:, 2:3])
    edge = 2.0 * n ** -0.5
    e = torch.randn(n, 2, 3, generator=gen, device=DEV, dtype=torch.float64) * edge
    e -= (e * d[:, None]).sum(-1, keepdim=True) * d[:, None]
    return torch.cat([d * r, e[:, 0], e[:, 1]], 1).float().contiguous()


def _pack(quv):
    """(n, 12) words of the device's triangle layout (native.pack_tris) on the device."""
    n = quv.shape[0]
    out = torch.zeros(n, 12, device=DEV)
    out[:, 0:3], out[:, 4:7], out[:, 8:11] = quv[:, 0:3], quv[:, 3:6], quv[:, 6:9]
    words = out.view(torch.int32)
    words[:, 3] = -1
    return out


def _boxes(case, gen):
    n = case["n"]
    out = torch.zeros(n, 8, device=DEV)
    if case["shape"] == "instances":
        c = torch.rand(n, 3, generator=gen, device=DEV) * torch.tensor([40.0, 3.0, 40.0], device=DEV)
        h = torch.rand(n, 3, generator=gen, device=DEV) * 0.7 + 0.3
        out[:, 0:3], out[:, 4:7] = c - h, c + h
        return out
    quv = _surface(n, gen) if case["shape"] == "surface" else _soup(n, 0, gen)
    q = quv[:, 0:3]
    p = torch.stack([q, q + quv[:, 3:6], q + quv[:, 6:9]], 1)
    out[:, 0:3], out[:, 4:7] = p.amin(1) - 1e-3, p.amax(1) + 1e-3
    return out


def _rays(n, quv, gen):
    """Origins on a sphere of radius 2 about the cube's middle; half the rays go to a triangle's
    middle, half to a point of the cube."""
    o = torch.randn(n, 3, generator=gen, device=DEV, dtype=torch.float64)
    o = 0.5 + 2.0 * o / o.norm(dim=1, keepdim=True)
    to = torch.rand(n, 3, generator=gen, device=DEV, dtype=torch.float64)
    k = n // 2
    at = quv[torch.randint(0, quv.shape[0], (k,), generator=gen, device=DEV)].double()
    to[:k] = at[:, 0:3] + (at[:, 3:6] + at[:, 6:9]) / 3.0
    o = o.float()
    d = to - o.double()
    return o.contiguous(), (d / d.norm(dim=1, keepdim=True)).float().contiguous()


def _scene(case, seed):
    """(the scene's dict, the scene on the device with its tree built)."""
    ctx, _ = _ctx()
    mask, tab = _kept["tables"]
    kind, seed = case.get("scene", "box"), int(seed) & 0xFFFFFF
    w, h = case.get("w", 256), case.get("h", case.get("w", 256))
    if kind == "field":
        sc = W.instanced_field(seed, n_instances=case["tris"], n_meshes=6, tri_range=(2_000, 20_000), width=w, height=h,
                               sky_w=512, sky_h=256)
        return sc, render.instanced_scene(ctx, sc, 1, 30, mask, tab)
    if kind == "foggy":
        sc = W.foggy_cornell(seed, w, h)
    elif kind == "textured":
        sc = W.textured_cornell(seed, w, h)
    else:
        sc = W.box_scene(seed, case["tris"], w, h)
    return sc, render.world_scene(ctx, sc, 1, 30, mask, tab)


def _params(sc, case, seed, move=0.0):
    cam = dict(sc["camera"])
    cam["from"] = (cam["from"][0] + move, cam["from"][1], cam["from"][2])
    return native.trace_params(W.camera(cam, sc["width"] / sc["height"]), sc["width"], sc["height"],
                               case.get("depth", 8), 1, 1, case.get("exact", 0), int(seed) & 0xFFFF)


def prepare(case, seed):
    ctx, stream = _ctx()
    gen = _gen(seed)
    torch.cuda.current_stream().synchronize()
    with torch.cuda.stream(stream):
        st = {"case": case, "ctx": ctx, "stream": stream}
        kind = case["kind"]
        if kind == "build":
            n = case["n"]
            st["boxes"] = _boxes(case, gen)
            lo, hi = st["boxes"][:, 0:3].amin(0), st["boxes"][:, 4:7].amax(0)
            st["params"] = ctx.params(n, lo.cpu().numpy(), hi.cpu().numpy(), case["key_bits"], case["builder"])
            st["nodes"] = torch.zeros(2 * n - 1, 8, device=DEV, dtype=torch.int32)
            st["aux"] = torch.zeros(n, device=DEV, dtype=torch.int32)
        elif kind == "query":
            n = case["rays"]
            quv = _soup(case["tris"], seed, gen)
            st["tris"] = _pack(quv)
            st["o"], st["d"] = _rays(n, quv, gen)
            st["tmax"] = torch.rand(n, generator=gen, device=DEV) * 2.0 + 1.0
            st["scene"] = s = native.Scene(ctx)
            s.set_triangles(None, st["tris"].data_ptr(), case["tris"])
            s.build(case["builder"], case["key_bits"])
            st["prim"] = torch.zeros(n, device=DEV, dtype=torch.int32)
            st["t"] = torch.zeros(n, device=DEV)
            st["hit"] = torch.zeros(n, device=DEV, dtype=torch.uint8)
        elif kind == "image":
            sc, st["scene"] = _scene(case, seed)
            st["params"] = _params(sc, case, seed)
            st["image"] = torch.zeros(case["h"], case["w"], 4, device=DEV)
        elif kind == "frame":
            sc, st["scene"] = _scene(case, seed)
            st["old"], st["new"] = _params(sc, case, seed), _params(sc, case, seed, 2.0)
            st["before"] = torch.zeros(4, case["h"], case["w"], 4, device=DEV)
            st["after"] = torch.zeros_like(st["before"])
            st["image"] = torch.zeros(case["h"], case["w"], 4, device=DEV)
            st["scene"].trace_frame_device(None, st["old"], 0, 4, 0, st["before"].data_ptr(), 32, 8)
        elif kind == "denoise":
            st["planes"] = _planes(case, gen)
            st["image"] = torch.zeros(case["h"], case["w"], 4, device=DEV)
        elif kind == "caustics":
            sc, st["scene"] = _scene({"scene": "box", "tris": 20_492, "w": case["w"]}, seed)
            st["params"] = _params(sc, case, seed)
            st["image"] = torch.zeros(case["w"], case["w"], 3, device=DEV)
        else:
            st["batch"] = b = native.Batch(ctx)
            st["scenes"], st["images"] = [], []
            for i, (tris, res) in enumerate(_batch(case)):
                sc, s = _scene({"scene": "box", "tris": tris, "w": res}, int(seed) * 64 + i)
                st["scenes"].append(s)
                st["images"].append(torch.zeros(res, res, 4, device=DEV))
                b.add(s, _params(sc, case, seed), case["spp"], st["images"][-1].data_ptr(), builder=2)
        stream.synchronize()
    return st


def _batch(case):
    """(triangles, resolution) of a batch's scenes: uneven, from 1k triangles to 130k."""
    return [(int(1_000 * 2 ** i), (128, 256, 200)[i % 3]) for i in range(case["scenes"])]


def _planes(case, gen):
    """The denoiser's planes of a made-up image: smooth surfaces with edges, a patch of lamp, noisy
    samples with their moments."""
    w, h, k = case["w"], case["h"], case["samples"]
    y, x = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float64), torch.arange(w, device=DEV, dtype=torch.float64),
                          indexing="ij")
    ph = torch.rand(4, generator=gen, device=DEV, dtype=torch.float64) * 6.28
    region = torch.floor(3 * torch.sin(x * 9.0 / w + ph[0]) + 2 * torch.cos(y * 7.0 / h + ph[1]))
    ang = region * 1.3 + 0.3 * torch.sin(x * 4.0 / w + ph[2])
    nrm = torch.stack([torch.cos(ang) * 0.8, torch.sin(ang) * 0.8, torch.full_like(ang, 0.6)], -1)
    dist = 600.0 + 80.0 * region + 50.0 * y / h + 30.0 * x / w
    alb = torch.stack([0.3 + 0.1 * torch.remainder(region, 5), 0.6 + 0.05 * torch.remainder(region, 3), 0.5 + 0 * region], -1)
    kind = torch.zeros(h, w, device=DEV, dtype=torch.float64)
    kind[h // 8:h // 6, w // 3:w // 2] = 1.0
    light = 0.6 + 0.4 * torch.sin(x * 5.0 / w + y * 3.0 / h + ph[3])
    planes = torch.zeros(4, h, w, 4, device=DEV)
    s, m = torch.zeros(h, w, 3, device=DEV, dtype=torch.float64), torch.zeros(h, w, 2, device=DEV, dtype=torch.float64)
    luma = torch.tensor([0.2126, 0.7152, 0.0722], device=DEV, dtype=torch.float64)
    for _ in range(k):
        g = -torch.log(torch.rand(h, w, generator=gen, device=DEV, dtype=torch.float64).clamp_min(1e-6))
        irr = (light * g)[..., None].expand(-1, -1, 3)
        s += irr * torch.where(kind[..., None] == 0, alb, torch.ones_like(alb))
        l = (irr * luma).sum(-1)
        m += torch.stack([l, l * l], -1)
    planes[0, ..., :3], planes[0, ..., 3] = s, k
    planes[1, ..., :2] = m
    planes[2, ..., :3], planes[2, ..., 3] = nrm, dist
    planes[3, ..., :3], planes[3, ..., 3] = alb, kind
    return planes


# ---- one pass -----------------------------------------------------------------------------------
def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    with torch.cuda.stream(st["stream"]):
        if kind == "build":
            ctx.build_device(st["params"], st["boxes"].data_ptr(), st["nodes"].data_ptr(), st["aux"].data_ptr())
            return {"nodes": st["nodes"], "aux": st["aux"]}
        if kind == "query":
            s, n = st["scene"], case["rays"]
            if case["rebuild"]:
                s.set_triangles(None, st["tris"].data_ptr(), case["tris"])
                s.build(case["builder"], case["key_bits"])
            s.intersect_device(st["o"].data_ptr(), st["d"].data_ptr(), n, st["prim"].data_ptr(), st["t"].data_ptr())
            ctx.check(ctx.L.lrc_scene_occluded(s.h, st["o"].data_ptr(), st["d"].data_ptr(), st["tmax"].data_ptr(), n, 0.0,
                                               st["hit"].data_ptr(), native.LRC_DEVICE))
            return {"prim": st["prim"], "t": st["t"], "blocked": st["hit"]}
        if kind == "image":
            st["image"].zero_()
            st["scene"].trace_device(st["params"], case["spp"], st["image"].data_ptr())
            return {"image": st["image"]}
        if kind == "frame":
            st["scene"].trace_frame_device(st["old"], st["new"], 4, 1, st["before"].data_ptr(), st["after"].data_ptr(), 32, 8)
            ctx.denoise_device(case["w"], case["h"], st["after"].data_ptr(), st["image"].data_ptr())
            return {"planes": st["after"], "image": st["image"]}
        if kind == "denoise":
            ctx.denoise_device(case["w"], case["h"], st["planes"].data_ptr(), st["image"].data_ptr(), case["passes"])
            return {"image": st["image"]}
        if kind == "caustics":
            st["image"].zero_()
            st["scene"].caustics_device(st["params"], case["photons"], 9, st["image"].data_ptr())
            return {"image": st["image"]}
        st["batch"].run(build=True, graph=True, zero=True)
        return {"images": st["images"]}


# ---- what a pass cannot do without ------------------------------------------------------------------
def _ray_flops(tris):
    """A closest or shadow ray: about two boxes a level of a balanced tree (18 operations each), a
    few triangles (50 each) and its share of the shading."""
    return 2 * 18 * math.log2(max(tris, 2)) + 4 * 50 + 300


def work(case):
    kind = case["kind"]
    if kind == "build":
        n, k, passes = case["n"], 4 if case["key_bits"] == 30 else 8, 4 if case["key_bits"] == 30 else 8
        return {"bytes": n * (32 + 64 + 4) + n * (k + passes * 2 * (k + 4)), "flops": n * (100 if case["builder"] == 0 else 1500)}
    if kind == "query":
        n, t = case["rays"], case["tris"]
        build = t * (48 + 48 + 32 + 68 + 64 + 4 + 64) if case["rebuild"] else t * (48 + 64)
        # a ray through a cube of n triangles passes about n^(1/3) leaf cells
        return {"bytes": build + n * (2 * 12 * 2 + 4 + 4 + 4 + 1), "flops": 2 * n * 18 * 4 * t ** (1 / 3)}
    if kind == "image":
        paths = case["w"] * case["h"] * case["spp"]
        tris = case["tris"] * (10_000 if case["scene"] == "field" else 1)
        return {"bytes": case["w"] * case["h"] * 32 + min(tris, 200_000) * 112, "flops": paths * 5 * _ray_flops(tris)}
    if kind == "frame":
        px = case["w"] * case["h"]
        return {"bytes": px * (64 * 2 + 16) + case["tris"] * 112, "flops": px * (7 * _ray_flops(case["tris"]) + 5 * 25 * 40)}
    if kind == "denoise":
        px = case["w"] * case["h"]
        return {"bytes": px * (64 + 16), "flops": px * case["passes"] * 25 * 40}
    if kind == "caustics":
        return {"bytes": case["w"] ** 2 * 24 + 20_492 * 112, "flops": case["photons"] * 3 * _ray_flops(20_492)}
    px = sum(r * r for _, r in _batch(case))
    tris = sum(t for t, _ in _batch(case))
    return {"bytes": px * 32 + 2 * tris * 270, "flops": px * case["spp"] * 5 * _ray_flops(20_000) + tris * 1600}


def tolerance(case):
    kind = case["kind"]
    if kind == "build":
        return "exact"                                  # the reference's tree, node for node
    if kind == "query":
        return {"rel": 1e-6, "max": 1e-5, "differ": 1e-5}   # t rounded as the C code rounds it; ties in t aside
    if kind == "denoise":
        # halves between the passes: a sum in another order turns a few of them to the next one
        return {"rel": 5e-5, "max": 4e-3}
    # paths: against the C code (another libm) the images' relRMSE is 3e-6 to 2e-5
    return {"rel": 1e-4, "max": 2e-2}


# ---- the same in 64 bits ------------------------------------------------------------------------------
def exact(case, seed):
    """The queries' t by testing every triangle (not of larger soups, whose triangles are so small that
    a ray aimed at one in 32 bits passes by it), the denoiser with its arithmetic in 64 bits. Trees
    are whole numbers; a random walk has no 64-bit value (one sample that goes another way is
    another image)."""
    if case["kind"] == "query":
        if case["tris"] > 100_000 or case["tris"] * case["rays"] > 3e9:
            return None
        return _exact_query(case, seed)
    if case["kind"] == "denoise":
        return {"image": _exact_denoise(_planes(case, _gen(seed)).double(), case["passes"])}
    return None


def _exact_query(case, seed):
    gen = _gen(seed)
    quv = _soup(case["tris"], seed, gen)
    o, d = _rays(case["rays"], quv, gen)
    quv, o, d = quv.double(), o.double(), d.double()
    q, u, v = quv[:, 0:3], quv[:, 3:6], quv[:, 6:9]
    best = torch.full((case["rays"],), math.inf, device=DEV, dtype=torch.float64)
    step = max(1, 30_000_000 // case["rays"])

    def cross(a, b):
        return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    dd, oo = [d[:, k, None] for k in range(3)], [o[:, k, None] for k in range(3)]
    for i in range(0, case["tris"], step):
        qq, uu, vv = ([x[None, i:i + step, k] for k in range(3)] for x in (q, u, v))
        pv = cross(dd, vv)
        det = dot(uu, pv)
        tv = [oo[k] - qq[k] for k in range(3)]
        b1 = dot(tv, pv) / det
        qv = cross(tv, uu)
        b2 = dot(dd, qv) / det
        t = dot(vv, qv) / det
        ok = (det.abs() >= 1e-12) & (b1 >= 0) & (b1 <= 1) & (b2 >= 0) & (b1 + b2 <= 1) & (t > 0)
        best = torch.minimum(best, torch.where(ok, t, torch.full_like(t, math.inf)).amin(1))
    return {"prim": None, "t": torch.where(best.isinf(), torch.full_like(best, -1.0), best), "blocked": None}


def _hash32(x):
    """lowbias32 on int64 tensors holding 32-bit values."""
    x = x ^ (x >> 16)
    x = (x * 0x7FEB352D) & 0xFFFFFFFF
    x = x ^ (x >> 15)
    x = (x * 0x846CA68B) & 0xFFFFFFFF
    return x ^ (x >> 16)


def _half(x):
    return x.half().double()


def _exact_denoise(px, passes):
    """The a-trous filter of the path tracer's planes (h x w x 4 each): the image packed as halves
    between passes, as the format has it; everything else in 64 bits."""
    h, w = px.shape[1:3]
    a, mom, n, g = px[0], px[1], px[2], px[3]
    luma = torch.tensor([0.2126, 0.7152, 0.0722], device=DEV, dtype=torch.float64)
    kind = g[..., 3] - 4 * torch.floor(g[..., 3] / 4)
    surface = kind == 0
    # the normals through their octahedral 16-bit code
    e = n[..., :2] / n[..., :3].abs().sum(-1, keepdim=True).clamp_min(1e-6)
    sgn = torch.where(e >= 0, 1.0, -1.0)
    e = torch.where((n[..., 2] < 0)[..., None], (1 - e.flip(-1).abs()) * sgn, e)
    e = torch.round(e.float().clamp(-1, 1) * 32767).double() / 32767
    z = 1 - e.abs().sum(-1)
    t = (-z).clamp_min(0)[..., None]
    e = e + torch.where(e >= 0, -t, t)
    nrm = torch.cat([e, z[..., None]], -1)
    nrm = nrm / nrm.norm(dim=-1, keepdim=True)
    dist = n[..., 3]
    irr = a[..., :3] / a[..., 3:].clamp_min(1)
    irr = torch.where(surface[..., None], irr / g[..., :3].clamp_min(1e-3), irr)
    lum = (irr * luma).sum(-1)
    ys, xs = torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing="ij")

    def at(qy, qx):
        ok = (qy >= 0) & (qx >= 0) & (qy < h) & (qx < w)
        return ok, qy.clamp(0, h - 1) * w + qx.clamp(0, w - 1)

    def get(x, i):
        return x.reshape(h * w, *x.shape[2:])[i]

    c = a[..., 3].clamp_min(1)
    var = (mom[..., 1] / c - (mom[..., 0] / c) ** 2).clamp_min(0) / c
    s1, s2, cn = (torch.zeros(h, w, device=DEV, dtype=torch.float64) for _ in range(3))
    for dy in range(-3, 4):
        for dx in range(-3, 4):
            ok, i = at(ys + dy, xs + dx)
            ok &= (get(a, i)[..., 3] != 0) & (get(kind, i) == kind)
            ok &= ~(surface & ((get(n, i)[..., :3] * n[..., :3]).sum(-1) < 0.9))
            l = torch.where(ok, get(lum, i), 0.0)
            s1, s2, cn = s1 + l, s2 + l * l, cn + ok
    near = (s2 / cn - (s1 / cn) ** 2).clamp_min(0)
    var = torch.where(a[..., 3] >= 4, var, near)
    var = torch.where(kind == 1, 0.0, var)
    img = torch.cat([_half(irr.clamp_max(6e4)), _half(var.clamp(-1, 6e4))[..., None]], -1)
    img[a[..., 3] == 0] = torch.tensor([0.0, 0.0, 0.0, -1.0], device=DEV, dtype=torch.float64)
    b3 = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
    k = ys * w + xs
    for p in range(passes):
        step, last = 1 << p, p == passes - 1
        keep = (img[..., 3] < 0) | (kind == 1)
        v, vw = (torch.zeros(h, w, device=DEV, dtype=torch.float64) for _ in range(2))
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                s = get(img, at(ys + dy, xs + dx)[1])[..., 3]
                wt = (0.25 if dx else 0.5) * (0.25 if dy else 0.5)
                v, vw = v + torch.where(s < 0, 0.0, wt * s), vw + torch.where(s < 0, 0.0, wt)
        v = v / vw.clamp_min(1e-6)
        lp = (img[..., :3] * luma).sum(-1)

        def side(dy, dx):
            return (dist - get(dist, at(ys + dy, xs + dx)[1])).abs()

        gx, gy = torch.minimum(side(0, -1), side(0, 1)), torch.minimum(side(-1, 0), side(1, 0))
        seed = _hash32(((k * 0x9E3779B9) & 0xFFFFFFFF) ^ ((step * 0x85EBCA6B) & 0xFFFFFFFF))
        jit = step // 2
        acc = torch.zeros(h, w, 5, device=DEV, dtype=torch.float64)
        for j in range(5):
            for i in range(5):
                ox, oy = torch.full_like(xs, (i - 2) * step), torch.full_like(xs, (j - 2) * step)
                if jit and (i != 2 or j != 2):
                    seed = _hash32(seed)
                    ox = ox + (((seed & 0xFFFF) * (2 * jit + 1)) >> 16) - jit
                    oy = oy + (((seed >> 16) * (2 * jit + 1)) >> 16) - jit
                ok, q = at(ys + oy, xs + ox)
                s, gq = get(img, q), get(kind, q)
                centre = q == k
                ok &= centre | ((s[..., 3] >= 0) & (gq == kind))
                wl = torch.exp(-(lp - (s[..., :3] * luma).sum(-1)).abs() / (4.0 * torch.maximum(v, s[..., 3]).clamp_min(0).sqrt() + 1e-6))
                wn = (get(nrm, q) * nrm).sum(-1).clamp_min(0) ** 128
                wz = torch.exp(-(dist - get(dist, q)).abs() / (gx * ox.abs() + gy * oy.abs() + 1e-3 * dist + 1e-6))
                wt = torch.where(centre, 1.0, wl * torch.where(surface, wn * wz, 1.0)) * b3[i] * b3[j]
                wt = torch.where(ok, wt, 0.0)
                acc += torch.cat([wt[..., None] * s[..., :3], (wt * wt * s[..., 3])[..., None], wt[..., None]], -1)
        out = acc[..., :3] / acc[..., 4:]
        if last:
            res = torch.ones(h, w, 4, device=DEV, dtype=torch.float64)
            res[..., :3] = torch.where(surface[..., None], out * g[..., :3], out)
            res[..., :3] = torch.where(keep[..., None], img[..., :3], res[..., :3])
            res[img[..., 3] < 0] = 0.0
            return res
        nxt = torch.cat([_half(out.clamp_max(6e4)), _half((acc[..., 3] / acc[..., 4] ** 2).clamp(-1, 6e4))[..., None]], -1)
        img = torch.where(keep[..., None], img, nxt)
