// pathtrace.cu - the path tracer on sm_100a: the light transport of the reference's
// trace_path_sampled (engine/rt/tracer.c:364-545) and trace_image (:329-356), which its WGSL
// megakernel `main`/`trace()` restate (engine/gpu/shaders/trace/trace.wgsl:1125-1316).
//
// Per bounce: the closest hit through the world's BVH (shape ids: primitives, then triangles, as
// scene_intersect numbers them, engine/rt/accel.c:252), the hit (engine/rt/intersect.c set_hit,
// finish_*), the lamp counted by its emit mode (FULL / NONE / MIS), next event estimation of the
// lamp quad with a shadow ray to dist - RT_SHADOW_MARGIN (sample_direct_light, tracer.c:56) and
// the power heuristic, the BSDF's lobe pick and sample (bsdf.cuh), Russian roulette after 3
// bounces. Float build constants: RT_EPS 2e-3, RT_SHADOW_MARGIN 2e-2 (tracer.c:14-23).
//
// Two launch modes:
//   exact: one thread per pixel, its samples in order from the CPU's per-pixel PCG32 stream and
//          sampler (trace_image's seeding): the image is the CPU's up to transcendental rounding
//          (the parity mode);
//   fast:  one thread per (pixel, sample), each sample its own PCG32 stream (seeded from pixel,
//          sample and image seed) and the same Owen-Sobol dimensions; a pixel's samples sit in
//          neighbouring lanes and are summed by warp shuffles in a fixed order (deterministic).

#include "pt_device.cuh"
#include <algorithm>

namespace lrc {
namespace pt {

// Every lane on its own way, through the binary nodes: scenes with media (their shadow rays are traced in
// place, path_shade), scenes without wide nodes and calls of more paths than PT_WARP_PATHS (below).
// exact mode: one thread per pixel of rows [y0, y0 + rows), samples [0, spp) in order from the
// CPU's per-pixel stream (trace_image, tracer.c:337-353)
template <bool MEDIA, bool GUIDED>
__global__ void __launch_bounds__(128) exact_kernel(PtScene S, PtParams P, float4 *accum, unsigned long long *ray_count,
                                                    uint32_t *err) {
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t x = idx % P.W, yy = idx / P.W;
    uint32_t rays = 0;
    if (yy < (uint32_t)P.rows) {
        const uint32_t y = P.y0 + yy;
        const uint64_t pixel = (uint64_t)y * P.W + x;
        Rng rng;
        rng_seed(rng, 0x853c49e6748fea9bull ^ (pixel * 0x9E3779B97F4A7C15ull) ^ (P.seed * 0xD1B54A32D192ED03ull), pixel);
        V3 sum = v3(0, 0, 0);
        float ml = 0.0f, ml2 = 0.0f, l_last = 0.0f;
        for (int k = 0; k < P.spp; k++) {
            Sampler sm{&rng, (uint32_t)k, (uint32_t)P.seed * 0x9e3779b9u, (int)x, (int)y, P.sampler_on, S.mask};
            float jx, jy;
            sampler_2d(sm, 0, jx, jy);
            float u = dvd(add((float)x, jx), (float)P.W), v = dvd(add((float)y, jy), (float)P.H);
            V3 o, d;
            camera_ray(P, u, v, o, d);
            V3 c = trace_path<MEDIA>(S, P, o, d, sm, err, rays);
            if (!is_number(c)) {
                if (GUIDED) l_last = 0.0f;           // (a dropped sample counts as black)
                continue;
            }
            c = clamp_sample(c, P.clamp);
            sum = vadd(sum, c);
            if (GUIDED) {
                const float l = sample_luma(c, P.guide[pixel]);
                ml += l;
                ml2 += l * l;
                l_last = l;
            }
        }
        float4 a = accum[pixel];
        accum[pixel] = make_float4(a.x + sum.x, a.y + sum.y, a.z + sum.z, a.w + (float)P.spp);
        if (GUIDED) {                                // (z, w: the last sample's luminance and number + 1)
            const float4 m = P.moments[pixel];
            P.moments[pixel] = make_float4(m.x + ml, m.y + ml2, l_last, last_sample_tag(P));
        }
    }
    if (ray_count) {
        unsigned long long r = rays;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if ((threadIdx.x & 31) == 0 && r) atomicAdd(ray_count, r);
    }
}

// fast mode: P.group lanes (a power of 2 dividing 32) per pixel, lane s tracing samples s, s + g,
// s + 2g, ... of [spp0, spp0 + spp), each from its own PCG32 stream; the group's sums are then added
// in a fixed order (deterministic)
template <bool MEDIA, bool GUIDED>
__global__ void __launch_bounds__(128) fast_kernel(PtScene S, PtParams P, float4 *accum, unsigned long long *ray_count,
                                                   uint32_t *err) {
    const uint32_t g = P.group;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t pix_local = tid / g;
    const uint32_t lane_s = (uint32_t)(tid % g);
    const uint64_t npix = (uint64_t)P.W * P.rows;
    uint32_t rays = 0;
    V3 c = v3(0, 0, 0);
    float cnt = 0.0f, ml = 0.0f, ml2 = 0.0f, l_last = 0.0f;
    const bool live = pix_local < npix;
    uint64_t pixel = 0;
    if (live) {
        const uint32_t x = (uint32_t)(pix_local % P.W), y = P.y0 + (uint32_t)(pix_local / P.W);
        pixel = (uint64_t)y * P.W + x;
        for (uint32_t k = lane_s; k < (uint32_t)P.spp; k += g) {
            const uint32_t kk = P.spp0 + k;
            Rng rng;
            rng_seed(rng, mix64(pixel * 0x9E3779B97F4A7C15ull ^ ((uint64_t)kk << 40) ^ P.seed), pixel);
            Sampler sm{&rng, kk, (uint32_t)P.seed * 0x9e3779b9u, (int)x, (int)y, P.sampler_on, S.mask};
            float jx, jy;
            sampler_2d(sm, 0, jx, jy);
            float u = dvd(add((float)x, jx), (float)P.W), v = dvd(add((float)y, jy), (float)P.H);
            V3 o, d;
            camera_ray(P, u, v, o, d);
            V3 s = trace_path<MEDIA>(S, P, o, d, sm, err, rays);
            s = is_number(s) ? clamp_sample(s, P.clamp) : v3(0, 0, 0);
            c = vadd(c, s);
            cnt += 1.0f;
            if (GUIDED) {
                const float l = sample_luma(s, P.guide[pixel]);
                ml += l;
                ml2 += l * l;
                l_last = l;
            }
        }
    }
    // (the pixel's last sample, spp0 + spp - 1, is lane (spp - 1) % g's last)
    if (GUIDED) l_last = __shfl_sync(0xffffffffu, l_last, (uint32_t)(P.spp - 1) % g, g);
    for (uint32_t o = 1; o < g; o <<= 1) {               // fixed-order tree sum over the group
        c.x += __shfl_down_sync(0xffffffffu, c.x, o, g);
        c.y += __shfl_down_sync(0xffffffffu, c.y, o, g);
        c.z += __shfl_down_sync(0xffffffffu, c.z, o, g);
        cnt += __shfl_down_sync(0xffffffffu, cnt, o, g);
        if (GUIDED) {
            ml += __shfl_down_sync(0xffffffffu, ml, o, g);
            ml2 += __shfl_down_sync(0xffffffffu, ml2, o, g);
        }
    }
    if (live && lane_s == 0) {
        float4 a = accum[pixel];
        accum[pixel] = make_float4(a.x + c.x, a.y + c.y, a.z + c.z, a.w + cnt);
        if (GUIDED) {                                // (z, w: the last sample's luminance and number + 1)
            const float4 m = P.moments[pixel];
            P.moments[pixel] = make_float4(m.x + ml, m.y + ml2, l_last, last_sample_tag(P));
        }
    }
    if (ray_count) {
        unsigned long long r = rays;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if ((threadIdx.x & 31) == 0 && r) atomicAdd(ray_count, r);
    }
}

// The same through the wide nodes, in calls of at most PT_WARP_PATHS paths on scenes without media: the
// lanes of a warp meet before every walk (warp_bounce), and a lane whose path ends starts its next sample
// there. With few warps an SM the length of the walks decides, which the wide nodes cut to a third;
// with more, the instructions: 128 x 128 pixels at 1 spp of 4k / 20k / 200k triangles 0.55 / 0.83 / 1.21 ms
// by lanes on their own, 0.47 / 0.75 / 0.80 by warps; 256 x 256: 0.83 / 1.13 / 1.36, 0.97 / 1.34 / 1.26.
// spread: only every spread-th lane has a path, in calls of so few paths that most of the chip's warps
// are idle (64 x 64 pixels of 20k triangles: 0.66 -> 0.5 ms; beyond SPREAD_LANES lanes the warps take the
// instruction cache from one another: 128 x 128 with 4 lanes a path 0.67 ms, with one 0.47).
constexpr uint64_t PT_WARP_PATHS = 24u << 10;
constexpr uint64_t SPREAD_LANES = 1u << 14;
constexpr uint32_t SPREAD_MOST = 8;
struct PathLane {
    uint64_t index;                                  // the lane's path among all (pixels x group)
    bool has;                                        // this lane is one of those with a path
};
__device__ __forceinline__ PathLane path_lane(uint32_t spread) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    return PathLane{tid / spread, threadIdx.x % spread == 0};
}
__device__ __forceinline__ void add_rays(unsigned long long *ray_count, uint32_t rays) {
    if (!ray_count) return;
    unsigned long long r = rays;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if ((threadIdx.x & 31) == 0 && r) atomicAdd(ray_count, r);
}

// exact mode: one lane per pixel of rows [y0, y0 + rows), samples [0, spp) in order from the CPU's
// per-pixel stream (trace_image, tracer.c:337-353)
template <bool GUIDED>
__global__ void __launch_bounds__(128, 4) exact_paths_kernel(const __grid_constant__ PtScene S, const __grid_constant__ PtParams P,
                                                             uint32_t spread, float4 *accum, unsigned long long *ray_count,
                                                             uint32_t *err) {
    const PathLane L = path_lane(spread);
    const uint32_t x = (uint32_t)(L.index % (uint32_t)P.W), yy = (uint32_t)(L.index / (uint32_t)P.W);
    const bool live = L.has && yy < (uint32_t)P.rows;
    const uint32_t y = P.y0 + yy;
    const uint64_t pixel = (uint64_t)y * (uint32_t)P.W + x;
    uint32_t rays = 0;
    Rng rng;
    rng_seed(rng, 0x853c49e6748fea9bull ^ (pixel * 0x9E3779B97F4A7C15ull) ^ (P.seed * 0xD1B54A32D192ED03ull), pixel);
    V3 sum = v3(0, 0, 0);
    float ml = 0.0f, ml2 = 0.0f, l_last = 0.0f;
    int k = 0;
    bool on = false;
    PathState ps;
    path_begin(0, v3(0, 0, 0), v3(0, 0, 1), ps, 0, 0.0f);
    for (;;) {
        Sampler sm{&rng, (uint32_t)k, (uint32_t)P.seed * 0x9e3779b9u, (int)x, (int)y, P.sampler_on, S.mask};
        if (!on && live && k < P.spp) {
            float jx, jy;
            sampler_2d(sm, 0, jx, jy);
            const float u = dvd(add((float)x, jx), (float)P.W), v = dvd(add((float)y, jy), (float)P.H);
            V3 o, d;
            camera_ray(P, u, v, o, d);
            path_begin(P.mis, o, d, ps, P.skip_caustics, P.indirect_clamp);
            on = true;
        }
        if (!__any_sync(0xffffffffu, on)) break;
        const bool cont = warp_bounce(S, P.max_depth, P.mis, ps, on, sm, err, rays);
        if (on && !cont) {
            V3 c = ps.radiance;
            on = false;
            k++;
            if (!is_number(c)) {
                if (GUIDED) l_last = 0.0f;           // (a dropped sample counts as black)
                continue;
            }
            c = clamp_sample(c, P.clamp);
            sum = vadd(sum, c);
            if (GUIDED) {
                const float l = sample_luma(c, P.guide[pixel]);
                ml += l;
                ml2 += l * l;
                l_last = l;
            }
        }
    }
    if (live) {
        const float4 a = accum[pixel];
        accum[pixel] = make_float4(a.x + sum.x, a.y + sum.y, a.z + sum.z, a.w + (float)P.spp);
        if (GUIDED) {                                // (z, w: the last sample's luminance and number + 1)
            const float4 m = P.moments[pixel];
            P.moments[pixel] = make_float4(m.x + ml, m.y + ml2, l_last, last_sample_tag(P));
        }
    }
    add_rays(ray_count, rays);
}

// fast mode, as fast_kernel
template <bool GUIDED>
__global__ void __launch_bounds__(128, 4) fast_paths_kernel(const __grid_constant__ PtScene S, const __grid_constant__ PtParams P,
                                                            uint32_t spread, float4 *accum, unsigned long long *ray_count,
                                                            uint32_t *err) {
    const uint32_t g = P.group;
    const PathLane L = path_lane(spread);
    const uint64_t pix_local = L.index / g;
    const uint32_t lane_s = (uint32_t)(L.index % g);
    const bool live = L.has && pix_local < (uint64_t)P.W * P.rows;
    const uint32_t x = (uint32_t)(pix_local % (uint32_t)P.W), y = P.y0 + (uint32_t)(pix_local / (uint32_t)P.W);
    const uint64_t pixel = (uint64_t)y * (uint32_t)P.W + x;
    uint32_t rays = 0, k = lane_s;
    V3 c = v3(0, 0, 0);
    float cnt = 0.0f, ml = 0.0f, ml2 = 0.0f, l_last = 0.0f;
    bool on = false;
    Rng rng;
    rng.state = 0;
    rng.inc = 1;
    PathState ps;
    path_begin(0, v3(0, 0, 0), v3(0, 0, 1), ps, 0, 0.0f);
    for (;;) {
        const uint32_t kk = P.spp0 + k;
        Sampler sm{&rng, kk, (uint32_t)P.seed * 0x9e3779b9u, (int)x, (int)y, P.sampler_on, S.mask};
        if (!on && live && k < (uint32_t)P.spp) {
            rng_seed(rng, mix64(pixel * 0x9E3779B97F4A7C15ull ^ ((uint64_t)kk << 40) ^ P.seed), pixel);
            float jx, jy;
            sampler_2d(sm, 0, jx, jy);
            const float u = dvd(add((float)x, jx), (float)P.W), v = dvd(add((float)y, jy), (float)P.H);
            V3 o, d;
            camera_ray(P, u, v, o, d);
            path_begin(P.mis, o, d, ps, P.skip_caustics, P.indirect_clamp);
            on = true;
        }
        if (!__any_sync(0xffffffffu, on)) break;
        const bool cont = warp_bounce(S, P.max_depth, P.mis, ps, on, sm, err, rays);
        if (on && !cont) {
            const V3 s = is_number(ps.radiance) ? clamp_sample(ps.radiance, P.clamp) : v3(0, 0, 0);
            c = vadd(c, s);
            cnt += 1.0f;
            if (GUIDED) {
                const float l = sample_luma(s, P.guide[pixel]);
                ml += l;
                ml2 += l * l;
                l_last = l;
            }
            on = false;
            k += g;
        }
    }
    // the pixel's lanes summed in the fixed order of fast_kernel's shuffles (spread: they are at most 128
    // threads, a block's)
    if (spread == 1) {
        if (GUIDED) l_last = __shfl_sync(0xffffffffu, l_last, (uint32_t)(P.spp - 1) % g, g);
        for (uint32_t o = 1; o < g; o <<= 1) {
            c.x += __shfl_down_sync(0xffffffffu, c.x, o, g);
            c.y += __shfl_down_sync(0xffffffffu, c.y, o, g);
            c.z += __shfl_down_sync(0xffffffffu, c.z, o, g);
            cnt += __shfl_down_sync(0xffffffffu, cnt, o, g);
            if (GUIDED) {
                ml += __shfl_down_sync(0xffffffffu, ml, o, g);
                ml2 += __shfl_down_sync(0xffffffffu, ml2, o, g);
            }
        }
    } else {
        __shared__ float s_sum[64][7];
        const uint32_t i = threadIdx.x / spread;
        if (L.has) {
            s_sum[i][0] = c.x; s_sum[i][1] = c.y; s_sum[i][2] = c.z; s_sum[i][3] = cnt;
            s_sum[i][4] = ml; s_sum[i][5] = ml2; s_sum[i][6] = l_last;
        }
        __syncthreads();
        if (live && lane_s == 0) {
            l_last = s_sum[i + (uint32_t)(P.spp - 1) % g][6];
            for (uint32_t o = 1; o < g; o <<= 1)
                for (uint32_t q = 0; q + o < g; q += 2 * o)
                    for (int w = 0; w < 6; w++) s_sum[i + q][w] += s_sum[i + q + o][w];
            c = v3(s_sum[i][0], s_sum[i][1], s_sum[i][2]);
            cnt = s_sum[i][3];
            ml = s_sum[i][4];
            ml2 = s_sum[i][5];
        }
    }
    if (live && lane_s == 0) {
        const float4 a = accum[pixel];
        accum[pixel] = make_float4(a.x + c.x, a.y + c.y, a.z + c.z, a.w + cnt);
        if (GUIDED) {                                // (z, w: the last sample's luminance and number + 1)
            const float4 m = P.moments[pixel];
            P.moments[pixel] = make_float4(m.x + ml, m.y + ml2, l_last, last_sample_tag(P));
        }
    }
    add_rays(ray_count, rays);
}

// closest hits over shape ids (primitives, then triangles): lrc_scene_intersect for world scenes
__global__ void __launch_bounds__(128) shapes_closest_kernel(const __grid_constant__ PtScene S, const float *__restrict__ orig,
                                                             const float *__restrict__ dir, uint64_t n, float tmin, float tmax,
                                                             int32_t *__restrict__ prim, int32_t *__restrict__ inst_out,
                                                             float *__restrict__ tout, uint32_t *err) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = i < n;
    V3 o = v3(0, 0, 0), d = v3(0, 0, 1);
    if (on) {
        o = v3(orig[3 * i], orig[3 * i + 1], orig[3 * i + 2]);
        d = v3(dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]);
    }
    float best = tmax;
    int32_t id = warp_walk<false>(S, on, o, d, tmin, best, err), inst = -1;
    if (!on) return;
    if (S.ninst) {
        int ii = -1, tri = -1;
        if (walk_instances<false>(S, o, d, tmin, best, ii, tri, err)) {
            id = tri;
            inst = ii;
        }
    }
    prim[i] = id;
    if (inst_out) inst_out[i] = inst;
    tout[i] = id >= 0 ? best : -1.0f;
}

// primitive_bounds (scene.c:47-63) of each primitive (6 float4 each) into boxes (8 floats each)
__global__ void prim_boxes_kernel(const float4 *__restrict__ prims, uint32_t n, float4 *__restrict__ boxes) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 *pr = prims + 6 * (size_t)i;
    float4 c = __ldg(pr), q = __ldg(pr + 1), u = __ldg(pr + 2), v = __ldg(pr + 3);
    float lo[3], hi[3];
    if (q.w == 0.0f) {
        lo[0] = sub(c.x, c.w); lo[1] = sub(c.y, c.w); lo[2] = sub(c.z, c.w);
        hi[0] = add(c.x, c.w); hi[1] = add(c.y, c.w); hi[2] = add(c.z, c.w);
    } else {
        float p[4][3] = {{q.x, q.y, q.z},
                         {add(q.x, u.x), add(q.y, u.y), add(q.z, u.z)},
                         {add(q.x, v.x), add(q.y, v.y), add(q.z, v.z)},
                         {add(q.x, add(u.x, v.x)), add(q.y, add(u.y, v.y)), add(q.z, add(u.z, v.z))}};
        for (int k = 0; k < 3; k++) {
            lo[k] = p[0][k];
            hi[k] = p[0][k];
            for (int j = 1; j < 4; j++) { lo[k] = rmin(lo[k], p[j][k]); hi[k] = rmax(hi[k], p[j][k]); }
        }
    }
    boxes[2 * (size_t)i] = make_float4(sub(lo[0], 1e-3f), sub(lo[1], 1e-3f), sub(lo[2], 1e-3f), 0.0f);
    boxes[2 * (size_t)i + 1] = make_float4(add(hi[0], 1e-3f), add(hi[1], 1e-3f), add(hi[2], 1e-3f), 0.0f);
}

}  // namespace pt

cudaError_t pt_prim_boxes(const float *d_prims, uint32_t n, float *d_boxes, cudaStream_t st) {
    if (!n) return cudaSuccess;
    pt::prim_boxes_kernel<<<(n + 127) / 128, 128, 0, st>>>(reinterpret_cast<const float4 *>(d_prims), n,
                                                           reinterpret_cast<float4 *>(d_boxes));
    return cudaGetLastError();
}

uint64_t pt_paths(const PtParams &P) { return (uint64_t)P.W * P.rows * (P.exact ? 1 : P.group); }

bool pt_walks_wide(const PtParams &P, bool media) { return !media && pt_paths(P) <= pt::PT_WARP_PATHS; }
bool pt_gradients_walk_wide(uint32_t ntiles, bool media) { return !media && ntiles <= pt::PT_WARP_PATHS; }

cudaError_t pt_trace(const PtScene &S, const PtParams &P, float *d_accum, unsigned long long *d_rays, uint32_t *d_status,
                     cudaStream_t st) {
    if (P.rows <= 0 || P.spp <= 0 || P.W <= 0) return cudaSuccess;
    float4 *acc = reinterpret_cast<float4 *>(d_accum);
    const uint64_t paths = pt_paths(P);
    const int k = P.moments ? 1 : 0, x = P.exact ? 1 : 0;
    if (!pt_walks_wide(P, S.nvol != 0) || !S.wide.nodes) {
        // (kernels compiled with and without the media's tracking and the denoiser's moments: each
        // holds registers that a scene or an image without them would pay for)
        using Fn = void (*)(PtScene, PtParams, float4 *, unsigned long long *, uint32_t *);
        static const Fn fns[2][4] = {{pt::fast_kernel<false, false>, pt::fast_kernel<false, true>, pt::fast_kernel<true, false>,
                                      pt::fast_kernel<true, true>},
                                     {pt::exact_kernel<false, false>, pt::exact_kernel<false, true>,
                                      pt::exact_kernel<true, false>, pt::exact_kernel<true, true>}};
        fns[x][(S.nvol ? 2 : 0) + k]<<<(unsigned)((paths + 127) / 128), 128, 0, st>>>(S, P, acc, d_rays, d_status);
        return cudaGetLastError();
    }
    using Fn = void (*)(PtScene, PtParams, uint32_t, float4 *, unsigned long long *, uint32_t *);
    static const Fn fns[2][2] = {{pt::fast_paths_kernel<false>, pt::fast_paths_kernel<true>},
                                 {pt::exact_paths_kernel<false>, pt::exact_paths_kernel<true>}};
    uint32_t spread = 1;
    while (spread < pt::SPREAD_MOST && paths * spread * 2 <= pt::SPREAD_LANES) spread *= 2;
    fns[x][k]<<<(unsigned)((paths * spread + 127) / 128), 128, 0, st>>>(S, P, spread, acc, d_rays, d_status);
    return cudaGetLastError();
}

namespace pt {

// a tile's gradient sample (trace.wgsl main with T.txl.w = 1): old pixel o's sample kk traced again
// in the new scene from the same random numbers (the fast kernel's stream of (o, kk, seed) and the
// sampler's dimensions of o), through the new pixel k moved by the old one's offset (dx, dy); lam[0]
// = |l - old l| / max(l, old l, 1e-3) of the two samples' luminance over their albedo, -1 where
// there is no sample or the new one is not a number
template <bool MEDIA, bool WARP>
__global__ void __launch_bounds__(128) grad_kernel(const __grid_constant__ PtScene S, const __grid_constant__ PtParams P,
                                                   GradTile *tiles, uint32_t ntiles, uint32_t spread,
                                                   const float4 *__restrict__ guide, unsigned long long *ray_count,
                                                   uint32_t *err) {
    const PathLane lane = path_lane(spread);
    const uint32_t t = (uint32_t)lane.index;
    uint32_t rays = 0;
    const bool live = lane.has && t < ntiles && tiles[t].o >= 0;
    if (WARP ? __any_sync(0xffffffffu, live) : live) {
        GradTile T{};
        if (live) T = tiles[t];
        const uint32_t W = (uint32_t)P.W;
        const uint32_t ox = (uint32_t)T.o % W, oy = (uint32_t)T.o / W;
        const uint32_t kx = (uint32_t)T.k % W, ky = (uint32_t)T.k / W;
        const uint64_t opix = (uint64_t)(uint32_t)T.o;
        Rng rng;
        rng_seed(rng, mix64(opix * 0x9E3779B97F4A7C15ull ^ ((uint64_t)T.kk << 40) ^ P.seed), opix);
        Sampler sm{&rng, T.kk, (uint32_t)P.seed * 0x9e3779b9u, (int)ox, (int)oy, P.sampler_on, S.mask};
        float jx, jy;
        sampler_2d(sm, 0, jx, jy);
        const float u = dvd(add(add((float)kx, T.dx), jx), (float)P.W);
        const float v = dvd(add(add((float)ky, T.dy), jy), (float)P.H);
        V3 o, d;
        camera_ray(P, u, v, o, d);
        V3 c;
        if (!WARP) {
            c = trace_path<MEDIA>(S, P, o, d, sm, err, rays);
        } else {
            PathState ps;
            path_begin(P.mis, o, d, ps, P.skip_caustics, P.indirect_clamp);
            for (bool on = live; __any_sync(0xffffffffu, on);)
                if (!warp_bounce(S, P.max_depth, P.mis, ps, on, sm, err, rays)) on = false;
            c = ps.radiance;
        }
        float lam = -1.0f;
        if (live && is_number(c) && vmax3(c) >= 0.0f) {
            c = clamp_sample(c, P.clamp);
            const float l = sample_luma(c, guide[T.k]);
            lam = fabsf(l - T.l) / fmaxf(fmaxf(l, T.l), 1e-3f);
        }
        if (live) tiles[t].lam[0] = lam;
    }
    if (ray_count) {
        unsigned long long r = rays;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if ((threadIdx.x & 31) == 0 && r) atomicAdd(ray_count, r);
    }
}

}  // namespace pt

cudaError_t pt_gradients(const PtScene &S, const PtParams &P, GradTile *d_tiles, uint32_t ntiles, const float4 *d_guide,
                         unsigned long long *d_rays, uint32_t *d_status, cudaStream_t st) {
    if (!ntiles) return cudaSuccess;
    const bool warp = pt_gradients_walk_wide(ntiles, S.nvol != 0) && S.wide.nodes;
    uint32_t spread = 1;
    while (warp && spread < pt::SPREAD_MOST && (uint64_t)ntiles * spread * 2 <= pt::SPREAD_LANES) spread *= 2;
    (S.nvol ? pt::grad_kernel<true, false> : warp ? pt::grad_kernel<false, true> : pt::grad_kernel<false, false>)
        <<<(unsigned)(((uint64_t)ntiles * spread + 127) / 128), 128, 0, st>>>(S, P, d_tiles, ntiles, spread, d_guide, d_rays,
                                                                              d_status);
    return cudaGetLastError();
}

cudaError_t pt_intersect(const PtScene &S, const float *d_orig, const float *d_dir, uint64_t n, float tmin, float tmax,
                         int32_t *d_prim, int32_t *d_inst, float *d_t, uint32_t *d_status, cudaStream_t st) {
    if (!n) return cudaSuccess;
    pt::shapes_closest_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(S, d_orig, d_dir, n, tmin, tmax, d_prim, d_inst,
                                                                           d_t, d_status);
    return cudaGetLastError();
}

// the instances' world boxes (records' words 24-26, 28-30) as builder boxes (8 floats each)
__global__ void inst_boxes_kernel(const float4 *__restrict__ rec, uint32_t n, float4 *__restrict__ boxes) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 lo = __ldg(&rec[8 * (size_t)i + 6]), hi = __ldg(&rec[8 * (size_t)i + 7]);
    boxes[2 * (size_t)i] = make_float4(lo.x, lo.y, lo.z, 0.0f);
    boxes[2 * (size_t)i + 1] = make_float4(hi.x, hi.y, hi.z, 0.0f);
}

cudaError_t pt_inst_boxes(const float *d_rec, uint32_t n, float *d_boxes, cudaStream_t st) {
    if (!n) return cudaSuccess;
    inst_boxes_kernel<<<(n + 127) / 128, 128, 0, st>>>(reinterpret_cast<const float4 *>(d_rec), n,
                                                       reinterpret_cast<float4 *>(d_boxes));
    return cudaGetLastError();
}

}  // namespace lrc
