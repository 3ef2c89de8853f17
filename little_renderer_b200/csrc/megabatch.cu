// megabatch.cu - the batch's persistent megakernel (engine 0: one path a lane, the next sample begun when
// a path ends) and the pass that adds a batch's per-task sums into its images (both engines').
#include "pt_device.cuh"
#include <algorithm>

namespace lrc {
namespace pt {

// ---- the batch: one persistent kernel over the tasks of many jobs --------------------------------

// Each lane holds one task (a pixel's lane slot) and one path of it at a time. A loop pass is
// one bounce for every lane with a path; a lane whose path ends adds it to its task's sum and
// starts the task's next sample, and a lane whose task is done writes it out and takes the next
// task of the queue (one atomic per warp and pass for all such lanes). The lanes thus stay busy
// however the path lengths and the samples per task differ, within a job and across jobs, and
// the grid drains the queue with no launch per job and no tail per job.
template <int BLOCK, int MINB, bool MEDIA>
__global__ void __launch_bounds__(BLOCK, MINB) batch_kernel(const BatchJob *__restrict__ jobs, uint32_t njobs,
                                                      unsigned long long ntasks, unsigned long long *next, uint32_t *err) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    int j = -1;                       // the job of the lane's task (-1: none)
    unsigned long long task = 0;
    uint64_t pixel = 0;               // the pixel's index in its image
    uint32_t x = 0, y = 0, slot = 0, kk = 0, kend = 0, g = 1, rays = 0;
    V3 c = v3(0, 0, 0);
    float cnt = 0.0f, ml = 0.0f, ml2 = 0.0f, l_last = 0.0f;   // the task's sum, samples, luminance moments
    bool active = false, done = false;
    PathState ps;
    Rng rng;
    rng.state = 0;
    rng.inc = 1;
    for (;;) {
        if (j >= 0 && !active && kk >= kend) {       // the task is done
            const BatchJob &J = jobs[j];
            const unsigned long long l = task - J.task0;
            J.partial[l] = make_float4(c.x, c.y, c.z, cnt);
            J.prays[l] = rays;
            if (J.pmom) J.pmom[l] = make_float4(ml, ml2, l_last, 0.0f);
            j = -1;
        }
        const bool need = !done && j < 0;
        const uint32_t m = __ballot_sync(0xffffffffu, need);
        if (m) {
            const int leader = __ffs(m) - 1;
            unsigned long long base = 0;
            if ((int)lane == leader) base = atomicAdd(next, (unsigned long long)__popc(m));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (need) {
                task = base + __popc(m & lt_mask);
                if (task >= ntasks) {
                    done = true;
                } else {
                    j = (int)batch_job_of(jobs, njobs, task);
                    const BatchJob &J = jobs[j];
                    const unsigned long long l = task - J.task0;
                    g = (uint32_t)J.P.group;
                    const unsigned long long pl = l / g;
                    slot = (uint32_t)(l - pl * g);
                    x = (uint32_t)(pl % (uint32_t)J.P.W);
                    y = (uint32_t)J.P.y0 + (uint32_t)(pl / (uint32_t)J.P.W);
                    pixel = (uint64_t)y * (uint32_t)J.P.W + x;
                    kk = (uint32_t)J.P.spp0 + slot;
                    kend = (uint32_t)(J.P.spp0 + J.P.spp);
                    c = v3(0, 0, 0);
                    cnt = 0.0f;
                    ml = ml2 = l_last = 0.0f;
                    rays = 0;
                    if (J.P.exact)                    // trace_image's per-pixel stream, all samples in order
                        rng_seed(rng, 0x853c49e6748fea9bull ^ (pixel * 0x9E3779B97F4A7C15ull) ^ (J.P.seed * 0xD1B54A32D192ED03ull),
                                 pixel);
                }
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
        if (j < 0) continue;                         // (only lanes that ran out of tasks)
        const BatchJob &J = jobs[j];
        Sampler sm{&rng, kk, (uint32_t)J.P.seed * 0x9e3779b9u, (int)x, (int)y, J.P.sampler_on, J.S.mask};
        if (!active) {                               // the task's next sample: its camera ray
            if (!J.P.exact)
                rng_seed(rng, mix64(pixel * 0x9E3779B97F4A7C15ull ^ ((uint64_t)kk << 40) ^ J.P.seed), pixel);
            float jx, jy;
            sampler_2d(sm, 0, jx, jy);
            float u = dvd(add((float)x, jx), (float)J.P.W), v = dvd(add((float)y, jy), (float)J.P.H);
            V3 o, d;
            camera_ray(J.P, u, v, o, d);
            path_begin(J.P.mis || (MEDIA && J.S.nvol), o, d, ps, J.P.skip_caustics, J.P.indirect_clamp);
            active = true;
        }
        if (!path_bounce<MEDIA>(J.S, J.P.max_depth, J.P.mis, ps, sm, err, rays)) {
            V3 s = is_number(ps.radiance) ? clamp_sample(ps.radiance, J.P.clamp) : v3(0, 0, 0);
            c = vadd(c, s);
            cnt += 1.0f;
            if (J.P.moments) {
                const float l = sample_luma(s, J.P.guide[pixel]);
                ml += l;
                ml2 += l * l;
                l_last = l;
            }
            active = false;
            kk += g;
        }
    }
}

// pixel i of all the batch's bands (a whole warp calls it together): the pixel's slots summed in
// the fast kernel's shuffle order (pairs, then pairs of pairs, ...) and added to its image, its rays
// to its job
__device__ __forceinline__ void resolve_pixel(const BatchJob *__restrict__ jobs, uint32_t njobs, unsigned long long npix,
                                              unsigned long long i) {
    uint32_t jj = 0xffffffffu;
    unsigned long long r = 0;
    if (i < npix) {
        uint32_t lo = 0, hi = njobs - 1;
        while (lo < hi) {
            uint32_t mid = (lo + hi + 1) >> 1;
            if (__ldg(&jobs[mid].pix0) <= i) lo = mid;
            else hi = mid - 1;
        }
        jj = lo;
        const BatchJob &J = jobs[jj];
        const unsigned long long pl = i - J.pix0;
        const uint32_t g = (uint32_t)J.P.group;
        float4 v[16];
        for (uint32_t s = 0; s < 16; s++) {
            if (s < g) {
                v[s] = J.partial[pl * g + s];
                r += J.prays[pl * g + s];
            }
        }
        for (uint32_t o = 1; o < 16; o <<= 1)
            for (uint32_t s = 0; s + o < 16; s += 2 * o)
                if (s + o < g) {
                    v[s].x += v[s + o].x;
                    v[s].y += v[s + o].y;
                    v[s].z += v[s + o].z;
                    v[s].w += v[s + o].w;
                }
        const uint32_t x = (uint32_t)(pl % (uint32_t)J.P.W), y = (uint32_t)J.P.y0 + (uint32_t)(pl / (uint32_t)J.P.W);
        const uint64_t pixel = (uint64_t)y * (uint32_t)J.P.W + x;
        float4 *a = J.accum + pixel;
        float4 av = *a;
        *a = make_float4(av.x + v[0].x, av.y + v[0].y, av.z + v[0].z, av.w + v[0].w);
        if (J.pmom) {                                // the moments, in the same order; the last sample's
            float2 mv[16];                           // (spp0 + spp - 1) from slot (spp - 1) % g
            for (uint32_t s = 0; s < 16; s++)
                if (s < g) {
                    const float4 q = J.pmom[pl * g + s];
                    mv[s] = make_float2(q.x, q.y);
                }
            for (uint32_t o = 1; o < 16; o <<= 1)
                for (uint32_t s = 0; s + o < 16; s += 2 * o)
                    if (s + o < g) {
                        mv[s].x += mv[s + o].x;
                        mv[s].y += mv[s + o].y;
                    }
            const float4 m = J.P.moments[pixel];
            const float lz = J.pmom[pl * g + (uint32_t)(J.P.spp - 1) % g].z;
            J.P.moments[pixel] = make_float4(m.x + mv[0].x, m.y + mv[0].y, lz, last_sample_tag(J.P));
        }
    }
    // the rays of the warp's pixels, one atomic per job present
    const uint32_t peers = __match_any_sync(0xffffffffu, jj);
    const uint32_t sum = __reduce_add_sync(peers, (uint32_t)r);
    if (jj != 0xffffffffu && (threadIdx.x & 31) == (uint32_t)(__ffs(peers) - 1) && sum)
        atomicAdd(jobs[jj].rays, (unsigned long long)sum);
}

// one thread per pixel
__global__ void __launch_bounds__(128) batch_resolve_kernel(const BatchJob *__restrict__ jobs, uint32_t njobs,
                                                            unsigned long long npix) {
    resolve_pixel(jobs, njobs, npix, (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// the same over a fixed grid, the job and pixel counts read from the run block (run[1], run[3]):
// a graph captured once resolves any run
__global__ void __launch_bounds__(128) batch_resolve_run_kernel(const BatchJob *__restrict__ jobs,
                                                                const unsigned long long *__restrict__ run) {
    const uint32_t njobs = (uint32_t)run[1];
    const unsigned long long npix = run[3];
    if (!njobs) return;
    for (unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x; base < npix;
         base += (unsigned long long)gridDim.x * blockDim.x)
        resolve_pixel(jobs, njobs, npix, base + threadIdx.x);
}

}  // namespace pt

// the batch kernel's launch shapes: threads per block and the blocks per SM its registers are
// capped for (65536 / (threads x blocks) registers a thread)
namespace {
using BatchFn = void (*)(const BatchJob *, uint32_t, unsigned long long, unsigned long long *, uint32_t *);
struct BatchVariant {
    int block, minb;
    BatchFn fn, media;   // (media: the kernel compiled with the media's tracking, for batches that have some)
};
#define LRC_BATCH_VARIANT(B, M) {B, M, pt::batch_kernel<B, M, false>, pt::batch_kernel<B, M, true>}
const BatchVariant kBatchVariants[] = {
    LRC_BATCH_VARIANT(128, 4), LRC_BATCH_VARIANT(128, 3), LRC_BATCH_VARIANT(128, 5),
    LRC_BATCH_VARIANT(256, 2), LRC_BATCH_VARIANT(64, 8),  LRC_BATCH_VARIANT(256, 3),
};
#undef LRC_BATCH_VARIANT
}  // namespace

int batch_variants() { return (int)(sizeof(kBatchVariants) / sizeof(kBatchVariants[0])); }

int batch_variant_shape(int v, int *block, int *minb) {
    if (v < 0 || v >= batch_variants()) return -1;
    *block = kBatchVariants[v].block;
    *minb = kBatchVariants[v].minb;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kBatchVariants[v].fn, kBatchVariants[v].block, 0)) return -1;
    return n;
}

cudaError_t batch_trace(const BatchJob *d_jobs, uint32_t njobs, unsigned long long ntasks, unsigned long long *d_next,
                        uint32_t *d_status, int variant, int grid, bool media, cudaStream_t st) {
    if (!njobs || !ntasks) return cudaSuccess;
    if (grid < 1 || variant < 0 || variant >= batch_variants()) return cudaErrorInvalidValue;
    void *args[] = {(void *)&d_jobs, (void *)&njobs, (void *)&ntasks, (void *)&d_next, (void *)&d_status};
    const BatchVariant &V = kBatchVariants[variant];
    return cudaLaunchKernel((const void *)(media ? V.media : V.fn), dim3(grid), dim3(V.block), args, 0, st);
}

cudaError_t batch_resolve(const BatchJob *d_jobs, uint32_t njobs, unsigned long long npix, cudaStream_t st) {
    if (!njobs || !npix) return cudaSuccess;
    pt::batch_resolve_kernel<<<(unsigned)((npix + 127) / 128), 128, 0, st>>>(d_jobs, njobs, npix);
    return cudaGetLastError();
}

cudaError_t batch_resolve_run(const BatchJob *d_jobs, const unsigned long long *d_run, int num_sms, cudaStream_t st) {
    pt::batch_resolve_run_kernel<<<16 * num_sms, 128, 0, st>>>(d_jobs, d_run);
    return cudaGetLastError();
}

}  // namespace lrc
