// wide.cuh - the walk over 8-wide nodes with quantised child boxes, shared by the path tracer
// (pt_device.cuh) and the ray queries (wide.cu, which also makes the nodes). The node is the compressed
// wide node of Ylitie, Karras and Laine ("Efficient incoherent ray traversal on GPUs through compressed
// wide BVHs", HPG 2017) in a layout of our own, and the walk theirs: slots ordered by octant
// instead of sorted by distance, a node's hit children kept as one stack entry, triangles put off
// while few of a warp's lanes have one.
//
// Node (5 x 16 bytes): the grid's origin p and the three axes' scale exponents (scale = a power of
// two, its float exponent field) with the mask of inner slots; the first inner child, the first leaf
// entry, the mask of leaf slots; then the 8 slots' boxes as bytes, lo x, y, z, then hi x, y, z: lo = p +
// q_lo scale, hi = p + q_hi scale hold the binary node's box with 1/64 of a step to spare (the
// walk's rounding: below). A slot's place says where its box lies in the node (bit a set: on axis a's
// upper side), so that a ray that goes up on the axes in m meets slot s ^ m before slot s. Inner
// children lie one after another in slot order, leaf entries too. An empty slot's box is inverted.
// A leaf entry (3 x 16 bytes) is one shape: its id and a triangle's q, u, v.
//
// The closest hits of the binary walk of the tree the nodes were made from: every shape whose
// boxes the ray meets there is tested here, by the same operations, and where two shapes are hit at
// the same t - the one case in which the order of the tests decides - `tie` says so and the caller
// asks the binary walk. Rays that a shape could be hit by at a t that is no number (the binary walk then
// takes whatever it meets next) go to the binary walk (wide_plain): at once, or when the wide walk found none.
// The other way round, the boxes here being larger, a shape may be tested whose box the binary walk's slab test
// rounds away from the ray: a sliver, whose t is mostly rounding and lies outside its box (1 of 4M hits on a soup
// of 4M triangles is another triangle, its t the same to 1e-8; holding each hit against its binary box
// took 27 us more of 72 in a query of 16384 rays, for the binary walks of the few that failed).
#pragma once
#include "lrc_internal.cuh"

namespace lrc {
namespace pt {

constexpr int WD_STACK = 96;                 // pending groups of children a ray (one a level; triangles put off)
constexpr int WD_PUT_OFF_BELOW = 48;         // (triangles are put off only while the stack has room for every level)
constexpr uint32_t WD_INNER = 0xff000000u;   // a group's hit inner children, the nearest at the top bit

// the scale that brings a byte of a node's box to a float without a conversion: placed below the
// exponent of 1.0 it reads 1 + byte 2^-15
constexpr float WD_BYTE = 32768.0f;

struct WideRay {
    V3 o, d;
    float ix, iy, iz, ax, ay, az;            // 1 / d (a zero component made tiny first), o / d
    uint32_t up;                             // bit a: d goes up on axis a (or is +0)
};

__device__ __forceinline__ WideRay wide_ray(V3 o, V3 d) {
    auto inv = [](float x) { return 1.0f / (fabsf(x) < 1e-20f ? copysignf(1e-20f, x) : x); };
    WideRay r;
    r.o = o;
    r.d = d;
    r.ix = inv(d.x); r.iy = inv(d.y); r.iz = inv(d.z);
    r.ax = o.x * r.ix; r.ay = o.y * r.iy; r.az = o.z * r.iz;
    r.up = (r.ix < 0.0f ? 0u : 1u) | (r.iy < 0.0f ? 0u : 2u) | (r.iz < 0.0f ? 0u : 4u);
    return r;
}

// three-input minimum and maximum, and two fused multiply-adds in one instruction (sm_100)
__device__ __forceinline__ float wd_max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float wd_min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ uint64_t wd_pair(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void wd_split(uint64_t v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t wd_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
template <int B>
__device__ __forceinline__ float wd_byte(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x3f800000u, 0x7604 | (B << 4)));
}
// bit s of m to bit s ^ up
__device__ __forceinline__ uint32_t wd_by_octant(uint32_t m, uint32_t up) {
    if (up & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (up & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (up & 4u) m = ((m & 0x0fu) << 4) | ((m >> 4) & 0x0fu);
    return m;
}

// slots 4 h + J and 4 h + J + 1 of a node: their bits of the hit mask. A plane's t is byte' S + C with
// byte' = 1 + byte 2^-15, S = 2^15 scale / d and C = (p - o) / d - S: the rounding of C is 2^-9 of a
// grid step, within the 1/64 step the boxes are widened by.
template <int J>
__device__ __forceinline__ uint32_t wd_slots(uint32_t nx, uint32_t ny, uint32_t nz, uint32_t fx, uint32_t fy, uint32_t fz,
                                             uint64_t sx, uint64_t sy, uint64_t sz, uint64_t cx, uint64_t cy, uint64_t cz,
                                             float tmin, float best) {
    float a0, a1, b0, b1, c0, c1, d0, d1, e0, e1, f0, f1;
    wd_split(wd_fma2(wd_pair(wd_byte<J>(nx), wd_byte<J + 1>(nx)), sx, cx), a0, a1);
    wd_split(wd_fma2(wd_pair(wd_byte<J>(ny), wd_byte<J + 1>(ny)), sy, cy), b0, b1);
    wd_split(wd_fma2(wd_pair(wd_byte<J>(nz), wd_byte<J + 1>(nz)), sz, cz), c0, c1);
    wd_split(wd_fma2(wd_pair(wd_byte<J>(fx), wd_byte<J + 1>(fx)), sx, cx), d0, d1);
    wd_split(wd_fma2(wd_pair(wd_byte<J>(fy), wd_byte<J + 1>(fy)), sy, cy), e0, e1);
    wd_split(wd_fma2(wd_pair(wd_byte<J>(fz), wd_byte<J + 1>(fz)), sz, cz), f0, f1);
    uint32_t m = 0;
    if (fmaxf(wd_max3(a0, b0, c0), tmin) <= fminf(wd_min3(d0, e0, f0), best)) m |= 1u << J;
    if (fmaxf(wd_max3(a1, b1, c1), tmin) <= fminf(wd_min3(d1, e1, f1), best)) m |= 2u << J;
    return m;
}

// node ni against the ray in [tmin, best]: ng = (first inner child, hit inner slots by octant << 24 |
// inner slots), tg = (first leaf entry, leaf slots << 8 | hit leaf slots)
__device__ __forceinline__ void wide_node(const float4 *__restrict__ nodes, uint32_t ni, const WideRay &r, float tmin, float best,
                                          uint2 &ng, uint2 &tg) {
    const float4 *np = nodes + 5 * (size_t)ni;
    const float4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3), n4 = __ldg(np + 4);
    const uint32_t ex = __float_as_uint(n0.w), inner = ex >> 24, leaves = __float_as_uint(n1.z) & 0xffu;
    const float sx = __uint_as_float((ex & 0xffu) << 23) * r.ix * WD_BYTE;
    const float sy = __uint_as_float(((ex >> 8) & 0xffu) << 23) * r.iy * WD_BYTE;
    const float sz = __uint_as_float(((ex >> 16) & 0xffu) << 23) * r.iz * WD_BYTE;
    const float cx = fmaf(n0.x, r.ix, -r.ax) - sx, cy = fmaf(n0.y, r.iy, -r.ay) - sy, cz = fmaf(n0.z, r.iz, -r.az) - sz;
    const uint64_t sx2 = wd_pair(sx, sx), sy2 = wd_pair(sy, sy), sz2 = wd_pair(sz, sz);
    const uint64_t cx2 = wd_pair(cx, cx), cy2 = wd_pair(cy, cy), cz2 = wd_pair(cz, cz);
    // the near and far planes by the direction's sign
    const bool ux = r.up & 1u, uy = r.up & 2u, uz = r.up & 4u;
    const uint32_t lx0 = __float_as_uint(n2.x), lx1 = __float_as_uint(n2.y), ly0 = __float_as_uint(n2.z),
                   ly1 = __float_as_uint(n2.w), lz0 = __float_as_uint(n3.x), lz1 = __float_as_uint(n3.y);
    const uint32_t hx0 = __float_as_uint(n3.z), hx1 = __float_as_uint(n3.w), hy0 = __float_as_uint(n4.x),
                   hy1 = __float_as_uint(n4.y), hz0 = __float_as_uint(n4.z), hz1 = __float_as_uint(n4.w);
    const uint32_t nx0 = ux ? lx0 : hx0, ny0 = uy ? ly0 : hy0, nz0 = uz ? lz0 : hz0;
    const uint32_t fx0 = ux ? hx0 : lx0, fy0 = uy ? hy0 : ly0, fz0 = uz ? hz0 : lz0;
    const uint32_t nx1 = ux ? lx1 : hx1, ny1 = uy ? ly1 : hy1, nz1 = uz ? lz1 : hz1;
    const uint32_t fx1 = ux ? hx1 : lx1, fy1 = uy ? hy1 : ly1, fz1 = uz ? hz1 : lz1;
    uint32_t m = wd_slots<0>(nx0, ny0, nz0, fx0, fy0, fz0, sx2, sy2, sz2, cx2, cy2, cz2, tmin, best);
    m |= wd_slots<2>(nx0, ny0, nz0, fx0, fy0, fz0, sx2, sy2, sz2, cx2, cy2, cz2, tmin, best);
    m |= wd_slots<0>(nx1, ny1, nz1, fx1, fy1, fz1, sx2, sy2, sz2, cx2, cy2, cz2, tmin, best) << 4;
    m |= wd_slots<2>(nx1, ny1, nz1, fx1, fy1, fz1, sx2, sy2, sz2, cx2, cy2, cz2, tmin, best) << 4;
    ng = make_uint2(__float_as_uint(n1.x), wd_by_octant(m & inner, r.up) << 24 | inner);
    tg = make_uint2(__float_as_uint(n1.y), leaves << 8 | (m & leaves));
}

// Moller-Trumbore (intersect.h:96-112) of a leaf entry's triangle, rounded as the C code rounds it: a
// hit with t in (tmin, tmax]
__device__ __forceinline__ bool wide_tri(float4 q, float4 u, float4 v, V3 o, V3 d, float tmin, float tmax, float &tout) {
    const V3 vv = v3(v.x, v.y, v.z), uu = v3(u.x, u.y, u.z);
    const V3 pvec = vcross(d, vv);
    const float det = vdot(uu, pvec);
    if (fabsf(det) < 1e-12f) return false;
    const float inv = dvd(1.0f, det);
    const V3 tvec = vsub(o, v3(q.x, q.y, q.z));
    const float b1 = mul(vdot(tvec, pvec), inv);
    if (b1 < 0.0f || b1 > 1.0f) return false;
    const V3 qvec = vcross(tvec, uu);
    const float b2 = mul(vdot(d, qvec), inv);
    if (b2 < 0.0f || add(b1, b2) > 1.0f) return false;
    const float t = mul(vdot(vv, qvec), inv);
    if (t <= tmin || t > tmax) return false;
    tout = t;
    return true;
}

// A ray's walk: begun by wide_begin, one wide_step a node (and its hit leaves) until it returns true.
struct WideWalk {
    uint2 ng;                                // the group walked: hit inner children left
    int sp;
    int32_t hit;                             // the closest shape's id so far (-1: none)
    float best;                              // its t (at first the ray's end)
    bool tie;                                // another shape was hit at t = best (or wide_odd, wide_full): ask the binary walk
};
__device__ __forceinline__ void wide_begin(WideWalk &w, float tmax) {
    w.ng = make_uint2(0u, 0x80000000u);      // (the root: its relative index comes out 0 of no inner slots)
    w.sp = 0;
    w.hit = -1;
    w.best = tmax;
    w.tie = false;
}

// Whether the shape tests of a ray give numbers: with o, d and the shapes (collapse_kernel's bound) within 1e9
// and d not (nearly) zero, the products of hit_sphere_t ((6 |d| |c - o|)^2) and wide_tri (24 |q|^3) stay
// finite and no zero is divided by zero.
constexpr float WD_FAR = 1e9f;
__device__ __forceinline__ bool wide_plain(V3 o, V3 d) {
    const float dd = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
    return fabsf(o.x) + fabsf(o.y) + fabsf(o.z) <= WD_FAR && dd <= WD_FAR && dd >= 1e-18f;   // (not so for a NaN)
}
// a walk that ends with its first step, the binary one to be asked
__device__ __forceinline__ void wide_odd(WideWalk &w) {
    w.ng.y = 0u;
    w.tie = true;
}

// A walk whose stack is full ends: the binary walk, whose pending nodes are others, is asked. ASK = false (the
// wavefront's kernels): it is reported, as the path tracer's binary walk reports its 64 (a group waits for a
// node of which that walk holds one or more back, so that it would be full first).
template <bool ASK>
__device__ __forceinline__ bool wide_full(bool &tie, uint32_t *err) {
    if (ASK) tie = true;
    else atomicOr(err, ST_STACK_OVERFLOW);
    return true;
}

// with: how many lanes of the warp take this step together (they are to be reconverged before each step:
// wide_run, or the refilling loops' ballots; left to themselves the lanes of a warp part at their first
// triangle and stay apart).
// Shapes: shape(entry's id, its first 16 bytes' place, o, d, tmin, tmax, t) tests one leaf entry with t
// in (tmin, tmax]. ANY: the first hit before best ends the walk; otherwise lanes whose triangles
// would be tested by fewer than a quarter of the lanes at it keep them for later (triangles tested with a
// few lanes are what a divergent walk loses most by; an any-hit walk is better off testing them).
// COUNT: cnt[0] += nodes (80 bytes each), cnt[1] += leaf entries. True: the walk is over.
template <bool ANY, bool COUNT, bool ASK = true, typename Shape>
__device__ __forceinline__ bool wide_step(const WideScene &S, const WideRay &r, WideWalk &w, uint2 *stack, float tmin, int with,
                                          uint32_t *err, Shape &&shape, uint32_t *cnt = nullptr) {
    uint2 tg;
    if (w.ng.y & WD_INNER) {
        const uint32_t bit = 31 - __clz(w.ng.y);
        w.ng.y &= ~(1u << bit);
        const uint32_t slot = (bit - 24u) ^ r.up;
        const uint32_t ni = w.ng.x + __popc(w.ng.y & 0xffu & ((1u << slot) - 1u));
        if (w.ng.y & WD_INNER) {
            if (w.sp >= WD_STACK) return wide_full<ASK>(w.tie, err);
            stack[w.sp++] = w.ng;
        }
        if (ni >= S.nnodes) { atomicOr(err, ST_BAD_TREE); return true; }
        if constexpr (COUNT) cnt[0]++;
        wide_node(S.nodes, ni, r, tmin, w.best, w.ng, tg);
    } else {                                 // (triangles put off)
        tg = w.ng;
        w.ng.y = 0u;
    }
    while (tg.y & 0xffu) {
        if (!ANY && 4 * __popc(__activemask()) < with && (w.ng.y & WD_INNER) && w.sp < WD_PUT_OFF_BELOW) {
            stack[w.sp++] = make_uint2(tg.x, tg.y & 0xffffu);
            break;
        }
        const uint32_t slot = 31 - __clz(tg.y & 0xffu);
        tg.y &= ~(1u << slot);
        const uint32_t e = tg.x + __popc((tg.y >> 8) & ((1u << slot) - 1u));
        if (e >= S.nleaves) { atomicOr(err, ST_BAD_TREE); return true; }
        if constexpr (COUNT) cnt[1]++;
        const float4 *lp = S.leaves + 3 * (size_t)e;
        const float4 q = __ldg(lp);
        const int32_t id = (int32_t)__float_as_uint(q.w);
        float t;
        if (!shape((uint32_t)id, q, lp, r, tmin, w.best, t)) continue;
        if (t < w.best) {
            w.best = t;
            w.hit = id;
            w.tie = false;
            if (ANY) return true;
        } else if (!ANY && w.hit >= 0 && w.hit != id) {
            w.tie = true;
        }
    }
    if (!(w.ng.y & WD_INNER)) {
        if (w.sp == 0) return true;
        w.ng = stack[--w.sp];
    }
    return false;
}

// a whole walk by one lane, its steps in step with the other lanes that walk now
template <bool ANY, bool COUNT, typename Shape>
__device__ __forceinline__ void wide_run(const WideScene &S, const WideRay &r, WideWalk &w, float tmin, uint32_t *err,
                                         Shape &&shape, uint32_t *cnt = nullptr) {
    uint2 stack[WD_STACK];
    uint32_t with = __activemask();
    while (true) {
        const bool over = wide_step<ANY, COUNT>(S, r, w, stack, tmin, __popc(with), err, shape, cnt);
        with = __ballot_sync(with, !over);
        if (over) return;
    }
}

// whether the nodes can be walked (the collapse marks the root of a tree whose boxes the grid cannot hold)
__device__ __forceinline__ bool wide_walked(const WideScene &S) { return __float_as_uint(__ldg(&S.nodes[1].w)) == 0u; }

// The walk with 8 lanes a ray (a warp: 4 rays), for so few rays that their walks' length and not their
// number decides: lane s of the 8 tests slot s of a node and, when it is a leaf, its shape, so a
// node costs a fifth of the instructions one after another and its shapes are tested together. All 8
// lanes hold the same ray and walk; they call together.
template <bool ANY, typename Shape>
__device__ __forceinline__ int32_t wide_walk8(const WideScene &S, const WideRay &r, float tmin, float &best, bool &tie,
                                              uint32_t *err, Shape &&shape) {
    const uint32_t lane = threadIdx.x & 31u, s = lane & 7u, sh = lane & 24u, peers = 0xffu << sh;
    uint2 stack[WD_STACK];
    int sp = 0;
    int32_t hit = -1;
    uint32_t ni = 0;
    tie = false;
    const uint32_t far_x = r.up & 1u ? 24u : 0u, far_y = r.up & 2u ? 24u : 0u, far_z = r.up & 4u ? 24u : 0u;
    while (true) {
        if (ni >= S.nnodes) { atomicOr(err, ST_BAD_TREE); return -1; }
        const float4 *np = S.nodes + 5 * (size_t)ni;
        const float4 n0 = __ldg(np), n1 = __ldg(np + 1);
        const uint8_t *qb = reinterpret_cast<const uint8_t *>(np + 2) + s;
        const float nx = (float)__ldg(qb + (24u - far_x)), ny = (float)__ldg(qb + 8 + (24u - far_y)),
                    nz = (float)__ldg(qb + 16 + (24u - far_z));
        const float fx = (float)__ldg(qb + far_x), fy = (float)__ldg(qb + 8 + far_y), fz = (float)__ldg(qb + 16 + far_z);
        const uint32_t ex = __float_as_uint(n0.w), inner = ex >> 24, leaves = __float_as_uint(n1.z) & 0xffu;
        const float sx = __uint_as_float((ex & 0xffu) << 23) * r.ix, sy = __uint_as_float(((ex >> 8) & 0xffu) << 23) * r.iy,
                    sz = __uint_as_float(((ex >> 16) & 0xffu) << 23) * r.iz;
        const float cx = fmaf(n0.x, r.ix, -r.ax), cy = fmaf(n0.y, r.iy, -r.ay), cz = fmaf(n0.z, r.iz, -r.az);
        const float tn = fmaxf(wd_max3(fmaf(nx, sx, cx), fmaf(ny, sy, cy), fmaf(nz, sz, cz)), tmin);
        const float tf = fminf(wd_min3(fmaf(fx, sx, cx), fmaf(fy, sy, cy), fmaf(fz, sz, cz)), best);
        const uint32_t m = (__ballot_sync(peers, tn <= tf) >> sh) & 0xffu;
        if (m & leaves) {
            float t = 0.0f;
            int32_t id = -1;
            bool found = false;
            if ((m & leaves) >> s & 1u) {
                const uint32_t e = __float_as_uint(n1.y) + __popc(leaves & ((1u << s) - 1u));
                if (e < S.nleaves) {
                    const float4 *lp = S.leaves + 3 * (size_t)e;
                    const float4 q = __ldg(lp);
                    id = (int32_t)__float_as_uint(q.w);
                    found = shape((uint32_t)id, q, lp, r, tmin, best, t) && (t < best || hit >= 0);
                } else {
                    atomicOr(err, ST_BAD_TREE);
                }
            }
            const uint32_t hits = __ballot_sync(peers, found);
            if (hits) {
                float tt = found ? t : __int_as_float(0x7f800000);
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) tt = fminf(tt, __shfl_xor_sync(peers, tt, o));
                if (ANY) {
                    if (tt < best) { best = tt; return 1; }
                } else {
                    const uint32_t first = __ballot_sync(peers, found && t == tt);
                    const int32_t who = __shfl_sync(peers, id, __ffs(first) - 1);
                    if (tt < best) {
                        best = tt;
                        hit = who;
                        tie = __popc(first) > 1;
                    } else if (who != hit || __popc(first) > 1) {
                        tie = true;
                    }
                }
            }
        }
        uint2 ng = make_uint2(__float_as_uint(n1.x), wd_by_octant(m & inner, r.up) << 24 | inner);
        if (!(ng.y & WD_INNER)) {
            if (sp == 0) return hit;
            ng = stack[--sp];
        }
        const uint32_t bit = 31 - __clz(ng.y);
        ng.y &= ~(1u << bit);
        const uint32_t slot = (bit - 24u) ^ r.up;
        ni = ng.x + __popc(ng.y & 0xffu & ((1u << slot) - 1u));
        if (ng.y & WD_INNER) {
            if (sp >= WD_STACK) { tie = true; return -1; }   // (wide_full)
            stack[sp++] = ng;
        }
    }
}

}  // namespace pt
}  // namespace lrc
