// wide.cu - the 8-wide nodes (wide.cuh) made on the device from a binary tree, and the ray queries
// over them: closest hit (scene_intersect, engine/rt/accel.c:252) and any hit (scene_occluded, :280)
// of a scene of triangles.
//
// Collapse: one launch, 8 lanes a wide node. A wide node takes its binary node's two children and
// opens the one with the largest surface area while fewer than 8 slots are used; a leaf of several
// entries opens into one slot per entry (or, where they do not fit, gets a node of its own). The nodes
// are numbered as they are found, and node i's binary node is posted at items[i]: groups of lanes
// take numbers in order and wait for theirs to be posted, so a tree's levels follow one another
// without a launch or the host between them (the wait is bounded, and a group whose number is never
// posted leaves when every node posted has been made). Bound by the chain of node reads a level (an
// opened child's record, 7 times) times the levels: 4M soup triangles 1.0 ms, 200k triangles 55 us.
#include "pt_device.cuh"
#include <algorithm>

namespace lrc {

namespace {

using namespace pt;

constexpr int WD_THREADS = 128;
enum { CT_HEAD = 0, CT_MADE = 2, CT_STOP = 3, CT_ALLOC = 4 };   // words of the counters (CT_ALLOC: 64 bits)

struct Collapse {
    const Node *bin;
    uint32_t root, nn;
    const uint32_t *aux;
    uint32_t naux;
    uint32_t entries;                            // the tree's leaf entries (of aux's naux)
    const float4 *tris;
    uint32_t nprims, ntris;
    float widen;                                 // every box is widened by this share of the root box's largest coordinate
    float4 *nodes;
    uint32_t ncap;
    uint32_t *wild;                              // set when a box is none the grid can hold
    float4 *leaves;
    uint32_t *items;
    uint32_t *ctr;
    uint32_t *err;
};

__device__ __forceinline__ uint32_t ld_now(const uint32_t *p) { return *(const volatile uint32_t *)p; }

enum { K_NONE = 0, K_INNER = 1, K_GROUP = 2, K_ENTRY = 3 };   // nothing, an inner node, a leaf of several, one entry

struct Child {
    int kind;
    uint32_t ref;                                // K_INNER, K_GROUP: the binary node; K_ENTRY: its place in aux
    uint32_t a, b;                               // K_INNER, K_GROUP: the binary node's words
    float lo[3], hi[3];
    bool shut;                                   // (a leaf of several that does not fit)
};

__device__ __forceinline__ void take_node(const Collapse &C, uint32_t c, Child &o) {
    o.kind = K_NONE;
    o.shut = false;
    if (c >= C.nn) {
        atomicOr(C.err, ST_BAD_TREE);
        return;
    }
    const float4 *p = reinterpret_cast<const float4 *>(&C.bin[c]);
    const float4 l = __ldg(p), h = __ldg(p + 1);
    o.lo[0] = l.x; o.lo[1] = l.y; o.lo[2] = l.z;
    o.hi[0] = h.x; o.hi[1] = h.y; o.hi[2] = h.z;
    o.a = __float_as_uint(l.w);
    o.b = __float_as_uint(h.w);
    o.ref = c;
    if (!(o.b & LEAF_BIT)) {
        o.kind = K_INNER;
        return;
    }
    const uint32_t n = o.b & ~LEAF_BIT;
    if (o.a > C.naux || n > C.naux - o.a) {
        atomicOr(C.err, ST_BAD_TREE);
    } else if (n == 1) {
        o.kind = K_ENTRY;
        o.ref = o.a;
    } else if (n) {
        o.kind = K_GROUP;
    }
}

// the scale's exponent field for an axis from lo to hi: 253 steps hold it, and a step is no smaller
// than the floats there, so that the grid's origin one step below lo costs at most half a step
__device__ __forceinline__ uint32_t scale_field(float lo, float hi) {
    const uint32_t e = (__float_as_uint(__fdiv_ru(__fsub_ru(hi, lo), 253.0f)) >> 23) + 1u;
    const uint32_t u = __float_as_uint(fmaxf(fabsf(lo), fabsf(hi))) >> 23;
    return min(max(max(e, u > 23u ? u - 23u : 0u), 1u), 253u);
}

__global__ void __launch_bounds__(WD_THREADS) collapse_kernel(const __grid_constant__ Collapse C) {
    const uint32_t all = 0xffffffffu, lane = threadIdx.x & 31u, s = lane & 7u;
    // (the root box's largest coordinate: its widening, none where it is no number a grid holds)
    const float4 rl = __ldg(reinterpret_cast<const float4 *>(&C.bin[C.root])), rh = __ldg(reinterpret_cast<const float4 *>(&C.bin[C.root]) + 1);
    float pad = C.widen * fmaxf(fmaxf(fmaxf(fabsf(rl.x), fabsf(rl.y)), fabsf(rl.z)), fmaxf(fmaxf(fabsf(rh.x), fabsf(rh.y)), fabsf(rh.z)));
    if (!(pad < WD_FAR)) pad = 0.0f;
    uint32_t idx = 0, spins = 0, made = 0;       // made: the nodes this warp made, not yet counted in CT_MADE
    bool claimed = false;
    for (;;) {
        // the groups without a number take the next ones
        const uint32_t want = __ballot_sync(all, !claimed && s == 0u);
        if (want) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&C.ctr[CT_HEAD], (uint32_t)__popc(want));
            base = __shfl_sync(all, base, 0);
            if (!claimed) idx = base + __popc(want & ((1u << (lane & 24u)) - 1u));
            claimed = true;
        }
        uint32_t item = 0;
        if (s == 0u && idx < C.ncap) item = idx ? ld_now(&C.items[idx]) : C.root + 1u;
        item = __shfl_sync(all, item, 0, 8);
        const bool ready = item != 0u;
        if (!__any_sync(all, ready)) {
            uint32_t done = 0;
            if (lane == 0) {
                if (made) {
                    __threadfence();
                    atomicAdd(&C.ctr[CT_MADE], made);
                    made = 0;
                }
                // (made first: a node counted there had its children's numbers taken before)
                const uint32_t m = ld_now(&C.ctr[CT_MADE]);
                __threadfence();
                const uint32_t n = ld_now(&C.ctr[CT_ALLOC]) + 1u;   // (the root has no number taken)
                done = m == n || ld_now(&C.ctr[CT_STOP]) ? 1u : 0u;
                if (!done && ++spins > SPIN_LIMIT) {
                    atomicOr(C.err, ST_TIMEOUT_BARRIER);
                    done = 1u;
                }
            }
            if (__shfl_sync(all, done, 0)) return;
            __nanosleep(40);
            continue;
        }
        spins = 0;
        // the node's two children (or a leaf's entries), one a lane
        Child c;
        c.kind = K_NONE;
        c.shut = false;
        uint32_t n = 0;
        if (ready) {
            const Node &x = C.bin[item - 1u];
            const uint32_t xa = x.a, xb = x.b;
            if (xb & LEAF_BIT) {
                n = min(xb & ~LEAF_BIT, 8u);
                if (s < n) {
                    take_node(C, item - 1u, c);
                    if (c.kind != K_NONE) {
                        c.kind = K_ENTRY;
                        c.ref = xa + s;
                    }
                }
            } else {
                n = 2;
                if (s < 2u) take_node(C, s ? xb : xa, c);
            }
        }
        // the largest one opened while there is room
        for (int round = 0; round < 16; round++) {
            float area = -1.0f;
            if (n < 8u && (c.kind == K_INNER || (c.kind == K_GROUP && !c.shut))) {
                const float dx = c.hi[0] - c.lo[0], dy = c.hi[1] - c.lo[1], dz = c.hi[2] - c.lo[2];
                area = fmaxf(dx * dy + dy * dz + dz * dx, 0.0f);
            }
            uint32_t who = s;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const float oa = __shfl_xor_sync(all, area, o, 8);
                const uint32_t ow = __shfl_xor_sync(all, who, o, 8);
                if (oa > area || (oa == area && ow < who)) { area = oa; who = ow; }
            }
            const bool open = area >= 0.0f;
            if (!__any_sync(all, open)) break;
            const uint32_t wa = __shfl_sync(all, c.a, who, 8), wb = __shfl_sync(all, c.b, who, 8),
                           wr = __shfl_sync(all, c.ref, who, 8);
            if (!open) continue;
            if (!(wb & LEAF_BIT)) {
                if (s == who) take_node(C, wa, c);
                else if (s == n) take_node(C, wb, c);
                n++;
            } else {
                const uint32_t cnt = wb & ~LEAF_BIT;
                if (n - 1u + cnt <= 8u) {
                    if (s == who || (s >= n && s < n - 1u + cnt)) {
                        take_node(C, wr, c);
                        c.kind = K_ENTRY;
                        c.ref = wa + (s == who ? 0u : s - n + 1u);
                    }
                    n += cnt - 1u;
                } else if (s == who) {
                    c.shut = true;
                }
            }
        }
        // the node's box
        const bool have = c.kind != K_NONE;
        const float inf = __int_as_float(0x7f800000);
        float lo[3], hi[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            lo[a] = have ? c.lo[a] : inf;
            hi[a] = have ? c.hi[a] : -inf;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(all, lo[a], o, 8));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(all, hi[a], o, 8));
            }
        }
        // boxes of a NaN or an infinity, which the grid cannot hold, or beyond WD_FAR (wide_plain): the tree is not
        // walked (C.wild: the root's last word, or the mark a scene's meshes share, says so; the callers
        // walk the binary one)
        bool plain = true;
#pragma unroll
        for (int a = 0; a < 3; a++) plain = plain && (!have || (fabsf(c.lo[a]) <= WD_FAR && fabsf(c.hi[a]) <= WD_FAR));
        if (!plain) atomicOr(C.wild, 1u);
        // a slot for each child: of the pairs left the one that lies best (its middle farthest to the
        // slot's corner), again and again
        float e[3];
#pragma unroll
        for (int a = 0; a < 3; a++) e[a] = have ? (c.lo[a] + c.hi[a]) - (lo[a] + hi[a]) : 0.0f;
        uint32_t taken = 0, slot = 0;
        bool placed = !have;
        for (int round = 0; round < 8; round++) {
            float best = -inf;
            uint32_t at = 0;
            if (!placed) {
#pragma unroll
                for (uint32_t k = 0; k < 8; k++) {
                    const float v = (k & 1u ? e[0] : -e[0]) + (k & 2u ? e[1] : -e[1]) + (k & 4u ? e[2] : -e[2]);
                    if (!(taken >> k & 1u) && (v > best || best == -inf)) { best = v; at = k; }
                }
            }
            float v = placed ? -inf : fmaxf(best, -3e38f);
            uint32_t who = s;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const float ov = __shfl_xor_sync(all, v, o, 8);
                const uint32_t ow = __shfl_xor_sync(all, who, o, 8);
                if (ov > v || (ov == v && ow < who)) { v = ov; who = ow; }
            }
            const uint32_t got = __shfl_sync(all, at, who, 8);
            if (v > -inf) {
                taken |= 1u << got;
                if (s == who) { slot = got; placed = true; }
            }
        }
        // lanes without a child: the slots left, in order
        const uint32_t idle = (__ballot_sync(all, !have) >> (lane & 24u)) & 0xffu;
        if (!have) {
            uint32_t left = ~taken & 0xffu;
            for (uint32_t k = __popc(idle & ((1u << s) - 1u)); k; k--) left &= left - 1u;
            slot = __ffs(left) - 1;
        }
        uint32_t inner = 0, leaf = 0;
        if (c.kind == K_INNER || c.kind == K_GROUP) inner = 1u << slot;
        if (c.kind == K_ENTRY) leaf = 1u << slot;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            inner |= __shfl_xor_sync(all, inner, o, 8);
            leaf |= __shfl_xor_sync(all, leaf, o, 8);
        }
        // numbers for the warp's children and leaf entries, one addition for its 4 nodes
        uint32_t sum = ready ? (uint32_t)__popc(inner) | (uint32_t)__popc(leaf) << 16 : 0u, before = 0;
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const uint32_t v = __shfl_sync(all, sum, 8 * g);
            if (8u * g < (lane & 24u)) before += v;
        }
        const uint32_t total = __shfl_sync(all, before + sum, 31);
        unsigned long long base = 0;
        if (lane == 0)
            base = atomicAdd(reinterpret_cast<unsigned long long *>(&C.ctr[CT_ALLOC]),
                             (unsigned long long)(total & 0xffffu) | (unsigned long long)(total >> 16) << 32);
        base = __shfl_sync(all, base, 0);
        const uint32_t child0 = 1u + (uint32_t)base + (before & 0xffffu), leaf0 = (uint32_t)(base >> 32) + (before >> 16);
        const bool fits = child0 + __popc(inner) <= C.ncap && leaf0 + __popc(leaf) <= C.entries;
        if (ready && !fits) {                    // (more nodes than a tree of this size has)
            atomicOr(C.err, ST_BAD_TREE);
            C.ctr[CT_STOP] = 1u;
        }
        if (ready && fits) {
            // the grid and the slot's bytes
            uint8_t *out = reinterpret_cast<uint8_t *>(C.nodes + 5 * (size_t)idx);
            uint32_t field[3];
            float p[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const float l0 = __fsub_rd(lo[a], pad), h0 = __fadd_ru(hi[a], pad);
                field[a] = scale_field(l0, h0);
                const float step = __uint_as_float(field[a] << 23);
                p[a] = __fsub_rd(l0, step);
                const double per = (double)__uint_as_float((254u - field[a]) << 23);   // 1 / step
                const double l = ((double)c.lo[a] - pad - (double)p[a]) * per - 0x1p-6;
                const double h = ((double)c.hi[a] + pad - (double)p[a]) * per + 0x1p-6;
                out[32 + 8 * a + slot] = have ? (uint8_t)fmin(fmax(floor(l), 0.0), 255.0) : (uint8_t)255;
                out[56 + 8 * a + slot] = have ? (uint8_t)fmin(fmax(ceil(h), 0.0), 255.0) : (uint8_t)0;
            }
            if (s == 0u) {
                C.nodes[5 * (size_t)idx] =
                    make_float4(p[0], p[1], p[2], __uint_as_float(field[0] | field[1] << 8 | field[2] << 16 | inner << 24));
                uint32_t *w = reinterpret_cast<uint32_t *>(out) + 4;
                w[0] = child0;
                w[1] = leaf0;
                w[2] = leaf;                     // (the last word is the root's alone: above)
            }
            if (c.kind == K_ENTRY) {
                const uint32_t at = leaf0 + __popc(leaf & ((1u << slot) - 1u)), id = __ldg(&C.aux[c.ref]);
                float4 q = make_float4(0, 0, 0, 0), u = q, v = q;
                if (id >= C.nprims && id - C.nprims < C.ntris) {
                    const float4 *t = C.tris + 3 * (size_t)(id - C.nprims);
                    q = __ldg(t);
                    u = __ldg(t + 1);
                    v = __ldg(t + 2);
                } else if (id >= C.nprims) {
                    atomicOr(C.err, ST_BAD_TREE);
                }
                q.w = __uint_as_float(id);
                C.leaves[3 * (size_t)at] = q;
                C.leaves[3 * (size_t)at + 1] = u;
                C.leaves[3 * (size_t)at + 2] = v;
            } else if (have) {
                *(volatile uint32_t *)&C.items[child0 + __popc(inner & ((1u << slot) - 1u))] = c.ref + 1u;
            }
        }
        made += __popc(__ballot_sync(all, ready && s == 0u));
        if (ready) claimed = false;
    }
}

// ---- the queries ---------------------------------------------------------------------------------
// A block takes `chunk` rays; its lanes whose ray is done take the block's next ones once fewer than
// WD_REFILL of a warp's lanes are at work (the walks of a warp's rays differ in length several times
// over).
constexpr int WD_REFILL = 20;
constexpr uint32_t WD_CHUNK = 2048;
// Up to this many rays 8 lanes walk a ray: with fewer rays than the chip holds lanes the walks' length
// decides, not their number (closest hits over 4M triangles, 8 lanes a ray and one: 20480 rays 330 and
// 294 us, 32768 417 and 340; over 20k triangles 57 and 55, 71 and 57).
constexpr uint64_t WD_EIGHT_LANES_TO = 1u << 14;

struct Query {
    WideScene W;
    TraceTables tt;                              // the binary tree
    const float *orig, *dir, *tmaxs;             // (tmaxs: any hit)
    uint64_t n;
    float tmin, tmax;
    int32_t *prim;
    float *t;
    uint8_t *blocked;
    uint32_t chunk;
    uint32_t *err;
};

// a triangle's leaf entry (the scenes of the queries hold nothing else)
struct TriLeaf {
    __device__ __forceinline__ bool operator()(uint32_t, float4 q, const float4 *lp, const WideRay &r, float tmin, float tmax,
                                               float &t) const {
        return wide_tri(q, __ldg(lp + 1), __ldg(lp + 2), r.o, r.d, tmin, tmax, t);
    }
};

__device__ __forceinline__ V3 query_v3(const float *p, uint64_t i) { return v3(p[3 * i], p[3 * i + 1], p[3 * i + 2]); }
__device__ __forceinline__ WideRay query_ray(const Query &Q, uint64_t i) { return wide_ray(query_v3(Q.orig, i), query_v3(Q.dir, i)); }
// Whether the wide walk tests all that the binary walk meets: both find a box within 4 (|o| + m) 2^-24 in all (m: the
// tree's largest coordinate; the binary slab test rounds once, the wide one three times), and the wide boxes are
// WD_WIDEN_TIGHT = 2^-16 of m larger, so for origins within 60 m. (Rays from farther off take the binary walk,
// whose rounding loses hits there too: the same ones.)
__device__ __forceinline__ bool query_plain(const Query &Q, const WideRay &r) {
    const float4 *root = reinterpret_cast<const float4 *>(Q.tt.nodes + Q.tt.root);
    const float4 l = __ldg(root), h = __ldg(root + 1);
    const float m = fmaxf(fmaxf(fmaxf(fabsf(l.x), fabsf(l.y)), fmaxf(fabsf(l.z), fabsf(h.x))), fmaxf(fabsf(h.y), fabsf(h.z)));
    return wide_plain(r.o, r.d) && fmaxf(fmaxf(fabsf(r.o.x), fabsf(r.o.y)), fabsf(r.o.z)) <= 60.0f * m;
}

// ray i through the binary tree: where two triangles are hit at the same t (the binary walk's order
// decides), and where the tree is not walked wide. Its stack is as deep as traverse.cu's, that the queries
// of any tree are answered as they are there (LBVH trees over 63-bit keys reach 93 levels).
constexpr int QUERY_STACK = 96;
template <bool ANY>
__device__ __noinline__ void query_binary(const Query &Q, uint64_t i) {
    float best = ANY ? Q.tmaxs[i] : Q.tmax;
    int32_t hit = -1;
    const V3 o = query_v3(Q.orig, i), d = query_v3(Q.dir, i);
    bvh_walk<false, QUERY_STACK>(reinterpret_cast<const float4 *>(Q.tt.nodes), Q.tt.root, Q.tt.nnodes, Q.tt.aux, Q.tt.naux, o, d, Q.tmin,
                    best, Q.err, [&](uint32_t id) {
        if (id >= Q.tt.ntris) { atomicOr(Q.err, ST_BAD_TREE); return true; }
        float t;
        if (!hit_tri_t(Q.tt.tris + 3 * (size_t)id, o, d, Q.tmin, best, t)) return false;
        best = t;
        hit = (int32_t)id;
        return ANY;
    });
    if (ANY) {
        Q.blocked[i] = hit >= 0 ? 1 : 0;
    } else {
        Q.prim[i] = hit;
        Q.t[i] = hit >= 0 ? best : -1.0f;
    }
}

template <bool ANY>
__device__ __forceinline__ void query_done(const Query &Q, uint64_t i, int32_t hit, float best, bool tie) {
    if (tie) {
        query_binary<ANY>(Q, i);
    } else if (ANY) {
        Q.blocked[i] = hit >= 0 ? 1 : 0;
    } else {
        Q.prim[i] = hit;
        Q.t[i] = hit >= 0 ? best : -1.0f;
    }
}

template <bool ANY>
__global__ void __launch_bounds__(WD_THREADS, 8) wide_query_kernel(const __grid_constant__ Query Q) {
    constexpr int32_t TIE = (int32_t)0x80000000;
    constexpr uint8_t ASK = 2;
    __shared__ uint32_t s_next, s_tie;
    const uint32_t all = 0xffffffffu, lane = threadIdx.x & 31u;
    const uint64_t first = (uint64_t)blockIdx.x * Q.chunk;
    const uint32_t n = (uint32_t)(Q.n - first < Q.chunk ? Q.n - first : Q.chunk);
    if (!wide_walked(Q.W)) {
        for (uint32_t k = threadIdx.x; k < n; k += WD_THREADS) query_binary<ANY>(Q, first + k);
        return;
    }
    if (threadIdx.x == 0) s_next = s_tie = 0;
    __syncthreads();
    uint2 stack[WD_STACK];
    WideRay r = wide_ray(v3(0, 0, 0), v3(0, 0, 0));
    WideWalk w;
    wide_begin(w, 0.0f);
    uint64_t i = 0;
    bool at = false, more = true;
    bool over = false;
    while (!over) {
        uint32_t m = __ballot_sync(all, at);
        if (more && __popc(m) < WD_REFILL) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&s_next, (uint32_t)__popc(~m));
            base = __shfl_sync(all, base, 0);
            more = base + __popc(~m) < n;
            if (!at) {
                const uint32_t k = base + __popc(~m & ((1u << lane) - 1u));
                if (k < n) {
                    at = true;
                    i = first + k;
                    r = query_ray(Q, i);
                    wide_begin(w, ANY ? Q.tmaxs[i] : Q.tmax);
                    if (!query_plain(Q, r)) wide_odd(w);
                }
            }
            m = __ballot_sync(all, at);
        }
        over = !m;
        if (at && wide_step<ANY, false>(Q.W, r, w, stack, Q.tmin, __popc(m), Q.err, TriLeaf{})) {
            at = false;
            if (!w.tie) {
                query_done<ANY>(Q, i, w.hit, w.best, false);
            } else {
                if (ANY) Q.blocked[i] = ASK;
                else Q.prim[i] = TIE;
                s_tie = 1;
            }
        }
    }
    // (the binary walk's code and registers stay out of the loop above)
    __syncthreads();
    if (s_tie)
        for (uint32_t k = threadIdx.x; k < n; k += WD_THREADS)
            if (ANY ? Q.blocked[first + k] == ASK : Q.prim[first + k] == TIE) query_binary<ANY>(Q, first + k);
}

template <bool ANY>
__global__ void __launch_bounds__(WD_THREADS, 8) wide_query8_kernel(const __grid_constant__ Query Q) {
    const uint64_t i = ((uint64_t)blockIdx.x * WD_THREADS + threadIdx.x) >> 3;
    if (i >= Q.n) return;
    const bool one = (threadIdx.x & 7u) == 0u;
    const WideRay r = query_ray(Q, i);
    if (!wide_walked(Q.W) || !query_plain(Q, r)) {
        if (one) query_binary<ANY>(Q, i);
        return;
    }
    float best = ANY ? Q.tmaxs[i] : Q.tmax;
    bool tie;
    const int32_t hit = wide_walk8<ANY>(Q.W, r, Q.tmin, best, tie, Q.err, TriLeaf{});
    if (one) query_done<ANY>(Q, i, hit, best, tie);
}

// the closest-hit walk's box tests in halves of 32-byte records (an 80-byte node: 5) and triangle tests: [0] and [1];
// of the binary walk where that is walked
__global__ void __launch_bounds__(WD_THREADS) wide_count_kernel(const __grid_constant__ Query Q, unsigned long long *stats) {
    const uint64_t i = (uint64_t)blockIdx.x * WD_THREADS + threadIdx.x;
    uint32_t cnt[2] = {0, 0};
    if (i < Q.n) {
        const WideRay r = query_ray(Q, i);
        if (wide_walked(Q.W) && query_plain(Q, r)) {
            WideWalk w;
            wide_begin(w, Q.tmax);
            wide_run<false, true>(Q.W, r, w, Q.tmin, Q.err, TriLeaf{}, cnt);
            cnt[0] *= 5u;
        } else {
            float best = Q.tmax;
            bvh_walk<true, QUERY_STACK>(reinterpret_cast<const float4 *>(Q.tt.nodes), Q.tt.root, Q.tt.nnodes, Q.tt.aux, Q.tt.naux,
                                        r.o, r.d, Q.tmin, best, Q.err, [&](uint32_t id) {
                if (id >= Q.tt.ntris) { atomicOr(Q.err, ST_BAD_TREE); return true; }
                float t;
                if (hit_tri_t(Q.tt.tris + 3 * (size_t)id, r.o, r.d, Q.tmin, best, t)) best = t;
                return false;
            }, cnt);
            cnt[0] *= 2u;
        }
    }
    unsigned long long a = cnt[0], b = cnt[1];
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0 && (a | b)) {
        atomicAdd(&stats[0], a);
        atomicAdd(&stats[1], b);
    }
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }

// Wide nodes of a tree with naux leaf entries: with one entry a leaf a node has 8 children, or all of
// its subtree's entries (2 to 7): at most 4 / 7 of the entries; else fewer than the entries.
uint32_t node_cap(uint32_t naux, bool single) { return single ? (uint32_t)((uint64_t)naux * 4 / 7 + 2) : naux + 1; }

template <bool ANY>
cudaError_t query(Query &Q, cudaStream_t st) {
    if (!Q.n) return cudaSuccess;
    if (Q.n <= WD_EIGHT_LANES_TO) {
        wide_query8_kernel<ANY><<<(unsigned)((Q.n * 8 + WD_THREADS - 1) / WD_THREADS), WD_THREADS, 0, st>>>(Q);
        return cudaGetLastError();
    }
    // A block's rays: enough to refill from, few enough that the last blocks end together (1M rays on 20k
    // triangles: 256 a block 0.57 ms, 864 0.63).
    Q.chunk = (uint32_t)std::min<uint64_t>(WD_CHUNK, std::max<uint64_t>(WD_THREADS, Q.n / 4096 / 32 * 32));
    wide_query_kernel<ANY><<<(unsigned)((Q.n + Q.chunk - 1) / Q.chunk), WD_THREADS, 0, st>>>(Q);
    return cudaGetLastError();
}

}  // namespace

size_t wide_bytes(uint32_t naux, bool single) {
    const size_t cap = node_cap(naux, single);
    return up256(cap * 80) + up256((size_t)naux * 48) + up256(cap * 4) + 256;
}

WideScene wide_view(void *buf, uint32_t naux, bool single) {
    WideScene W{};
    W.nnodes = node_cap(naux, single);
    W.nleaves = naux;
    W.nodes = static_cast<const float4 *>(buf);
    W.leaves = reinterpret_cast<const float4 *>(static_cast<char *>(buf) + up256((size_t)W.nnodes * 80));
    return W;
}

cudaError_t wide_build_part(const Node *d_bin, uint32_t root, uint32_t nn, const uint32_t *d_aux, uint32_t naux,
                            uint32_t entries, uint32_t nprims, const float *d_tris, uint32_t ntris, float widen, void *buf,
                            bool single, uint32_t *d_wild, uint32_t *d_status, int num_sms, cudaStream_t st) {
    if (!nn || !entries) return cudaErrorInvalidValue;
    const WideScene W = wide_view(buf, entries, single);
    Collapse C{};
    C.bin = d_bin;
    C.root = root;
    C.nn = nn;
    C.aux = d_aux;
    C.naux = naux;
    C.entries = entries;
    C.widen = widen;
    C.tris = reinterpret_cast<const float4 *>(d_tris);
    C.nprims = nprims;
    C.ntris = ntris;
    C.nodes = const_cast<float4 *>(W.nodes);
    C.ncap = W.nnodes;
    C.wild = d_wild ? d_wild : static_cast<uint32_t *>(buf) + 7;
    C.leaves = const_cast<float4 *>(W.leaves);
    char *items = static_cast<char *>(buf) + up256((size_t)C.ncap * 80) + up256((size_t)entries * 48);
    const size_t item_bytes = up256((size_t)C.ncap * 4);
    C.items = reinterpret_cast<uint32_t *>(items);
    C.ctr = reinterpret_cast<uint32_t *>(items + item_bytes);
    C.err = d_status;
    cudaError_t e = cudaMemsetAsync(items, 0, item_bytes + 256, st);
    if (!e) e = cudaMemsetAsync(buf, 0, 80, st);
    if (e) return e;
    // 16 nodes a block at once; no more blocks than are resident together (they wait for one another's nodes)
    const uint32_t blocks = std::min<uint32_t>((uint32_t)num_sms * 4u, std::max<uint32_t>(entries / 64u, 1u));
    collapse_kernel<<<blocks, WD_THREADS, 0, st>>>(C);
    return cudaGetLastError();
}

cudaError_t wide_build(const Node *d_bin, uint32_t nn, const uint32_t *d_aux, uint32_t naux, uint32_t nprims,
                       const float *d_tris, uint32_t ntris, float widen, void *buf, bool single, uint32_t *d_status, int num_sms,
                       cudaStream_t st) {
    return wide_build_part(d_bin, 0, nn, d_aux, naux, naux, nprims, d_tris, ntris, widen, buf, single, nullptr, d_status, num_sms,
                           st);
}

cudaError_t wide_intersect(const WideScene &W, const TraceTables &tt, const float *d_orig, const float *d_dir, uint64_t nrays,
                           float tmin, float tmax, int32_t *d_prim, float *d_t, uint32_t *d_status, cudaStream_t st) {
    Query Q{};
    Q.W = W;
    Q.tt = tt;
    Q.orig = d_orig;
    Q.dir = d_dir;
    Q.n = nrays;
    Q.tmin = tmin;
    Q.tmax = tmax;
    Q.prim = d_prim;
    Q.t = d_t;
    Q.err = d_status;
    return query<false>(Q, st);
}

cudaError_t wide_occluded(const WideScene &W, const TraceTables &tt, const float *d_orig, const float *d_dir,
                          const float *d_tmax, uint64_t nrays, float tmin, uint8_t *d_out, uint32_t *d_status,
                          cudaStream_t st) {
    Query Q{};
    Q.W = W;
    Q.tt = tt;
    Q.orig = d_orig;
    Q.dir = d_dir;
    Q.tmaxs = d_tmax;
    Q.n = nrays;
    Q.tmin = tmin;
    Q.blocked = d_out;
    Q.err = d_status;
    return query<true>(Q, st);
}

cudaError_t wide_count(const WideScene &W, const TraceTables &tt, const float *d_orig, const float *d_dir, uint64_t nrays,
                       float tmin, float tmax, unsigned long long *d_stats, uint32_t *d_status, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(d_stats, 0, 16, st);
    if (e || !nrays) return e;
    Query Q{};
    Q.W = W;
    Q.tt = tt;
    Q.orig = d_orig;
    Q.dir = d_dir;
    Q.n = nrays;
    Q.tmin = tmin;
    Q.tmax = tmax;
    Q.err = d_status;
    wide_count_kernel<<<(unsigned)((nrays + WD_THREADS - 1) / WD_THREADS), WD_THREADS, 0, st>>>(Q, d_stats);
    return cudaGetLastError();
}

}  // namespace lrc
