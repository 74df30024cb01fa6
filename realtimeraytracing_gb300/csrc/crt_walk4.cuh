// The 64-byte compressed 4-wide nodes and the persistent closest-hit / any-hit
// walk over them (crt_trace.cu).  Compiled with -fmad=false.
//
// Record of binary internal node i: its subtree's top opened twice, the internal
// child of largest area first, so up to four children.  The array is indexed by the
// binary rank; a walk enters at rank 0 and follows references, so the records of
// ranks that were opened away lie between those it reads.
//   words 0-2   origin (minimum corner over the children) * 2^-60
//   words 3, 10, 11  step * 2^73 per axis (a power of two)
//   words 4-9   8-bit steps of the children's planes: min x, y, z, max x, y, z;
//               byte c of a word belongs to child c
//   words 12-15 child references (leaf flag | place in tree order, or rank;
//               kNoChild in an empty slot, whose planes are inverted)
// The planes origin + q * step enclose, as real numbers, the child's box grown
// by 4 * abs_eps (crt_build.cu rounds every step outward).
//
// Decoding.  A float whose bits are q << 16 is exactly q * 2^-133 (denormal up
// to q = 127, the first normals above, same spacing), so one byte permute and
// one fused multiply-add give a slab distance with a single rounding: with
// R = 2^-40 / d, A = step * 2^73 * R and B = origin * 2^-60 * R - o * 2^-60 * R,
// fma(q * 2^-133, A, B) is the distance times 2^-100.  All distances the walk
// compares (entry distances, the pruning bound) carry that factor.
//
// Exactness.  B and the product round once each, as slab_wt's form does; with
// origins within 8 times the scene's range the error stays below
// 26 * 2^-24 of that range, and the shader's own slab form adds at most
// 18 * 2^-24, both inside the 4 * abs_eps = 2^-18 the boxes are grown by.
// So every box the binary walk enters is entered here, and
//   * the watertight predicate needs no more (its hits do not depend on boxes);
//   * the shader's predicate tests a leaf only if its exact box passes the
//     shader's slab test (leaf_box_passes), which is the shader's tested set.
// A ray parallel to an axis plane (1/d infinite) meets the shader's NaNs where a
// box plane passes through its origin.  They reject a box of which every box
// inside is rejected too, but for leaves flat in the ray's own plane, whose
// triangles the shader's predicate rejects (a = 0): the tested leaves that can
// hit are still those whose own box passes.
// That holds for trees whose leaf boxes are their triangles' and whose children lie
// inside their parents, as builds and refits make them; other imported trees keep to
// the binary nodes (crt_import.cu).  Rays outside that range (far origins, extreme
// scales, negative tmin), scenes whose boxes cannot be quantised and walks that
// outgrow their stack are left to the binary walk: closest hits to trace_pool_kernel
// (crt_pool.cuh), any hits and pixels to a thread each.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "crt_build.cuh"
#include "crt_common.cuh"
#include "crt_traverse.cuh"

namespace crt {

struct Walk4Node {
    float ox, oy, oz, sx, sy, sz;
    uint32_t nx, ny, nz, xx, xy, xz;
    uint32_t ref[4];
};

__device__ __forceinline__ Walk4Node load_walk4(const uint4* __restrict__ node) {
    uint32_t w[16];
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
        : "l"(node));
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(w[8]), "=r"(w[9]), "=r"(w[10]), "=r"(w[11]), "=r"(w[12]), "=r"(w[13]), "=r"(w[14]), "=r"(w[15])
        : "l"(node + 2));
    Walk4Node n;
    n.ox = __uint_as_float(w[0]);
    n.oy = __uint_as_float(w[1]);
    n.oz = __uint_as_float(w[2]);
    n.sx = __uint_as_float(w[3]);
    n.sy = __uint_as_float(w[10]);
    n.sz = __uint_as_float(w[11]);
    n.nx = w[4]; n.ny = w[5]; n.nz = w[6];
    n.xx = w[7]; n.xy = w[8]; n.xz = w[9];
#pragma unroll
    for (int c = 0; c < 4; ++c) n.ref[c] = w[12 + c];
    return n;
}

constexpr float kWalk4TScale = 7.888609052210118e-31f;  // 2^-100: slab distances
constexpr float kWalk4RScale = 9.094947017729282e-13f;  // 2^-40: 1/d
constexpr float kWalk4OScale = 8.673617379884035e-19f;  // 2^-60: origins

// A ray's constants: R = 2^-40 / d per axis and -(o * 2^-60) * R.
struct Walk4Ray {
    float rx, ry, rz;
    float bx, by, bz;
};

// False: this ray takes the binary walk.  Components below 2^-40 of the largest
// count as that much: over the scene (t * |d| <= 10 ranges) it moves the ray by
// 10 * 2^-40 of the range, far inside the boxes' growth.
__device__ __forceinline__ bool walk4_setup(Walk4Ray& w, float3 o, float3 d, float tmin, float abs_eps) {
    const float range = abs_eps * 1048576.f;  // largest coordinate or extent (scene_abs_eps)
    const float far = fmaxf(fabsf(o.x), fmaxf(fabsf(o.y), fabsf(o.z)));
    const float big = fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z)));
    const float least = big * 9.094947017729282e-13f;
    w.rx = kWalk4RScale / copysignf(fmaxf(fabsf(d.x), least), d.x);
    w.ry = kWalk4RScale / copysignf(fmaxf(fabsf(d.y), least), d.y);
    w.rz = kWalk4RScale / copysignf(fmaxf(fabsf(d.z), least), d.z);
    w.bx = -((o.x * kWalk4OScale) * w.rx);
    w.by = -((o.y * kWalk4OScale) * w.ry);
    w.bz = -((o.z * kWalk4OScale) * w.rz);
    // NaNs fail the comparisons or the tests after them; range / big, the distance
    // unit, lies in 2^-20 .. 2^20, so every product above and below is normal
    return tmin >= 0.f && far <= 8.f * range && big <= range * 1048576.f && range <= big * 1048576.f &&
           isfinite(o.x) && isfinite(o.y) && isfinite(o.z) && !isnan(d.x) && !isnan(d.y) && !isnan(d.z);
}

// Distance of the plane in byte C of word; SAT: clamped to [0, 1], which is free
// (distances carry 2^-100, so only negative ones, and NaN, change: to 0).  Steps
// stored as floats instead of exponent bytes, this clamp and three-operand minima
// take 17 ALU operations off a visit: 1920x1080 frames with shadow rays over 1.31 M
// triangles 838 -> 795 us, 8.4 M bounce rays 6.32 -> 6.16 ms (memory latency bounds those).
template <int C, bool SAT = false>
__device__ __forceinline__ float walk4_plane(uint32_t word, float a, float b) {
    // byte C of word to bits 16-23, zeros elsewhere
    const float q = __uint_as_float(__byte_perm(word, 0u, 0x4044u | (static_cast<uint32_t>(C) << 8)));
    if (!SAT) return __fmaf_rn(q, a, b);
    float t;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(q), "f"(a), "f"(b));
    return t;
}

// Entry distance (clamped to 0) of child C if the ray meets its box no farther
// than bound, else +inf.
template <int C>
__device__ __forceinline__ float walk4_child(const uint32_t (&near)[3], const uint32_t (&far)[3], const float (&a)[3],
                                             const float (&b)[3], float bound) {
    const float t0 = fmaxf(fmaxf(walk4_plane<C, true>(near[0], a[0], b[0]), walk4_plane<C>(near[1], a[1], b[1])),
                           walk4_plane<C>(near[2], a[2], b[2]));
    const float t1 = fminf(fminf(fminf(walk4_plane<C>(far[0], a[0], b[0]), walk4_plane<C>(far[1], a[1], b[1])),
                                 walk4_plane<C>(far[2], a[2], b[2])), bound);
    return t0 <= t1 ? t0 : __int_as_float(0x7F800000);
}

__device__ __forceinline__ void walk4_children(const Walk4Node& n, const Walk4Ray& w, float bound, float (&t)[4]) {
    const float a[3] = {n.sx * w.rx, n.sy * w.ry, n.sz * w.rz};
    const float b[3] = {__fmaf_rn(n.ox, w.rx, w.bx), __fmaf_rn(n.oy, w.ry, w.by), __fmaf_rn(n.oz, w.rz, w.bz)};
    const bool sx = w.rx < 0.f, sy = w.ry < 0.f, sz = w.rz < 0.f;
    const uint32_t near[3] = {sx ? n.xx : n.nx, sy ? n.xy : n.ny, sz ? n.xz : n.nz};
    const uint32_t far[3] = {sx ? n.nx : n.xx, sy ? n.ny : n.xy, sz ? n.nz : n.xz};
    t[0] = walk4_child<0>(near, far, a, b, bound);
    t[1] = walk4_child<1>(near, far, a, b, bound);
    t[2] = walk4_child<2>(near, far, a, b, bound);
    t[3] = walk4_child<3>(near, far, a, b, bound);
}

// Orders the four (distance, reference) pairs, nearest first (FARTHEST: the
// farthest met child first); missed children (+inf) go last either way.
template <bool FARTHEST>
__device__ __forceinline__ void walk4_sort(float (&t)[4], uint32_t (&r)[4]) {
    const float inf = __int_as_float(0x7F800000);
    if (FARTHEST)
#pragma unroll
        for (int c = 0; c < 4; ++c) t[c] = t[c] == inf ? inf : -t[c];
#define CRT_CSWAP(x, y)                                   \
    {                                                     \
        const bool s = t[y] < t[x];                       \
        const float tx = t[x], ty = t[y];                 \
        const uint32_t rx = r[x], ry = r[y];              \
        t[x] = s ? ty : tx; t[y] = s ? tx : ty;           \
        r[x] = s ? ry : rx; r[y] = s ? rx : ry;           \
    }
    CRT_CSWAP(0, 1) CRT_CSWAP(2, 3) CRT_CSWAP(0, 2) CRT_CSWAP(1, 3) CRT_CSWAP(1, 2)
#undef CRT_CSWAP
}

// The shader's predicate tests a leaf only if its exact box (that of its
// stored triangle) passes the shader's slab test.
__device__ __forceinline__ bool leaf_box_passes(const RayCtx& r, float4 a, float4 b, float4 c, float bound) {
    const float4 mn = make_float4(min_std(a.x, min_std(b.x, c.x)), min_std(a.y, min_std(b.y, c.y)),
                                  min_std(a.z, min_std(b.z, c.z)), 0.f);
    const float4 mx = make_float4(max_std(a.x, max_std(b.x, c.x)), max_std(a.y, max_std(b.y, c.y)),
                                  max_std(a.z, max_std(b.z, c.z)), 0.f);
    float te;
    return slab<false>(r, mn, mx, 0.f, te) && te <= bound;
}

// The binary walk of one ray (see the head of this file).
template <bool ANY, bool WT, int STACK>
__device__ __noinline__ uint4 trace_binary(const TraceParams& p, uint32_t i, float4 r0, float4 r1) {
    return trace_one<ANY, WT, STACK, false, 0>(p, i, r0, r1);
}

// Stack entries in shared memory per thread, entries beyond them in local
// memory, blocked lanes that start the warp's leaf tests, idle lanes that
// refill, resident blocks per SM.  GB300, 8.4 M bounce rays over 4.19 M triangles
// in caller order (64 uneven scenes built and traced): 14 / 20 / 22 entries 8.17 /
// 6.67 / 6.53 ms (28 drop a resident block: 10.8); leaf tests at 3 / 4 / 6 / 12
// lanes 6.67 / 6.67 / 6.78 / 7.56; refill at 4 / 6 / 8 / 12 idle lanes 6.68 / 6.63
// / 6.67 / 7.43 (6.79 / 6.64 / 6.60 / 7.25); two or three pops per step instead
// of one 7.05 / 7.49; 56 registers for 9 blocks per SM with 18 entries 6.54 (6.73).
constexpr int kWalk4Shared = 22, kWalk4Local = 64, kWalk4Flush = 4, kWalk4Refill = 6, kWalk4Blocks = 8;
constexpr int kWalk4Block = 128;
constexpr uint32_t kWalk4Row = kWalk4Block * 8, kWalk4Spill = 8;
static_assert(kWalk4Shared >= kWalk4Spill + 4 && kWalk4Local % kWalk4Spill == 0, "stack shape");

// The scene whose ray range holds ray i.
__device__ __forceinline__ uint32_t batch_scene_of(const uint32_t* ray_off, uint32_t n_scenes, uint32_t i) {
    uint32_t lo = 0, hi = n_scenes - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (ray_off[mid] <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ uint2 walk4_lds(uint32_t a) {
    uint2 e;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(e.x), "=r"(e.y) : "r"(a));
    return e;
}
__device__ __forceinline__ void walk4_sts(uint32_t a, uint2 e) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(e.x), "r"(e.y) : "memory");
}

// One lane's walk.  cur: the internal node to visit next, or -1 (pop one); pend:
// a parked leaf.  The stack's newest entries sit in shared memory (a column per
// thread, so any mix of depths is free of bank conflicts), older ones move to
// local memory eight at a time.  An entry is (reference, entry distance).
// Closest hit: the low two distance bits count the siblings pushed just below it,
// which are farther, so one too-far entry drops them all (the count can raise a
// distance by 3 ulp, far inside the bound's slack of 2^-14).  Any hit: the
// siblings below are nearer and the bound stays where it was when they were
// pushed, so entries are taken without another look at their distance.
struct Walk4Lane {
    static constexpr uint32_t kNoLeaf = 0xFFFFFFFFu;
    const uint4* cw;      // the scene: nodes, leaf triangles, slack
    const float4* xtri;
    float abs_eps;
    Walk4Ray w;           // the ray
    WRay wt;
    float3 o, d;
    float tmin;
    float bt, bu, bv, bound;  // best hit (bt: tmax until there is one), pruning bound
    uint32_t btri, bleaf;     // bleaf: the shader's tie order
    int cur;
    uint32_t pend, top, spilled;
    float pend_t;
    bool redo;                // the walk outgrew its stack: to be done on the binary nodes
    uint32_t fetched, tested; // nodes and triangles (walk4_run with COUNT)

    __device__ __forceinline__ void stop(uint32_t s_base) {
        cur = -1;
        top = s_base;
        spilled = 0;
        pend = kNoLeaf;
    }
    __device__ __forceinline__ void set_bound() { bound = prune_bound(bt, abs_eps) * kWalk4TScale; }
    // Starts ray (r0, r1) at the root (whose children are tested, not its own
    // box); false for a ray of the binary walk, which is then stopped.
    template <bool WT>
    __device__ __forceinline__ bool start(uint32_t s_base, float4 r0, float4 r1, bool walkable) {
        o = make_float3(r0.x, r0.y, r0.z);
        d = make_float3(r1.x, r1.y, r1.z);
        tmin = r0.w;
        bt = r1.w;
        bu = bv = 0.f;
        btri = CRT_MISS;
        redo = false;
        stop(s_base);
        set_bound();
        if (WT) wt = wt_setup(d);
        if (!(tmin <= bt)) return true;  // an empty ray
        if (!walk4_setup(w, o, d, tmin, abs_eps) || !walkable) return false;
        cur = 0;
        return true;
    }
    template <bool WT>
    __device__ __forceinline__ void test_leaf(uint32_t leaf) {
        if (leaf == kNoChild) return;  // an empty slot whose planes collapsed in rounding
        const uint32_t L = leaf & ~kLeafRef;
        const float4* t = xtri + 3 * static_cast<size_t>(L);
        const float4 a = __ldg(t), b = __ldg(t + 1), c = __ldg(t + 2);
        if (!WT) {
            RayCtx r;
            r.o = o;
            r.d = d;
            r.inv = make_float3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
            r.exact = !(isfinite(r.inv.x) && isfinite(r.inv.y) && isfinite(r.inv.z));
            if (!leaf_box_passes(r, a, b, c, prune_bound(bt, abs_eps))) return;
        }
        const float3 A = make_float3(a.x, a.y, a.z), B = make_float3(b.x, b.y, b.z), C = make_float3(c.x, c.y, c.z);
        // accepted only up to the best hit (bt <= tmax)
        const HitRes h = WT ? tri_watertight(o, tmin, bt, wt, A, B, C) : tri_reference(o, d, tmin, bt, A, B, C);
        if (!h.did) return;
        const uint32_t tri = __float_as_uint(a.w);
        if (btri == CRT_MISS || h.t < bt || (h.t == bt && (WT ? tri < btri : L > bleaf))) {
            bt = h.t; bu = h.u; bv = h.v; btri = tri;
            if (!WT) bleaf = L;
            set_bound();
        }
    }
    __device__ __forceinline__ uint4 hit() const {
        return btri != CRT_MISS ? make_uint4(btri, __float_as_uint(bt), __float_as_uint(bu), __float_as_uint(bv))
                                : make_uint4(CRT_MISS, 0u, 0u, 0u);
    }
};

// Steps the warp's walks until at least `limit` lanes are over (lanes without a
// ray are) and returns their mask.  In a step each lane without a node pops one
// stack entry: an internal node becomes cur, the first leaf is parked, a second
// leaf stays on the stack and blocks the lane; then each lane with a node visits
// it.  The warp tests its parked leaves together once FLUSH lanes are blocked (or
// hold one with nothing else left), or no lane has a node.
// s_base: the lane's first shared entry (the row below it is readable).
template <bool ANY, bool WT, int FLUSH, bool COUNT = false>
__device__ __forceinline__ uint32_t walk4_run(Walk4Lane& L, uint32_t s_base, uint2* __restrict__ st, int limit) {
    constexpr uint32_t kRow = kWalk4Row, kNoLeaf = Walk4Lane::kNoLeaf;
#pragma unroll 1
    while (true) {
        bool blocked = false, over = false;
        if (L.cur < 0) {
            if (L.spilled) {  // rare: older entries come back
                if (L.top == s_base) {
                    const uint32_t n = min(L.spilled, kWalk4Spill);
                    L.spilled -= n;
                    for (uint32_t k = 0; k < n; ++k, L.top += kRow) walk4_sts(L.top, st[L.spilled + k]);
                }
            }
            const uint2 e = walk4_lds(L.top - kRow);
            const bool some = L.top != s_base, full = L.pend != kNoLeaf;
            const bool near = ANY || __uint_as_float(e.y) <= L.bound;
            const bool leaf = static_cast<int>(e.x) < 0;
            blocked = full && (!some || (near && leaf));
            over = !some && !full;
            if (some && near && !leaf) L.cur = static_cast<int>(e.x);
            if (some && near && leaf && !full) {
                L.pend = e.x;
                L.pend_t = __uint_as_float(e.y);
            }
            uint32_t drop = near ? kRow : kRow + kRow * (e.y & 3u);
            if (!some || blocked) drop = 0u;
            if (L.spilled) {  // rare: some of the siblings were moved
                const uint32_t have = L.top - s_base;
                if (have < drop) {
                    L.spilled -= (drop - have) / kRow;
                    drop = have;
                }
            }
            L.top -= drop;
        }
        const uint32_t wm = __ballot_sync(0xFFFFFFFFu, L.cur >= 0);
        const uint32_t bm = __ballot_sync(0xFFFFFFFFu, blocked);
        if (__popc(bm) >= FLUSH || !wm) {
            if (L.pend != kNoLeaf) {
                if (ANY || L.pend_t <= L.bound) {
                    L.template test_leaf<WT>(L.pend);
                    if (COUNT) ++L.tested;
                }
                L.pend = kNoLeaf;
                if (ANY && L.btri != CRT_MISS) {
                    L.stop(s_base);
                    over = true;
                }
            }
        }
        const uint32_t om = __ballot_sync(0xFFFFFFFFu, over);
        if (__popc(om) >= limit) return om;
        if (L.cur >= 0) {
            Walk4Node n = load_walk4(L.cw + 4 * static_cast<size_t>(static_cast<uint32_t>(L.cur)));
            if (COUNT) ++L.fetched;
            if (L.top > s_base + (kWalk4Shared - 4) * kRow) {  // rare: the oldest entries move to local memory
                if (L.spilled + kWalk4Spill > kWalk4Local) {
                    L.redo = true;
                    L.stop(s_base);
                    continue;
                }
                for (uint32_t k = 0; k < kWalk4Spill; ++k) st[L.spilled + k] = walk4_lds(s_base + k * kRow);
                for (uint32_t q = s_base; q + kWalk4Spill * kRow < L.top; q += kRow)
                    walk4_sts(q, walk4_lds(q + kWalk4Spill * kRow));
                L.top -= kWalk4Spill * kRow;
                L.spilled += kWalk4Spill;
            }
            float t[4];
            walk4_children(n, L.w, L.bound, t);
            walk4_sort<ANY>(t, n.ref);
            const float inf = __int_as_float(0x7F800000);
            uint32_t below = 0;
            // each entry is stored where the next one goes unless it counts: four rows are free above top
#pragma unroll
            for (int c = 3; c >= 1; --c) {
                walk4_sts(L.top, make_uint2(n.ref[c], (__float_as_uint(t[c]) & ~3u) | below));
                if (t[c] < inf) {
                    L.top += kRow;
                    if (!ANY) ++below;
                }
            }
            // the nearest child is entered; a leaf goes through the stack
            walk4_sts(L.top, make_uint2(n.ref[0], (__float_as_uint(t[0]) & ~3u) | below));
            const bool met = t[0] < inf;
            L.cur = met ? static_cast<int>(n.ref[0]) : -1;
            if (met && L.cur < 0) L.top += kRow;
        }
    }
}

// A persistent walk's counters in device memory.  The launch's last block zeroes
// them for the next one (no clear in between) and hands the number of rays left
// over (above kWalkLeft they are not all on the list; kWalkAll: it gave up) to the
// device, last_left, and where given to page-locked host memory, with the nodes' bad
// flag after it, so that a caller that waits for the launch anyway starts the kernel
// for them only when there are any, and knows a scene that cannot be quantised from
// then on.
struct Walk4Counters {
    uint32_t taken, left, blocks, last_left, gave_up, pad[3];
};
static_assert(sizeof(Walk4Counters) == kWalkCounterBytes, "walk scratch");

// Puts ray i on the list of what is left to the binary walk (the compiler makes it
// one atomic a warp).  An overflowing list makes a launch give up where what it took
// so far is little use, where 9 in 16 of the first quarter of the rays were left over.
// 4.2 M rays over 4.19 M triangles, 1/64, 1/16, 1/4, 1/2, 3/4 and all of them from far
// away, in runs of neighbours: 3.4, 3.9, 4.3, 5.4, 6.2, 5.9 ms (every other one: 6.2);
// on the binary nodes from the start 5.6 to 5.9.  Giving up from 7 in 16 on costs the
// half 0.8 ms, later than the first quarter up to 2 ms.  On giving up the counter gets
// the number of rays, so that every warp finds nothing more to take.
__device__ __forceinline__ void walk4_leave(Walk4Counters* ctr, uint32_t* __restrict__ left, uint32_t i, uint32_t n_rays) {
    const uint32_t k = atomicAdd(&ctr->left, 1u);
    if (k < kWalkLeft) {
        left[k] = i;
        return;
    }
    const uint32_t taken = *reinterpret_cast<volatile uint32_t*>(&ctr->taken);
    if (k >= taken / 2u + taken / 16u && taken < n_rays / 4u) {
        atomicMax(&ctr->taken, n_rays);
        *reinterpret_cast<volatile uint32_t*>(&ctr->gave_up) = 1u;
    }
}

// The hit record of a ray that was left over, until the binary walk writes its hit
// (a miss otherwise has a distance of 0): where the rays left are more than the list
// holds, these marks are what names them.
constexpr uint32_t kLeftMark = 0x7FFFFFFFu;
__device__ __forceinline__ uint4 left_mark() { return make_uint4(CRT_MISS, kLeftMark, 0u, 0u); }
__device__ __forceinline__ bool left_marked(const crt_hit* hits, uint32_t i) {
    const uint2 h = *reinterpret_cast<const uint2*>(hits + i);
    return h.x == CRT_MISS && h.y == kLeftMark;
}

__device__ __forceinline__ void walk4_finish(Walk4Counters* ctr, uint32_t* host_left, const uint32_t* bad) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicInc(&ctr->blocks, gridDim.x - 1) != gridDim.x - 1) return;
    __threadfence();
    // every other block is done with the counters: three loads in flight at once
    const uint32_t listed = ld_relaxed_u32(&ctr->left), gave_up = ld_relaxed_u32(&ctr->gave_up);
    const uint32_t unquantised = host_left ? __ldg(bad) : 0u;
    const uint32_t n = gave_up != 0u ? kWalkAll : listed;
    if (host_left)  // both words in one store
        *reinterpret_cast<volatile unsigned long long*>(host_left) = static_cast<unsigned long long>(unquantised) << 32 | n;
    ctr->taken = ctr->left = ctr->gave_up = 0u;
    ctr->last_left = n;
}

// Persistent warps over a ray pool, one ray per lane; lanes whose ray is done take
// new rays from the counter once kWalk4Refill of them wait.
//
// What bounds it (ncu, 1 M rays): the ALU pipe (68 % busy: byte permutes,
// minima, selects; issue slots 65 %), about 21 of 32 lanes visiting in a step.
// The walk over the binary nodes with persistent warps it replaces was bound by
// L1 wavefronts (65-70 % busy, one per lane and 16-byte load, four per visit)
// at 12.7 active threads per instruction: 8.4 M bounce rays over 4.19 M
// triangles 12.7 -> 6.5 ms in caller order (660 -> 1290 Mrays/s), 12.2 -> 7.1
// in predicted order with its inference and sort; 1.5 M sorted rays over 0.3 M
// triangles 1.60 -> 1.04 ms.  Any hit, one thread per ray before: 4.2 M rays
// 6.70 -> 2.69 ms.  Walk4Demand (crt_host.h) says when deriving the nodes pays.
//
// Rays the compressed walk cannot take (walk4_setup, unquantised scenes, one-leaf
// trees, walks deeper than the stack) go to the list `left` and are marked.
// ctr (Walk4Counters, zero between launches): the rays taken and left.
template <bool ANY, bool WT, bool BATCH>
__global__ void __launch_bounds__(kWalk4Block, kWalk4Blocks)
    trace_walk4_kernel(const TraceParams p, Walk4Counters* ctr, uint32_t* __restrict__ left, uint32_t* host_left,
                       const BatchScene* __restrict__ scenes, uint32_t n_scenes) {
    constexpr uint32_t kIdle = 0xFFFFFFFFu, kDone = 0xFFFFFFFEu;
    __shared__ uint2 s_st[kWalk4Shared + 1][kWalk4Block];  // row 0 is read (and ignored) below an empty stack
    __shared__ uint32_t s_ray_off[BATCH ? kMaxBatchScenes + 1 : 1];
    __shared__ uint32_t s_bad[BATCH ? kMaxBatchScenes / 32 : 1];  // a bit a scene: unquantised, or one leaf
    if (BATCH) {
        for (uint32_t k = threadIdx.x; k <= n_scenes; k += kWalk4Block)
            s_ray_off[k] = k < n_scenes ? scenes[k].ray_off : scenes[n_scenes - 1].ray_off + scenes[n_scenes - 1].n_rays;
        for (uint32_t k = threadIdx.x; k < kMaxBatchScenes; k += kWalk4Block) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, k < n_scenes && (__ldg(p.cw_bad + k) != 0u || scenes[k].n_tris < 2u));
            if ((k & 31u) == 0u) s_bad[k >> 5] = m;
        }
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t s_base = static_cast<uint32_t>(__cvta_generic_to_shared(&s_st[1][threadIdx.x]));
    uint2 st[kWalk4Local];
    Walk4Lane L{};
    L.cw = p.cwide;
    L.xtri = p.xtri;
    L.abs_eps = p.abs_eps;
    L.stop(s_base);
    bool walkable = !BATCH && __ldg(p.cw_bad) == 0u && p.n_nodes > 2;
    uint32_t i = kIdle;
    bool pool_left = true;
    while (true) {
        const uint32_t need = __ballot_sync(0xFFFFFFFFu, i == kIdle);
        if (need && pool_left) {
            const uint32_t take = static_cast<uint32_t>(__popc(need));
            const int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if (lane == static_cast<uint32_t>(leader)) base = atomicAdd(&ctr->taken, take);
            base = __shfl_sync(0xFFFFFFFFu, base, leader);
            pool_left = base < p.n_rays && p.n_rays - base > take;
            const uint32_t k = base + static_cast<uint32_t>(__popc(need & ((1u << lane) - 1u)));
            if (i == kIdle && k < p.n_rays && k >= base) {
                i = p.order ? __ldg(p.order + k) : k;
                if (i >= p.n_rays) {
                    raise_corrupt(p.err, 7, k, i);
                    i = kIdle;
                } else {
                    if (BATCH) {
                        const uint32_t k_scene = batch_scene_of(s_ray_off, n_scenes, i);
                        const BatchScene bs = scenes[k_scene];
                        L.cw = p.cwide + 4 * static_cast<size_t>(bs.wide_off);
                        L.xtri = p.xtri + 3 * static_cast<size_t>(bs.tri_off);
                        L.abs_eps = bs.abs_eps;
                        walkable = (s_bad[k_scene >> 5] >> (k_scene & 31u) & 1u) == 0u;
                    }
                    const float4 r0 = __ldg(reinterpret_cast<const float4*>(p.rays + i));
                    const float4 r1 = __ldg(reinterpret_cast<const float4*>(p.rays + i) + 1);
                    L.redo = !L.template start<WT>(s_base, r0, r1, walkable);
                }
            }
        }
        if (i == kIdle && !pool_left) i = kDone;
        if (__all_sync(0xFFFFFFFFu, i == kDone)) break;
        const uint32_t om = walk4_run<ANY, WT, kWalk4Flush>(L, s_base, st, pool_left ? kWalk4Refill : 32);
        const bool done = (om >> lane & 1u) && i < kDone;
        if (done) {
            uint4 h = L.hit();
            if (L.redo) {
                walk4_leave(ctr, left, i, p.n_rays);
                h = left_mark();
            }
            reinterpret_cast<uint4*>(p.hits)[i] = h;
            i = kIdle;
        }
    }
    walk4_finish(ctr, host_left, p.cw_bad);
}

// The binary walk of the any-hit rays a trace_walk4_kernel launch left over, a thread
// each: n of them, or as many as *count says; where they are more than the list holds,
// all rays are looked at for marks (kWalkAll: all are walked).  Closest hits: trace_pool_kernel (crt_pool.cuh).
template <bool ANY, bool WT, int STACK, bool BATCH>
__global__ void __launch_bounds__(kWalk4Block)
    walk4_left_kernel(const TraceParams p, const uint32_t* __restrict__ count, uint32_t n,
                      const uint32_t* __restrict__ left, const BatchScene* __restrict__ scenes, uint32_t n_scenes) {
    if (count) n = *count;
    const bool all = n > kWalkLeft;
    const uint64_t total = all ? p.n_rays : n;
    for (uint64_t k = static_cast<uint64_t>(blockIdx.x) * kWalk4Block + threadIdx.x; k < total;
         k += static_cast<uint64_t>(gridDim.x) * kWalk4Block) {
        const uint32_t i = !all ? left[k] : p.order ? __ldg(p.order + k) : static_cast<uint32_t>(k);
        if (i >= p.n_rays) { raise_corrupt(p.err, 7, static_cast<uint32_t>(k), i); continue; }
        if (all && n != kWalkAll && !left_marked(p.hits, i)) continue;
        TraceParams q = p;
        if (BATCH) {
            uint32_t lo = 0, hi = n_scenes - 1;
            while (lo < hi) {
                const uint32_t mid = (lo + hi + 1) >> 1;
                if (__ldg(&scenes[mid].ray_off) <= i) lo = mid; else hi = mid - 1;
            }
            const BatchScene bs = scenes[lo];
            q.nodes = p.nodes + bs.node_off;
            q.wide = p.wide + 4 * static_cast<size_t>(bs.wide_off);
            q.xtri = p.xtri + 3 * static_cast<size_t>(bs.tri_off);
            q.abs_eps = bs.abs_eps;
            q.n_nodes = 2 * bs.n_tris - 1;
        }
        trace_ray<ANY, WT, STACK, false, 0>(q, i);
    }
}

// One thread's whole walk over the compressed nodes (leaves tested as they are
// met), with the binary walk where walk4_setup or the stack asks for it.
template <bool ANY, bool WT, int STACK>
__device__ __forceinline__ uint4 trace_walk4_one(const TraceParams& p, const uint32_t i, const float4 r0,
                                                 const float4 r1) {
    const float3 o = make_float3(r0.x, r0.y, r0.z), d = make_float3(r1.x, r1.y, r1.z);
    const float tmin = r0.w, tmax = r1.w;
    if (!(tmin <= tmax)) return make_uint4(CRT_MISS, 0u, 0u, 0u);
    const uint32_t n_leaves = (p.n_nodes + 1) / 2;
    Walk4Ray w;
    if (!walk4_setup(w, o, d, tmin, p.abs_eps) || n_leaves < 2 || __ldg(p.cw_bad) != 0u)
        return trace_binary<ANY, WT, STACK>(p, i, r0, r1);
    WRay wt{};
    if (WT) wt = wt_setup(d);
    float bt = tmax, bu = 0.f, bv = 0.f, bound = prune_bound(bt, p.abs_eps) * kWalk4TScale;
    uint32_t bkey = 0xFFFFFFFFu, btri = CRT_MISS, cur = 0, fetched = 0, tested = 0;
    bool corrupt = false;
    constexpr int kCap = 64;
    uint2 st[kCap];
    int sp = 0;
    auto test_leaf = [&](uint32_t leaf) {
        const uint32_t L = leaf & ~kLeafRef;
        if (L >= n_leaves) { corrupt = true; return; }
        const float4* t = p.xtri + 3 * static_cast<size_t>(L);
        const float4 a = __ldg(t), b = __ldg(t + 1), c = __ldg(t + 2);
        if (!WT) {
            RayCtx r;
            r.o = o;
            r.d = d;
            r.inv = make_float3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
            r.exact = !(isfinite(r.inv.x) && isfinite(r.inv.y) && isfinite(r.inv.z));
            if (!leaf_box_passes(r, a, b, c, prune_bound(bt, p.abs_eps))) return;
        }
        ++tested;
        const float3 A = make_float3(a.x, a.y, a.z), B = make_float3(b.x, b.y, b.z), C = make_float3(c.x, c.y, c.z);
        const HitRes h = WT ? tri_watertight(o, tmin, tmax, wt, A, B, C) : tri_reference(o, d, tmin, tmax, A, B, C);
        if (!h.did) return;
        const uint32_t tri = __float_as_uint(a.w);
        const uint32_t key = WT ? tri : ~L;
        if (btri == CRT_MISS || h.t < bt || (h.t == bt && key < bkey)) {
            bt = h.t; bu = h.u; bv = h.v; bkey = key; btri = tri;
            bound = prune_bound(bt, p.abs_eps) * kWalk4TScale;
        }
    };
    const float inf = __int_as_float(0x7F800000);
    while (true) {
        if (cur & kLeafRef) {
            if (cur != kNoChild) test_leaf(cur);
            if (ANY && btri != CRT_MISS) break;
        } else {
            if (cur >= n_leaves - 1) { corrupt = true; break; }
            if (sp + 3 > kCap) return trace_binary<ANY, WT, STACK>(p, i, r0, r1);
            ++fetched;
            Walk4Node n = load_walk4(p.cwide + 4 * static_cast<size_t>(cur));
            float t[4];
            walk4_children(n, w, bound, t);
            walk4_sort<ANY>(t, n.ref);
#pragma unroll
            for (int c = 3; c >= 1; --c)
                if (t[c] < inf) st[sp++] = make_uint2(n.ref[c], __float_as_uint(t[c]));
            if (t[0] < inf) { cur = n.ref[0]; continue; }
        }
        bool more = false;
        while (sp > 0) {
            const uint2 e = st[--sp];
            if (fabsf(__uint_as_float(e.y)) <= bound) { cur = e.x; more = true; break; }
        }
        if (!more) break;
    }
    if (corrupt) raise_corrupt(p.err, 5, i, 0u);
    if (p.stats) {
        atomicAdd(p.stats + 0, static_cast<unsigned long long>(fetched));
        atomicAdd(p.stats + 1, static_cast<unsigned long long>(tested));
    }
    return btri != CRT_MISS ? make_uint4(btri, __float_as_uint(bt), __float_as_uint(bu), __float_as_uint(bv))
                            : make_uint4(CRT_MISS, 0u, 0u, 0u);
}

}  // namespace crt
