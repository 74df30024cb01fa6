// The persistent closest-hit walk over the binary nodes: rays the walk over the
// compressed nodes (crt_walk4.cuh) leaves over, and large batches of rays over
// scenes it cannot take at all.  Compiled with -fmad=false.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "crt_build.cuh"
#include "crt_common.cuh"
#include "crt_traverse.cuh"
#include "crt_walk4.cuh"

namespace crt {

// The scene a lane's ray is walked in: nodes, leaf triangles, the watertight slack
// and the leaf count (one scene, or the ray's scene of a batch).
struct PoolScene {
    const crt_bvh_node* nodes;
    const float4* wide;
    const float4* xtri;
    float abs_eps;
    uint32_t n_leaves;
};

// One lane's ray, walked as trace_one's binary walk but for its leaf tests, which
// may be put off (pend).
template <bool WT, int STACK>
struct PoolRay {
    static constexpr uint32_t kNoLeaf = 0xFFFFFFFFu;
    RayCtx r;
    WRay w;
    float tmin, tmax, bt, bu, bv, bound;
    uint32_t bkey, btri, cur;
    int sp;
    bool have;
    uint32_t pend;  // one postponed leaf (kNoLeaf: none)

    __device__ __forceinline__ void test_leaf(const PoolScene& sc, uint32_t L, bool& corrupt) {
        if (L >= sc.n_leaves) { corrupt = true; return; }
        const float4* t = sc.xtri + 3 * static_cast<size_t>(L);
        const float4 a = __ldg(t), b = __ldg(t + 1), c = __ldg(t + 2);
        const float3 A = make_float3(a.x, a.y, a.z), B = make_float3(b.x, b.y, b.z), C = make_float3(c.x, c.y, c.z);
        const HitRes h = WT ? tri_watertight(r.o, tmin, tmax, w, A, B, C) : tri_reference(r.o, r.d, tmin, tmax, A, B, C);
        if (!h.did) return;
        const uint32_t tri = __float_as_uint(a.w);
        const uint32_t key = WT ? tri : ~L;
        if (!have || h.t < bt || (h.t == bt && key < bkey)) {
            have = true; bt = h.t; bu = h.u; bv = h.v; bkey = key; btri = tri;
            bound = prune_bound(bt, sc.abs_eps);
        }
    }

    // Sets up ray (r0, r1) and enters the root; false when the ray is already finished.
    __device__ __forceinline__ bool start(const PoolScene& sc, float4 r0, float4 r1, bool& corrupt) {
        r.o = make_float3(r0.x, r0.y, r0.z);
        r.d = make_float3(r1.x, r1.y, r1.z);
        tmin = r0.w;
        tmax = r1.w;
        have = false;
        bt = tmax; bu = 0.f; bv = 0.f;
        bkey = 0xFFFFFFFFu; btri = CRT_MISS;
        sp = 0;
        cur = 0xFFFFFFFFu;
        pend = kNoLeaf;
        if (!(tmin <= tmax) || sc.n_leaves == 0) return false;
        r.inv = make_float3(1.0f / r.d.x, 1.0f / r.d.y, 1.0f / r.d.z);
        r.oi = make_float3(r.o.x * r.inv.x, r.o.y * r.inv.y, r.o.z * r.inv.z);
        r.exact = !(isfinite(r.inv.x) && isfinite(r.inv.y) && isfinite(r.inv.z) && r.inv.x != 0.f && r.inv.y != 0.f &&
                    r.inv.z != 0.f);
        if (WT) w = wt_setup(r.d);
        bound = prune_bound(bt, sc.abs_eps);
        const float4* n4 = reinterpret_cast<const float4*>(sc.nodes);
        const uint4 lr = __ldg(reinterpret_cast<const uint4*>(n4 + 2));
        float te;
        if (!slab<WT>(r, __ldg(n4), __ldg(n4 + 1), WT ? sc.abs_eps : 0.f, te) || te > bound) return false;
        if (lr.y == 0u && lr.z == 0u) {  // a one-leaf tree
            test_leaf(sc, 0u, corrupt);
            return false;
        }
        cur = 0u;
        return true;
    }

    __device__ __forceinline__ void flush(const PoolScene& sc, bool& corrupt) {
        if (pend == kNoLeaf) return;
        test_leaf(sc, pend, corrupt);
        pend = kNoLeaf;
    }

    // One node visit; false when the walk has finished.
    __device__ __forceinline__ bool step(const PoolScene& sc, uint2* st, bool& corrupt, bool& overflow) {
        if (cur >= sc.n_leaves - 1) { corrupt = true; return false; }
        const float4* nd = sc.wide + 4 * static_cast<size_t>(cur);
        const float4 w0 = __ldg(nd), w1 = __ldg(nd + 1), w2 = __ldg(nd + 2), w3 = __ldg(nd + 3);
        const uint32_t ref0 = __float_as_uint(w0.w), ref1 = __float_as_uint(w1.w);
        float t0, t1;
        bool h0, h1;
        if (WT) {
            h0 = slab_wt(r, w0, w1, t0);
            h1 = slab_wt(r, w2, w3, t1);
        } else {
            h0 = slab<false>(r, w0, w1, 0.f, t0);
            h1 = slab<false>(r, w2, w3, 0.f, t1);
        }
        const float bnd = bound;
        h0 = h0 && t0 <= bnd;
        h1 = h1 && t1 <= bnd;
        const bool leaf0 = (ref0 & kLeafRef) != 0u, leaf1 = (ref1 & kLeafRef) != 0u;
        if ((h0 && leaf0) || (h1 && leaf1)) {
            // the parked leaf comes first, and then the bound trace_one has here: the
            // same leaves are tested in the same order, which decides where distances
            // are not numbers or far less exact than the bound's slack
            flush(sc, corrupt);
            h0 = h0 && t0 <= bound;
            h1 = h1 && t1 <= bound;
            if (h0 && leaf0) { pend = ref0 & ~kLeafRef; h0 = false; }
            if (h1 && leaf1) {
                flush(sc, corrupt);
                pend = ref1 & ~kLeafRef;
                h1 = false;
            }
        }
        if (h0 || h1) {
            const float bnd2 = bound;
            h0 = h0 && t0 <= bnd2;
            h1 = h1 && t1 <= bnd2;
        }
        if (h0 && h1) {
            const bool near1 = t1 < t0;
            if (sp < STACK) {  // (node, entry distance) as one 8-byte entry
                st[sp] = make_uint2(near1 ? ref0 : ref1, __float_as_uint(near1 ? t0 : t1));
                ++sp;
            } else {
                overflow = true;
            }
            cur = near1 ? ref1 : ref0;
            return true;
        }
        if (h0) { cur = ref0; return true; }
        if (h1) { cur = ref1; return true; }
        const float bnd3 = bound;
        while (sp > 0) {
            --sp;
            const uint2 e = st[sp];
            if (__uint_as_float(e.y) <= bnd3) { cur = e.x; return true; }
        }
        return false;
    }

    __device__ __forceinline__ uint4 hit() const {
        return have ? make_uint4(btri, __float_as_uint(bt), __float_as_uint(bu), __float_as_uint(bv))
                    : make_uint4(CRT_MISS, 0u, 0u, 0u);
    }
};

// Node visits between refills, and the parked leaves that trigger a warp's leaf
// tests (measured over 8 M incoherent bounce rays).
constexpr int kPoolBurst = 16, kPoolFlush = 6;

// The n rays of the list (as many as *count says, if given), or the marked ones of
// all rays where they are more than the list holds, or all rays (kWalkAll), in caller
// order or p.order.  The warps are persistent: after kPoolBurst visits the lanes whose
// ray has finished take the next ones from the counter, and leaf tests are run for the
// whole warp at once when enough lanes hold a parked leaf, or a lane that has nothing
// else left does.
//
// Against one thread a ray: 4.2 M rays over 4.19 M clustered triangles from 30 scene
// sizes away 9.1 -> 5.9 ms (shader's predicate 47.5 -> 24.6), the same rays over a
// scene with a vertex at infinity 9.1 -> 5.9; the walk over the compressed nodes,
// which takes neither, does such rays in 2.7 from close by.
template <bool WT, int STACK, bool BATCH>
__global__ void __launch_bounds__(kWalk4Block)
    trace_pool_kernel(const TraceParams p, Walk4Counters* ctr, const uint32_t* __restrict__ count, uint32_t n,
                      const uint32_t* __restrict__ left, const BatchScene* __restrict__ scenes, uint32_t n_scenes) {
    constexpr uint32_t kIdle = 0xFFFFFFFFu, kDone = 0xFFFFFFFEu;
    __shared__ uint32_t s_ray_off[BATCH ? kMaxBatchScenes + 1 : 1];
    if (count) n = *count;
    if (n == 0u) return;
    const bool all = n > kWalkLeft, marks = all && n != kWalkAll;
    const uint32_t total = all ? p.n_rays : n;
    if (BATCH) {
        for (uint32_t k = threadIdx.x; k <= n_scenes; k += kWalk4Block)
            s_ray_off[k] = k < n_scenes ? scenes[k].ray_off : scenes[n_scenes - 1].ray_off + scenes[n_scenes - 1].n_rays;
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
    PoolScene sc{p.nodes, p.wide, p.xtri, p.abs_eps, (p.n_nodes + 1) / 2};
    PoolRay<WT, STACK> ray;
    ray.pend = PoolRay<WT, STACK>::kNoLeaf;
    uint2 st[STACK];
    uint32_t i = kIdle;
    bool corrupt = false, overflow = false;
    while (true) {
        while (const uint32_t need = __ballot_sync(0xFFFFFFFFu, i == kIdle)) {
            const int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if (lane == static_cast<uint32_t>(leader)) base = atomicAdd(&ctr->taken, static_cast<uint32_t>(__popc(need)));
            base = __shfl_sync(0xFFFFFFFFu, base, leader);
            if (i != kIdle) continue;
            const uint32_t k = base + static_cast<uint32_t>(__popc(need & lt_mask));
            if (k >= total) { i = kDone; continue; }
            const uint32_t ri = !all ? __ldg(left + k) : p.order ? __ldg(p.order + k) : k;
            if (ri >= p.n_rays) { raise_corrupt(p.err, 7, k, ri); i = kDone; continue; }
            if (marks && !left_marked(p.hits, ri)) continue;
            if (BATCH) {
                const BatchScene bs = scenes[batch_scene_of(s_ray_off, n_scenes, ri)];
                sc.nodes = p.nodes + bs.node_off;
                sc.wide = p.wide + 4 * static_cast<size_t>(bs.wide_off);
                sc.xtri = p.xtri + 3 * static_cast<size_t>(bs.tri_off);
                sc.abs_eps = bs.abs_eps;
                sc.n_leaves = bs.n_tris;
            }
            const float4 r0 = __ldg(reinterpret_cast<const float4*>(p.rays + ri));
            const float4 r1 = __ldg(reinterpret_cast<const float4*>(p.rays + ri) + 1);
            if (ray.start(sc, r0, r1, corrupt)) i = ri;
            else reinterpret_cast<uint4*>(p.hits)[ri] = ray.hit();
        }
        if (__all_sync(0xFFFFFFFFu, i == kDone)) break;
        bool walking = i < kDone;
#pragma unroll 1
        for (int s = 0; s < kPoolBurst; ++s) {
            if (walking) walking = ray.step(sc, st, corrupt, overflow);
            const bool parked = i < kDone && ray.pend != PoolRay<WT, STACK>::kNoLeaf;
            const uint32_t pm = __ballot_sync(0xFFFFFFFFu, parked);
            if (__popc(pm) >= kPoolFlush || __any_sync(0xFFFFFFFFu, parked && !walking)) {
                if (parked) ray.flush(sc, corrupt);
            }
            if (!__any_sync(0xFFFFFFFFu, walking)) break;
        }
        if (i < kDone && !walking) {
            reinterpret_cast<uint4*>(p.hits)[i] = ray.hit();
            i = kIdle;
        }
    }
    if (corrupt) raise_corrupt(p.err, 5, blockIdx.x, threadIdx.x);
    else if (overflow) raise_error(p.err, kDevStackOverflow);
    walk4_finish(ctr, nullptr, nullptr);
}

}  // namespace crt
