// Trace kernels of libcrt: rays from memory to hits (crt_trace, batched
// scenes), ray ordering for CRT_TRACE_SORT_RAYS, ray generation and shadow
// rays.  The traversal itself is in crt_traverse.cuh.  Compiled with
// -fmad=false: every float operation rounds once, in the shader's order.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "crt_build.cuh"
#include "crt_common.cuh"
#include "crt_pool.cuh"
#include "crt_traverse.cuh"
#include "crt_walk4.cuh"

namespace crt {

template <bool ANY, bool WT, int STACK, bool SEED, int WALK, int BLOCK>
__global__ void __launch_bounds__(BLOCK) trace_kernel(TraceParams p) {
    const uint32_t t_id = blockIdx.x * BLOCK + threadIdx.x;
    if (t_id >= p.n_rays) return;
    const uint32_t i = p.order ? __ldg(p.order + t_id) : ray_of_thread(t_id, p.tile_width);
    if (i >= p.n_rays) { raise_corrupt(p.err, 7, t_id, i); return; }
    if (WALK == 2) {
        const float4 r0 = __ldg(reinterpret_cast<const float4*>(p.rays + i));
        const float4 r1 = __ldg(reinterpret_cast<const float4*>(p.rays + i) + 1);
        reinterpret_cast<uint4*>(p.hits)[i] = trace_walk4_one<ANY, WT, STACK>(p, i, r0, r1);
    } else {
        trace_ray<ANY, WT, STACK, SEED, WALK>(p, i);
    }
}

// Many scenes in one launch: ray i belongs to the scene whose ray range holds
// it and is traced against that scene's BVH (same walk as above).
// SEED: learned seeding in a batch; base.pred_class holds every ray's class,
// base.treelets / base.n_treelets every scene's cut (scene k's at 128 k / k).
template <bool ANY, bool WT, int STACK, bool SEED, int BLOCK>
__global__ void __launch_bounds__(BLOCK) trace_batch_kernel(TraceParams base, const BatchScene* __restrict__ scenes,
                                                            uint32_t n_scenes, uint32_t n_rays_total) {
    __shared__ uint32_t s_ray_off[kMaxBatchScenes + 1];
    for (uint32_t k = threadIdx.x; k <= n_scenes; k += BLOCK) s_ray_off[k] = scenes[k < n_scenes ? k : n_scenes - 1].ray_off +
                                                                            (k < n_scenes ? 0u : scenes[n_scenes - 1].n_rays);
    __syncthreads();
    const uint32_t t = blockIdx.x * BLOCK + threadIdx.x;
    if (t >= n_rays_total) return;
    const uint32_t i = base.order ? __ldg(base.order + t) : t;
    if (i >= n_rays_total) { raise_corrupt(base.err, 7, t, i); return; }
    uint32_t lo = 0, hi = n_scenes - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (s_ray_off[mid] <= i) lo = mid; else hi = mid - 1;
    }
    const BatchScene sc = scenes[lo];
    TraceParams p = base;
    p.nodes = base.nodes + sc.node_off;
    p.wide = base.wide + 4 * static_cast<size_t>(sc.wide_off);
    p.xtri = base.xtri + 3 * static_cast<size_t>(sc.tri_off);
    p.n_nodes = 2 * sc.n_tris - 1;
    p.abs_eps = sc.abs_eps;
    if (SEED) {
        p.treelets = base.treelets + 128 * static_cast<size_t>(lo);
        p.n_treelets = base.n_treelets + lo;
    }
    trace_ray<ANY, WT, STACK, SEED, 0>(p, i);
}

// ------------------------------------------------------ ray ordering
// CRT_TRACE_SORT_RAYS: rays are traced in the order of a 24-bit coherence
// key — Morton code of the cell, on a 32^3 grid of the scene box, where the
// ray enters the box (its origin if it starts inside; 15 bits), then an
// octahedral direction bin (32 x 16, 9 bits) — so warps hold rays that
// reach the scene close together and point the same way.  In a batch
// the scene index (8 bits) goes on top, which keeps every ray inside its
// scene's range.  A stable LSD radix sort (the build's digit pass) makes the
// order; every ray still gets its own hit.
__device__ __forceinline__ uint32_t spread5_bits(uint32_t v) {
    v &= 31u;
    return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6) | ((v & 16u) << 8);
}

__device__ __forceinline__ uint32_t coherence_key(float4 r0, float4 r1, float4 mn, float4 mx) {
    // entry distance into the box (a key only: any rounding is harmless)
    const float ix = 1.f / r1.x, iy = 1.f / r1.y, iz = 1.f / r1.z;
    const float tx1 = (mn.x - r0.x) * ix, tx2 = (mx.x - r0.x) * ix;
    const float ty1 = (mn.y - r0.y) * iy, ty2 = (mx.y - r0.y) * iy;
    const float tz1 = (mn.z - r0.z) * iz, tz2 = (mx.z - r0.z) * iz;
    float te = fmaxf(fmaxf(fminf(tx1, tx2), fminf(ty1, ty2)), fminf(tz1, tz2));
    if (!(te > 0.f) || !isfinite(te)) te = 0.f;
    const float ex = r0.x + te * r1.x, ey = r0.y + te * r1.y, ez = r0.z + te * r1.z;
    const float sx = 32.f / fmaxf(mx.x - mn.x, 1e-20f), sy = 32.f / fmaxf(mx.y - mn.y, 1e-20f);
    const float sz = 32.f / fmaxf(mx.z - mn.z, 1e-20f);
    const int cx = min(max(static_cast<int>(floorf((ex - mn.x) * sx)), 0), 31);
    const int cy = min(max(static_cast<int>(floorf((ey - mn.y) * sy)), 0), 31);
    const int cz = min(max(static_cast<int>(floorf((ez - mn.z) * sz)), 0), 31);
    const uint32_t m = (spread5_bits(cx) << 2) | (spread5_bits(cy) << 1) | spread5_bits(cz);
    const float a = fabsf(r1.x) + fabsf(r1.y) + fabsf(r1.z);
    float px = a > 0.f ? r1.x / a : 0.f, py = a > 0.f ? r1.y / a : 0.f;
    if (r1.z < 0.f) {
        const float qx = (1.f - fabsf(py)) * (px >= 0.f ? 1.f : -1.f);
        const float qy = (1.f - fabsf(px)) * (py >= 0.f ? 1.f : -1.f);
        px = qx;
        py = qy;
    }
    const int bu = min(max(static_cast<int>((px + 1.f) * 16.f), 0), 31);
    const int bv = min(max(static_cast<int>((py + 1.f) * 8.f), 0), 15);
    return (m << 9) | (static_cast<uint32_t>(bu) << 4) | static_cast<uint32_t>(bv);
}

// Keys of all rays and the histograms of their PASSES 8-bit digits; with
// scenes, ray i belongs to the scene whose ray range holds it and is keyed
// on that scene's root box.
template <int PASSES>
__global__ void __launch_bounds__(256) ray_key_kernel(const crt_ray* __restrict__ rays, uint32_t n,
                                                      const crt_bvh_node* __restrict__ nodes,
                                                      const BatchScene* __restrict__ scenes, uint32_t n_scenes,
                                                      uint32_t* __restrict__ keys, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[PASSES * 256];
    __shared__ uint32_t s_ray_off[kMaxBatchScenes + 1];
    for (int k = threadIdx.x; k < PASSES * 256; k += blockDim.x) h[k] = 0u;
    if (scenes)
        for (uint32_t k = threadIdx.x; k <= n_scenes; k += blockDim.x)
            s_ray_off[k] = k < n_scenes ? scenes[k].ray_off : scenes[n_scenes - 1].ray_off + scenes[n_scenes - 1].n_rays;
    __syncthreads();
    float4 mn = __ldg(reinterpret_cast<const float4*>(nodes)), mx = __ldg(reinterpret_cast<const float4*>(nodes) + 1);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t top = 0;
        if (scenes) {
            uint32_t lo = 0, hi = n_scenes - 1;
            while (lo < hi) {
                const uint32_t mid = (lo + hi + 1) >> 1;
                if (s_ray_off[mid] <= i) lo = mid; else hi = mid - 1;
            }
            const float4* root = reinterpret_cast<const float4*>(nodes + scenes[lo].node_off);
            mn = __ldg(root);
            mx = __ldg(root + 1);
            top = lo << 24;
        }
        const float4 r0 = __ldg(reinterpret_cast<const float4*>(rays + i));
        const float4 r1 = __ldg(reinterpret_cast<const float4*>(rays + i) + 1);
        const uint32_t key = top | coherence_key(r0, r1, mn, mx);
        keys[i] = key;
#pragma unroll
        for (int p = 0; p < PASSES; ++p) atomicAdd(&h[p * 256 + ((key >> (8 * p)) & 255u)], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < PASSES * 256; k += blockDim.x)
        if (h[k]) atomicAdd(&hist[k], h[k]);
}

__global__ void __launch_bounds__(256) raygen_kernel(const crt_camera* __restrict__ cam, uint32_t width, uint32_t height,
                                                     crt_ray* __restrict__ rays) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t y = blockIdx.y;
    if (x >= width) return;
    float4 r0, r1;
    camera_ray(cam, x, y, width, height, r0, r1);
    float4* o = reinterpret_cast<float4*>(rays + static_cast<size_t>(y) * width + x);
    o[0] = r0;
    o[1] = r1;
}


__global__ void __launch_bounds__(256) shadow_kernel(const crt_ray* __restrict__ prim, const crt_hit* __restrict__ hits,
                                                     uint32_t n, float lx, float ly, float lz, crt_ray* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint4 h = __ldg(reinterpret_cast<const uint4*>(hits) + i);
    const float4 r0 = __ldg(reinterpret_cast<const float4*>(prim + i));
    const float4 r1 = __ldg(reinterpret_cast<const float4*>(prim + i) + 1);
    float4 s0, s1;
    shadow_ray(r0, r1, h, lx, ly, lz, s0, s1);
    float4* o = reinterpret_cast<float4*>(out + i);
    o[0] = s0;
    o[1] = s1;
}


template <bool ANY, bool WT, int BLOCK>
static void launch_trace_b(const TraceParams& p, bool deep, bool seed, int walk, cudaStream_t s) {
    const uint32_t grid = (p.n_rays + BLOCK - 1) / BLOCK;
    if (grid == 0) return;
    if (seed) {
        if (deep) trace_kernel<ANY, WT, 1024, true, 0, BLOCK><<<grid, BLOCK, 0, s>>>(p);
        else trace_kernel<ANY, WT, 64, true, 0, BLOCK><<<grid, BLOCK, 0, s>>>(p);
    } else if (walk == 1) {
        if (deep) trace_kernel<ANY, WT, 1024, false, 1, BLOCK><<<grid, BLOCK, 0, s>>>(p);
        else trace_kernel<ANY, WT, 96, false, 1, BLOCK><<<grid, BLOCK, 0, s>>>(p);
    } else if (walk == 2) {
        if (deep) trace_kernel<ANY, WT, 1024, false, 2, BLOCK><<<grid, BLOCK, 0, s>>>(p);
        else trace_kernel<ANY, WT, 96, false, 2, BLOCK><<<grid, BLOCK, 0, s>>>(p);
    } else {
        if (deep) trace_kernel<ANY, WT, 1024, false, 0, BLOCK><<<grid, BLOCK, 0, s>>>(p);
        else trace_kernel<ANY, WT, 64, false, 0, BLOCK><<<grid, BLOCK, 0, s>>>(p);
    }
}

template <bool ANY, bool WT>
static void launch_trace_t(const TraceParams& p, int block, bool deep, bool seed, int walk, cudaStream_t s) {
    if (block == 256) launch_trace_b<ANY, WT, 256>(p, deep, seed, walk, s);
    else if (block == 64) launch_trace_b<ANY, WT, 64>(p, deep, seed, walk, s);
    else launch_trace_b<ANY, WT, 128>(p, deep, seed, walk, s);
}

// trace_pool_kernel over the n rays left over (*count of them, if given), or over all
// rays (kWalkAll).
template <bool WT, int STACK, bool BATCH>
static void launch_pool_s(const TraceParams& p, const WalkScratch& w, const uint32_t* count, uint32_t n,
                          const BatchScene* scenes, uint32_t n_scenes, cudaStream_t s) {
    static const uint32_t grid = [] {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trace_pool_kernel<WT, STACK, BATCH>, kWalk4Block, 0);
        return static_cast<uint32_t>(kNumSms * (per_sm > 0 ? per_sm : 1));
    }();
    const uint32_t items = count || n > kWalkLeft ? p.n_rays : n;
    trace_pool_kernel<WT, STACK, BATCH><<<std::min((items - 1) / kWalk4Block + 1, grid), kWalk4Block, 0, s>>>(
        p, reinterpret_cast<Walk4Counters*>(w.ctr), count, n, w.left, scenes, n_scenes);
}

template <bool WT, bool BATCH>
static void launch_pool(const TraceParams& p, bool deep, const WalkScratch& w, const uint32_t* count, uint32_t n,
                        const BatchScene* scenes, uint32_t n_scenes, cudaStream_t s) {
    if (deep) launch_pool_s<WT, 1024, BATCH>(p, w, count, n, scenes, n_scenes, s);
    else launch_pool_s<WT, 64, BATCH>(p, w, count, n, scenes, n_scenes, s);
}

template <bool ANY, bool WT, bool BATCH>
static void launch_walk4_t(const TraceParams& p, bool deep, const WalkScratch& w, uint32_t left, const BatchScene* scenes,
                           uint32_t n_scenes, cudaStream_t s) {
    static int grid = 0;
    if (grid == 0) {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trace_walk4_kernel<ANY, WT, BATCH>, kWalk4Block, 0);
        grid = kNumSms * (per_sm > 0 ? per_sm : 1);
    }
    Walk4Counters* ctr = reinterpret_cast<Walk4Counters*>(w.ctr);
    const uint32_t want = (p.n_rays + kWalk4Block - 1) / kWalk4Block;
    if (left == 0) {
        trace_walk4_kernel<ANY, WT, BATCH><<<std::min(want, static_cast<uint32_t>(grid)), kWalk4Block, 0, s>>>(
            p, ctr, w.left, w.host_left, scenes, n_scenes);
        if (w.host_left) return;
    }
    const uint32_t* count = left == 0 ? &ctr->last_left : nullptr;
    if (!ANY) {
        launch_pool<WT, BATCH>(p, deep, w, count, left, scenes, n_scenes, s);
        return;
    }
    // a thread an item where their number is known
    const uint32_t items = left == 0 || left > kWalkLeft ? p.n_rays : left;
    const uint32_t full = (items - 1) / kWalk4Block + 1;
    const uint32_t few = left == 0 ? std::min(full, static_cast<uint32_t>(kNumSms * 16)) : full;
    if (deep) walk4_left_kernel<ANY, WT, 1024, BATCH><<<few, kWalk4Block, 0, s>>>(p, count, left, w.left, scenes, n_scenes);
    else walk4_left_kernel<ANY, WT, 64, BATCH><<<few, kWalk4Block, 0, s>>>(p, count, left, w.left, scenes, n_scenes);
}

template <bool BATCH>
static void launch_walk4(const TraceParams& p, uint32_t flags, bool deep, const WalkScratch& w, uint32_t left,
                         const BatchScene* scenes, uint32_t n_scenes, cudaStream_t s) {
    const bool any = flags & CRT_TRACE_ANY, wt = flags & CRT_TRI_WATERTIGHT;
    if (any && wt) launch_walk4_t<true, true, BATCH>(p, deep, w, left, scenes, n_scenes, s);
    else if (any) launch_walk4_t<true, false, BATCH>(p, deep, w, left, scenes, n_scenes, s);
    else if (wt) launch_walk4_t<false, true, BATCH>(p, deep, w, left, scenes, n_scenes, s);
    else launch_walk4_t<false, false, BATCH>(p, deep, w, left, scenes, n_scenes, s);
}

void launch_trace_pool(const TraceParams& p, uint32_t flags, const WalkScratch& w, cudaStream_t s) {
    if (p.n_rays != 0) launch_walk4<false>(p, flags, (flags >> 16) != 0, w, 0, nullptr, 0, s);
}

void launch_trace_left(const TraceParams& p, uint32_t flags, const WalkScratch& w, uint32_t n, cudaStream_t s) {
    if (n != 0) launch_walk4<false>(p, flags, (flags >> 16) != 0, w, n, nullptr, 0, s);
}

void launch_trace_binary_pool(const TraceParams& p, uint32_t flags, const WalkScratch& w, cudaStream_t s) {
    if (p.n_rays == 0) return;
    const bool deep = (flags >> 16) != 0;
    if (flags & CRT_TRI_WATERTIGHT) launch_pool<true, false>(p, deep, w, nullptr, kWalkAll, nullptr, 0, s);
    else launch_pool<false, false>(p, deep, w, nullptr, kWalkAll, nullptr, 0, s);
}

void launch_trace_batch_binary_pool(const TraceParams& p, const BatchScene* scenes, uint32_t n_scenes, uint32_t flags,
                                    bool deep, const WalkScratch& w, cudaStream_t s) {
    if (p.n_rays == 0 || n_scenes == 0) return;
    if (flags & CRT_TRI_WATERTIGHT) launch_pool<true, true>(p, deep, w, nullptr, kWalkAll, scenes, n_scenes, s);
    else launch_pool<false, true>(p, deep, w, nullptr, kWalkAll, scenes, n_scenes, s);
}

void launch_trace_batch_pool(const TraceParams& p, const BatchScene* scenes, uint32_t n_scenes, uint32_t flags,
                             bool deep, const WalkScratch& w, cudaStream_t s) {
    if (p.n_rays != 0 && n_scenes != 0) launch_walk4<true>(p, flags, deep, w, 0, scenes, n_scenes, s);
}

void launch_trace(const TraceParams& p, uint32_t flags, int block, cudaStream_t s) {
    const bool any = flags & CRT_TRACE_ANY, wt = flags & CRT_TRI_WATERTIGHT;
    const bool deep = (flags >> 16) != 0;  // set by the host when the tree may be deeper than the stacks allow
    const bool seed = p.pred_class != nullptr;
    const int walk = ((flags & CRT_TRACE_COMPRESSED) && p.cwide) ? 2 : ((flags & CRT_TRACE_WIDE) && p.wide4) ? 1 : 0;
    if (any && wt) launch_trace_t<true, true>(p, block, deep, seed, walk, s);
    else if (any) launch_trace_t<true, false>(p, block, deep, seed, walk, s);
    else if (wt) launch_trace_t<false, true>(p, block, deep, seed, walk, s);
    else launch_trace_t<false, false>(p, block, deep, seed, walk, s);
}

template <bool ANY, bool WT, int BLOCK>
static void launch_batch_b(const TraceParams& p, const BatchScene* scenes, uint32_t n_scenes, uint32_t n_rays,
                           bool deep, cudaStream_t s) {
    const uint32_t grid = (n_rays + BLOCK - 1) / BLOCK;
    if (grid == 0) return;
    if (p.pred_class) {
        if (deep) trace_batch_kernel<ANY, WT, 1024, true, BLOCK><<<grid, BLOCK, 0, s>>>(p, scenes, n_scenes, n_rays);
        else trace_batch_kernel<ANY, WT, 64, true, BLOCK><<<grid, BLOCK, 0, s>>>(p, scenes, n_scenes, n_rays);
    } else {
        if (deep) trace_batch_kernel<ANY, WT, 1024, false, BLOCK><<<grid, BLOCK, 0, s>>>(p, scenes, n_scenes, n_rays);
        else trace_batch_kernel<ANY, WT, 64, false, BLOCK><<<grid, BLOCK, 0, s>>>(p, scenes, n_scenes, n_rays);
    }
}

template <bool ANY, bool WT>
static void launch_batch_t(const TraceParams& p, const BatchScene* scenes, uint32_t n_scenes, uint32_t n_rays,
                           int block, bool deep, cudaStream_t s) {
    if (block == 512) launch_batch_b<ANY, WT, 512>(p, scenes, n_scenes, n_rays, deep, s);
    else if (block == 256) launch_batch_b<ANY, WT, 256>(p, scenes, n_scenes, n_rays, deep, s);
    else launch_batch_b<ANY, WT, 128>(p, scenes, n_scenes, n_rays, deep, s);
}

void launch_trace_batch(const TraceParams& p, const BatchScene* scenes, uint32_t n_scenes, uint32_t n_rays,
                        uint32_t flags, int block, bool deep, cudaStream_t s) {
    const bool any = flags & CRT_TRACE_ANY, wt = flags & CRT_TRI_WATERTIGHT;
    if (any && wt) launch_batch_t<true, true>(p, scenes, n_scenes, n_rays, block, deep, s);
    else if (any) launch_batch_t<true, false>(p, scenes, n_scenes, n_rays, block, deep, s);
    else if (wt) launch_batch_t<false, true>(p, scenes, n_scenes, n_rays, block, deep, s);
    else launch_batch_t<false, false>(p, scenes, n_scenes, n_rays, block, deep, s);
}

size_t ray_order_scratch_bytes(uint32_t n) {
    const size_t tiles = (n + sort_tile_keys(8) - 1) / sort_tile_keys(8);
    return 4 * (3 * static_cast<size_t>(n) + 4 * 256 + 4 * (tiles * 256 + 1) + 64);
}

void launch_ray_order(const crt_ray* rays, uint32_t n, const crt_bvh_node* nodes, const BatchScene* scenes,
                      uint32_t n_scenes, uint32_t* order, void* scratch, uint32_t* err, uint32_t spin_limit,
                      cudaStream_t s) {
    if (n == 0) return;
    const int passes = scenes ? 4 : 3;
    uint32_t* ka = static_cast<uint32_t*>(scratch);
    uint32_t* kb = ka + n;
    uint32_t* vt = kb + n;
    uint32_t* hist = vt + n;
    uint32_t* lb = hist + 4 * 256;  // per pass: ticket, then the look-back words
    const size_t tiles = (n + sort_tile_keys(8) - 1) / sort_tile_keys(8);
    const size_t lb_words = tiles * 256 + 1;
    cudaMemsetAsync(hist, 0, 4 * (4 * 256 + 4 * lb_words), s);
    const uint32_t grid = std::min<uint32_t>((n + 255) / 256, kNumSms * 8);
    if (scenes) ray_key_kernel<4><<<grid, 256, 0, s>>>(rays, n, nodes, scenes, n_scenes, ka, hist);
    else ray_key_kernel<3><<<grid, 256, 0, s>>>(rays, n, nodes, nullptr, 0, ka, hist);
    // stable 8-bit passes; the values alternate between order and vt so
    // that the last pass writes order
    const uint32_t* kin = ka;
    const uint32_t* vin = nullptr;
    for (int p = 0; p < passes; ++p) {
        uint32_t* kout = (p & 1) ? ka : kb;
        uint32_t* vout = ((passes - 1 - p) & 1) ? vt : order;
        uint32_t* l = lb + p * lb_words;
        launch_onesweep(kin, vin, kout, vout, n, 8 * p, 8, hist + 256 * p, l + 1, l, err, spin_limit, s);
        kin = kout;
        vin = vout;
    }
}

void launch_raygen(const crt_camera* cam_dev, uint32_t width, uint32_t height, crt_ray* rays, cudaStream_t s) {
    dim3 grid((width + 255) / 256, height);
    raygen_kernel<<<grid, 256, 0, s>>>(cam_dev, width, height, rays);
}

void launch_shadow_rays(const crt_ray* prim, const crt_hit* hits, uint32_t n, float lx, float ly, float lz, crt_ray* out,
                        cudaStream_t s) {
    if (n == 0) return;
    shadow_kernel<<<(n + 255) / 256, 256, 0, s>>>(prim, hits, n, lx, ly, lz, out);
}

}  // namespace crt
