// One-launch frames and the shading pass of libcrt: camera ray, closest hit
// and, per option, the shadow ray's any hit and the shaded texel of every
// pixel.  Compiled with -fmad=false: every float operation rounds once, in
// the shader's order, as in the CPU oracle.
//
// Shading restates srcCommon/shaders/raytracer.glsl:
//   getColor                        :159-179
//   intersectBVH with border test   :182-236
//   bvhColor of getClosestHitBVH    :246-277 (the depth-uDepthDisplayBVH box)
//   main's initial value, imageStore :299-331
#include <cstdint>
#include <cuda_runtime.h>

#include "crt_build.cuh"
#include "crt_common.cuh"
#include "crt_traverse.cuh"
#include "crt_walk4.cuh"

namespace crt {

// ------------------------------------------------------------- shading
// intersectBVH (raytracer.glsl:182-236): 0 = miss, 1 = hit, 2 = hit whose
// entry point lies within `line` of a face of the box on at least two axes
// (near a box edge).  GLSL min/max, its early exits and its entry point
// o + d * tMin, each operation rounded once.
__device__ __forceinline__ uint32_t display_slab(float3 o, float3 d, float4 mn, float4 mx, float line) {
    const float ix = 1.0f / d.x;
    const float tx1 = (mn.x - o.x) * ix, tx2 = (mx.x - o.x) * ix;
    float tMin = min_std(tx1, tx2), tMax = max_std(tx1, tx2);
    if (tMax < 0.f || tMin > tMax) return 0u;
    const float iy = 1.0f / d.y;
    const float ty1 = (mn.y - o.y) * iy, ty2 = (mx.y - o.y) * iy;
    tMin = max_std(tMin, min_std(ty1, ty2));
    tMax = min_std(tMax, max_std(ty1, ty2));
    if (tMax < 0.f || tMin > tMax) return 0u;
    const float iz = 1.0f / d.z;
    const float tz1 = (mn.z - o.z) * iz, tz2 = (mx.z - o.z) * iz;
    tMin = max_std(tMin, min_std(tz1, tz2));
    tMax = min_std(tMax, max_std(tz1, tz2));
    if (!(tMax >= 0.f && tMin <= tMax)) return 0u;
    const float ex = o.x + d.x * tMin, ey = o.y + d.y * tMin, ez = o.z + d.z * tMin;
    const bool cx = fabsf(ex - mn.x) < line || fabsf(ex - mx.x) < line;
    const bool cy = fabsf(ey - mn.y) < line || fabsf(ey - mx.y) < line;
    const bool cz = fabsf(ez - mn.z) < line || fabsf(ez - mx.z) < line;
    return ((cx && cy) || (cx && cz) || (cy && cz)) ? 2u : 1u;
}

// bvhColor.  The shader's walk pops right children first, enters every box
// the ray intersects and overwrites bvhColor at each intersected node of
// depth D, so the last such node decides.  A left-child-first walk meets the
// nodes of one depth in exactly the reverse order, so that node is the FIRST
// intersected depth-D node of a left-first walk that descends only through
// intersected boxes: this walk stops there and never goes below depth D.
// Returns display_slab's value for that node, 0 when there is none.
__device__ __noinline__ uint32_t bvh_display(const TraceParams& p, uint32_t depth_d, float3 o, float3 d) {
    const float line = 0.05f / (static_cast<float>(depth_d) + 1.f);  // BVH_LINE_WIDTH / (uDepthDisplayBVH + 1)
    uint32_t st_node[kShadeMaxDepth];
    uint32_t st_depth[kShadeMaxDepth];
    int sp = 0;
    uint32_t cur = 0, depth = 0;
    // each node is met at most once, so a walk longer than the tree is a bad tree
    for (uint32_t guard = 0; guard < p.n_nodes; ++guard) {
        if (cur >= p.n_nodes) { raise_corrupt(p.err, 10, cur, p.n_nodes); return 0u; }
        const float4* nd = reinterpret_cast<const float4*>(p.nodes + cur);
        const float4 mn = __ldg(nd), mx = __ldg(nd + 1);
        const uint4 k = __ldg(reinterpret_cast<const uint4*>(nd + 2));  // tri, left, right, pad
        const uint32_t hit = display_slab(o, d, mn, mx, line);
        if (hit != 0u) {
            if (depth == depth_d) return hit;
            if (k.y != 0u || k.z != 0u) {  // internal (isLeafBVH: left == right == 0)
                // pending right siblings have strictly increasing depths < D
                if (sp >= static_cast<int>(kShadeMaxDepth)) { raise_corrupt(p.err, 10, cur, depth); return 0u; }
                st_node[sp] = k.z;
                st_depth[sp] = depth + 1;
                ++sp;
                cur = k.y;
                ++depth;
                continue;
            }
        }
        if (sp == 0) return 0u;
        --sp;
        cur = st_node[sp];
        depth = st_depth[sp];
    }
    if (p.n_nodes != 0) raise_corrupt(p.err, 10, cur, p.n_nodes);
    return 0u;
}

// getColor + main's initial value for hit h of the ray (r0.xyz, r1.xyz).
__device__ __forceinline__ float4 shade_texel(const TraceParams& p, const ShadeParams& sp, uint4 h, float4 r0,
                                              float4 r1) {
    float4 c = make_float4(0.f, 0.f, 0.f, 1.f);
    if (sp.flags & CRT_SHADE_BVH) {
        const uint32_t b = bvh_display(p, sp.bvh_depth, make_float3(r0.x, r0.y, r0.z), make_float3(r1.x, r1.y, r1.z));
        c = b == 2u ? make_float4(0.7f, 0.f, 0.7f, 0.1f)      // BVH_AABB_LINE_COLOR
            : b == 1u ? make_float4(0.5f, 0.f, 0.5f, 0.1f)    // BVH_AABB_COLOR
                      : make_float4(0.f, 0.f, 0.f, 0.f);      // bvhColor's initial value
    }
    if (h.x == CRT_MISS) return c;
    if (h.x >= sp.n_tris) { raise_corrupt(p.err, 11, h.x, sp.n_tris); return c; }
    const uint32_t L = __ldg(sp.inv_perm + h.x);
    if (L >= sp.n_tris) { raise_corrupt(p.err, 11, h.x, L); return c; }
    const uint32_t model = __float_as_uint(__ldg(p.xtri + 3 * static_cast<size_t>(L) + 1).w);
    const uint32_t mat = model < sp.n_models ? __ldg(sp.models + 17 * model + 16) : 0u;
    const float4 m = mat < sp.n_materials ? __ldg(sp.materials + mat) : make_float4(0.f, 0.f, 0.f, 0.f);
    c = make_float4(c.x + m.x, c.y + m.y, c.z + m.z, c.w + m.w);
    if (sp.flags & CRT_SHADE_WIREFRAME) {
        const float u = __uint_as_float(h.z), v = __uint_as_float(h.w);
        const float w = 1.0f - u - v;  // _Coords.z as rayTriangleIntersection forms it
        if (u < 0.02f || v < 0.02f || w < 0.02f) c = make_float4(0.f, 0.f, 0.f, 1.f);  // WIREFRAME_LINE_WIDTH
    }
    return c;
}

__global__ void __launch_bounds__(256) shade_kernel(TraceParams p, ShadeParams sp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n_rays) return;
    const uint4 h = __ldg(reinterpret_cast<const uint4*>(p.hits) + i);
    float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0;
    if (sp.flags & CRT_SHADE_BVH) {
        r0 = __ldg(reinterpret_cast<const float4*>(p.rays + i));
        r1 = __ldg(reinterpret_cast<const float4*>(p.rays + i) + 1);
    }
    sp.image[i] = shade_texel(p, sp, h, r0, r1);
}

void launch_shade(const TraceParams& p, const ShadeParams& sp, cudaStream_t s) {
    if (p.n_rays == 0) return;
    shade_kernel<<<(p.n_rays + 255) / 256, 256, 0, s>>>(p, sp);
}

// ------------------------------------------------------------- frames
// One frame in one launch (crt_trace_frame, crt_render_frame): a thread
// generates pixel i's camera ray, traces it to the closest hit and, with a
// light, traces that hit's shadow ray to any hit at once, while the nodes
// around the hit are still cached; with SHADE it also writes the pixel's
// texel.  The rays, hits and texels are the ones the separate raygen, trace,
// shadow-ray and shade calls produce.
struct FrameParams {
    const crt_camera* cam;
    uint32_t width, height, y0, rows;
    int shadows;
    float lx, ly, lz;
    crt_hit* hits_shadow;
};

// Pixel i over the binary nodes.
template <bool WT, int STACK, bool SHADE>
__device__ __forceinline__ void frame_pixel(const TraceParams& p, const FrameParams& f, const ShadeParams& sp, uint32_t i) {
    const uint32_t y = i / f.width, x = i - y * f.width;
    float4 r0, r1;
    camera_ray(f.cam, x, y, f.width, f.height, r0, r1);
    const uint4 h = trace_one<false, WT, STACK, false, 0>(p, i, r0, r1);
    if (!SHADE || p.hits) reinterpret_cast<uint4*>(p.hits)[i] = h;
    if (SHADE) sp.image[i] = shade_texel(p, sp, h, r0, r1);
    if (!f.shadows) return;
    uint4 hs = make_uint4(CRT_MISS, 0u, 0u, 0u);
    if (h.x != CRT_MISS) {
        float4 s0, s1;
        shadow_ray(r0, r1, h, f.lx, f.ly, f.lz, s0, s1);
        hs = trace_one<true, WT, STACK, false, 0>(p, i, s0, s1);
    }
    reinterpret_cast<uint4*>(f.hits_shadow)[i] = hs;
}

// Thread t takes pixel ray_of_thread(t) of the image rows [y0, y0 + rows).
template <bool WT, int STACK, int BLOCK, bool SHADE>
__global__ void __launch_bounds__(BLOCK) frame_kernel(TraceParams p, FrameParams f, ShadeParams sp) {
    const uint32_t t_id = blockIdx.x * BLOCK + threadIdx.x;
    if (t_id >= f.width * f.rows) return;
    frame_pixel<WT, STACK, SHADE>(p, f, sp, f.y0 * f.width + ray_of_thread(t_id, p.tile_width));
}

// The same over the compressed nodes: a warp takes a tile of 32 pixels (warp w
// tile w, then tiles from the counter while there are any), walks its
// camera rays together, then their shadow rays, testing a leaf as soon as a
// lane holds one (coherent lanes reach theirs together; waiting for two: 3 %
// slower).  Pixels with a ray of the binary walk go to the list `left` for
// frame_left_kernel.
//
// Bound by the ALU pipe (65-71 % busy, 18-22 of 32 threads per instruction) and
// by the rays of the longest walks at the end (an SM is busy 82-86 % of the
// launch).  Against one thread per pixel over the binary nodes (41 %, 10-15
// threads): 160x120 over 2,003 triangles 36 -> 25 us, 512x512 over 65,536 (the
// shader's predicate) 244 -> 180 us, 1920x1080 with shadow rays over 1.31 M 831 ->
// 720 us, 1280x720 over 2.0 M clustered 540 -> 372 us.  One thread per pixel over
// these nodes, its stack in local memory, was slower than either (65,536: 414 us
// a call against 282).
template <bool WT, bool SHADE, bool COUNT>
__global__ void __launch_bounds__(kWalk4Block, kWalk4Blocks)
    frame_walk4_kernel(const TraceParams p, const FrameParams f, const ShadeParams sp, Walk4Counters* ctr,
                       uint32_t* __restrict__ left, uint32_t* host_left) {
    __shared__ uint2 s_st[kWalk4Shared + 1][kWalk4Block];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t s_base = static_cast<uint32_t>(__cvta_generic_to_shared(&s_st[1][threadIdx.x]));
    const uint32_t n = f.width * f.rows, tiles = (n + 31u) / 32u, warps = gridDim.x * (kWalk4Block / 32);
    const bool walkable = __ldg(p.cw_bad) == 0u && p.n_nodes > 2;
    uint2 st[kWalk4Local];
    Walk4Lane L{};
    L.cw = p.cwide;
    L.xtri = p.xtri;
    L.abs_eps = p.abs_eps;
    uint32_t tile = blockIdx.x * (kWalk4Block / 32) + (threadIdx.x >> 5);
    while (tile < tiles) {
        const uint32_t t = 32u * tile + lane;
        const bool valid = t < n;
        const uint32_t i = f.y0 * f.width + ray_of_thread(valid ? t : 0u, p.tile_width);
        const uint32_t y = i / f.width, x = i - y * f.width;
        float4 r0, r1;
        camera_ray(f.cam, x, y, f.width, f.height, r0, r1);
        bool redo = !L.template start<WT>(s_base, r0, r1, walkable);
        if (!valid) L.stop(s_base);
        walk4_run<false, WT, 1, COUNT>(L, s_base, st, 32);
        redo = redo || L.redo;
        const uint4 h = redo ? make_uint4(CRT_MISS, 0u, 0u, 0u) : L.hit();
        // the ray again: what the walk keeps of it
        r0 = make_float4(L.o.x, L.o.y, L.o.z, 0.f);
        r1 = make_float4(L.d.x, L.d.y, L.d.z, __int_as_float(0x7F800000));
        if (valid && !redo) {
            if (!SHADE || p.hits) reinterpret_cast<uint4*>(p.hits)[i] = h;
            if (SHADE) sp.image[i] = shade_texel(p, sp, h, r0, r1);
        }
        if (f.shadows) {
            float4 s0, s1;
            shadow_ray(r0, r1, h, f.lx, f.ly, f.lz, s0, s1);  // empty where the primary ray missed
            redo = !L.template start<WT>(s_base, s0, s1, walkable) || redo;
            if (!valid) L.stop(s_base);
            walk4_run<true, WT, 1, COUNT>(L, s_base, st, 32);
            redo = redo || L.redo;
            if (valid && !redo) reinterpret_cast<uint4*>(f.hits_shadow)[i] = L.hit();
        }
        if (valid && redo) {  // past the list the host does the whole image again
            const uint32_t k = atomicAdd(&ctr->left, 1u);
            if (k < kWalkLeft) left[k] = i;
        }
        uint32_t next = tiles;
        if (tiles > warps) {
            if (lane == 0) next = warps + atomicAdd(&ctr->taken, 1u);
            next = __shfl_sync(0xFFFFFFFFu, next, 0);
        }
        tile = next;
    }
    if (COUNT && p.stats) {
        atomicAdd(p.stats + 0, static_cast<unsigned long long>(L.fetched));
        atomicAdd(p.stats + 1, static_cast<unsigned long long>(L.tested));
    }
    walk4_finish(ctr, host_left, p.cw_bad);
}

template <bool WT, int STACK, bool SHADE>
__global__ void __launch_bounds__(kWalk4Block)
    frame_left_kernel(TraceParams p, FrameParams f, ShadeParams sp, uint32_t n, const uint32_t* __restrict__ left) {
    n = min(n, kWalkLeft);
    for (uint32_t k = blockIdx.x * kWalk4Block + threadIdx.x; k < n; k += gridDim.x * kWalk4Block) {
        const uint32_t i = left[k];
        if (i >= p.n_rays) raise_corrupt(p.err, 7, k, i);
        else frame_pixel<WT, STACK, SHADE>(p, f, sp, i);
    }
}

// The frame, or with left != 0 the pixels that its launch left over.
template <bool WT, bool SHADE>
static void launch_frame_walk4(const TraceParams& p, const FrameParams& f, const ShadeParams& sp, bool deep,
                               const WalkScratch& w, uint32_t left, cudaStream_t s) {
    static int grid = 0;
    if (grid == 0) {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, frame_walk4_kernel<WT, SHADE, false>, kWalk4Block, 0);
        grid = kNumSms * (per_sm > 0 ? per_sm : 1);
    }
    if (left != 0) {
        const uint32_t few = (left + kWalk4Block - 1) / kWalk4Block;
        if (deep) frame_left_kernel<WT, 1024, SHADE><<<few, kWalk4Block, 0, s>>>(p, f, sp, left, w.left);
        else frame_left_kernel<WT, 64, SHADE><<<few, kWalk4Block, 0, s>>>(p, f, sp, left, w.left);
        return;
    }
    Walk4Counters* ctr = reinterpret_cast<Walk4Counters*>(w.ctr);
    const uint32_t want = (f.width * f.rows + kWalk4Block - 1) / kWalk4Block;
    const uint32_t blocks = want < static_cast<uint32_t>(grid) ? want : static_cast<uint32_t>(grid);
    if (p.stats) frame_walk4_kernel<WT, SHADE, true><<<blocks, kWalk4Block, 0, s>>>(p, f, sp, ctr, w.left, w.host_left);
    else frame_walk4_kernel<WT, SHADE, false><<<blocks, kWalk4Block, 0, s>>>(p, f, sp, ctr, w.left, w.host_left);
}

template <bool WT, int BLOCK, bool SHADE>
static void launch_frame_s(const TraceParams& p, const crt_camera* cam, uint32_t width, uint32_t height, uint32_t y0,
                           uint32_t rows, const float* light, crt_hit* hits_shadow, bool deep, const ShadeParams& sp,
                           const WalkScratch& w, uint32_t left, cudaStream_t s) {
    const uint32_t grid = (width * rows + BLOCK - 1) / BLOCK;
    if (grid == 0) return;
    const int sh = light != nullptr;
    const FrameParams f{cam, width, height, y0, rows, sh, sh ? light[0] : 0.f, sh ? light[1] : 0.f, sh ? light[2] : 0.f,
                        hits_shadow};
    if (p.cwide) launch_frame_walk4<WT, SHADE>(p, f, sp, deep, w, left, s);
    else if (deep) frame_kernel<WT, 1024, BLOCK, SHADE><<<grid, BLOCK, 0, s>>>(p, f, sp);
    else frame_kernel<WT, 64, BLOCK, SHADE><<<grid, BLOCK, 0, s>>>(p, f, sp);
}

template <bool WT, int BLOCK>
static void launch_frame_b(const TraceParams& p, const crt_camera* cam, uint32_t width, uint32_t height, uint32_t y0,
                           uint32_t rows, const float* light, crt_hit* hits_shadow, bool deep, const ShadeParams* shade,
                           const WalkScratch& w, uint32_t left, cudaStream_t s) {
    if (shade) launch_frame_s<WT, BLOCK, true>(p, cam, width, height, y0, rows, light, hits_shadow, deep, *shade, w, left, s);
    else launch_frame_s<WT, BLOCK, false>(p, cam, width, height, y0, rows, light, hits_shadow, deep, ShadeParams{}, w, left, s);
}

void launch_frame(const TraceParams& p, const crt_camera* cam, uint32_t width, uint32_t height, uint32_t y0,
                  uint32_t rows, const float* light, crt_hit* hits_shadow, uint32_t flags, int block,
                  const ShadeParams* shade, const WalkScratch& w, uint32_t left, cudaStream_t s) {
    const bool wt = flags & CRT_TRI_WATERTIGHT;
    const bool deep = (flags >> 16) != 0;
    if (wt) {
        if (block == 256) launch_frame_b<true, 256>(p, cam, width, height, y0, rows, light, hits_shadow, deep, shade, w, left, s);
        else if (block == 64) launch_frame_b<true, 64>(p, cam, width, height, y0, rows, light, hits_shadow, deep, shade, w, left, s);
        else launch_frame_b<true, 128>(p, cam, width, height, y0, rows, light, hits_shadow, deep, shade, w, left, s);
    } else {
        if (block == 256) launch_frame_b<false, 256>(p, cam, width, height, y0, rows, light, hits_shadow, deep, shade, w, left, s);
        else if (block == 64) launch_frame_b<false, 64>(p, cam, width, height, y0, rows, light, hits_shadow, deep, shade, w, left, s);
        else launch_frame_b<false, 128>(p, cam, width, height, y0, rows, light, hits_shadow, deep, shade, w, left, s);
    }
}

}  // namespace crt
