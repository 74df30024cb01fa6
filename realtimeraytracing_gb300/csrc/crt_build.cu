// BVH build kernels of libcrt: scene box, Morton codes, Onesweep LSD radix
// sort of (code, index), PLOC iterations and the DFS node layout.
//
// Reference: srcCommon/scene/geometry/bvh.cpp (CPU, OpenMP) and the DFS
// flattening in srcOpenGL/scene/scene.cpp:189-208.  Every float result is
// bit-identical to the reference's (this file is compiled with -fmad=false).
#include <array>
#include <cooperative_groups.h>
#include <cstdint>
#include <cuda_runtime.h>
#include <map>
#include <mutex>

#include "crt_build.cuh"
#include "crt_common.cuh"
#include "crt_host.h"

namespace crt {

// =========================================================== K1: scene box
// getSceneAABB (bvh.cpp:235-251) folds max(cur, max(p0, max(p1, p2))) over
// all n_buffer records in order.  That fold ignores NaN candidates and keeps
// the earliest of equal values, so it equals the leftmost arg-max over
// non-NaN per-triangle values — an associative reduction.  Each candidate is
// keyed (ordered value, index); the winner's exact value (sign of zero
// included) is recomputed from its triangle.

struct TriExtent { float hi[3], lo[3]; };

__device__ __forceinline__ TriExtent tri_extent(const TriRec& t, const float* __restrict__ models) {
    const float* M = models + 16 * (t.model & (kMaxModels - 1));
    const float4 p0 = mat_vec(M, t.p0), p1 = mat_vec(M, t.p1), p2 = mat_vec(M, t.p2);
    TriExtent e;
    e.hi[0] = max_std(p0.x, max_std(p1.x, p2.x));
    e.hi[1] = max_std(p0.y, max_std(p1.y, p2.y));
    e.hi[2] = max_std(p0.z, max_std(p1.z, p2.z));
    e.lo[0] = min_std(p0.x, min_std(p1.x, p2.x));
    e.lo[1] = min_std(p0.y, min_std(p1.y, p2.y));
    e.lo[2] = min_std(p0.z, min_std(p1.z, p2.z));
    return e;
}

__device__ __forceinline__ unsigned long long shfl_xor_u64(unsigned long long v, int m) {
    return __shfl_xor_sync(0xFFFFFFFFu, v, m);
}

__global__ void __launch_bounds__(256) scene_box_kernel(const crt_triangle* __restrict__ tris, uint32_t n_buffer,
                                                        const float* __restrict__ models, SceneState* st,
                                                        uint32_t* err) {
    unsigned long long kmax[3] = {0ull, 0ull, 0ull};
    unsigned long long kmin[3] = {~0ull, ~0ull, ~0ull};
    bool bad = false;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_buffer; i += gridDim.x * blockDim.x) {
        const TriRec t = load_tri(tris, i);
        bad |= t.model >= kMaxModels;
        const TriExtent e = tri_extent(t, models);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (e.hi[a] == e.hi[a]) {
                const unsigned long long k = (static_cast<unsigned long long>(ordered_key(e.hi[a])) << 32) | (0xFFFFFFFFu - i);
                kmax[a] = k > kmax[a] ? k : kmax[a];
            }
            if (e.lo[a] == e.lo[a]) {
                const unsigned long long k = (static_cast<unsigned long long>(ordered_key(e.lo[a])) << 32) | i;
                kmin[a] = k < kmin[a] ? k : kmin[a];
            }
        }
    }
    if (bad) raise_error(err, kDevBadModel);
#pragma unroll
    for (int a = 0; a < 3; ++a)
        for (int m = 16; m > 0; m >>= 1) {
            const unsigned long long x = shfl_xor_u64(kmax[a], m), y = shfl_xor_u64(kmin[a], m);
            kmax[a] = x > kmax[a] ? x : kmax[a];
            kmin[a] = y < kmin[a] ? y : kmin[a];
        }
    __shared__ unsigned long long s_k[6][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int a = 0; a < 3; ++a) { s_k[a][warp] = kmax[a]; s_k[3 + a][warp] = kmin[a]; }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int a = threadIdx.x;
        const int nw = blockDim.x >> 5;
        unsigned long long v = s_k[a][0];
        for (int w = 1; w < nw; ++w) v = (a < 3) ? (s_k[a][w] > v ? s_k[a][w] : v) : (s_k[a][w] < v ? s_k[a][w] : v);
        if (a < 3) atomicMax(&st->key_max[a], v); else atomicMin(&st->key_min[a - 3], v);
    }
    // The last block to finish turns the keys into the box and the cube.
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(&st->blocks_done, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    const float kInf = __int_as_float(0x7F800000);
    float smin[3], smax[3];
    for (int a = 0; a < 3; ++a) {
        const unsigned long long kx = atomicAdd(&st->key_max[a], 0ull);
        const unsigned long long kn = atomicAdd(&st->key_min[a], 0ull);
        smax[a] = -kInf;
        smin[a] = kInf;
        if (kx != 0ull) smax[a] = tri_extent(load_tri(tris, 0xFFFFFFFFu - static_cast<uint32_t>(kx)), models).hi[a];
        if (kn != ~0ull) smin[a] = tri_extent(load_tri(tris, static_cast<uint32_t>(kn)), models).lo[a];
        st->key_max[a] = 0ull;
        st->key_min[a] = ~0ull;
    }
    st->blocks_done = 0u;
    // getCircumscribedCube (bvh.cpp:253-303): X is chosen whenever distX > 0.
    float cmn[3] = {smin[0], smin[1], smin[2]}, cmx[3] = {smax[0], smax[1], smax[2]};
    const float dX = smax[0] - smin[0], dY = smax[1] - smin[1], dZ = smax[2] - smin[2];
    float maxDist = 0.f;
    int axis;
    if (dX > maxDist) { maxDist = dX; axis = 0; }
    else if (dY > maxDist) { maxDist = dY; axis = 1; }
    else { maxDist = dZ; axis = 2; }
    const float dist[3] = {dX, dY, dZ};
    for (int a = 0; a < 3; ++a) {
        if (a == axis) continue;
        const float delta = (maxDist - dist[a]) / 2.f;
        cmx[a] += delta;
        cmn[a] -= delta;
    }
    for (int a = 0; a < 3; ++a) {
        st->scene_min[a] = smin[a];
        st->scene_max[a] = smax[a];
        st->cube_min[a] = cmn[a];
        st->cube_len[a] = cmx[a] - cmn[a];  // getNormalizedCentroids (bvh.cpp:319-321)
    }
    st->abs_eps = scene_abs_eps(smin, smax);
}

// ====================================================== K1: Morton codes
__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {  // bvh.cpp:350-356
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__device__ __forceinline__ uint32_t to_u10(float x) {  // bvh.cpp:363-367
    x = min_std(max_std(x * 1024.0f, 0.0f), 1023.0f);
    return __float2uint_rz(x);  // NaN -> 0, as on the reference's hosts
}

// The digit histograms of the radix passes: for each of PASSES digit places
// of BITS bits, one count per digit value, in shared memory (s_hist[p *
// 2^BITS + d]).  The sort's counting step — with 1-bit digits it is the
// reference's per-bit histogram (histogramOfGlobalDigitCounts.glsl:31-59).
template <int BITS, int PASSES>
__device__ __forceinline__ void add_digit_counts(uint32_t key, uint32_t* s_hist) {
    constexpr uint32_t RADIX = 1u << BITS;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) atomicAdd(&s_hist[p * RADIX + ((key >> (p * BITS)) & (RADIX - 1))], 1u);
}

// Block-wide inclusive scan, in thread order, of one 64-bit value per thread
// (the radix passes pack two 32-bit counts into it); s_wsum holds one entry
// per warp.  Every thread of the block must call it.
template <int BLOCK>
__device__ __forceinline__ unsigned long long block_inclusive_scan_u64(unsigned long long v,
                                                                       unsigned long long* s_wsum) {
    constexpr int WARPS = BLOCK / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) s_wsum[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long run = 0;
        for (int w = 0; w < WARPS; ++w) { const unsigned long long t = s_wsum[w]; s_wsum[w] = run; run += t; }
    }
    __syncthreads();
    return v + s_wsum[warp];
}

// Centroid (triangle.cpp:31-33), normalisation (bvh.cpp:314-328) and code
// (bvh.cpp:358-372), plus the digit histograms of all radix passes.
template <int BITS>
__global__ void __launch_bounds__(256) morton_kernel(const crt_triangle* __restrict__ tris, uint32_t n,
                                                     const float* __restrict__ models_third,
                                                     const SceneState* __restrict__ st,
                                                     uint32_t* __restrict__ codes, uint32_t* __restrict__ hist) {
    constexpr int RADIX = 1 << BITS;
    constexpr int PASSES = (30 + BITS - 1) / BITS;
    __shared__ uint32_t s_hist[PASSES * RADIX];
    for (int i = threadIdx.x; i < PASSES * RADIX; i += blockDim.x) s_hist[i] = 0u;
    __syncthreads();
    const float cmx = st->cube_min[0], cmy = st->cube_min[1], cmz = st->cube_min[2];
    const float lx = st->cube_len[0], ly = st->cube_len[1], lz = st->cube_len[2];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const TriRec t = load_tri(tris, i);
        const float* M3 = models_third + 16 * (t.model & (kMaxModels - 1));
        float4 s;
        s.x = t.p0.x + t.p1.x + t.p2.x;
        s.y = t.p0.y + t.p1.y + t.p2.y;
        s.z = t.p0.z + t.p1.z + t.p2.z;
        s.w = t.p0.w + t.p1.w + t.p2.w;
        const float4 c = mat_vec(M3, s);
        const float nx = (c.x - cmx) / lx, ny = (c.y - cmy) / ly, nz = (c.z - cmz) / lz;
        const uint32_t code = (expand_bits(to_u10(nx)) << 2) | (expand_bits(to_u10(ny)) << 1) | expand_bits(to_u10(nz));
        codes[i] = code;
        add_digit_counts<BITS, PASSES>(code, s_hist);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < PASSES * RADIX; i += blockDim.x)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// ============================================== K2: Onesweep digit binning
// One stable counting pass over digit (key >> shift) & (RADIX-1) of a tile
// of BLOCK*KPT keys (Adinets & Merrill, "Onesweep", 2022):
//  * warp multisplit: each lane ORs its bit into the warp's shared-memory
//    mask of its digit, so the lanes holding the same digit read their group
//    back (fewer instructions than BITS ballots, and than match.any, on this
//    part); every lane reads the warp's count of its digit, then the highest
//    of the group adds the group's size (no branch to a leader, no shuffle);
//  * chained-scan decoupled look-back across tiles for the global digit
//    offsets; each digit's thread reads a window of LB_WIN predecessor tiles
//    per round trip with relaxed loads (flag and count share one word);
//  * a shared-memory staged scatter, first of the digit-carrying array
//    (keys, or values for SEG) then of the other, so that every warp's
//    global stores fall in a few contiguous runs.
// Pass 0 synthesises the values (iota), which makes the result the
// reference's std::sort of (code, index) pairs (bvh.cpp:214-232).
constexpr uint32_t kLbAgg = 1u << 30, kLbPrefix = 2u << 30, kLbMask = (1u << 30) - 1u;
constexpr int kLbWindow = 4;

// SEG: the digit is not taken from the key but is the segment (scene) whose
// range [seg_off[d], seg_off[d+1]) holds the value — one extra stable pass
// that groups concatenated scenes back together after the code passes.
template <int BITS, int BLOCK, int KPT, bool SEG>
__global__ void __launch_bounds__(BLOCK, 3) onesweep_kernel(const uint32_t* __restrict__ keys_in,
                                                            const uint32_t* __restrict__ vals_in,
                                                            uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                                            uint32_t n, int shift, const uint32_t* __restrict__ pass_hist,
                                                            uint32_t* lookback, uint32_t* ticket, uint32_t* err,
                                                            uint32_t spin_limit, const uint32_t* __restrict__ seg_off,
                                                            uint32_t n_seg) {
    constexpr int RADIX = 1 << BITS;
    constexpr int WARPS = BLOCK / 32;
    constexpr int TILE = BLOCK * KPT;
    static_assert(BLOCK >= RADIX, "one thread per digit");
    __shared__ uint32_t s_buf[TILE];            // staging for the scatter
    __shared__ uint32_t s_whist[WARPS][RADIX];  // per-warp digit counters, then per-warp offsets
    __shared__ uint32_t s_match[WARPS][RADIX];  // per-warp lane masks of the key being ranked
    __shared__ uint32_t s_start[RADIX];         // block-local exclusive digit start
    __shared__ uint32_t s_adj[RADIX];           // global destination of sorted slot i is s_adj[d] + i
    __shared__ unsigned long long s_wsum[WARPS];
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_seg[SEG ? RADIX + 1 : 1];
    __shared__ uint32_t s_timeout;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(ticket, 1u);
        s_timeout = 0u;
    }
    for (int i = threadIdx.x; i < WARPS * RADIX; i += BLOCK) {
        (&s_whist[0][0])[i] = 0u;
        (&s_match[0][0])[i] = 0u;
    }
    if (SEG)
        for (int i = threadIdx.x; i <= RADIX; i += BLOCK) s_seg[i] = (static_cast<uint32_t>(i) <= n_seg) ? seg_off[i] : 0xFFFFFFFFu;
    __syncthreads();
    auto digit_of = [&](uint32_t key, uint32_t val) -> uint32_t {
        if (!SEG) return (key >> shift) & (RADIX - 1);
        uint32_t lo = 0, hi = n_seg - 1;  // last segment start <= val
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (s_seg[mid] <= val) lo = mid; else hi = mid - 1;
        }
        return lo;
    };
    const uint32_t tile = s_tile;
    const uint64_t tile_base = static_cast<uint64_t>(tile) * TILE;
    if (tile_base >= n) return;
    const uint64_t rem = n - tile_base;
    const uint32_t tile_n = rem < static_cast<uint64_t>(TILE) ? static_cast<uint32_t>(rem) : static_cast<uint32_t>(TILE);
    // Warp w ranks the contiguous keys [w*32*KPT, (w+1)*32*KPT) of the tile, j-major.
    const uint32_t wofs = static_cast<uint32_t>(warp) * 32u * KPT + lane;
    const uint32_t* kin = keys_in + tile_base;
    const uint32_t* vin = vals_in ? vals_in + tile_base : nullptr;
    const uint32_t ibase = static_cast<uint32_t>(tile_base);

    uint32_t key[KPT], val[KPT], pos[KPT];
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
        const uint32_t lo = wofs + j * 32u;
        key[j] = lo < tile_n ? __ldg(kin + lo) : 0u;
        val[j] = lo < tile_n ? (vin ? __ldg(vin + lo) : ibase + lo) : 0u;
    }
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t* my_hist = &s_whist[warp][0];
    uint32_t* my_match = &s_match[warp][0];
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
        const bool ok = wofs + j * 32u < tile_n;
        const uint32_t d = ok ? digit_of(key[j], val[j]) : 0u;
        // the lanes holding digit d: each sets its bit in the warp's mask of d
        if (ok) atomicOr(my_match + d, 1u << lane);
        __syncwarp();
        const uint32_t peers = ok ? my_match[d] : 0u;
        // every lane reads its digit's running count (the lanes of one digit
        // read one word: a broadcast); after the warp has read, the group's
        // highest lane alone adds the group's size and clears the mask
        const uint32_t base = my_hist[d];
        __syncwarp();
        if (ok && (peers >> lane) == 1u) {
            my_hist[d] = base + static_cast<uint32_t>(__popc(peers));
            my_match[d] = 0u;
        }
        pos[j] = base + __popc(peers & lt_mask);
        __syncwarp();
    }
    __syncthreads();

    // Per digit: exclusive over warps, tile total, publication.
    const int d = threadIdx.x;
    uint32_t total = 0, excl = 0;
    if (d < RADIX) {
        for (int w = 0; w < WARPS; ++w) {
            const uint32_t c = s_whist[w][d];
            s_whist[w][d] = total;
            total += c;
        }
        st_relaxed_u32(lookback + static_cast<size_t>(tile) * RADIX + d, (tile == 0 ? kLbPrefix : kLbAgg) | total);
    }
    // Block-wide exclusive scans over digits of (tile totals) and (global
    // histogram), packed as two 32-bit halves of one 64-bit scan.
    const uint32_t gh = (d < RADIX) ? pass_hist[d] : 0u;
    const uint32_t a = (d < RADIX) ? total : 0u;
    const unsigned long long packed =
        block_inclusive_scan_u64<BLOCK>((static_cast<unsigned long long>(gh) << 32) | a, s_wsum);
    if (d < RADIX) {
        if (tile > 0) {
            // Look-back: sum the predecessors' counts of digit d down to the
            // nearest inclusive prefix; tile 0 always publishes one.
            int64_t k = static_cast<int64_t>(tile) - 1;
            SpinBound spin(spin_limit);
            while (true) {
                uint32_t v[kLbWindow];
#pragma unroll
                for (int q = 0; q < kLbWindow; ++q)
                    v[q] = (k - q >= 0) ? ld_relaxed_u32(lookback + static_cast<size_t>(k - q) * RADIX + d) : kLbPrefix;
                int q = 0;
                bool done = false;
#pragma unroll
                for (; q < kLbWindow; ++q) {
                    const uint32_t f = v[q] & ~kLbMask;
                    if (f == 0u) break;
                    excl += v[q] & kLbMask;
                    if (f == kLbPrefix) { done = true; break; }
                }
                if (done) break;
                k -= q;
                if (q < kLbWindow && !spin.step()) {
                    raise_error(err, kDevTimeout);
                    s_timeout = 1u;
                    break;
                }
            }
            st_relaxed_u32(lookback + static_cast<size_t>(tile) * RADIX + d, kLbPrefix | (excl + total));
        }
        const uint32_t incl_a = static_cast<uint32_t>(packed & 0xFFFFFFFFull);
        const uint32_t incl_g = static_cast<uint32_t>(packed >> 32);
        s_start[d] = incl_a - a;
        s_adj[d] = (incl_g - gh) + excl - (incl_a - a);
    }
    __syncthreads();
    if (s_timeout) return;  // the prefix is incomplete: write nothing
    // Tile-local sorted slot of each element.
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
        const bool ok = wofs + j * 32u < tile_n;
        const uint32_t dd = ok ? digit_of(key[j], val[j]) : 0u;
        pos[j] += s_start[dd] + my_hist[dd];
        if (ok) s_buf[pos[j]] = SEG ? val[j] : key[j];
    }
    __syncthreads();
    uint32_t dst[KPT];
#pragma unroll
    for (int k = 0; k < KPT; ++k) {
        const uint32_t i = k * BLOCK + threadIdx.x;
        if (i < tile_n) {
            const uint32_t x = s_buf[i];
            dst[k] = s_adj[SEG ? digit_of(0u, x) : digit_of(x, 0u)] + i;
            if (dst[k] >= n) {  // only a corrupt histogram gets here
                raise_corrupt(err, 17, tile, dst[k]);
                dst[k] = 0xFFFFFFFFu;
                continue;
            }
            if (SEG) vals_out[dst[k]] = x;
            else keys_out[dst[k]] = x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < KPT; ++j)
        if (wofs + j * 32u < tile_n) s_buf[pos[j]] = SEG ? key[j] : val[j];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KPT; ++k) {
        const uint32_t i = k * BLOCK + threadIdx.x;
        if (i < tile_n && dst[k] != 0xFFFFFFFFu) {
            if (SEG) keys_out[dst[k]] = s_buf[i];
            else vals_out[dst[k]] = s_buf[i];
        }
    }
}

// A cluster record or node box, 32 aligned bytes in one access: two 16-byte ones
// move every sector twice.  (Leaf boxes, the layout's gathers and its traversal nodes:
// 16.8 M triangles, leaves and PLOC 5.09 -> 4.75 ms, layout 2.83 -> 2.74; 1.31 M
// triangles, layout 0.210 -> 0.181.)  Plain accesses: grid_barrier's release and acquire
// order them between iterations.
__device__ __forceinline__ void ld_record(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st_record(float4* p, const float4& a, const float4& b) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                 "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}
// The same from memory that no thread of the launch writes.
__device__ __forceinline__ void ld_record_nc(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

constexpr uint32_t kLayoutUnset = 0xFFFFFFFFu;  // a place not yet published (dataflow layout)

// ==================================================== leaf clusters
// plocPreprocessing (bvh.cpp:26-46): sorted position i holds the leaf of
// triangle perm[i] with AABB::buildFromTriangle's box (bvh.cpp:383-399).
// Also stores the model-transformed vertices the traversal tests against,
// in sorted order (the layout moves them into tree order).
__global__ void __launch_bounds__(256) leaf_init_kernel(const crt_triangle* __restrict__ tris, uint32_t n,
                                                        const float* __restrict__ models,
                                                        const uint32_t* __restrict__ perm,
                                                        float4* __restrict__ node_box, float4* __restrict__ clusters,
                                                        float4* __restrict__ xtri, uint2* it, uint2* __restrict__ pf,
                                                        uint32_t* err) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) it[0] = make_uint2(n, n);
    if (i >= n) return;
    pf[i] = make_uint2(kLayoutUnset, 0u);  // the layout's places arrive from each node's parent
    const uint32_t ti = perm[i];
    if (ti >= n) { raise_corrupt(err, 1, i, ti); return; }
    const TriRec t = load_tri(tris, ti);
    const float* M = models + 16 * (t.model & (kMaxModels - 1));
    const float4 p0 = mat_vec(M, t.p0), p1 = mat_vec(M, t.p1), p2 = mat_vec(M, t.p2);
    float4 mn, mx;
    mn.x = min_std(p0.x, min_std(p1.x, p2.x));
    mn.y = min_std(p0.y, min_std(p1.y, p2.y));
    mn.z = min_std(p0.z, min_std(p1.z, p2.z));
    mx.x = max_std(p0.x, max_std(p1.x, p2.x));
    mx.y = max_std(p0.y, max_std(p1.y, p2.y));
    mx.z = max_std(p0.z, max_std(p1.z, p2.z));
    mn.w = __uint_as_float(ti);
    mx.w = 0.f;
    st_record(node_box + 2 * static_cast<size_t>(i), mn, mx);
    mn.w = __uint_as_float(i);
    mx.w = __uint_as_float(1u);
    st_record(clusters + 2 * static_cast<size_t>(i), mn, mx);
    // sorted order: triangle id in the first .w, model id in the second
    // (read by the shading pass)
    xtri[3 * static_cast<size_t>(i) + 0] = make_float4(p0.x, p0.y, p0.z, __uint_as_float(ti));
    xtri[3 * static_cast<size_t>(i) + 1] = make_float4(p1.x, p1.y, p1.z, __uint_as_float(t.model));
    xtri[3 * static_cast<size_t>(i) + 2] = make_float4(p2.x, p2.y, p2.z, 0.f);
}

// ================================================ K3: one PLOC iteration
// For the n live clusters (Morton order, 32-byte records: min.xyz|node id,
// max.xyz|leaf count) a tile starting at position s with R = radius does:
//   nearest neighbour of the positions [s - R, e + R) in [i-R, i+R] by surface
//     area of the merged box, first strict minimum = lowest j on ties
//     (bvh.cpp:193-210);
//   merge decisions for its own ploc_own(R) = TILE-3R positions [s, e):
//     mutual pairs merge at the lower position (bvh.cpp:159-191);
//   exclusive scan of survivors and compaction (bvh.cpp:125-156), with the
//     scan across tiles done by decoupled look-back,
// so one launch is one reference iteration.  New nodes get ids it[iter].y +
// (merges before them); the last tile writes it[iter+1] = (live clusters,
// next id).
//
// Boxes of positions [s-2R, e+2R) are staged in shared memory as separate
// min/max coordinate arrays, position s-2R+w at index w; window entries
// outside [0, n) hold an infinite box (area +inf, never chosen under the strict
// minimum, as the reference never considers them).
//
// PLOC of 16.8 M uniform triangles 6.56 -> 5.09 ms, of 1.31 M 0.75 -> 0.66, by
// three changes: each pair's area is computed once (ploc_nearest_sym: 6.13 ms),
// tiles are opened and closed a tile apart (ploc_open: 5.31), and records move in
// 32-byte accesses, a window's all in flight at once.  A tile's 23.6 k cycles (three
// blocks an SM) are now: window 2.3, search 8.9, decisions 3.5, look-back 2.5,
// records 6.4; the search's instructions alone would take about 10.
//
// The search compares areas computed from fminf/fmaxf boxes; those differ
// from the std::min/max boxes only in the sign of a zero, which changes no
// difference max - min and no comparison, so the chosen neighbour is the
// reference's.  Stored boxes use std::min/max semantics.
constexpr unsigned long long kPlAgg = 1ull << 62, kPlPrefix = 2ull << 62;
constexpr unsigned long long kPlMask31 = (1ull << 31) - 1ull;

__device__ __forceinline__ float sa_merged(float4 amn, float4 amx, float4 bmn, float4 bmx) {
    const float dx = fmaxf(amx.x, bmx.x) - fminf(amn.x, bmn.x);
    const float dy = fmaxf(amx.y, bmx.y) - fminf(amn.y, bmn.y);
    const float dz = fmaxf(amx.z, bmx.z) - fminf(amn.z, bmn.z);
    return 2.0f * (dx * dy + dy * dz + dz * dx);
}

template <int TILE, int BLOCK, int MAXR>
struct __align__(16) PlocSmem {
    static_assert(TILE == 4 * BLOCK, "four nearest-neighbour positions per thread");
    static constexpr int kWin = TILE + 2 * MAXR;  // positions [s-2R, e+2R), e - s <= TILE - 2R
    static_assert(kWin % 4 == 0, "aligned coordinate arrays");
    float mnx[kWin], mny[kWin], mnz[kWin], mxx[kWin], mxy[kWin], mxz[kWin];
    uint32_t id[kWin], lc[kWin];
    __align__(16) uint32_t nn[TILE];  // nearest neighbour of position s - R + i
    unsigned long long wsum[BLOCK / 32];
    unsigned long long prefix;
};

__device__ __forceinline__ float2 lds2(const float* a) { return *reinterpret_cast<const float2*>(a); }

// Nearest neighbours of this thread's positions q0..q0+3, q0 = s - R + 4t (radii
// without a compiled search, and the cluster kernel).  Each thread keeps the boxes
// of its 4 positions in registers and walks the 2R+4 boxes around them once,
// reading two consecutive entries per 8-byte shared load.
// RC > 0: the radius is the compile-time RC (even); RC == 0:
// runtime radius R, scalar loads.
template <int RC, int TILE, int BLOCK, int MAXR>
__device__ __forceinline__ void ploc_nearest(PlocSmem<TILE, BLOCK, MAXR>& S, int s, int e, int n, int R_rt) {
    const int R = RC > 0 ? RC : R_rt;
    const int q0 = s - R + 4 * static_cast<int>(threadIdx.x);
    if (q0 >= e + R) return;  // none of its positions is stored (no barrier in here)
    const int wq = 4 * static_cast<int>(threadIdx.x) + R;  // window index of q0
    float amnx[4], amny[4], amnz[4], amxx[4], amxy[4], amxz[4], best[4];
    int bj[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        amnx[i] = S.mnx[wq + i]; amny[i] = S.mny[wq + i]; amnz[i] = S.mnz[wq + i];
        amxx[i] = S.mxx[wq + i]; amxy[i] = S.mxy[wq + i]; amxz[i] = S.mxz[wq + i];
        best[i] = __int_as_float(0x7F800000);
        bj[i] = q0 + i;
    }
    // candidate at window offset d (position q0 + d) for own position i
    auto visit = [&](int d, int i, float bnx, float bny, float bnz, float bxx, float bxy, float bxz) {
        const float dx = fmaxf(amxx[i], bxx) - fminf(amnx[i], bnx);
        const float dy = fmaxf(amxy[i], bxy) - fminf(amny[i], bny);
        const float dz = fmaxf(amxz[i], bxz) - fminf(amnz[i], bnz);
        const float v = 2.0f * (dx * dy + dy * dz + dz * dx);
        if (v < best[i]) { best[i] = v; bj[i] = q0 + d; }
    };
    if (RC > 0) {
        static_assert(RC % 2 == 0, "aligned window pairs");
#pragma unroll
        for (int g = -RC; g <= RC + 2; g += 2) {
            const int w = wq + g;  // even: an 8-byte aligned pair of entries
            const float2 nx = lds2(S.mnx + w), ny = lds2(S.mny + w), nz = lds2(S.mnz + w);
            const float2 xx = lds2(S.mxx + w), xy = lds2(S.mxy + w), xz = lds2(S.mxz + w);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int d = g + u;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int k = d - i;
                    if (k != 0 && k >= -RC && k <= RC)
                        visit(d, i, u ? nx.y : nx.x, u ? ny.y : ny.x, u ? nz.y : nz.x, u ? xx.y : xx.x,
                              u ? xy.y : xy.x, u ? xz.y : xz.x);
                }
            }
            // keeps the next pair's loads below this pair's work: without it
            // every load of the unrolled walk is hoisted and the persistent
            // kernels (80 registers at 3 blocks per SM) spill
            asm volatile("" ::: "memory");
        }
    } else {
        for (int d = -R; d <= R + 3; ++d) {
            const int w = wq + d;
            const float bnx = S.mnx[w], bny = S.mny[w], bnz = S.mnz[w], bxx = S.mxx[w], bxy = S.mxy[w], bxz = S.mxz[w];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int k = d - i;
                if (k != 0 && k >= -R && k <= R) visit(d, i, bnx, bny, bnz, bxx, bxy, bxz);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int p = q0 + i;
        if (p >= 0 && p < n && p < e + R) S.nn[4 * threadIdx.x + i] = static_cast<uint32_t>(bj[i]);
    }
}

// Nearest neighbour of position p, whose box is at window index w (window
// entries outside [0, n) infinite): the 2R candidates in increasing j (strict
// minimum: lowest j on ties).  RC > 0: compile-time radius.
template <int RC, int TILE, int BLOCK, int MAXR>
__device__ __forceinline__ uint32_t ploc_nearest_at(const PlocSmem<TILE, BLOCK, MAXR>& S, int p, int w, int R_rt) {
    const int R = RC > 0 ? RC : R_rt;
    const float amnx = S.mnx[w], amny = S.mny[w], amnz = S.mnz[w], amxx = S.mxx[w], amxy = S.mxy[w], amxz = S.mxz[w];
    float best = __int_as_float(0x7F800000);
    int bj = p;
    auto visit = [&](int d) {
        const int wj = w + d;
        const float dx = fmaxf(amxx, S.mxx[wj]) - fminf(amnx, S.mnx[wj]);
        const float dy = fmaxf(amxy, S.mxy[wj]) - fminf(amny, S.mny[wj]);
        const float dz = fmaxf(amxz, S.mxz[wj]) - fminf(amnz, S.mnz[wj]);
        const float v = 2.0f * (dx * dy + dy * dz + dz * dx);
        if (v < best) { best = v; bj = p + d; }
    };
    if (RC > 0) {
#pragma unroll
        for (int d = -RC; d <= RC; ++d)
            if (d != 0) visit(d);
    } else {
        for (int d = -R; d <= R; ++d)
            if (d != 0) visit(d);
    }
    return static_cast<uint32_t>(bj);
}

// A tile's shared memory, with the hand-over of ploc_nearest_sym between warps.
template <int TILE, int BLOCK, int MAXR>
struct PlocTileSmem : PlocSmem<TILE, BLOCK, MAXR> {
    static constexpr int kEdges = MAXR / 4 * (MAXR / 4 + 1) / 2;  // of a warp: 1 + 2 + ... groups of four
    float4 edge_v[BLOCK / 32][kEdges];
    uint32_t edge_i[BLOCK / 32][kEdges];
};

// Nearest neighbours of the positions [s - R, e + R) of a tile, each pair's area
// computed once.  Thread t has the positions q0 .. q0 + 3, q0 = s - 2R + 4t, and
// walks the groups of four after them as far as R reaches: an area counts for its
// own position (forward: the candidate is higher) and for the candidate
// (backward), whose best over this thread's four goes to the thread that owns it,
// d lanes up, or through shared memory into the next warp.  Ties go to the lowest
// j: backward over forward, farther backward groups over nearer ones, strict
// minima in ascending order otherwise.
//
// What bounds it: issue slots and the ALU pipe (six minima and maxima and two
// updates an area, against one update for each of two areas before).
template <int RC, int TILE, int BLOCK, int MAXR>
__device__ __forceinline__ void ploc_nearest_sym(PlocTileSmem<TILE, BLOCK, MAXR>& S, int s, int e, int n) {
    static_assert(RC % 4 == 0 && RC <= MAXR, "whole groups of four");
    constexpr int D = RC / 4;  // groups after its own that a thread's positions reach
    const int t = static_cast<int>(threadIdx.x), lane = t & 31, warp = t >> 5;
    const int q0 = s - 2 * RC + 4 * t, w0 = 4 * t;
    const float inf = __int_as_float(0x7F800000);
    float fb[4], bb[4];  // least area forward and backward
    int fj[4], bj[4];    // its candidate, from q0
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        fb[i] = bb[i] = inf;
        fj[i] = bj[i] = i;
    }
    const bool live = q0 - 4 * lane < e + RC;  // whole warps: some position is stored (candidates only go up)
    if (live) {
        auto four = [&](const float* a, int w, float (&r)[4]) {
            const float4 v = *reinterpret_cast<const float4*>(a + w);
            r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
        };
        float anx[4], any[4], anz[4], axx[4], axy[4], axz[4];
        four(S.mnx, w0, anx); four(S.mny, w0, any); four(S.mnz, w0, anz);
        four(S.mxx, w0, axx); four(S.mxy, w0, axy); four(S.mxz, w0, axz);
#pragma unroll
        for (int k = 1; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < k; ++i) {
                const float dx = fmaxf(axx[i], axx[k]) - fminf(anx[i], anx[k]);
                const float dy = fmaxf(axy[i], axy[k]) - fminf(any[i], any[k]);
                const float dz = fmaxf(axz[i], axz[k]) - fminf(anz[i], anz[k]);
                const float v = 2.0f * (dx * dy + dy * dz + dz * dx);
                if (v < fb[i]) { fb[i] = v; fj[i] = k; }
                if (v < bb[k]) { bb[k] = v; bj[k] = i; }
            }
#pragma unroll
        for (int g = 1; g <= D; ++g) {
            float bnx[4], bny[4], bnz[4], bxx[4], bxy[4], bxz[4], pv[4];
            four(S.mnx, w0 + 4 * g, bnx); four(S.mny, w0 + 4 * g, bny); four(S.mnz, w0 + 4 * g, bnz);
            four(S.mxx, w0 + 4 * g, bxx); four(S.mxy, w0 + 4 * g, bxy); four(S.mxz, w0 + 4 * g, bxz);
            uint32_t pi = 0u;  // the candidates' best among this thread's positions, a byte each
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                pv[u] = inf;
                uint32_t pu = 0u;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (4 * g + u - i > RC) continue;
                    const float dx = fmaxf(axx[i], bxx[u]) - fminf(anx[i], bnx[u]);
                    const float dy = fmaxf(axy[i], bxy[u]) - fminf(any[i], bny[u]);
                    const float dz = fmaxf(axz[i], bxz[u]) - fminf(anz[i], bnz[u]);
                    const float v = 2.0f * (dx * dy + dy * dz + dz * dx);
                    if (v < fb[i]) { fb[i] = v; fj[i] = 4 * g + u; }
                    if (v < pv[u]) { pv[u] = v; pu = static_cast<uint32_t>(i) << (8 * u); }
                }
                pi |= pu;
            }
            const uint32_t ri = __shfl_up_sync(0xFFFFFFFFu, pi, g);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float rv = __shfl_up_sync(0xFFFFFFFFu, pv[u], g);
                if (lane >= g && rv <= bb[u]) { bb[u] = rv; bj[u] = static_cast<int>(ri >> (8 * u) & 3u) - 4 * g; }
            }
            if (lane >= 32 - g) {  // the next warp's lane + g - 32
                S.edge_v[warp][g * (g - 1) / 2 + lane + g - 32] = make_float4(pv[0], pv[1], pv[2], pv[3]);
                S.edge_i[warp][g * (g - 1) / 2 + lane + g - 32] = pi;
            }
            asm volatile("" ::: "memory");  // the next group's loads stay below this group's work
        }
    }
    __syncthreads();
    if (!live) return;
    if (warp > 0)
        for (int g = lane + 1; g <= D; ++g) {  // groups that lie in the warp before
            const float4 v = S.edge_v[warp - 1][g * (g - 1) / 2 + lane];
            const uint32_t ri = S.edge_i[warp - 1][g * (g - 1) / 2 + lane];
            const float rv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (rv[u] <= bb[u]) { bb[u] = rv[u]; bj[u] = static_cast<int>(ri >> (8 * u) & 3u) - 4 * g; }
        }
    uint32_t j[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) j[i] = static_cast<uint32_t>(q0 + (fb[i] < bb[i] ? fj[i] : (bb[i] < inf ? bj[i] : i)));
    // four positions from a multiple of four: stored or not together but for the
    // ends of the array, past which nothing is read
    if (w0 >= RC && q0 + 3 >= 0 && q0 < min(n, e + RC)) *reinterpret_cast<uint4*>(S.nn + w0 - RC) = make_uint4(j[0], j[1], j[2], j[3]);
}

// One warp: (survivors, merges) of the tiles before `tile` (> 0).
__device__ __forceinline__ void ploc_look_back(uint32_t tile, const unsigned long long* lb_cur, uint32_t* err,
                                               uint32_t spin_limit, unsigned long long& ev, unsigned long long& em) {
    const int lane = threadIdx.x & 31;
    ev = em = 0;
    // Lane l reads the status word of tile k0 - l (32 predecessors per
    // round trip, nearest first); the sum runs down to the nearest
    // inclusive prefix.  (Four words per lane was measured slower:
    // the nearest prefix is usually a few tiles back.)
    long long k0 = static_cast<long long>(tile) - 1;
    SpinBound spin(spin_limit);
    while (true) {
        const long long k = k0 - lane;
        const unsigned long long v = k >= 0 ? ld_relaxed_u64(&lb_cur[k]) : kPlPrefix;
        const unsigned long long f = v & (3ull << 62);
        const uint32_t pm = __ballot_sync(0xFFFFFFFFu, f == kPlPrefix);
        const uint32_t zm = __ballot_sync(0xFFFFFFFFu, f == 0ull);
        const int stop = pm ? __ffs(pm) - 1 : 31;  // lanes 0..stop are summed
        const uint32_t upto = stop == 31 ? 0xFFFFFFFFu : ((2u << stop) - 1u);
        if (zm & upto) {  // a tile before the nearest prefix has not published yet
            if (!spin.step()) { raise_error(err, kDevTimeout); break; }
            continue;
        }
        unsigned long long cv = lane <= stop ? ((v >> 31) & kPlMask31) : 0ull;
        unsigned long long cm = lane <= stop ? (v & kPlMask31) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            cv += __shfl_xor_sync(0xFFFFFFFFu, cv, o);
            cm += __shfl_xor_sync(0xFFFFFFFFu, cm, o);
        }
        ev += cv;
        em += cm;
        if (pm) break;
        k0 -= 32;
    }
}

// One tile of one PLOC iteration (see above).  Reads of data other blocks
// wrote (the cluster array) bypass L1 (__ldcg), so the same code is correct
// inside the persistent kernel, where no launch boundary separates iterations.
// IPT < 4: a tile owns ploc_own_ipt(R) = IPT*BLOCK - 2R positions and each
// thread searches IPT positions (instead of four): for iterations whose tiles
// all run at once, where a tile's latency is the iteration's.
template <int IPT, int BLOCK>
__host__ __device__ constexpr uint32_t ploc_own_ipt(int radius) {
    return static_cast<uint32_t>(IPT * BLOCK) - 2u * static_cast<uint32_t>(radius);
}
template <int TILE, int BLOCK, int MAXR, int IPT = 4>
__device__ __forceinline__ void ploc_tile(PlocTileSmem<TILE, BLOCK, MAXR>& S, uint32_t tile, const uint2 cur, int iter,
                                          const float4* __restrict__ cin, float4* __restrict__ cout,
                                          float4* __restrict__ node_box, uint4* __restrict__ node_kids, uint2* it,
                                          uint32_t N, int R, unsigned long long* lb_cur, unsigned long long* lb_next,
                                          uint32_t* err, uint32_t spin_limit) {
    static_assert(IPT == 1 || IPT == 2 || IPT == 4, "one, two or four positions per thread");
    constexpr bool SMALL = IPT < 4;
    const int own = static_cast<int>(SMALL ? ploc_own_ipt<IPT, BLOCK>(R) : ploc_own(R));
    const int n = static_cast<int>(cur.x);
    const int s = static_cast<int>(tile) * own;
    __syncthreads();  // the previous tile of this block is done with S
    if (threadIdx.x == 0) st_relaxed_u64(&lb_next[tile], 0ull);
    const int e = min(n, s + own);
    const int wbase = s - 2 * R;  // window index 0
    const int lo = max(0, wbase);
    const int hi = min(n, e + 2 * R);
    for (int p = lo + threadIdx.x; p < hi; p += BLOCK) {
        const float4 a = __ldcg(cin + 2 * static_cast<size_t>(p));
        const float4 b = __ldcg(cin + 2 * static_cast<size_t>(p) + 1);
        const int w = p - wbase;
        S.mnx[w] = a.x; S.mny[w] = a.y; S.mnz[w] = a.z; S.id[w] = __float_as_uint(a.w);
        S.mxx[w] = b.x; S.mxy[w] = b.y; S.mxz[w] = b.z; S.lc[w] = __float_as_uint(b.w);
    }
    {  // window entries of positions outside [0, n): infinite boxes
        const int kWin = SMALL ? IPT * BLOCK + 2 * R : PlocSmem<TILE, BLOCK, MAXR>::kWin;  // the entries the search reads
        const float inf = __int_as_float(0x7F800000);
        const int below = lo - wbase, above = hi - wbase;
        for (int w = threadIdx.x; w < kWin; w += BLOCK) {
            if (w >= below && w < above) continue;
            S.mnx[w] = -inf; S.mny[w] = -inf; S.mnz[w] = -inf;
            S.mxx[w] = inf; S.mxy[w] = inf; S.mxz[w] = inf;
        }
    }
    __syncthreads();
    if (SMALL) {
        // thread t: positions q = s - R + IPT*t + i at window index IPT*t + i + R;
        // [s - R, e + R) fits since e - s <= IPT*BLOCK - 2R
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const int t = IPT * static_cast<int>(threadIdx.x) + i, q = s - R + t;
            if (q >= 0 && q < n && q < e + R) {
                uint32_t j;
                switch (R) {
                    case 8: j = ploc_nearest_at<8>(S, q, t + R, R); break;
                    case 16: j = ploc_nearest_at<16>(S, q, t + R, R); break;
                    case 32: j = ploc_nearest_at<32>(S, q, t + R, R); break;
                    default: j = ploc_nearest_at<0>(S, q, t + R, R); break;
                }
                S.nn[t] = j;
            }
        }
    } else {
        switch (R) {
            case 8: ploc_nearest_sym<8>(S, s, e, n); break;
            case 16: ploc_nearest_sym<16>(S, s, e, n); break;
            case 32: ploc_nearest_sym<32>(S, s, e, n); break;
            default: ploc_nearest<0>(S, s, e, n, R); break;
        }
    }
    __syncthreads();

    // Decisions for the tile's own positions: thread t owns [s + t*IPT, +IPT).
    const int nbase = s - R;  // S.nn index 0
    uint32_t flags = 0;       // bit q: valid, bit 16+q: merge head
    uint32_t nv = 0, nm = 0;
#pragma unroll
    for (int q = 0; q < IPT; ++q) {
        const int p = s + static_cast<int>(threadIdx.x) * IPT + q;
        if (p >= e) break;
        const int j = static_cast<int>(S.nn[p - nbase]);
        const bool mutual = (j != p) && (static_cast<int>(S.nn[j - nbase]) == p);
        const bool head = mutual && p < j;
        const bool gone = mutual && p > j;
        if (!gone) { flags |= 1u << q; ++nv; }
        if (head) { flags |= 1u << (16 + q); ++nm; }
    }
    // Block exclusive scan of (nv, nm) packed as 16|16 bits.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t packed = (nv << 16) | nm;
    uint32_t incl = packed;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) S.wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        // Warp 0: exclusive scan of the warp sums, then the look-back over
        // the preceding tiles, 32 status words per round trip.
        uint32_t ws = lane < BLOCK / 32 ? static_cast<uint32_t>(S.wsum[lane]) : 0u, wi = ws;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
            if (lane >= o) wi += y;
        }
        if (lane < BLOCK / 32) S.wsum[lane] = wi - ws;
        const uint32_t run = __shfl_sync(0xFFFFFFFFu, wi, 31);
        const unsigned long long tv = run >> 16, tm = run & 0xFFFFu;
        unsigned long long ev = 0, em = 0;
        if (tile == 0) {
            if (lane == 0) st_relaxed_u64(&lb_cur[0], kPlPrefix | (tv << 31) | tm);
        } else {
            if (lane == 0) st_relaxed_u64(&lb_cur[tile], kPlAgg | (tv << 31) | tm);
            ploc_look_back(tile, lb_cur, err, spin_limit, ev, em);
            if (lane == 0) st_relaxed_u64(&lb_cur[tile], kPlPrefix | ((ev + tv) << 31) | (em + tm));
        }
        if (lane == 0) {
            S.prefix = (ev << 32) | em;
            if (e == n)  // last tile: size and id base of the next iteration
                it[iter + 1] = make_uint2(static_cast<uint32_t>(ev + tv), cur.y + static_cast<uint32_t>(em + tm));
        }
    }
    __syncthreads();
    const uint32_t excl = static_cast<uint32_t>(S.wsum[warp]) + (incl - packed);
    uint32_t out_v = static_cast<uint32_t>(S.prefix >> 32) + (excl >> 16);
    uint32_t out_m = cur.y + static_cast<uint32_t>(S.prefix & 0xFFFFFFFFull) + (excl & 0xFFFFu);
#pragma unroll
    for (int q = 0; q < IPT; ++q) {
        if (!(flags & (1u << q))) continue;
        const int p = s + static_cast<int>(threadIdx.x) * IPT + q;
        const int wp = p - wbase;
        float4 mn = make_float4(S.mnx[wp], S.mny[wp], S.mnz[wp], __uint_as_float(S.id[wp]));
        float4 mx = make_float4(S.mxx[wp], S.mxy[wp], S.mxz[wp], __uint_as_float(S.lc[wp]));
        if (flags & (1u << (16 + q))) {
            const int j = static_cast<int>(S.nn[p - nbase]);
            const int wj = j - wbase;
            const uint32_t id = out_m++;
            if (id >= 2 * N - 1 || id < N) { raise_corrupt(err, 2 + (iter << 8), p, id); continue; }
            float4 m0, m1;  // AABB::merge (bvh.cpp:401-413), first argument = lower position
            m0.x = min_std(mn.x, S.mnx[wj]); m0.y = min_std(mn.y, S.mny[wj]); m0.z = min_std(mn.z, S.mnz[wj]);
            m1.x = max_std(mx.x, S.mxx[wj]); m1.y = max_std(mx.y, S.mxy[wj]); m1.z = max_std(mx.z, S.mxz[wj]);
            m0.w = mn.w;                      // left child id
            m1.w = __uint_as_float(S.id[wj]); // right child id
            node_box[2 * static_cast<size_t>(id)] = m0;
            node_box[2 * static_cast<size_t>(id) + 1] = m1;
            const uint32_t lc = S.lc[wp] + S.lc[wj];
            // children and their leaf counts, read by the DFS layout
            node_kids[id - N] = make_uint4(S.id[wp], S.id[wj], S.lc[wp], S.lc[wj]);
            mn = make_float4(m0.x, m0.y, m0.z, __uint_as_float(id));
            mx = make_float4(m1.x, m1.y, m1.z, __uint_as_float(lc));
        }
        if (out_v >= static_cast<uint32_t>(n)) { raise_corrupt(err, 3 + (iter << 8), p, out_v); continue; }
        cout[2 * static_cast<size_t>(out_v)] = mn;
        cout[2 * static_cast<size_t>(out_v) + 1] = mx;
        ++out_v;
    }
}

// ---- Tiles of an iteration with more tiles than blocks, in two halves.
// ploc_open: window, search, decisions and the tile's totals, published at once;
// ploc_close: look-back, then the survivors' records.  A block opens its next tile
// before it closes the last one, so a tile's predecessors have a whole tile's time
// to publish: with both halves in one, a third of a tile's time went into waiting
// for the slowest of the several hundred tiles before it (10.4 k of 31 k cycles).
// Decisions wait as one word a position; close reads the records again (from L2).
template <int TILE, int BLOCK, int MAXR>
struct PlocPipeSmem {
    static constexpr int kWin = TILE + 2 * MAXR;
    PlocTileSmem<TILE, BLOCK, MAXR> tile;
    __align__(16) uint32_t dec[2][TILE];  // place among the tile's survivors | among its merges << 11 | partner - p << 21 | flags
    unsigned long long prefix;
    uint32_t ticket;
};
constexpr uint32_t kDecKeep = 1u << 27, kDecHead = 1u << 28;

template <int TILE, int BLOCK, int MAXR>
__device__ __forceinline__ uint32_t ploc_open(PlocPipeSmem<TILE, BLOCK, MAXR>& P, int buf, uint32_t tile, int n,
                                              const float4* __restrict__ cin, int R, unsigned long long* lb_cur,
                                              unsigned long long* lb_next) {
    PlocTileSmem<TILE, BLOCK, MAXR>& S = P.tile;
    const int own = static_cast<int>(ploc_own(R)), s = static_cast<int>(tile) * own, e = min(n, s + own);
    const int wbase = s - 2 * R, nbase = s - R;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) st_relaxed_u64(&lb_next[tile], 0ull);
    const float inf = __int_as_float(0x7F800000);
    {  // every load of the window in flight at once (the last round is a few threads')
        constexpr int kRounds = (PlocSmem<TILE, BLOCK, MAXR>::kWin + BLOCK - 1) / BLOCK;
        float4 a[kRounds], b[kRounds];
        const int first = static_cast<int>(threadIdx.x) + wbase, hi = min(n, e + 2 * R);
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            const int p = first + r * BLOCK;
            if (p >= 0 && p < hi) {
                ld_record(cin + 2 * static_cast<size_t>(p), a[r], b[r]);
            } else {
                a[r] = make_float4(-inf, -inf, -inf, 0.f);
                b[r] = make_float4(inf, inf, inf, 0.f);
            }
        }
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            const int w = static_cast<int>(threadIdx.x) + r * BLOCK;
            if (w >= PlocSmem<TILE, BLOCK, MAXR>::kWin) break;
            S.mnx[w] = a[r].x; S.mny[w] = a[r].y; S.mnz[w] = a[r].z;
            S.mxx[w] = b[r].x; S.mxy[w] = b[r].y; S.mxz[w] = b[r].z;
        }
    }
    __syncthreads();
    switch (R) {
        case 8: ploc_nearest_sym<8>(S, s, e, n); break;
        case 16: ploc_nearest_sym<16>(S, s, e, n); break;
        case 32: ploc_nearest_sym<32>(S, s, e, n); break;
        default: ploc_nearest<0>(S, s, e, n, R); break;
    }
    __syncthreads();
    // thread t decides positions s + 4t .. s + 4t + 3
    constexpr int IPT = TILE / BLOCK;
    uint32_t dec[IPT], nv = 0, nm = 0;
#pragma unroll
    for (int q = 0; q < IPT; ++q) {
        const int p = s + static_cast<int>(threadIdx.x) * IPT + q;
        dec[q] = 0u;
        if (p >= e) continue;
        const int j = static_cast<int>(S.nn[p - nbase]);
        const bool mutual = (j != p) && (static_cast<int>(S.nn[j - nbase]) == p);
        if (mutual && p > j) continue;
        dec[q] = kDecKeep | nv | nm << 11;
        ++nv;
        if (mutual) {
            dec[q] |= kDecHead | static_cast<uint32_t>(j - p) << 21;
            ++nm;
        }
    }
    const uint32_t packed = nv | nm << 11;
    uint32_t incl = packed;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) S.wsum[warp] = incl;
    __syncthreads();
    uint32_t before = 0u, total = 0u;  // at most 1,024 | 512: no carry between the two
#pragma unroll
    for (int w = 0; w < BLOCK / 32; ++w) {
        const uint32_t v = static_cast<uint32_t>(S.wsum[w]);
        if (w < warp) before += v;
        total += v;
    }
    if (threadIdx.x == 0)
        st_relaxed_u64(&lb_cur[tile], (tile == 0 ? kPlPrefix : kPlAgg) |
                                          static_cast<unsigned long long>(total & 0x7FFu) << 31 | total >> 11);
    before += incl - packed;
#pragma unroll
    for (int q = 0; q < IPT; ++q) dec[q] = dec[q] ? dec[q] + before : 0u;
    static_assert(IPT == 4, "one vector a thread");
    *reinterpret_cast<uint4*>(&P.dec[buf][4 * threadIdx.x]) = make_uint4(dec[0], dec[1], dec[2], dec[3]);
    return total;
}

template <int TILE, int BLOCK, int MAXR>
__device__ __forceinline__ void ploc_close(PlocPipeSmem<TILE, BLOCK, MAXR>& P, int buf, uint32_t tile, uint32_t total,
                                           const uint2 cur, int iter, const float4* __restrict__ cin,
                                           float4* __restrict__ cout, float4* __restrict__ node_box,
                                           uint4* __restrict__ node_kids, uint2* it, uint32_t N, int R,
                                           unsigned long long* lb_cur, uint32_t* err, uint32_t spin_limit) {
    constexpr int IPT = TILE / BLOCK;
    const int n = static_cast<int>(cur.x), own = static_cast<int>(ploc_own(R));
    const int s = static_cast<int>(tile) * own, e = min(n, s + own);
    if (threadIdx.x < 32) {
        const unsigned long long tv = total & 0x7FFu, tm = total >> 11;
        unsigned long long ev = 0, em = 0;
        if (tile > 0) {
            ploc_look_back(tile, lb_cur, err, spin_limit, ev, em);
            if (threadIdx.x == 0) st_relaxed_u64(&lb_cur[tile], kPlPrefix | ((ev + tv) << 31) | (em + tm));
        }
        if (threadIdx.x == 0) {
            P.prefix = (ev << 32) | em;
            if (e == n)  // last tile: size and id base of the next iteration
                it[iter + 1] = make_uint2(static_cast<uint32_t>(ev + tv), cur.y + static_cast<uint32_t>(em + tm));
        }
    }
    __syncthreads();
    const uint32_t base_v = static_cast<uint32_t>(P.prefix >> 32), base_m = cur.y + static_cast<uint32_t>(P.prefix);
    // Neighbouring threads take neighbouring positions, one at a time: two or four
    // positions' records in flight cost registers (16.8 M clusters 5.45 and 6.51 ms
    // against 5.09; all four during the look-back 6.35).
#pragma unroll
    for (int q = 0; q < IPT; ++q) {
        const int x = q * BLOCK + static_cast<int>(threadIdx.x);
        const uint32_t d = x < e - s ? P.dec[buf][x] : 0u;
        if (!d) continue;
        const uint32_t p = static_cast<uint32_t>(s + x), out_v = base_v + (d & 0x7FFu);
        const float4* r = cin + 2 * static_cast<size_t>(p);
        float4 mn, mx;
        ld_record(r, mn, mx);
        if (d & kDecHead) {
            float4 jn, jx, m0, m1;
            ld_record(r + 2 * (d >> 21 & 0x3Fu), jn, jx);
            const uint32_t id = base_m + (d >> 11 & 0x3FFu);
            if (id >= 2 * N - 1 || id < N) { raise_corrupt(err, 2 + (iter << 8), p, id); continue; }
            // AABB::merge (bvh.cpp:401-413), first argument = lower position
            m0.x = min_std(mn.x, jn.x); m0.y = min_std(mn.y, jn.y); m0.z = min_std(mn.z, jn.z);
            m1.x = max_std(mx.x, jx.x); m1.y = max_std(mx.y, jx.y); m1.z = max_std(mx.z, jx.z);
            m0.w = mn.w;  // left child id
            m1.w = jn.w;  // right child id
            st_record(node_box + 2 * static_cast<size_t>(id), m0, m1);
            const uint32_t lca = __float_as_uint(mx.w), lcb = __float_as_uint(jx.w);
            // children and their leaf counts, read by the DFS layout
            node_kids[id - N] = make_uint4(__float_as_uint(mn.w), __float_as_uint(jn.w), lca, lcb);
            mn = make_float4(m0.x, m0.y, m0.z, __uint_as_float(id));
            mx = make_float4(m1.x, m1.y, m1.z, __uint_as_float(lca + lcb));
        }
        if (out_v >= static_cast<uint32_t>(n)) { raise_corrupt(err, 3 + (iter << 8), p, out_v); continue; }
        st_record(cout + 2 * static_cast<size_t>(out_v), mn, mx);
    }
}

template <int TILE, int BLOCK, int MAXR>
__global__ void __launch_bounds__(BLOCK) ploc_iteration_kernel(const float4* __restrict__ cin, float4* __restrict__ cout,
                                                               float4* __restrict__ node_box, uint4* __restrict__ node_kids,
                                                               uint2* it, int iter, uint32_t N,
                                                               int R, unsigned long long* lookback, uint32_t* tickets,
                                                               uint32_t n_tiles_cap, uint32_t* err, uint32_t spin_limit) {
    __shared__ PlocTileSmem<TILE, BLOCK, MAXR> S;
    __shared__ uint32_t s_tile;
    const uint2 cur = it[iter];
    const uint32_t n = cur.x;
    if (n <= 1u) {
        // Finished: carry the state forward so a later launch of this build
        // never reads an entry left over from an earlier build.
        if (blockIdx.x == 0 && threadIdx.x == 0) it[iter + 1] = cur;
        return;
    }
    unsigned long long* lb_cur = lookback + static_cast<size_t>(iter & 1) * n_tiles_cap;
    unsigned long long* lb_next = lookback + static_cast<size_t>((iter + 1) & 1) * n_tiles_cap;
    if (threadIdx.x == 0) s_tile = atomicAdd(&tickets[iter & 1], 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile * ploc_own(R) >= n) return;
    if (tile == 0 && threadIdx.x == 0) tickets[(iter + 1) & 1] = 0u;
    ploc_tile<TILE, BLOCK, MAXR>(S, tile, cur, iter, cin, cout, node_box, node_kids, it, N, R, lb_cur, lb_next, err,
                                 spin_limit);
}

// ================================================== K4: DFS node layout
// Scene::recursiveTopDownTraversalBVH (scene.cpp:189-201): pre-order, left
// subtree first, root (the last merge, id 2N-2) at 0.  A node at position p
// puts its left child at p+1 and its right child at p + 2*leaves(left).
//
// Two passes.  (a) Top-down: nodes created in PLOC iteration k only have
// parents from later iterations, so levels run from the last iteration
// down; a node reads its (DFS position, first leaf below, depth parity),
// passes them to its children and records dfs[p] = node id for itself and
// for its leaf children.  Only these few words move per node.  (b) One
// parallel pass over the DFS positions in order writes every output record
// once, so the node array and the traversal nodes are written coalesced.
//
// Output (b) also writes the traversal's own node format: one 64-byte record
// per internal node holding both children's boxes and references, indexed by
// the node's rank among internal nodes in DFS order (position minus the
// leaves before it, i.e. minus its first leaf).  Leaves are referenced by
// their position in the tree's left-to-right leaf order (the number of
// leaves before them in DFS order) — which is not their sorted position:
// PLOC merges clusters that are not adjacent in Morton order, so subtrees
// interleave there — and the parent of each leaf moves that leaf's
// transformed triangle into that order.  The traversal's tie rule (equal t:
// the leaf later in DFS order, which the shader visits first) and every
// subtree's leaves forming one contiguous range rest on this order.
__device__ __forceinline__ uint2 layout_place(uint32_t X, const uint2* __restrict__ pf, uint32_t N) {
    // (DFS position, first leaf below | depth parity << 31) of X; the root sits at (0, 0)
    return (X == 2 * N - 2) ? make_uint2(0u, 0u) : __ldcg(pf + (X - N));
}

// Position pass for internal node X placed at me = (position, first leaf |
// parity << 31).  PUBLISH: each internal child's record goes out as one
// 64-bit relaxed store, which a thread polling for it (the dataflow layout
// below) reads whole; the record is all it needs from the parent.
// kids: X's node_kids record (left id, right id, their leaf counts), which the
// dataflow pass loads before it waits for X's position.
template <bool PUBLISH>
__device__ __forceinline__ void layout_down_at(uint32_t X, uint2 me, const uint4 kids, uint2* __restrict__ pf,
                                               uint32_t N, uint32_t* __restrict__ dfs, uint32_t* err) {
    const uint32_t p = me.x, f = me.y & 0x7FFFFFFFu, odd = me.y >> 31;
    const uint32_t a = kids.x, b = kids.y, lca = kids.z;
    const uint32_t pl = p + 1, pr = p + 2 * lca;
    if (pr >= 2 * N - 1 || p < f || p - f >= N - 1 || (b >= N && b - N >= N - 1) || (a >= N && a - N >= N - 1)) {
        raise_corrupt(err, 4, X, pr);
        return;
    }
    dfs[p] = X;
    const uint32_t nodd = (odd ^ 1u) << 31;
    if (PUBLISH) {
        auto word = [](uint32_t pos, uint32_t first) {
            return (static_cast<unsigned long long>(first) << 32) | pos;
        };
        if (a < N) dfs[pl] = a;
        else st_relaxed_u64(reinterpret_cast<unsigned long long*>(pf + (a - N)), word(pl, f | nodd));
        if (b < N) dfs[pr] = b;
        else st_relaxed_u64(reinterpret_cast<unsigned long long*>(pf + (b - N)), word(pr, (f + lca) | nodd));
        return;
    }
    if (a < N) dfs[pl] = a; else pf[a - N] = make_uint2(pl, f | nodd);
    if (b < N) dfs[pr] = b; else pf[b - N] = make_uint2(pr, (f + lca) | nodd);
}

// The dataflow pass also publishes the places of X's grandchildren (from its
// children's node_kids records kc[0], kc[1], loaded while X waited), so
// places travel two levels per round trip through L2.  X's internal child
// later publishes the same words (the same arithmetic on the same inputs);
// whichever store lands first, the word is the same.  Out-of-range records
// are skipped here: the child's own pass reports them.
__device__ __forceinline__ void layout_publish_grandchildren(uint2 me, const uint4 kids, const uint4 kc[2],
                                                            uint2* __restrict__ pf, uint32_t N) {
    const uint32_t p = me.x, f = me.y & 0x7FFFFFFFu, odd = me.y >> 31;
    const uint32_t cp[2] = {p + 1, p + 2 * kids.z}, cf[2] = {f, f + kids.z};
    const uint32_t gpar = odd << 31;  // two levels down: X's own depth parity
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const uint32_t id = c ? kids.y : kids.x;
        if (id < N || id - N >= N - 1) continue;  // a leaf child (or corrupt)
        const uint32_t ga = kc[c].x, gb = kc[c].y, lga = kc[c].z;
        const uint32_t gpl = cp[c] + 1, gpr = cp[c] + 2 * lga;
        if (gpr >= 2 * N - 1) continue;
        if (ga >= N && ga - N < N - 1)
            st_relaxed_u64(reinterpret_cast<unsigned long long*>(pf + (ga - N)),
                           (static_cast<unsigned long long>(cf[c] | gpar) << 32) | gpl);
        if (gb >= N && gb - N < N - 1)
            st_relaxed_u64(reinterpret_cast<unsigned long long*>(pf + (gb - N)),
                           (static_cast<unsigned long long>((cf[c] + lga) | gpar) << 32) | gpr);
    }
}

__device__ __forceinline__ void layout_down(uint32_t X, const uint4* __restrict__ node_kids, uint2* __restrict__ pf,
                                            uint32_t N, uint32_t* __restrict__ dfs, uint32_t* err) {
    layout_down_at<false>(X, layout_place(X, pf, N), __ldcg(node_kids + (X - N)), pf, N, dfs, err);
}

// grow: the scene's abs_eps; wide_wt receives the traversal nodes with every
// child box grown by it (min - grow, max + grow, rounded as the traversal's
// own box growth would round them), for watertight traces.
__device__ __forceinline__ void layout_emit(uint32_t p, const float4* __restrict__ node_box,
                                            const uint4* __restrict__ node_kids, const uint2* __restrict__ pf,
                                            uint32_t N, const uint32_t* __restrict__ dfs, crt_bvh_node* __restrict__ out,
                                            float4* __restrict__ wide, float4* __restrict__ wide_wt,
                                            uint8_t* __restrict__ depth_odd, const LeafOut& lv, float grow,
                                            uint32_t* err) {
    const uint32_t X = __ldcg(dfs + p);
    if (X >= 2 * N - 1) { raise_corrupt(err, 5, p, X); return; }
    float4 mn, mx;
    ld_record_nc(node_box + 2 * static_cast<size_t>(X), mn, mx);
    float4* o = reinterpret_cast<float4*>(out + p);
    o[0] = make_float4(mn.x, mn.y, mn.z, 0.f);
    o[1] = make_float4(mx.x, mx.y, mx.z, 0.f);
    if (X < N) {  // leaf: its triangle
        reinterpret_cast<uint4*>(o)[2] = make_uint4(__float_as_uint(mn.w), 0u, 0u, 0u);
        return;
    }
    const uint2 me = layout_place(X, pf, N);
    const uint32_t f = me.y & 0x7FFFFFFFu, odd = me.y >> 31;
    const uint4 kids = __ldcg(node_kids + (X - N));
    const uint32_t a = kids.x, b = kids.y, lca = kids.z, lcb = kids.w;
    const uint32_t pl = p + 1, pr = p + 2 * lca;
    if (p < f || p - f >= N - 1) { raise_corrupt(err, 6, p, f); return; }
    reinterpret_cast<uint4*>(o)[2] = make_uint4(0u, pl, pr, 0u);
    const uint32_t ch[2] = {a, b}, cp[2] = {pl, pr}, cf[2] = {f, f + lca};
    float4 cmn[2], cmx[2];
    uint32_t cref[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        ld_record_nc(node_box + 2 * static_cast<size_t>(ch[c]), cmn[c], cmx[c]);
        cref[c] = (ch[c] < N) ? (kLeafRef | cf[c])  // leaf: its position in tree order
                              : (cp[c] - cf[c]);    // internal: its rank among internal nodes in DFS order
        if (ch[c] < N) {  // move the leaf's triangle from sorted to tree order
            if (cf[c] >= N) { raise_corrupt(err, 6, p, cf[c]); continue; }
            const float4* src = lv.xtri_sorted + 3 * static_cast<size_t>(ch[c]);
            float4* dst = lv.xtri + 3 * static_cast<size_t>(cf[c]);
            const float4 t0 = __ldcg(src), t1 = __ldcg(src + 1), t2 = __ldcg(src + 2);
            dst[0] = t0;
            dst[1] = t1;
            dst[2] = t2;
            const uint32_t ti = __float_as_uint(t0.w);
            if (ti < N) lv.leaf_of_tri[ti] = cf[c];
            else raise_corrupt(err, 6, p, ti);
        }
    }
    if (depth_odd) depth_odd[p - f] = static_cast<uint8_t>(odd);
    float4* w = wide + 4 * static_cast<size_t>(p - f);
    st_record(w, make_float4(cmn[0].x, cmn[0].y, cmn[0].z, __uint_as_float(cref[0])),
              make_float4(cmx[0].x, cmx[0].y, cmx[0].z, __uint_as_float(cref[1])));
    st_record(w + 2, make_float4(cmn[1].x, cmn[1].y, cmn[1].z, __uint_as_float(lca)),  // leaf counts of the children
              make_float4(cmx[1].x, cmx[1].y, cmx[1].z, __uint_as_float(lcb)));
    float4* g = wide_wt + 4 * static_cast<size_t>(p - f);
    st_record(g, make_float4(cmn[0].x - grow, cmn[0].y - grow, cmn[0].z - grow, __uint_as_float(cref[0])),
              make_float4(cmx[0].x + grow, cmx[0].y + grow, cmx[0].z + grow, __uint_as_float(cref[1])));
    st_record(g + 2, make_float4(cmn[1].x - grow, cmn[1].y - grow, cmn[1].z - grow, __uint_as_float(lca)),
              make_float4(cmx[1].x + grow, cmx[1].y + grow, cmx[1].z + grow, __uint_as_float(lcb)));
}

__global__ void __launch_bounds__(256) layout_level_kernel(const uint4* __restrict__ node_kids,
                                                           uint2* __restrict__ pf, uint32_t id_begin, uint32_t id_end,
                                                           uint32_t N, uint32_t* __restrict__ dfs, uint32_t* err) {
    const uint32_t X = id_begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (X >= id_end) return;
    layout_down(X, node_kids, pf, N, dfs, err);
}

__global__ void __launch_bounds__(256) layout_emit_kernel(const float4* __restrict__ node_box,
                                                          const uint4* __restrict__ node_kids,
                                                          const uint2* __restrict__ pf, uint32_t N,
                                                          const uint32_t* __restrict__ dfs, crt_bvh_node* __restrict__ out,
                                                          float4* __restrict__ wide, float4* __restrict__ wide_wt,
                                                          uint8_t* __restrict__ depth_odd, LeafOut lv,
                                                          const SceneState* __restrict__ st, uint32_t* err) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= 2 * N - 1 || build_failed(err)) return;
    layout_emit(p, node_box, node_kids, pf, N, dfs, out, wide, wide_wt, depth_odd, lv, st->abs_eps, err);
}

// ============================ K3 and K4 in a few launches (the default)
// PLOC iterations separated by a grid-wide barrier (co-residency guaranteed by a
// cooperative launch; every wait is bounded and a timeout ends every block), the
// last ones on a cluster, then the layout's two passes.  Saves the per-iteration
// launch and the host round trips the multi-launch path needs.
__device__ __forceinline__ bool grid_barrier(unsigned long long* bar, unsigned long long& target, uint32_t* err,
                                             uint32_t spin_limit) {
    // A 64-bit arrival counter that only grows (zeroed before the launch):
    // barrier k is complete when it reaches k * gridDim, so a block needs one
    // fence and one atomic, then polls; no reset and no release step.
    // `target` is this block's running count (thread 0's copy is used).
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        __threadfence();
        atomicAdd(bar, 1ull);
        SpinBound spin(spin_limit);
        while (ld_acquire_u64(bar) < target)
            if (!spin.step()) { raise_error(err, kDevTimeout); break; }
    }
    __syncthreads();
    return (ld_acquire_u32(err) & kDevTimeout) == 0u;
}

// =============================== K3 on a cluster: the last PLOC iterations
// Once the live clusters fit in the shared memory of one thread-block cluster
// (n <= 16 (2048 - 2R)), it runs the remaining iterations there: block c holds
// the positions [c seg, (c + 1) seg) and a halo of 2R on each side in the window
// layout of a tile that starts at its first position.  An iteration is the
// reference's, as in ploc_tile: nearest neighbours, mutual pairs merged at the
// lower position, exclusive scan of survivors and merges (over the block, then
// over the blocks' totals, which every block stores to every other), compaction
// (each survivor stored straight into the window, and the halos, of the blocks
// that hold its new position).  Two cluster barriers separate the steps, so no
// iteration waits for the grid, a look-back or global memory; only new nodes and
// the iteration records are written out.  When one segment holds every cluster the
// other blocks leave and block 0 finishes alone.
//
// Bound by the latency of an iteration's chain: a search of 0.7-1.2 k cycles (2 R
// candidates over four, two or one threads a position), two scans, and two cluster
// barriers of ~1.3 k each; warps without positions only take the barriers.  What
// it replaces (one grid barrier an iteration down to 992 clusters, then one block)
// took 9-20 us an iteration, this 2.3-4.  PLOC of N clusters, us: 1,000 78, 4,000
// 98, 16,000 127, 32,000 168, 65,536 227 (before, 20,011: 258, now 135).  With
// 1,024 threads of two positions: 86, 113, 145, 186, 244 (more warps to wait for
// at each barrier); with 8 blocks of 512 32,000 217 and 65,536 260.  Beyond 32,256
// clusters (radius 16) the whole GPU's search is faster than sixteen SMs'.
constexpr int kClusterBlocks = 16, kClusterThreads = 512, kClusterTile = 4 * kClusterThreads;
constexpr int kClusterMinSeg = 64;  // >= 2 * kPlocMaxRadius: a halo reaches only the adjacent segment
static_assert(kClusterMinSeg >= 2 * kPlocMaxRadius, "halo");
struct ClusterSmem : PlocSmem<kClusterTile, kClusterThreads, kPlocMaxRadius> {
    __align__(16) uint32_t totals[2][kClusterBlocks];  // every block's survivors << 16 | merges
    uint32_t gsum[kClusterTile / 32];                  // the same per 32 positions
};

// Nearest neighbours of the positions [s - R, e + R) into nn (position s - R
// first).  PARTS threads share a position's 2R candidates, in ascending runs; the
// strict minimum, lowest j on ties, is the lexicographic minimum of (area, j).
template <int RC, int PARTS>
__device__ __forceinline__ void cluster_nearest(ClusterSmem& S, int s, int e, int n, int R_rt) {
    const int R = RC > 0 ? RC : R_rt;
    const int cnt = e - s + 2 * R, part = static_cast<int>(threadIdx.x) % PARTS;
    // whole warps enter together (they exchange below)
    for (int t0 = static_cast<int>(threadIdx.x & ~31u) / PARTS; t0 < cnt; t0 += kClusterThreads / PARTS) {
        const int t = t0 + static_cast<int>(threadIdx.x & 31u) / PARTS, q = s - R + t, w = t + R;
        float best = __int_as_float(0x7F800000);
        int bj = q;
        if (t < cnt) {
            const float amnx = S.mnx[w], amny = S.mny[w], amnz = S.mnz[w], amxx = S.mxx[w], amxy = S.mxy[w], amxz = S.mxz[w];
            auto visit = [&](int k) {  // candidate k of the offsets -R .. -1, 1 .. R
                const int d = k < R ? k - R : k - R + 1;
                const int wj = w + d;
                const float dx = fmaxf(amxx, S.mxx[wj]) - fminf(amnx, S.mnx[wj]);
                const float dy = fmaxf(amxy, S.mxy[wj]) - fminf(amny, S.mny[wj]);
                const float dz = fmaxf(amxz, S.mxz[wj]) - fminf(amnz, S.mnz[wj]);
                const float v = 2.0f * (dx * dy + dy * dz + dz * dx);
                if (v < best) { best = v; bj = q + d; }
            };
            if (RC > 0) {
                static_assert((2 * RC) % PARTS == 0, "equal runs");
#pragma unroll
                for (int u = 0; u < 2 * RC / PARTS; ++u) visit(part * (2 * RC / PARTS) + u);
            } else {
                const int per = (2 * R + PARTS - 1) / PARTS;
                for (int k = part * per; k < min(2 * R, (part + 1) * per); ++k) visit(k);
            }
        }
#pragma unroll
        for (int m = 1; m < PARTS; m <<= 1) {
            const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, m);
            const int oj = __shfl_xor_sync(0xFFFFFFFFu, bj, m);
            if (ov < best || (ov == best && oj < bj)) { best = ov; bj = oj; }
        }
        if (t < cnt && part == 0 && q >= 0 && q < n) S.nn[t] = static_cast<uint32_t>(bj);
    }
}

template <int RC>
__device__ __forceinline__ void ploc_cluster_r(ClusterSmem& S, int iter, const float4* __restrict__ cin,
                                               float4* __restrict__ node_box, uint4* __restrict__ node_kids, uint2* it,
                                               uint32_t N, int R_rt, uint32_t* iters_out, uint32_t* err) {
    namespace cg = cooperative_groups;
    auto cluster = cg::this_cluster();
    constexpr int PMAX = kClusterTile / kClusterThreads, WARPS = kClusterThreads / 32;
    static_assert(kClusterTile / 32 == 64, "the block scan takes 64 groups of positions in two rounds of lanes");
    const int R = RC > 0 ? RC : R_rt;
    const int rank = static_cast<int>(cluster.block_rank()), blocks = static_cast<int>(cluster.num_blocks());
    const int log_blocks = 31 - __clz(blocks);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const float inf = __int_as_float(0x7F800000);
    auto segment = [&](int n) { return max((n + blocks - 1) >> log_blocks, kClusterMinSeg); };
    const uint2 cur = __ldcg(it + iter);
    int n = static_cast<int>(cur.x);
    uint32_t idb = cur.y;
    int seg = segment(n);
    if (seg + 2 * R > kClusterTile) {  // the caller checked n <= blocks * (tile - 2R); only corruption gets here
        if (rank == 0 && threadIdx.x == 0) raise_corrupt(err, 12, static_cast<uint32_t>(iter), static_cast<uint32_t>(n));
        return;
    }
    int s = min(n, rank * seg), e = min(n, s + seg);
    for (int w = threadIdx.x; w < seg + 4 * R; w += kClusterThreads) {
        const int p = s + w - 2 * R;
        if (p >= 0 && p < n) {
            const float4 a = __ldcg(cin + 2 * static_cast<size_t>(p));
            const float4 b = __ldcg(cin + 2 * static_cast<size_t>(p) + 1);
            S.mnx[w] = a.x; S.mny[w] = a.y; S.mnz[w] = a.z; S.id[w] = __float_as_uint(a.w);
            S.mxx[w] = b.x; S.mxy[w] = b.y; S.mxz[w] = b.z; S.lc[w] = __float_as_uint(b.w);
        } else {
            S.mnx[w] = -inf; S.mny[w] = -inf; S.mnz[w] = -inf;
            S.mxx[w] = inf; S.mxy[w] = inf; S.mxz[w] = inf;
        }
    }
    if (threadIdx.x < 2 * kClusterBlocks) (&S.totals[0][0])[threadIdx.x] = 0u;
    // one segment holds everything: this block alone
    bool solo = n <= seg;
    cluster.sync();  // every block has started (its memory may be stored to), or is not needed
    if (solo && rank != 0) return;
    for (int par = 0; n > 1; par ^= 1) {
        if (static_cast<uint32_t>(iter) + 1 >= N) {  // uniform over the cluster
            if (rank == 0 && threadIdx.x == 0) raise_error(err, kDevIterLimit);
            break;
        }
        if (s < e) {
            const int cnt = e - s + 2 * R;
            if (cnt <= kClusterThreads / 4) cluster_nearest<RC, 4>(S, s, e, n, R);
            else if (cnt <= kClusterThreads / 2) cluster_nearest<RC, 2>(S, s, e, n, R);
            else if (cnt <= 2 * kClusterThreads) cluster_nearest<RC, 1>(S, s, e, n, R);
            else ploc_nearest<RC>(S, s, e, n, R);
        }
        __syncthreads();
        // Thread t decides positions s + t, s + 512 + t, ...: what survives, what
        // merges, and the prefix counts of both, by groups of 32 positions.
        // Warps without positions only take part in the barriers: an iteration is
        // bound by the instructions its blocks issue.
        const int own = e - s, groups = (own + 31) >> 5;
        uint32_t keep[PMAX], head[PMAX];  // the warp's lanes that survive / that merge
        int nb[PMAX];                     // neighbour's window index
#pragma unroll
        for (int q = 0; q < PMAX; ++q) {
            keep[q] = head[q] = 0u;
            nb[q] = 0;
            if (q * WARPS + warp >= groups) continue;
            const int p = s + q * kClusterThreads + static_cast<int>(threadIdx.x);
            bool kp = false, hd = false;
            if (p < e) {
                const int j = static_cast<int>(S.nn[p - s + R]);
                const bool mutual = (j != p) && (static_cast<int>(S.nn[j - s + R]) == p);
                kp = !(mutual && p > j);
                hd = mutual && p < j;
                nb[q] = j - s + 2 * R;
            }
            keep[q] = __ballot_sync(0xFFFFFFFFu, kp);
            head[q] = __ballot_sync(0xFFFFFFFFu, hd);
            if (lane == 0) S.gsum[q * WARPS + warp] = (static_cast<uint32_t>(__popc(keep[q])) << 16) | __popc(head[q]);
        }
        __syncthreads();
        // each such warp scans the groups' totals (survivors << 16 | merges)
        uint32_t excl[PMAX] = {};
        if (warp < groups || warp == 0) {
            uint32_t total = 0;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (r > 0 && groups <= 32) break;
                const uint32_t v = 32 * r + lane < groups ? S.gsum[32 * r + lane] : 0u;
                uint32_t incl = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += y;
                }
#pragma unroll
                for (int q = 0; q < PMAX; ++q) {
                    const int g = q * WARPS + warp;  // this warp's groups are every WARPS-th
                    const uint32_t x = __shfl_sync(0xFFFFFFFFu, incl - v, g & 31);
                    if (g >> 5 == r) excl[q] = total + x;
                }
                total += __shfl_sync(0xFFFFFFFFu, incl, 31);
            }
            if (warp == 0 && lane < (solo ? 1 : blocks)) cluster.map_shared_rank(&S.totals[par][0], lane)[rank] = total;
        }
        // the survivors' records, from this iteration's window
        float4 omn[PMAX], omx[PMAX];
        uint32_t right[PMAX], right_lc[PMAX];  // a merge's right child and its leaves
#pragma unroll
        for (int q = 0; q < PMAX; ++q) {
            if (!(keep[q] >> lane & 1u)) continue;
            const int wp = q * kClusterThreads + static_cast<int>(threadIdx.x) + 2 * R;
            omn[q] = make_float4(S.mnx[wp], S.mny[wp], S.mnz[wp], __uint_as_float(S.id[wp]));
            omx[q] = make_float4(S.mxx[wp], S.mxy[wp], S.mxz[wp], __uint_as_float(S.lc[wp]));
            if (head[q] >> lane & 1u) {  // AABB::merge (bvh.cpp:401-413), first argument = lower position
                const int wj = nb[q];
                omn[q].x = min_std(omn[q].x, S.mnx[wj]); omn[q].y = min_std(omn[q].y, S.mny[wj]); omn[q].z = min_std(omn[q].z, S.mnz[wj]);
                omx[q].x = max_std(omx[q].x, S.mxx[wj]); omx[q].y = max_std(omx[q].y, S.mxy[wj]); omx[q].z = max_std(omx[q].z, S.mxz[wj]);
                right[q] = S.id[wj];
                right_lc[q] = S.lc[wj];
            }
        }
        uint32_t n_next = 0u, merges = 0u, bv = 0u, bm = 0u;
        if (solo) {
            __syncthreads();  // every read of the window is done, the total is in
            n_next = S.totals[par][0] >> 16;
            merges = S.totals[par][0] & 0xFFFFu;
        } else {
            cluster.sync();
#pragma unroll
            for (int r = 0; r < kClusterBlocks; r += 4) {
                const uint4 t = *reinterpret_cast<const uint4*>(&S.totals[par][r]);  // 0 past the cluster's blocks
                const uint32_t v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (r + u == rank) { bv = n_next; bm = merges; }
                    n_next += v[u] >> 16;
                    merges += v[u] & 0xFFFFu;
                }
            }
        }
        const int seg2 = solo ? seg : segment(static_cast<int>(n_next));
        const float per_seg = 1.0f / static_cast<float>(seg2);
        auto put = [&](int b, int w, const float4& mn, const float4& mx) {
            ClusterSmem& D = solo ? S : *cluster.map_shared_rank(&S, b);
            D.mnx[w] = mn.x; D.mny[w] = mn.y; D.mnz[w] = mn.z; D.id[w] = __float_as_uint(mn.w);
            D.mxx[w] = mx.x; D.mxy[w] = mx.y; D.mxz[w] = mx.z; D.lc[w] = __float_as_uint(mx.w);
        };
#pragma unroll
        for (int q = 0; q < PMAX; ++q) {
            if (!(keep[q] >> lane & 1u)) continue;
            const uint32_t out_v = bv + (excl[q] >> 16) + __popc(keep[q] & lt_mask);
            float4 mn = omn[q], mx = omx[q];
            if (head[q] >> lane & 1u) {
                const uint32_t id = idb + bm + (excl[q] & 0xFFFFu) + __popc(head[q] & lt_mask);
                if (id >= 2 * N - 1 || id < N) {
                    raise_corrupt(err, 13 + (iter << 8), out_v, id);
                } else {
                    const uint32_t left_lc = __float_as_uint(mx.w);
                    node_box[2 * static_cast<size_t>(id)] = mn;  // .w: left child, then right child
                    node_box[2 * static_cast<size_t>(id) + 1] = make_float4(mx.x, mx.y, mx.z, __uint_as_float(right[q]));
                    node_kids[id - N] = make_uint4(__float_as_uint(mn.w), right[q], left_lc, right_lc[q]);
                    mn.w = __uint_as_float(id);
                    mx.w = __uint_as_float(left_lc + right_lc[q]);
                }
            }
            if (out_v >= n_next) { raise_corrupt(err, 14 + (iter << 8), out_v, n_next); continue; }
            if (solo) {
                put(0, static_cast<int>(out_v) + 2 * R, mn, mx);
                continue;
            }
            int owner = __float2int_rz(static_cast<float>(out_v) * per_seg);  // the quotient, or next to it
            int at = static_cast<int>(out_v) - owner * seg2;                  // place in its segment
            if (at < 0) { --owner; at += seg2; }
            if (at >= seg2) { ++owner; at -= seg2; }
            put(owner, at + 2 * R, mn, mx);
            if (at < 2 * R && owner > 0) put(owner - 1, at + seg2 + 2 * R, mn, mx);
            if (at >= seg2 - 2 * R && (owner + 1) * seg2 < static_cast<int>(n_next)) put(owner + 1, at - seg2 + 2 * R, mn, mx);
        }
        s = min(static_cast<int>(n_next), rank * seg2);
        e = min(static_cast<int>(n_next), s + seg2);
        if (s < e)  // window entries past the last cluster
            for (int w = static_cast<int>(n_next) - s + 2 * R + static_cast<int>(threadIdx.x); w < seg2 + 4 * R; w += kClusterThreads) {
                S.mnx[w] = -inf; S.mny[w] = -inf; S.mnz[w] = -inf;
                S.mxx[w] = inf; S.mxy[w] = inf; S.mxz[w] = inf;
            }
        n = static_cast<int>(n_next);
        idb += merges;
        seg = seg2;
        ++iter;
        if (rank == 0 && threadIdx.x == 0) it[iter] = make_uint2(n_next, idb);
        if (solo) {
            __syncthreads();
        } else {
            cluster.sync();
            solo = n <= seg;
            if (solo && rank != 0) return;
        }
    }
    if (rank == 0 && threadIdx.x == 0) iters_out[0] = static_cast<uint32_t>(iter);
}

template <int MAXR>
__global__ void __launch_bounds__(kClusterThreads) ploc_cluster_kernel(const float4* ca, const float4* cb,
                                                                       float4* __restrict__ node_box,
                                                                       uint4* __restrict__ node_kids, uint2* it, uint32_t N,
                                                                       int R, uint32_t* iters_out, uint32_t* err) {
    extern __shared__ __align__(16) unsigned char cluster_smem[];
    ClusterSmem& C = *reinterpret_cast<ClusterSmem*>(cluster_smem);
    const int iter = static_cast<int>(__ldcg(iters_out));
    const float4* cin = (iter & 1) ? cb : ca;
    switch (R) {
        case 8: ploc_cluster_r<8>(C, iter, cin, node_box, node_kids, it, N, R, iters_out, err); break;
        case 16: ploc_cluster_r<16>(C, iter, cin, node_box, node_kids, it, N, R, iters_out, err); break;
        case 32: ploc_cluster_r<32>(C, iter, cin, node_box, node_kids, it, N, R, iters_out, err); break;
        default: ploc_cluster_r<0>(C, iter, cin, node_box, node_kids, it, N, R, iters_out, err); break;
    }
}

// The iterations of more tiles than one_wave_tiles; iters_out: their number.
template <int TILE, int BLOCK, int MAXR>
__global__ void __launch_bounds__(BLOCK, kPlocBlocksPerSm) ploc_wide_kernel(float4* ca, float4* cb, float4* __restrict__ node_box,
                                                           uint4* __restrict__ node_kids, uint2* it, uint32_t N, int R,
                                                           uint32_t one_wave_tiles, unsigned long long* lookback,
                                                           uint32_t* tickets, uint32_t n_tiles_cap, unsigned long long* bar,
                                                           uint32_t* iters_out, uint32_t* err, uint32_t spin_limit) {
    __shared__ PlocPipeSmem<TILE, BLOCK, MAXR> P;
    unsigned long long bar_target = 0;  // grid barriers passed x gridDim (thread 0)
    int iter = 0;
    for (;; ++iter) {
        const uint2 cur = __ldcg(it + iter);
        const uint32_t n_tiles = (cur.x + ploc_own(R) - 1) / ploc_own(R);
        if (n_tiles <= one_wave_tiles) break;
        const float4* cin = (iter & 1) ? cb : ca;
        float4* cout = (iter & 1) ? ca : cb;
        unsigned long long* lb_cur = lookback + static_cast<size_t>(iter & 1) * n_tiles_cap;
        unsigned long long* lb_next = lookback + static_cast<size_t>((iter + 1) & 1) * n_tiles_cap;
        // A block takes its next ticket when it has opened a tile, and then closes
        // the tile before.  Tickets follow the order of these starts, and the
        // smallest unpublished tile's block only waits for smaller ones, so every
        // look-back wait ends.
        if (threadIdx.x == 0) P.ticket = atomicAdd(&tickets[iter & 1], 1u);
        uint32_t open = 0u, open_total = 0u;
        bool some = false;  // a tile is open
        for (int buf = 0;; buf ^= 1) {
            __syncthreads();
            const uint32_t tile = P.ticket;
            const bool more = tile < n_tiles;
            uint32_t total = 0u;
            if (more) {
                total = ploc_open(P, buf, tile, static_cast<int>(cur.x), cin, R, lb_cur, lb_next);
                if (threadIdx.x == 32) {  // not the warp that looks back
                    P.ticket = atomicAdd(&tickets[iter & 1], 1u);
                    if (tile == 0) tickets[(iter + 1) & 1] = 0u;
                }
            }
            if (some)
                ploc_close(P, buf ^ 1, open, open_total, cur, iter, cin, cout, node_box, node_kids, it, N, R, lb_cur, err,
                           spin_limit);
            if (!more) break;
            some = true;
            open = tile;
            open_total = total;
        }
        if (!grid_barrier(bar, bar_target, err, spin_limit)) return;
        if (static_cast<uint32_t>(iter) + 1 >= N) { raise_error(err, kDevIterLimit); return; }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) iters_out[0] = static_cast<uint32_t>(iter);
}

// The iterations of at most a tile a block, down to stop_n clusters.  Two blocks
// an SM: an iteration is a chain of latencies and its grid barrier, which fewer
// blocks shorten (65,536 clusters 225 -> 213 us of PLOC, 300,000 379 -> 369).
// wide_grid: the blocks of ploc_wide_kernel, which counted its barriers in bar too.
template <int TILE, int BLOCK, int MAXR>
__global__ void __launch_bounds__(BLOCK, kPlocOneWaveBlocksPerSm) ploc_persistent_kernel(float4* ca, float4* cb, float4* __restrict__ node_box,
                                                                uint4* __restrict__ node_kids, uint2* it, uint32_t N,
                                                                int R, uint32_t stop_n, unsigned long long* lookback,
                                                                uint32_t n_tiles_cap, uint32_t wide_grid,
                                                                unsigned long long* bar, uint32_t* iters_out,
                                                                uint32_t* err, uint32_t spin_limit) {
    __shared__ PlocTileSmem<TILE, BLOCK, MAXR> S;
    int iter = static_cast<int>(__ldcg(iters_out));
    unsigned long long bar_target = static_cast<unsigned long long>(iter) * wide_grid;
    for (;; ++iter) {
        const uint2 cur = __ldcg(it + iter);
        if (cur.x <= stop_n) break;  // every block reads the same record; the cluster kernel takes over
        const float4* cin = (iter & 1) ? cb : ca;
        float4* cout = (iter & 1) ? ca : cb;
        unsigned long long* lb_cur = lookback + static_cast<size_t>(iter & 1) * n_tiles_cap;
        unsigned long long* lb_next = lookback + static_cast<size_t>((iter + 1) & 1) * n_tiles_cap;
        const uint32_t n_tiles = (cur.x + ploc_own(R) - 1) / ploc_own(R);
        const uint32_t n_t1 = (cur.x + ploc_own_ipt<1, BLOCK>(R) - 1) / ploc_own_ipt<1, BLOCK>(R);
        const uint32_t n_t2 = (cur.x + ploc_own_ipt<2, BLOCK>(R) - 1) / ploc_own_ipt<2, BLOCK>(R);
        if (n_tiles > gridDim.x) {  // the first kernel stops below that; only corruption gets here
            if (blockIdx.x == 0 && threadIdx.x == 0) raise_corrupt(err, 15, static_cast<uint32_t>(iter), cur.x);
            return;
        }
        // One wave: block b runs tile b (all tiles are co-resident, so every
        // look-back wait ends).  One (two) positions per thread while those smaller
        // tiles fit the grid and the look-back arrays: the iteration then costs one
        // short tile's latency.  Every block clears its word of the next iteration's
        // look-back array: the next iteration may cut its (fewer) clusters into
        // more, smaller tiles than this one has, and a tile clears only its own
        // word (the grid barrier below orders these stores before any read).
        if (threadIdx.x == 0 && blockIdx.x < n_tiles_cap) st_relaxed_u64(&lb_next[blockIdx.x], 0ull);
        if (n_t1 <= gridDim.x && n_t1 <= n_tiles_cap) {
            if (blockIdx.x < n_t1)
                ploc_tile<TILE, BLOCK, MAXR, 1>(S, blockIdx.x, cur, iter, cin, cout, node_box, node_kids, it, N, R, lb_cur,
                                                lb_next, err, spin_limit);
        } else if (n_t2 <= gridDim.x && n_t2 <= n_tiles_cap) {
            if (blockIdx.x < n_t2)
                ploc_tile<TILE, BLOCK, MAXR, 2>(S, blockIdx.x, cur, iter, cin, cout, node_box, node_kids, it, N, R, lb_cur,
                                                lb_next, err, spin_limit);
        } else if (blockIdx.x < n_tiles) {
            ploc_tile<TILE, BLOCK, MAXR>(S, blockIdx.x, cur, iter, cin, cout, node_box, node_kids, it, N, R, lb_cur, lb_next,
                                         err, spin_limit);
        }
        if (!grid_barrier(bar, bar_target, err, spin_limit)) return;
        if (static_cast<uint32_t>(iter) + 1 >= N) { raise_error(err, kDevIterLimit); return; }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) iters_out[0] = static_cast<uint32_t>(iter);
}

// One internal node of the layout's dataflow pass: waits (bounded) for the
// place of node X, lays X out and publishes its children's places; top: also
// its grandchildren's.  False: the wait ran out.
__device__ __forceinline__ bool layout_place_node(uint32_t X, bool top, uint32_t* __restrict__ dfs,
                                                  const uint4* __restrict__ node_kids, uint32_t N, uint2* pf,
                                                  uint32_t* err, uint32_t spin_limit) {
    // X's record (and, at the top of the tree, where the chain of places is the
    // latency that counts, its internal children's), in flight while X's place
    // is awaited
    const uint4 kids = __ldcg(node_kids + (X - N));
    uint4 kc[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
    if (top && kids.x >= N && kids.x - N < N - 1) kc[0] = __ldcg(node_kids + (kids.x - N));
    if (top && kids.y >= N && kids.y - N < N - 1) kc[1] = __ldcg(node_kids + (kids.y - N));
    uint2 me = make_uint2(0u, 0u);  // the root's place
    if (X != 2 * N - 2) {
        const unsigned long long* w = reinterpret_cast<const unsigned long long*>(pf + (X - N));
        unsigned long long v = ld_relaxed_u64(w);
        SpinBound spin(spin_limit);
        while (static_cast<uint32_t>(v) == kLayoutUnset) {
            if (!spin.step()) {
                raise_error(err, kDevTimeout);
                return false;
            }
            v = ld_relaxed_u64(w);
        }
        me = make_uint2(static_cast<uint32_t>(v), static_cast<uint32_t>(v >> 32));
    }
    if (top) layout_publish_grandchildren(me, kids, kc, pf, N);
    layout_down_at<true>(X, me, kids, pf, N, dfs, err);
    return true;
}

// The layout's position pass in one cooperative launch.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) layout_places_kernel(uint32_t* __restrict__ dfs, const uint4* __restrict__ node_kids,
                                                              uint32_t N, uint2* pf, uint32_t* err, uint32_t spin_limit) {
    // DFS layout, position pass as dataflow: internal node ids grow with the
    // PLOC iteration that made them, so a parent's id is larger than its
    // children's and decreasing ids are a top-down order.  Every thread takes
    // the ids 2N-2, 2N-3, ... in grid-stride order and, before laying node X
    // out, waits (bounded) until X's parent has published X's position.  The
    // unfinished node with the largest id never waits (its parent is done), so
    // the co-resident grid always progresses, with no barrier per PLOC level.
    if (build_failed(err)) return;  // places that no parent hands out: nothing to wait for
    for (uint32_t t = blockIdx.x * BLOCK + threadIdx.x; t + 1 < N; t += gridDim.x * BLOCK)
        if (!layout_place_node(2 * N - 2 - t, t < gridDim.x * BLOCK, dfs, node_kids, N, pf, err, spin_limit)) return;
}

__global__ void single_leaf_kernel(const float4* __restrict__ node_box, crt_bvh_node* __restrict__ out, LeafOut lv) {
    const float4 mn = node_box[0], mx = node_box[1];
    float4* o = reinterpret_cast<float4*>(out);
    o[0] = make_float4(mn.x, mn.y, mn.z, 0.f);
    o[1] = make_float4(mx.x, mx.y, mx.z, 0.f);
    reinterpret_cast<uint4*>(o)[2] = make_uint4(__float_as_uint(mn.w), 0u, 0u, 0u);
    for (int k = 0; k < 3; ++k) lv.xtri[k] = lv.xtri_sorted[k];
    lv.leaf_of_tri[0] = 0u;
}

// ========================================== K4b: 4-wide traversal nodes
// Every internal node at even depth becomes a 128-byte 4-wide node holding
// its children's children (a leaf child stays itself): SoA boxes (min x of
// the four, min y, ..., max z) and the four references; empty slots carry
// kNoChild and an empty box.  Nodes keep the binary node's index (odd-depth
// slots stay unused), so references are unchanged and exact boxes stay exact.
__global__ void __launch_bounds__(256) wide4_kernel(const float4* __restrict__ wide, const uint8_t* __restrict__ depth_odd,
                                                    uint32_t n_internal, float4* __restrict__ wide4) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_internal || depth_odd[i]) return;
    float mnx[4], mny[4], mnz[4], mxx[4], mxy[4], mxz[4];
    uint32_t ref[4];
    int k = 0;
    const float4* w = wide + 4 * static_cast<size_t>(i);
    const float4 w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
    const float4 cmn[2] = {w0, w2}, cmx[2] = {w1, w3};
    const uint32_t cref[2] = {__float_as_uint(w0.w), __float_as_uint(w1.w)};
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        if (cref[c] & kLeafRef) {
            mnx[k] = cmn[c].x; mny[k] = cmn[c].y; mnz[k] = cmn[c].z;
            mxx[k] = cmx[c].x; mxy[k] = cmx[c].y; mxz[k] = cmx[c].z;
            ref[k++] = cref[c];
        } else {
            const float4* g = wide + 4 * static_cast<size_t>(cref[c]);
            const float4 g0 = g[0], g1 = g[1], g2 = g[2], g3 = g[3];
            mnx[k] = g0.x; mny[k] = g0.y; mnz[k] = g0.z; mxx[k] = g1.x; mxy[k] = g1.y; mxz[k] = g1.z;
            ref[k++] = __float_as_uint(g0.w);
            mnx[k] = g2.x; mny[k] = g2.y; mnz[k] = g2.z; mxx[k] = g3.x; mxy[k] = g3.y; mxz[k] = g3.z;
            ref[k++] = __float_as_uint(g1.w);
        }
    }
    const float inf = __int_as_float(0x7F800000);
    for (; k < 4; ++k) {
        mnx[k] = mny[k] = mnz[k] = inf;
        mxx[k] = mxy[k] = mxz[k] = -inf;
        ref[k] = kNoChild;
    }
    float4* o = wide4 + 8 * static_cast<size_t>(i);
    o[0] = make_float4(mnx[0], mnx[1], mnx[2], mnx[3]);
    o[1] = make_float4(mny[0], mny[1], mny[2], mny[3]);
    o[2] = make_float4(mnz[0], mnz[1], mnz[2], mnz[3]);
    o[3] = make_float4(mxx[0], mxx[1], mxx[2], mxx[3]);
    o[4] = make_float4(mxy[0], mxy[1], mxy[2], mxy[3]);
    o[5] = make_float4(mxz[0], mxz[1], mxz[2], mxz[3]);
    reinterpret_cast<uint4*>(o)[6] = make_uint4(ref[0], ref[1], ref[2], ref[3]);
    o[7] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// ================================= K4c: compressed 4-wide traversal nodes
// One 64-byte record per binary internal node (format: crt_walk4.cuh): the
// node's two children, then twice the internal child of largest area opened
// into its own two.  Every step is rounded outward by directed float rounding:
// the child's box grown by g = 4 * abs_eps, the origin the least corner, the
// step the least power of two with 255 of them covering the node's extent.
// Every rank gets a record, also those a walk never enters because they were opened
// away (64 B read in order, at most two more gathered from L2, 64 B written per node);
// opening by area fills the slots better than taking the grandchildren (which leave a
// slot empty beside every leaf) and visits fewer nodes.
__device__ __forceinline__ float half_area(float4 mn, float4 mx) {
    const float x = mx.x - mn.x, y = mx.y - mn.y, z = mx.z - mn.z;
    return x * y + y * z + z * x;
}

__device__ __forceinline__ void cwide_node(const float4* __restrict__ wide, uint32_t i, uint32_t n_internal,
                                           float abs_eps, uint4* __restrict__ out, uint32_t* bad) {
    float4 mn[4], mx[4];
    uint32_t ref[4];
    const float4* w = wide + 4 * static_cast<size_t>(i);
    const float4 w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3);
    mn[0] = w0; mx[0] = w1; ref[0] = __float_as_uint(w0.w);
    mn[1] = w2; mx[1] = w3; ref[1] = __float_as_uint(w1.w);
    const float inf = __int_as_float(0x7F800000);
#pragma unroll
    for (int c = 2; c < 4; ++c) {
        mn[c] = make_float4(inf, inf, inf, 0.f);
        mx[c] = make_float4(-inf, -inf, -inf, 0.f);
        ref[c] = kNoChild;
    }
#pragma unroll
    for (int c = 2; c < 4; ++c) {  // slots 0 .. c-1 are taken
        int best = -1;
        float area = -1.f;
#pragma unroll
        for (int k = 0; k < c; ++k) {
            const float a = half_area(mn[k], mx[k]);
            if (!(ref[k] & kLeafRef) && a > area) { area = a; best = k; }
        }
        uint32_t open = kNoChild;
#pragma unroll
        for (int k = 0; k < c; ++k)
            if (k == best) open = ref[k];
        if (open >= n_internal) continue;  // no internal child (or a non-finite area)
        const float4* g = wide + 4 * static_cast<size_t>(open);
        const float4 g0 = __ldg(g), g1 = __ldg(g + 1), g2 = __ldg(g + 2), g3 = __ldg(g + 3);
#pragma unroll
        for (int k = 0; k < c; ++k)
            if (k == best) { mn[k] = g0; mx[k] = g1; ref[k] = __float_as_uint(g0.w); }
        mn[c] = g2; mx[c] = g3; ref[c] = __float_as_uint(g1.w);
    }
    bool ok = walk4_scene(abs_eps);
#pragma unroll
    for (int c = 0; c < 4; ++c)  // the walk follows references unchecked
        ok = ok && (ref[c] == kNoChild || ((ref[c] & kLeafRef) ? (ref[c] & ~kLeafRef) <= n_internal : ref[c] < n_internal));
    const float grow = 4.f * abs_eps;
    const float lo[3][4] = {{mn[0].x, mn[1].x, mn[2].x, mn[3].x}, {mn[0].y, mn[1].y, mn[2].y, mn[3].y},
                            {mn[0].z, mn[1].z, mn[2].z, mn[3].z}};
    const float hi[3][4] = {{mx[0].x, mx[1].x, mx[2].x, mx[3].x}, {mx[0].y, mx[1].y, mx[2].y, mx[3].y},
                            {mx[0].z, mx[1].z, mx[2].z, mx[3].z}};
    float org[3];
    uint32_t step[3], q[6];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // NaN coordinates must not be skipped by fminf: they fail the isfinite tests below
        const float l = __fadd_rd(fminf(fminf(lo[a][0], lo[a][1]), fminf(lo[a][2], lo[a][3])), -grow);
        const float h = __fadd_ru(fmaxf(fmaxf(hi[a][0], hi[a][1]), fmaxf(hi[a][2], hi[a][3])), grow);
        ok = ok && isfinite(l) && isfinite(h);
        // the least biased exponent whose power of two is >= extent / 255 (1/255 rounded up)
        const float need = __fmul_ru(__fsub_ru(h, l), 0.00392156886f);
        const uint32_t e = min(max((__float_as_uint(need) + 0x7FFFFFu) >> 23, 1u), 180u);
        const float inv_step = __uint_as_float((254u - e) << 23);  // 2^(127 - e)
        org[a] = l * 8.673617379884035e-19f;
        step[a] = (e + 73u) << 23;  // as a float: step * 2^73
        uint32_t ql = 0, qh = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t bl = 255u, bh = 0u;  // an empty slot: inverted planes
            if (ref[c] != kNoChild) {
                ok = ok && isfinite(lo[a][c]) && isfinite(hi[a][c]);
                const float dl = __fsub_rd(__fadd_rd(lo[a][c], -grow), l), dh = __fsub_ru(__fadd_ru(hi[a][c], grow), l);
                bl = static_cast<uint32_t>(fminf(fmaxf(floorf(dl * inv_step), 0.f), 255.f));
                const float up = ceilf(dh * inv_step);
                ok = ok && up >= 0.f && up <= 255.f;
                bh = static_cast<uint32_t>(fminf(fmaxf(up, 0.f), 255.f));
            }
            ql |= bl << (8 * c);
            qh |= bh << (8 * c);
        }
        q[a] = ql;
        q[3 + a] = qh;
    }
    if (!ok) atomicOr(bad, 1u);
    uint4* o = out + 4 * static_cast<size_t>(i);
    o[0] = make_uint4(__float_as_uint(org[0]), __float_as_uint(org[1]), __float_as_uint(org[2]), step[0]);
    o[1] = make_uint4(q[0], q[1], q[2], q[3]);
    o[2] = make_uint4(q[4], q[5], step[1], step[2]);
    o[3] = make_uint4(ref[0], ref[1], ref[2], ref[3]);
}

__global__ void __launch_bounds__(256) cwide_kernel(const float4* __restrict__ wide, uint32_t n_internal, float abs_eps,
                                                    uint4* __restrict__ cwide, uint32_t* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_internal) cwide_node(wide, i, n_internal, abs_eps, cwide, bad);
}

__global__ void __launch_bounds__(256) cwide_batch_kernel(const float4* __restrict__ wide,
                                                          const BatchScene* __restrict__ scenes, uint32_t n_scenes,
                                                          uint32_t n_total, uint4* __restrict__ cwide, uint32_t* bad) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_total) return;
    uint32_t lo = 0, hi = n_scenes - 1;  // the last scene whose first triangle is <= j
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(&scenes[mid].tri_off) <= j) lo = mid; else hi = mid - 1;
    }
    const BatchScene sc = scenes[lo];
    const uint32_t i = j - sc.tri_off;
    if (i + 1 >= sc.n_tris) return;
    const size_t base = 4 * static_cast<size_t>(sc.wide_off);
    cwide_node(wide + base, i, sc.n_tris - 1, sc.abs_eps, cwide + base, bad + lo);
}

void launch_cwide(const float4* wide, uint32_t n_internal, float abs_eps, uint4* cwide, uint32_t* bad, cudaStream_t s) {
    cudaMemsetAsync(bad, 0, 4, s);
    if (n_internal == 0) return;
    cwide_kernel<<<(n_internal + 255) / 256, 256, 0, s>>>(wide, n_internal, abs_eps, cwide, bad);
}

void launch_cwide_batch(const float4* wide, const BatchScene* scenes, uint32_t n_scenes, uint32_t n_total, uint4* cwide,
                        uint32_t* bad, cudaStream_t s) {
    cudaMemsetAsync(bad, 0, 4ull * n_scenes, s);
    cwide_batch_kernel<<<(n_total + 255) / 256, 256, 0, s>>>(wide, scenes, n_scenes, n_total, cwide, bad);
}

void launch_wide4(const float4* wide, const uint8_t* depth_odd, uint32_t n_internal, float4* wide4, cudaStream_t s) {
    if (n_internal == 0) return;
    wide4_kernel<<<(n_internal + 255) / 256, 256, 0, s>>>(wide, depth_odd, n_internal, wide4);
}

// ============================================================ launchers
void launch_scene_box(const crt_triangle* tris, uint32_t n_buffer, const float* models, SceneState* st, uint32_t* err,
                      cudaStream_t s) {
    const uint32_t want = (n_buffer + 255) / 256;
    const uint32_t grid = want < static_cast<uint32_t>(kNumSms * 8) ? (want ? want : 1u) : kNumSms * 8;
    scene_box_kernel<<<grid, 256, 0, s>>>(tris, n_buffer, models, st, err);
}

void launch_morton(const crt_triangle* tris, uint32_t n, const float* models_third, const SceneState* st,
                   uint32_t* codes, uint32_t* hist, int bits, cudaStream_t s) {
    const uint32_t want = (n + 255) / 256;
    const uint32_t grid = want < static_cast<uint32_t>(kNumSms * 8) ? (want ? want : 1u) : kNumSms * 8;
    if (bits == 4) morton_kernel<4><<<grid, 256, 0, s>>>(tris, n, models_third, st, codes, hist);
    else morton_kernel<8><<<grid, 256, 0, s>>>(tris, n, models_third, st, codes, hist);
}

uint32_t sort_tile_keys(int bits) { return bits == 4 ? 256u * 16u : 256u * 16u; }

void launch_onesweep(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out, uint32_t n,
                     int shift, int bits, const uint32_t* pass_hist, uint32_t* lookback, uint32_t* ticket, uint32_t* err,
                     uint32_t spin_limit, cudaStream_t s) {
    const uint32_t tiles = (n + sort_tile_keys(bits) - 1) / sort_tile_keys(bits);
    if (bits == 4)
        onesweep_kernel<4, 256, 16, false><<<tiles, 256, 0, s>>>(keys_in, vals_in, keys_out, vals_out, n, shift,
                                                                  pass_hist, lookback, ticket, err, spin_limit, nullptr, 0);
    else
        onesweep_kernel<8, 256, 16, false><<<tiles, 256, 0, s>>>(keys_in, vals_in, keys_out, vals_out, n, shift,
                                                                  pass_hist, lookback, ticket, err, spin_limit, nullptr, 0);
}

void launch_onesweep_segments(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                              uint32_t n, const uint32_t* seg_off, uint32_t n_seg, const uint32_t* seg_hist,
                              uint32_t* lookback, uint32_t* ticket, uint32_t* err, uint32_t spin_limit, cudaStream_t s) {
    const uint32_t tiles = (n + sort_tile_keys(8) - 1) / sort_tile_keys(8);
    onesweep_kernel<8, 256, 16, true><<<tiles, 256, 0, s>>>(keys_in, vals_in, keys_out, vals_out, n, 0, seg_hist,
                                                             lookback, ticket, err, spin_limit, seg_off, n_seg);
}

// The sort's counting and digit-offset steps alone, on caller keys and
// counts (the reference's sort-shader known-answer tests drive them).
template <int BITS>
__global__ void __launch_bounds__(256) digit_counts_kernel(const uint32_t* __restrict__ keys, uint32_t n,
                                                           uint32_t* __restrict__ counts) {
    constexpr int RADIX = 1 << BITS;
    constexpr int PASSES = (32 + BITS - 1) / BITS;
    __shared__ uint32_t s_hist[PASSES * RADIX];
    for (int i = threadIdx.x; i < PASSES * RADIX; i += blockDim.x) s_hist[i] = 0u;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        add_digit_counts<BITS, PASSES>(keys[i], s_hist);
    __syncthreads();
    for (int i = threadIdx.x; i < PASSES * RADIX; i += blockDim.x)
        if (s_hist[i]) atomicAdd(&counts[i], s_hist[i]);
}

// One block per digit place: where each digit's keys start in the pass's
// output, the exclusive scan over digits that the radix pass takes of its
// global histogram (the same packed block scan, the global counts in the
// high half).
template <int BITS, int BLOCK>
__global__ void __launch_bounds__(BLOCK) digit_offsets_kernel(const uint32_t* __restrict__ counts,
                                                              uint32_t* __restrict__ offsets) {
    constexpr int RADIX = 1 << BITS;
    static_assert(BLOCK >= RADIX, "one thread per digit");
    __shared__ unsigned long long s_wsum[BLOCK / 32];
    const int d = threadIdx.x;
    const size_t base = static_cast<size_t>(blockIdx.x) * RADIX;
    const uint32_t gh = d < RADIX ? counts[base + d] : 0u;
    const unsigned long long incl = block_inclusive_scan_u64<BLOCK>(static_cast<unsigned long long>(gh) << 32, s_wsum);
    if (d < RADIX) offsets[base + d] = static_cast<uint32_t>(incl >> 32) - gh;
}

bool launch_digit_counts(const uint32_t* keys, uint32_t n, int bits, uint32_t* counts, cudaStream_t s) {
    const uint32_t want = (n + 255) / 256;
    const uint32_t grid = want < static_cast<uint32_t>(kNumSms * 8) ? (want ? want : 1u) : kNumSms * 8;
    switch (bits) {
        case 1: digit_counts_kernel<1><<<grid, 256, 0, s>>>(keys, n, counts); return true;
        case 2: digit_counts_kernel<2><<<grid, 256, 0, s>>>(keys, n, counts); return true;
        case 4: digit_counts_kernel<4><<<grid, 256, 0, s>>>(keys, n, counts); return true;
        case 8: digit_counts_kernel<8><<<grid, 256, 0, s>>>(keys, n, counts); return true;
        default: return false;
    }
}

bool launch_digit_offsets(const uint32_t* counts, uint32_t places, int bits, uint32_t* offsets, cudaStream_t s) {
    if (places == 0) return true;
    switch (bits) {
        case 1: digit_offsets_kernel<1, 32><<<places, 32, 0, s>>>(counts, offsets); return true;
        case 2: digit_offsets_kernel<2, 32><<<places, 32, 0, s>>>(counts, offsets); return true;
        case 4: digit_offsets_kernel<4, 32><<<places, 32, 0, s>>>(counts, offsets); return true;
        case 8: digit_offsets_kernel<8, 256><<<places, 256, 0, s>>>(counts, offsets); return true;
        default: return false;
    }
}

void launch_leaf_init(const crt_triangle* tris, uint32_t n, const float* models, const uint32_t* perm, float4* node_box,
                      float4* clusters, float4* xtri_sorted, uint2* it, uint2* pf, uint32_t* err, cudaStream_t s) {
    leaf_init_kernel<<<(n + 255) / 256, 256, 0, s>>>(tris, n, models, perm, node_box, clusters, xtri_sorted, it, pf, err);
}

void launch_ploc_iteration(const float4* cin, float4* cout, float4* node_box, uint4* node_kids, uint2* it,
                           int iter, uint32_t N, int radius, uint32_t n_upper,
                           unsigned long long* lookback, uint32_t* tickets, uint32_t n_tiles_cap, uint32_t* err,
                           uint32_t spin_limit, cudaStream_t s) {
    const uint32_t tiles = (n_upper + ploc_own(radius) - 1) / ploc_own(radius);
    ploc_iteration_kernel<kPlocSpan, 256, kPlocMaxRadius><<<tiles ? tiles : 1u, 256, 0, s>>>(
        cin, cout, node_box, node_kids, it, iter, N, radius, lookback, tickets, n_tiles_cap, err, spin_limit);
}

void launch_layout_level(const uint4* node_kids, uint2* pf, uint32_t id_begin,
                         uint32_t id_end, uint32_t N, uint32_t* dfs, uint32_t* err, cudaStream_t s) {
    if (id_end <= id_begin || id_end > 2 * N - 1) return;
    const uint32_t cnt = id_end - id_begin;
    layout_level_kernel<<<(cnt + 255) / 256, 256, 0, s>>>(node_kids, pf, id_begin, id_end, N, dfs, err);
}

void launch_layout_emit(const float4* node_box, const uint4* node_kids, const uint2* pf, uint32_t N,
                        const uint32_t* dfs, crt_bvh_node* out, float4* wide, float4* wide_wt, uint8_t* depth_odd,
                        LeafOut lv, const SceneState* st, uint32_t* err, cudaStream_t s) {
    const uint32_t cnt = 2 * N - 1;
    layout_emit_kernel<<<(cnt + 255) / 256, 256, 0, s>>>(node_box, node_kids, pf, N, dfs, out, wide, wide_wt, depth_odd,
                                                         lv, st, err);
}

// Blocks of a cooperative 256-thread launch of f on the current device, at most
// per_sm_max an SM (0: none).
static int cooperative_grid(const void* f, int per_sm_max) {
    int per_sm = 0, dev = 0, sms = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, 256, 0) != cudaSuccess) per_sm = 0;
    cudaGetLastError();
    return resident_blocks(coop != 0, per_sm, per_sm_max, sms);
}
constexpr int kAnyPerSm = 1 << 10;

// make()'s result for the current device, made once for each.
template <class Value, class Make>
static Value per_device(Make make) {
    static std::mutex mutex;
    static std::map<int, Value> made;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> hold(mutex);
    auto at = made.find(dev);
    if (at == made.end()) at = made.emplace(dev, make()).first;
    return at->second;
}

// Launch of a PLOC cluster kernel: `clusters` clusters of `blocks` blocks.
struct ClusterLaunch {
    cudaLaunchConfig_t c{};
    cudaLaunchAttribute a{};
    ClusterLaunch(int blocks, uint32_t clusters, cudaStream_t s) {
        a.id = cudaLaunchAttributeClusterDimension;
        a.val.clusterDim.x = blocks;
        a.val.clusterDim.y = a.val.clusterDim.z = 1;
        c.gridDim = dim3(blocks * clusters);
        c.blockDim = dim3(kClusterThreads);
        c.dynamicSmemBytes = sizeof(ClusterSmem);
        c.stream = s;
        c.attrs = &a;
        c.numAttrs = 1;
    }
    // Allows the kernel f clusters of kClusterBlocks on the current device (in the
    // current CUDA context: build_prepare repeats it for every library context).
    static void allow(const void* f) {
        cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(ClusterSmem)));
        cudaGetLastError();
    }
    // The clusters of `blocks` blocks that the device holds at once (0: it cannot run).
    static int active(const void* f, int blocks) {
        allow(f);
        ClusterLaunch l(blocks, 1, nullptr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, f, &l.c) != cudaSuccess) n = 0;
        cudaGetLastError();
        return n;
    }
};

static const void* const kWideFn = reinterpret_cast<const void*>(ploc_wide_kernel<kPlocSpan, 256, kPlocMaxRadius>);
static const void* const kWaveFn = reinterpret_cast<const void*>(ploc_persistent_kernel<kPlocSpan, 256, kPlocMaxRadius>);
static const void* const kPlacesFn = reinterpret_cast<const void*>(layout_places_kernel<256>);

// The grids of launch_ploc_layout on the current device.
static PlocGrids ploc_grids() {
    return per_device<PlocGrids>([] {
        PlocGrids g;
        g.wide = cooperative_grid(kWideFn, kPlocBlocksPerSm);
        g.wave = cooperative_grid(kWaveFn, kPlocOneWaveBlocksPerSm);
        g.places = cooperative_grid(kPlacesFn, kAnyPerSm);
        for (int b = kClusterBlocks; b >= 8 && g.cluster == 0; b /= 2)
            if (ClusterLaunch::active(reinterpret_cast<const void*>(ploc_cluster_kernel<kPlocMaxRadius>), b) > 0) g.cluster = b;
        return g;
    });
}

cudaError_t launch_ploc_layout(float4* ca, float4* cb, float4* node_box, uint4* node_kids, uint2* it, uint32_t N,
                               int radius, unsigned long long* lookback, uint32_t* tickets, uint32_t n_tiles_cap,
                               uint2* pf, crt_bvh_node* out, float4* wide, float4* wide_wt, uint8_t* depth_odd,
                               LeafOut lv, const SceneState* st, unsigned long long* bar, uint32_t* iters_out,
                               uint32_t* err, uint32_t spin_limit, cudaEvent_t ploc_done, bool* enqueued,
                               cudaStream_t s) {
    *enqueued = false;
    const PlocGrids grids = ploc_grids();
    if (!grids.supported()) return cudaErrorNotSupported;
    uint32_t stop_n = static_cast<uint32_t>(grids.cluster * (kClusterTile - 2 * radius));
    uint32_t one_wave = static_cast<uint32_t>(grids.wave), wide_grid = static_cast<uint32_t>(grids.wide);
    cudaError_t e = cudaSuccess;
    if ((N + ploc_own(radius) - 1) / ploc_own(radius) > one_wave) {
        void* args[] = {&ca, &cb, &node_box, &node_kids, &it, &N, &radius, &one_wave, &lookback, &tickets, &n_tiles_cap,
                        &bar, &iters_out, &err, &spin_limit};
        e = cudaLaunchCooperativeKernel(kWideFn, dim3(wide_grid), dim3(256), args, 0, s);
        if (e != cudaSuccess) return e;
        *enqueued = true;
    }
    if (N > stop_n) {
        void* args[] = {&ca, &cb, &node_box, &node_kids, &it, &N, &radius, &stop_n, &lookback, &n_tiles_cap, &wide_grid,
                        &bar, &iters_out, &err, &spin_limit};
        e = cudaLaunchCooperativeKernel(kWaveFn, dim3(one_wave), dim3(256), args, 0, s);
        if (e != cudaSuccess) return e;
        *enqueued = true;
    }
    ClusterLaunch l(grids.cluster, 1, s);
    e = cudaLaunchKernelEx(&l.c, ploc_cluster_kernel<kPlocMaxRadius>, static_cast<const float4*>(ca),
                           static_cast<const float4*>(cb), node_box, node_kids, it, N, radius, iters_out, err);
    if (e != cudaSuccess) return e;
    *enqueued = true;
    cudaEventRecord(ploc_done, s);
    const uint32_t want = (N + 254) / 256;  // N - 1 internal nodes
    uint32_t* dfs = reinterpret_cast<uint32_t*>(ca);
    void* args[] = {&dfs, &node_kids, &N, &pf, &err, &spin_limit};
    e = cudaLaunchCooperativeKernel(kPlacesFn, dim3(want < static_cast<uint32_t>(grids.places) ? want : grids.places),
                                    dim3(256), args, 0, s);
    if (e != cudaSuccess) return e;
    launch_layout_emit(node_box, node_kids, pf, N, dfs, out, wide, wide_wt, depth_odd, lv, st, err, s);
    return cudaGetLastError();
}

// A wait on a flag, bounded like every look-back and grid-barrier wait: on
// exhaustion the error word records the timeout and the kernel returns.
__global__ void wait_probe_kernel(const unsigned int* flag, uint32_t spin_limit, uint32_t* err) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    SpinBound spin(spin_limit);
    while (ld_acquire_u32(flag) == 0u)
        if (!spin.step()) { raise_error(err, kDevTimeout); return; }
}

void launch_wait_probe(const unsigned int* flag, uint32_t spin_limit, uint32_t* err, cudaStream_t s) {
    wait_probe_kernel<<<1, 32, 0, s>>>(flag, spin_limit, err);
}

void launch_single_leaf(const float4* node_box, crt_bvh_node* out, LeafOut lv, cudaStream_t s) {
    single_leaf_kernel<<<1, 1, 0, s>>>(node_box, out, lv);
}

}  // namespace crt

#include "crt_batch_kernels.cuh"
