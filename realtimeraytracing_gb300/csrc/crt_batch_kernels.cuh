// Included at the end of crt_build.cu (it reuses that file's PLOC tile,
// layout and grid-barrier device code).
//
// Many scenes in one pipeline (config 2): every stage is one launch over all
// scenes: the PLOC iterations run in lockstep inside one persistent cooperative
// kernel while a scene is larger than its thread-block cluster holds, then one
// cluster a scene, then the layout, and the whole build + trace can be captured
// into a CUDA graph and replayed.  Each scene's BVH is bit-identical to the
// one crt_build makes for that scene alone (same codes, same sort order,
// same PLOC decisions), because every kernel only sees its scene's data
// through per-scene offsets.
#pragma once

namespace crt {

// Per-scene reduction state of the scene box (all-zero initial state: the
// minimum keys are stored inverted so a memset resets them).
struct BatchBoxState {
    unsigned long long key_max[3];
    unsigned long long key_min_inv[3];
    unsigned int blocks_done;
    unsigned int pad0;
    float cube_min[3];
    float cube_len[3];
    float pad[2];
};

struct Chunk {
    uint32_t scene, begin, end, pad;
};

constexpr uint32_t kBoxChunk = 256 * 16;

__device__ __forceinline__ uint32_t scene_of(const uint32_t* off, uint32_t n, uint32_t i) {
    uint32_t lo = 0, hi = n - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (off[mid] <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ void tri_extent_b(const TriRec& t, const float* __restrict__ models, float hi[3], float lo[3]) {
    const float* M = models + 16 * (t.model & (kMaxModels - 1));
    const float4 p0 = mat_vec(M, t.p0), p1 = mat_vec(M, t.p1), p2 = mat_vec(M, t.p2);
    hi[0] = max_std(p0.x, max_std(p1.x, p2.x));
    hi[1] = max_std(p0.y, max_std(p1.y, p2.y));
    hi[2] = max_std(p0.z, max_std(p1.z, p2.z));
    lo[0] = min_std(p0.x, min_std(p1.x, p2.x));
    lo[1] = min_std(p0.y, min_std(p1.y, p2.y));
    lo[2] = min_std(p0.z, min_std(p1.z, p2.z));
}

// Scene boxes (bvh.cpp:235-251 per scene, leftmost arg-max as in the single
// scene kernel), then the cube (bvh.cpp:253-303) by each scene's last chunk.
__global__ void __launch_bounds__(256) batch_box_kernel(const crt_triangle* __restrict__ tris, const Chunk* __restrict__ chunks,
                                                        const float* __restrict__ models, BatchBoxState* states,
                                                        BatchScene* scenes, uint32_t* err) {
    const Chunk ch = chunks[blockIdx.x];
    BatchBoxState* st = states + ch.scene;
    unsigned long long kmax[3] = {0ull, 0ull, 0ull}, kmin[3] = {0ull, 0ull, 0ull};  // kmin inverted
    bool bad = false;
    for (uint32_t i = ch.begin + threadIdx.x; i < ch.end; i += 256) {
        const TriRec t = load_tri(tris, i);
        bad |= t.model >= kMaxModels;
        float hi[3], lo[3];
        tri_extent_b(t, models, hi, lo);
        const uint32_t li = i - scenes[ch.scene].tri_off;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (hi[a] == hi[a]) {
                const unsigned long long k = (static_cast<unsigned long long>(ordered_key(hi[a])) << 32) | (0xFFFFFFFFu - li);
                kmax[a] = k > kmax[a] ? k : kmax[a];
            }
            if (lo[a] == lo[a]) {
                const unsigned long long k = ~((static_cast<unsigned long long>(ordered_key(lo[a])) << 32) | li);
                kmin[a] = k > kmin[a] ? k : kmin[a];
            }
        }
    }
    if (bad) raise_error(err, kDevBadModel);
#pragma unroll
    for (int a = 0; a < 3; ++a)
        for (int m = 16; m > 0; m >>= 1) {
            const unsigned long long x = __shfl_xor_sync(0xFFFFFFFFu, kmax[a], m), y = __shfl_xor_sync(0xFFFFFFFFu, kmin[a], m);
            kmax[a] = x > kmax[a] ? x : kmax[a];
            kmin[a] = y > kmin[a] ? y : kmin[a];
        }
    __shared__ unsigned long long s_k[6][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int a = 0; a < 3; ++a) { s_k[a][warp] = kmax[a]; s_k[3 + a][warp] = kmin[a]; }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int a = threadIdx.x;
        unsigned long long v = s_k[a][0];
        for (int w = 1; w < 8; ++w) v = s_k[a][w] > v ? s_k[a][w] : v;
        if (a < 3) atomicMax(&st->key_max[a], v); else atomicMax(&st->key_min_inv[a - 3], v);
    }
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(&st->blocks_done, 1u) == scenes[ch.scene].n_chunks - 1);
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    const uint32_t base = scenes[ch.scene].tri_off;
    const float kInf = __int_as_float(0x7F800000);
    float smin[3], smax[3];
    for (int a = 0; a < 3; ++a) {
        const unsigned long long kx = atomicAdd(&st->key_max[a], 0ull);
        const unsigned long long kn = ~atomicAdd(&st->key_min_inv[a], 0ull);
        smax[a] = -kInf;
        smin[a] = kInf;
        float hi[3], lo[3];
        if (kx != 0ull) {
            tri_extent_b(load_tri(tris, base + (0xFFFFFFFFu - static_cast<uint32_t>(kx))), models, hi, lo);
            smax[a] = hi[a];
        }
        if (kn != ~0ull) {
            tri_extent_b(load_tri(tris, base + static_cast<uint32_t>(kn)), models, hi, lo);
            smin[a] = lo[a];
        }
    }
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
        st->cube_min[a] = cmn[a];
        st->cube_len[a] = cmx[a] - cmn[a];
    }
    scenes[ch.scene].abs_eps = scene_abs_eps(smin, smax);
}

__device__ __forceinline__ uint32_t expand_bits_b(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__device__ __forceinline__ uint32_t to_u10_b(float x) {
    x = min_std(max_std(x * 1024.0f, 0.0f), 1023.0f);
    return __float2uint_rz(x);
}

template <int BITS>
__global__ void __launch_bounds__(256) batch_morton_kernel(const crt_triangle* __restrict__ tris, const Chunk* __restrict__ chunks,
                                                           const float* __restrict__ models_third,
                                                           const BatchBoxState* __restrict__ states,
                                                           uint32_t* __restrict__ codes, uint32_t* __restrict__ hist) {
    constexpr int RADIX = 1 << BITS;
    constexpr int PASSES = (30 + BITS - 1) / BITS;
    __shared__ uint32_t s_hist[PASSES * RADIX];
    for (int i = threadIdx.x; i < PASSES * RADIX; i += blockDim.x) s_hist[i] = 0u;
    __syncthreads();
    const Chunk ch = chunks[blockIdx.x];
    const BatchBoxState* st = states + ch.scene;
    const float cmx = st->cube_min[0], cmy = st->cube_min[1], cmz = st->cube_min[2];
    const float lx = st->cube_len[0], ly = st->cube_len[1], lz = st->cube_len[2];
    for (uint32_t i = ch.begin + threadIdx.x; i < ch.end; i += 256) {
        const TriRec t = load_tri(tris, i);
        const float* M3 = models_third + 16 * (t.model & (kMaxModels - 1));
        float4 s;
        s.x = t.p0.x + t.p1.x + t.p2.x;
        s.y = t.p0.y + t.p1.y + t.p2.y;
        s.z = t.p0.z + t.p1.z + t.p2.z;
        s.w = t.p0.w + t.p1.w + t.p2.w;
        const float4 c = mat_vec(M3, s);
        const float nx = (c.x - cmx) / lx, ny = (c.y - cmy) / ly, nz = (c.z - cmz) / lz;
        const uint32_t code = (expand_bits_b(to_u10_b(nx)) << 2) | (expand_bits_b(to_u10_b(ny)) << 1) | expand_bits_b(to_u10_b(nz));
        codes[i] = code;
#pragma unroll
        for (int p = 0; p < PASSES; ++p) atomicAdd(&s_hist[p * RADIX + ((code >> (p * BITS)) & (RADIX - 1))], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < PASSES * RADIX; i += blockDim.x)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// Leaf clusters per scene (as leaf_init_kernel), plus each scene's first
// PLOC record and, for one-triangle scenes, their single output node.
__global__ void __launch_bounds__(256) batch_leaf_init_kernel(const crt_triangle* __restrict__ tris, uint32_t n_total,
                                                              BatchScene* scenes, uint32_t n_scenes,
                                                              const float* __restrict__ models,
                                                              const uint32_t* __restrict__ perm_global,
                                                              uint32_t* __restrict__ perm_local, float4* __restrict__ node_box,
                                                              float4* __restrict__ clusters,
                                                              float4* __restrict__ xtri_sorted, float4* __restrict__ xtri,
                                                              uint32_t* __restrict__ leaf_of_tri, uint2* __restrict__ it,
                                                              crt_bvh_node* __restrict__ nodes, uint2* __restrict__ pf,
                                                              uint32_t* err) {
    __shared__ uint32_t s_off[kMaxBatchScenes];
    for (uint32_t k = threadIdx.x; k < n_scenes; k += 256) s_off[k] = scenes[k].tri_off;
    __syncthreads();
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n_total) return;
    const uint32_t s = scene_of(s_off, n_scenes, i);
    const BatchScene sc = scenes[s];
    const uint32_t li = i - sc.tri_off;
    const uint32_t tg = perm_global[i];
    const uint32_t tl = tg - sc.tri_off;
    if (tg < sc.tri_off || tl >= sc.n_tris) { raise_corrupt(err, 6, i, tg); return; }
    if (li == 0) {
        it[sc.it_off] = make_uint2(sc.n_tris, sc.n_tris);
        scenes[s].iters = sc.n_tris > 1 ? 0u : 1u;   // one-triangle scenes need no iteration
    }
    perm_local[i] = tl;
    pf[i] = make_uint2(kLayoutUnset, 0u);  // the layout's places arrive from each node's parent
    const TriRec t = load_tri(tris, tg);
    const float* M = models + 16 * (t.model & (kMaxModels - 1));
    const float4 p0 = mat_vec(M, t.p0), p1 = mat_vec(M, t.p1), p2 = mat_vec(M, t.p2);
    float4 mn, mx;
    mn.x = min_std(p0.x, min_std(p1.x, p2.x));
    mn.y = min_std(p0.y, min_std(p1.y, p2.y));
    mn.z = min_std(p0.z, min_std(p1.z, p2.z));
    mx.x = max_std(p0.x, max_std(p1.x, p2.x));
    mx.y = max_std(p0.y, max_std(p1.y, p2.y));
    mx.z = max_std(p0.z, max_std(p1.z, p2.z));
    const size_t nb = 2 * (static_cast<size_t>(sc.node_off) + li);
    st_record(node_box + nb, make_float4(mn.x, mn.y, mn.z, __uint_as_float(tl)), make_float4(mx.x, mx.y, mx.z, 0.f));
    st_record(clusters + 2 * static_cast<size_t>(i), make_float4(mn.x, mn.y, mn.z, __uint_as_float(li)),
              make_float4(mx.x, mx.y, mx.z, __uint_as_float(1u)));
    // sorted order; the layout moves them into tree order (a one-triangle
    // scene's single leaf is in both orders at once)
    float4* xo = (sc.n_tris == 1 ? xtri : xtri_sorted) + 3 * static_cast<size_t>(i);
    xo[0] = make_float4(p0.x, p0.y, p0.z, __uint_as_float(tl));
    xo[1] = make_float4(p1.x, p1.y, p1.z, __uint_as_float(t.model));
    xo[2] = make_float4(p2.x, p2.y, p2.z, 0.f);
    if (sc.n_tris == 1) {
        leaf_of_tri[sc.tri_off] = 0u;
        float4* o = reinterpret_cast<float4*>(nodes + sc.node_off);
        o[0] = make_float4(mn.x, mn.y, mn.z, 0.f);
        o[1] = make_float4(mx.x, mx.y, mx.z, 0.f);
        reinterpret_cast<uint4*>(o)[2] = make_uint4(tl, 0u, 0u, 0u);
    }
}

// The sum of v over the threads before this one, and over all (BLOCK threads).
template <int BLOCK>
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* s_warp, uint32_t& total) {
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if ((threadIdx.x & 31u) >= o) incl += y;
    }
    if ((threadIdx.x & 31u) == 31u) s_warp[threadIdx.x >> 5] = incl;
    __syncthreads();
    uint32_t before = 0u;
    total = 0u;
#pragma unroll
    for (uint32_t w = 0; w < BLOCK / 32; ++w) {
        if (w < threadIdx.x >> 5) before += s_warp[w];
        total += s_warp[w];
    }
    return before + incl - v;
}

// The PLOC iterations of the scenes of more than stop_n live clusters, in
// lockstep.  Each iteration: every block derives the running scenes' tile counts,
// takes tiles from one ticket counter, maps a ticket to (scene, tile) and runs the
// single-scene tile code (ploc_open, ploc_close) on that scene's slices.  A grid barrier separates
// iterations.  A scene leaves with its iteration count in scenes[].iters once it
// has stop_n clusters or fewer; batch_cluster_kernel finishes it.  Thread k of
// every block keeps scene k, and the tile counts are scanned by the whole block:
// a loop over the scenes in one thread cost 64 dependent steps an iteration.
// Whole batch builds before and with the three launches below, us: 64 scenes of
// 1,000-250,000 triangles 2,730 -> 1,446, 16 of 5,000-20,000 886 -> 394, 200 of
// 100-5,000 1,795 -> 442, 2 of 1-1.5 M 2,493 -> 1,642 (the first and the last were
// 1,566 and 1,836 with tiles that wait for their predecessors at once).
template <int TILE, int BLOCK, int MAXR>
__global__ void __launch_bounds__(BLOCK, kPlocBlocksPerSm) batch_ploc_kernel(BatchScene* scenes, uint32_t n_scenes, float4* ca, float4* cb,
                                                           float4* node_box, uint4* node_kids, uint2* it, int R,
                                                           uint32_t stop_n, unsigned long long* lookback, uint32_t lb_cap,
                                                           uint32_t* tickets, unsigned long long* bar, uint32_t max_iters,
                                                           uint32_t* err, uint32_t spin_limit) {
    static_assert(BLOCK >= static_cast<int>(kMaxBatchScenes), "a thread per scene");
    __shared__ PlocPipeSmem<TILE, BLOCK, MAXR> P;
    unsigned long long bar_target = 0;  // grid barriers passed x gridDim (thread 0)
    __shared__ uint32_t s_tile_pre[BLOCK];
    __shared__ uint32_t s_n[BLOCK];
    __shared__ uint32_t s_warp[BLOCK / 32];
    const uint32_t k = threadIdx.x;
    uint32_t n = k < n_scenes ? scenes[k].n_tris : 0u;  // scene k's live clusters; no longer read once <= stop_n
    const uint32_t it_off = k < n_scenes ? scenes[k].it_off : 0u;
    for (int iter = 0;; ++iter) {
        if (iter > 0 && n > stop_n) {
            n = __ldcg(it + it_off + iter).x;
            if (n <= stop_n && blockIdx.x == 0) scenes[k].iters = static_cast<uint32_t>(iter);
        }
        const uint32_t tiles = n > stop_n ? (n + ploc_own(R) - 1) / ploc_own(R) : 0u;
        s_n[k] = n;
        uint32_t total;
        s_tile_pre[k] = block_exclusive<BLOCK>(tiles, s_warp, total);
        if (total == 0u) break;  // uniform: every thread has the same total
        if (static_cast<uint32_t>(iter) >= max_iters) { raise_error(err, kDevIterLimit); return; }
        // as ploc_wide_kernel: a tile is opened before the last one is closed
        if (threadIdx.x == 0) P.ticket = atomicAdd(&tickets[iter & 1], 1u);
        uint32_t open = 0u, open_scene = 0u, open_total = 0u;
        bool some = false;  // a tile is open
        for (int buf = 0;; buf ^= 1) {
            __syncthreads();
            const uint32_t g = P.ticket;
            const bool more = g < total;
            uint32_t lo = 0, tile_total = 0u, tile = 0u;
            if (more) {
                uint32_t hi = n_scenes - 1;  // the scene whose tile range holds g
                while (lo < hi) {
                    const uint32_t mid = (lo + hi + 1) >> 1;
                    if (s_tile_pre[mid] <= g) lo = mid; else hi = mid - 1;
                }
                tile = g - s_tile_pre[lo];
                const BatchScene& B = scenes[lo];
                const float4* cin = ((iter & 1) ? cb : ca) + 2 * static_cast<size_t>(B.tri_off);
                unsigned long long* lb = lookback + B.lb_off;
                tile_total = ploc_open(P, buf, tile, static_cast<int>(s_n[lo]), cin, R, lb + static_cast<size_t>(iter & 1) * lb_cap,
                                       lb + static_cast<size_t>((iter + 1) & 1) * lb_cap);
                if (threadIdx.x == 32) {  // not the warp that looks back
                    P.ticket = atomicAdd(&tickets[iter & 1], 1u);
                    if (g == 0) tickets[(iter + 1) & 1] = 0u;
                }
            }
            if (some) {
                const BatchScene& B = scenes[open_scene];
                const uint2 cur = make_uint2(s_n[open_scene], __ldcg(it + B.it_off + iter).y);
                const float4* cin = ((iter & 1) ? cb : ca) + 2 * static_cast<size_t>(B.tri_off);
                float4* cout = ((iter & 1) ? ca : cb) + 2 * static_cast<size_t>(B.tri_off);
                ploc_close(P, buf ^ 1, open, open_total, cur, iter, cin, cout, node_box + 2 * static_cast<size_t>(B.node_off),
                           node_kids + B.tri_off, it + B.it_off, B.n_tris, R,
                           lookback + static_cast<size_t>(iter & 1) * lb_cap + B.lb_off, err, spin_limit);
            }
            if (!more) break;
            some = true;
            open = tile;
            open_scene = lo;
            open_total = tile_total;
        }
        if (!grid_barrier(bar, bar_target, err, spin_limit)) return;
    }
}

// Every scene's remaining PLOC iterations, one cluster a scene (ploc_cluster_r);
// scenes[].iters: iterations done before, then all of them.
__global__ void __launch_bounds__(kClusterThreads) batch_cluster_kernel(BatchScene* scenes, const float4* ca, const float4* cb,
                                                                        float4* node_box, uint4* node_kids, uint2* it, int R,
                                                                        uint32_t* err) {
    extern __shared__ __align__(16) unsigned char cluster_smem[];
    ClusterSmem& C = *reinterpret_cast<ClusterSmem*>(cluster_smem);
    BatchScene& B = scenes[blockIdx.x / cooperative_groups::this_cluster().num_blocks()];
    const uint32_t N = B.n_tris;
    if (N < 2) return;  // no node to make
    const int iter = static_cast<int>(__ldcg(&B.iters));
    const float4* cin = ((iter & 1) ? cb : ca) + 2 * static_cast<size_t>(B.tri_off);
    float4* box = node_box + 2 * static_cast<size_t>(B.node_off);
    uint4* kids = node_kids + B.tri_off;
    uint2* rec = it + B.it_off;
    switch (R) {
        case 8: ploc_cluster_r<8>(C, iter, cin, box, kids, rec, N, R, &B.iters, err); break;
        case 16: ploc_cluster_r<16>(C, iter, cin, box, kids, rec, N, R, &B.iters, err); break;
        case 32: ploc_cluster_r<32>(C, iter, cin, box, kids, rec, N, R, &B.iters, err); break;
        default: ploc_cluster_r<0>(C, iter, cin, box, kids, rec, N, R, &B.iters, err); break;
    }
}

// The layout's position pass (layout_places_kernel) over all scenes.  A scene
// has blocks of its own, one per `share` of its internal nodes, so the scenes'
// chains of places run side by side (blocks that also held the end of the scene
// before made one chain of them all: 64 scenes of 2.6 M triangles 1,350 us, now
// 94).  A grid barrier a PLOC level, with a loop over the scenes in one thread, was
// what both replace.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) batch_places_kernel(const BatchScene* __restrict__ scenes, uint32_t n_scenes,
                                                             uint32_t share, uint32_t* __restrict__ dfs,
                                                             const uint4* __restrict__ node_kids, uint2* pf, uint32_t* err,
                                                             uint32_t spin_limit) {
    static_assert(BLOCK >= static_cast<int>(kMaxBatchScenes), "a thread per scene");
    __shared__ uint32_t s_warp[BLOCK / 32];
    __shared__ uint32_t s_mine[3];  // this block's scene, its place among the scene's blocks, their number
    const uint32_t k = threadIdx.x;
    const uint32_t blocks = k < n_scenes ? (scenes[k].n_tris - 1 + share - 1) / share : 0u;
    uint32_t total;
    const uint32_t first = block_exclusive<BLOCK>(blocks, s_warp, total);
    if (blockIdx.x >= total) return;  // uniform
    if (blockIdx.x - first < blocks) {
        s_mine[0] = k;
        s_mine[1] = blockIdx.x - first;
        s_mine[2] = blocks;
    }
    __syncthreads();
    if (build_failed(err)) return;  // as layout_places_kernel
    const BatchScene B = scenes[s_mine[0]];
    const uint32_t N = B.n_tris, stride = s_mine[2] * BLOCK;
    for (uint32_t t = s_mine[1] * BLOCK + threadIdx.x; t + 1 < N; t += stride)
        if (!layout_place_node(2 * N - 2 - t, t < stride, dfs + B.node_off, node_kids + B.tri_off, N, pf + B.tri_off, err,
                               spin_limit))
            return;
}

// Every DFS position of every scene with more than one triangle, in order.
__global__ void __launch_bounds__(256) batch_emit_kernel(const BatchScene* __restrict__ scenes, uint32_t n_scenes,
                                                         uint32_t n_slots, const float4* __restrict__ node_box,
                                                         const uint4* __restrict__ node_kids, const uint2* __restrict__ pf,
                                                         const uint32_t* __restrict__ dfs, crt_bvh_node* __restrict__ nodes,
                                                         float4* __restrict__ wide, float4* __restrict__ wide_wt,
                                                         uint8_t* __restrict__ depth_odd, LeafOut lv, uint32_t* err) {
    const uint32_t q = blockIdx.x * 256 + threadIdx.x;
    if (q >= n_slots || build_failed(err)) return;
    uint32_t lo = 0, hi = n_scenes - 1;  // node_off: slots before the scene
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(&scenes[mid].node_off) <= q) lo = mid; else hi = mid - 1;
    }
    const BatchScene B = scenes[lo];
    if (B.n_tris < 2) return;  // written with the leaves
    const LeafOut slv{lv.xtri_sorted + 3 * static_cast<size_t>(B.tri_off), lv.xtri + 3 * static_cast<size_t>(B.tri_off),
                      lv.leaf_of_tri + B.tri_off};
    layout_emit(q - B.node_off, node_box + 2 * static_cast<size_t>(B.node_off), node_kids + B.tri_off, pf + B.tri_off,
                B.n_tris, dfs + B.node_off, nodes + B.node_off, wide + 4 * static_cast<size_t>(B.wide_off),
                wide_wt + 4 * static_cast<size_t>(B.wide_off), depth_odd + B.wide_off, slv, B.abs_eps, err);
}

// ------------------------------------------------------------------ launchers
void launch_batch_box(const crt_triangle* tris, const void* chunks, uint32_t n_chunks, const float* models, void* states,
                      BatchScene* scenes, uint32_t* err, cudaStream_t s) {
    batch_box_kernel<<<n_chunks, 256, 0, s>>>(tris, static_cast<const Chunk*>(chunks), models,
                                              static_cast<BatchBoxState*>(states), scenes, err);
}

void launch_batch_morton(const crt_triangle* tris, const void* chunks, uint32_t n_chunks, const float* models_third,
                         const void* states, uint32_t* codes, uint32_t* hist, int bits, cudaStream_t s) {
    if (bits == 4)
        batch_morton_kernel<4><<<n_chunks, 256, 0, s>>>(tris, static_cast<const Chunk*>(chunks), models_third,
                                                        static_cast<const BatchBoxState*>(states), codes, hist);
    else
        batch_morton_kernel<8><<<n_chunks, 256, 0, s>>>(tris, static_cast<const Chunk*>(chunks), models_third,
                                                        static_cast<const BatchBoxState*>(states), codes, hist);
}

void launch_batch_leaf_init(const crt_triangle* tris, uint32_t n_total, BatchScene* scenes, uint32_t n_scenes,
                            const float* models, const uint32_t* perm_global, uint32_t* perm_local, float4* node_box,
                            float4* clusters, float4* xtri_sorted, float4* xtri, uint32_t* leaf_of_tri, uint2* it,
                            crt_bvh_node* nodes, uint2* pf, uint32_t* err, cudaStream_t s) {
    batch_leaf_init_kernel<<<(n_total + 255) / 256, 256, 0, s>>>(tris, n_total, scenes, n_scenes, models, perm_global,
                                                                 perm_local, node_box, clusters, xtri_sorted, xtri,
                                                                 leaf_of_tri, it, nodes, pf, err);
}

void build_prepare() {
    ClusterLaunch::allow(reinterpret_cast<const void*>(ploc_cluster_kernel<kPlocMaxRadius>));
    ClusterLaunch::allow(reinterpret_cast<const void*>(batch_cluster_kernel));
}

// Blocks of a scene's cluster: the most for which every scene's cluster is
// resident at once (up to 16; 152 SMs hold 76 clusters of two, 8 of sixteen), so
// that the scenes' chains of iterations run side by side.
static int batch_cluster_blocks(uint32_t n_scenes) {
    const std::array<int, 5> active = per_device<std::array<int, 5>>([] {  // clusters of 1 << i blocks the device holds
        std::array<int, 5> a{};
        for (int i = 0; i < 5; ++i) a[i] = ClusterLaunch::active(reinterpret_cast<const void*>(batch_cluster_kernel), 1 << i);
        return a;
    });
    for (int i = 4; i >= 0; --i)
        if (active[i] > 0 && (static_cast<uint32_t>(active[i]) >= n_scenes || i == 0)) return 1 << i;
    return 0;
}

struct BatchGrids {
    int ploc = 0, places = 0;
};

cudaError_t launch_batch_ploc(BatchScene* scenes, uint32_t n_scenes, uint32_t n_total, uint32_t max_n, float4* ca,
                              float4* cb, float4* node_box, uint4* node_kids, uint2* it, int radius,
                              unsigned long long* lookback, uint32_t lb_cap, uint32_t* tickets, uint2* pf,
                              crt_bvh_node* nodes, float4* wide, float4* wide_wt, uint8_t* depth_odd, LeafOut lv,
                              unsigned long long* bar, uint32_t* err, uint32_t spin_limit, cudaStream_t s) {
    const void* ploc_fn = reinterpret_cast<const void*>(batch_ploc_kernel<kPlocSpan, 256, kPlocMaxRadius>);
    const void* places_fn = reinterpret_cast<const void*>(batch_places_kernel<256>);
    const BatchGrids grids = per_device<BatchGrids>([&] {
        return BatchGrids{cooperative_grid(ploc_fn, kPlocBlocksPerSm), cooperative_grid(places_fn, kAnyPerSm)};
    });
    const int grid = grids.ploc, blocks = batch_cluster_blocks(n_scenes);
    // a scene's places are laid out by whole blocks: at most inner / share + n_scenes of them, all resident
    if (grid <= 0 || blocks <= 0 || grids.places <= static_cast<int>(n_scenes)) return cudaErrorNotSupported;
    cudaError_t e = cudaSuccess;
    uint32_t stop_n = static_cast<uint32_t>(blocks * (kClusterTile - 2 * radius)), max_iters = max_n + 1;
    if (max_n > stop_n) {
        void* args[] = {&scenes, &n_scenes, &ca, &cb, &node_box, &node_kids, &it, &radius, &stop_n, &lookback, &lb_cap,
                        &tickets, &bar, &max_iters, &err, &spin_limit};
        e = cudaLaunchCooperativeKernel(ploc_fn, dim3(grid), dim3(256), args, 0, s);
        if (e != cudaSuccess) return e;
    }
    const uint32_t inner = n_total - n_scenes;  // internal nodes
    if (inner == 0) return cudaSuccess;
    ClusterLaunch l(blocks, n_scenes, s);
    e = cudaLaunchKernelEx(&l.c, batch_cluster_kernel, scenes, static_cast<const float4*>(ca), static_cast<const float4*>(cb),
                           node_box, node_kids, it, radius, err);
    if (e != cudaSuccess) return e;
    const uint32_t spread = static_cast<uint32_t>(grids.places) - n_scenes;
    uint32_t share = (inner + spread - 1) / spread;
    share = share > 256 ? share : 256;
    uint32_t* dfs = reinterpret_cast<uint32_t*>(ca);  // node ids by DFS position: the clusters are done with
    const BatchScene* cs = scenes;
    const uint4* ck = node_kids;
    void* args[] = {&cs, &n_scenes, &share, &dfs, &ck, &pf, &err, &spin_limit};
    e = cudaLaunchCooperativeKernel(places_fn, dim3(inner / share + n_scenes), dim3(256), args, 0, s);
    if (e != cudaSuccess) return e;
    const uint32_t slots = n_total + inner;
    batch_emit_kernel<<<(slots + 255) / 256, 256, 0, s>>>(cs, n_scenes, slots, node_box, node_kids, pf, dfs, nodes, wide,
                                                          wide_wt, depth_odd, lv, err);
    return cudaGetLastError();
}

size_t batch_box_state_bytes() { return sizeof(BatchBoxState); }
size_t batch_chunk_bytes() { return sizeof(Chunk); }
uint32_t batch_box_chunk() { return kBoxChunk; }

}  // namespace crt
