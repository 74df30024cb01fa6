"""The persistent walk over the compressed 4-wide nodes (crt_walk4.cuh), which
crt_trace takes for at least 65,536 rays: its hits are the binary walk's
(CRT_TRACE_PER_RAY_THREADS) and the oracle's bit for bit at the sizes and rays
where it can go wrong — trees of 1 to 5 leaves, chains deeper than its stack,
exact duplicates, scenes whose boxes cannot be quantised, and rays the
compressed walk hands to the binary one (zero, tiny, infinite or NaN direction
components, far origins, negative tmin)."""
import numpy as np
import pytest

from oracle import oracle as O
from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

from test_gpu_trace import _cmp_hits

pytestmark = pytest.mark.gpu

N_RAYS = 65536 + 37  # the smallest launch of the walk, and a remainder
FLAGS = [crt.TRI_WATERTIGHT, crt.TRI_REFERENCE, crt.TRI_WATERTIGHT | crt.TRACE_ANY, crt.TRI_REFERENCE | crt.TRACE_ANY]


def mixed_rays(tris, seed, n=N_RAYS):
    """Rays toward the triangles of a scene, from around and inside it, some of each kind above."""
    r = np.random.RandomState(seed)
    v = tris[:, 0:3]
    lo, hi = v.min(0).astype(np.float64), v.max(0).astype(np.float64)
    size = max(float((hi - lo).max()), float(np.abs(v).max()), 1e-30)
    o = (lo + hi) / 2 + r.uniform(-1.5, 1.5, (n, 3)) * size
    target = v[r.randint(0, len(v), n)] + r.normal(0, 0.01, (n, 3)) * size
    d = target - o
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-300)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = o, d, np.inf
    k = n // 16
    rays[0:k, 4 + r.randint(0, 3)] = 0.0                              # an axis-parallel plane
    rays[k:k + 64, 4:7] = (0.0, 0.0, 1.0)
    rays[2 * k:3 * k, 0:3] = v[r.randint(0, len(v), k)] - rays[2 * k:3 * k, 4:7] * (40 * size)  # far origins
    rays[3 * k:4 * k, 7] = r.uniform(0, 2, k) * size                  # finite tmax
    rays[4 * k:5 * k, 3] = r.uniform(0, 1, k) * size                  # tmin past the origin
    rays[5 * k:6 * k, 3] = -size                                      # negative tmin
    rays[6 * k:7 * k, 4:7] *= r.choice([1e-3, 1e3], (k, 1))           # unnormalised directions
    rays[7 * k:7 * k + 64, 4] = 1e-25
    rays[7 * k + 64:7 * k + 80, 5] = np.inf
    rays[7 * k + 80:7 * k + 96, 6] = np.nan
    rays[7 * k + 96:7 * k + 112, 0] = np.nan
    rays[7 * k + 112:7 * k + 128, 3:8:4] = (1.0, 0.0)                 # empty: tmin > tmax
    return rays


def scene(name):
    if name[1:].isdigit():
        return S.uniform_soup(int(name[1:]), seed=3, edge_lo=0.05, edge_hi=0.3)
    if name == "duplicates":  # equal t everywhere, and a chain of 4-wide nodes deeper than the stack
        return np.concatenate([S.uniform_soup(1, seed=4, edge_lo=0.1, edge_hi=0.3)] * 600)
    if name == "clustered":
        return S.clustered_soup(30000, 32, 0.03, 0.005, 0.5, seed=5)
    t = S.uniform_soup(3000, seed=6)
    for c in (0, 4, 8):
        if name == "offset":   # far from the origin of coordinates: few bits left for the extent
            t[:, c:c + 3] += 1000.0
        if name == "flat":     # zero extent on one axis
            t[:, c + 1] = 0.25
        if name == "huge":     # outside the range the nodes are quantised in
            t[:, c:c + 3] *= np.float32(2.0 ** 52)
        if name == "tiny":
            t[:, c:c + 3] *= np.float32(2.0 ** -44)
    return t


@pytest.mark.parametrize("flags", FLAGS)
@pytest.mark.parametrize("name", ["n1", "n2", "n3", "n4", "n5", "n1025", "clustered", "duplicates", "offset", "flat"])
def test_walk_matches_oracle(ctx, name, flags):
    tris = scene(name)
    models = S.identity_models(1)
    rays = mixed_rays(tris, seed=len(name))
    bvh = ctx.build(tris, models=models)
    got = ctx.trace(bvh, rays, flags)
    _cmp_hits(got, ctx.trace(bvh, rays, flags | crt.PER_RAY_THREADS), bool(flags & crt.TRACE_ANY))
    # the oracle's IEEE slabs: both walks decide as they do for rays of numbers from within 8 times the scene's
    # range (slab_wt) that look forward (a hit behind the origin hangs on the sign of a rounded exit distance)
    reach = 8 * np.abs(tris[:, [0, 1, 2, 4, 5, 6, 8, 9, 10]]).max()
    near = np.isfinite(rays[:, 0:7]).all(1) & (np.abs(rays[:, 0:3]).max(1) <= reach) & (rays[:, 3] >= 0)
    ref, _ = O.trace(bvh.nodes(), tris, models, rays[near], flags)
    _cmp_hits(got[near], ref, bool(flags & crt.TRACE_ANY))
    bvh.free()


@pytest.mark.parametrize("flags", FLAGS)
@pytest.mark.parametrize("name", ["huge", "tiny", "nonfinite", "clustered", "duplicates"])
def test_walk_matches_binary_walk(ctx, name, flags):
    """Every order and the one-thread form of the compressed walk against one thread per ray on the binary nodes."""
    tris = scene(name)
    rays = mixed_rays(tris, seed=7)
    bvh = ctx.build(tris, models=S.identity_models(1))
    if name == "nonfinite":  # boxes that a refit made infinite
        tris[17, 0], tris[18, 5] = np.inf, -np.inf
        bvh.refit(tris, models=S.identity_models(1))
    want = ctx.trace(bvh, rays, flags | crt.PER_RAY_THREADS)
    for extra in (0, crt.SORT_RAYS, crt.TRACE_COMPRESSED | crt.PER_RAY_THREADS):
        got = ctx.trace(bvh, rays, flags | extra)
        if flags & crt.TRACE_ANY:
            np.testing.assert_array_equal(got[:, 0].view(np.uint32) == crt.MISS, want[:, 0].view(np.uint32) == crt.MISS)
        else:
            np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32), err_msg=hex(extra))
    bvh.free()


@pytest.mark.parametrize("flags", FLAGS)
def test_batch_walk_matches_single_scenes(ctx, flags):
    """A batch of at least 65,536 rays: scenes of 1, 2 and 5 leaves and unquantised ones beside ordinary ones, traced
    after a build and by a captured graph."""
    torch = pytest.importorskip("torch")
    names = ["n1", "clustered", "n2", "n5", "n1025", "duplicates", "offset"]
    tris = [scene(k) for k in names]
    rays = [mixed_rays(t, seed=11 + k, n=16000 + 33 * k) for k, t in enumerate(tris)]
    batch = crt.Batch(ctx, [len(t) for t in tris], [len(r) for r in rays], models=S.identity_models(1))
    d_tris, d_rays = (torch.from_numpy(np.concatenate(x)).cuda() for x in (tris, rays))
    hits = torch.empty((d_rays.shape[0], 4), dtype=torch.float32, device="cuda")

    def check(what):
        got, off = hits.cpu().numpy(), 0
        for t, r in zip(tris, rays):
            bvh = ctx.build(t, models=S.identity_models(1))
            want = ctx.trace(bvh, r, flags | crt.PER_RAY_THREADS)
            g = got[off:off + len(r)]
            if flags & crt.TRACE_ANY:
                np.testing.assert_array_equal(g[:, 0].view(np.uint32) == crt.MISS, want[:, 0].view(np.uint32) == crt.MISS)
            else:
                np.testing.assert_array_equal(g.view(np.uint32), want.view(np.uint32), err_msg=what)
            off += len(r)
            bvh.free()

    batch.build(d_tris)
    batch.trace(d_rays, hits, flags)
    check("build, trace")
    for _ in range(2):  # captured, then replayed
        hits.zero_()
        batch.run(d_tris, d_rays, hits, flags, graph=True)
    check("graph")
    hits.zero_()
    batch.trace(d_rays, hits, flags | crt.SORT_RAYS)
    check("sorted")
    batch.free()
