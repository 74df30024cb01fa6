"""Imported trees (crt_bvh_from_nodes) whose stored boxes are not those of
their triangles: too large, too small, off by an ulp, or not nested.  The hits
of such a tree are decided by its stored boxes, so they must not depend on the
number of rays of a call, nor on the walk that number selects: large traces and
one-launch frames against one thread per ray on the binary nodes, bit for bit.
Where a box leaves out part of what it holds ("shrunk", "unnested"), its entry
distance is no bound for the hits below it, and which of several hits of a ray
survives pruning may depend on the order of the tests; whether there is one
does not, so large closest-hit traces of those compare hit and miss alone.  A
refit makes the boxes the triangles' own again."""
import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

from test_gpu_trace import _cmp_hits

pytestmark = pytest.mark.gpu

N_RAYS = 65536 + 5
MODES = ["shrunk", "grown", "ulp", "unnested"]


def changed_nodes(nodes, mode):
    """The array with the boxes of its leaves (or of some internal nodes) changed.  Columns 0:3 minimum, 4:7 maximum."""
    out = nodes.copy()
    kids = out.view(np.uint32)[:, 9:11]
    leaf = (kids == 0).all(1)
    lo, hi = out[:, 0:3], out[:, 4:7]
    mid, half = (lo + hi) / 2, (hi - lo) / 2
    if mode == "shrunk":
        lo[leaf], hi[leaf] = (mid - np.float32(0.4) * half)[leaf], (mid + np.float32(0.4) * half)[leaf]
    elif mode == "grown":
        lo[leaf], hi[leaf] = (mid - np.float32(2.0) * half)[leaf], (mid + np.float32(2.0) * half)[leaf]
    elif mode == "ulp":
        lo[leaf] = np.nextafter(lo[leaf], np.float32(np.inf))
        hi[leaf] = np.nextafter(hi[leaf], np.float32(-np.inf))
    else:  # internal boxes that cut off parts of the boxes below them
        cut = ~leaf & (np.arange(len(out)) > 0) & (np.arange(len(out)) % 3 == 0)
        hi[cut] = (mid + np.float32(0.5) * half)[cut]
    return out


@pytest.fixture(scope="module")
def scene():
    tris = S.uniform_soup(5000, seed=31, edge_lo=0.02, edge_hi=0.1)
    rays = S.sphere_rays(N_RAYS, seed=32)
    half = N_RAYS // 2  # these graze: aimed at vertices, which are corners or edges of their triangles' boxes
    d = tris[np.arange(half) % len(tris), 0:3].astype(np.float64) - rays[:half, 0:3]
    rays[:half, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return tris, S.identity_models(1), rays


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("predicate", [crt.TRI_REFERENCE, crt.TRI_WATERTIGHT])
def test_hits_do_not_depend_on_the_number_of_rays(ctx, scene, mode, predicate):
    tris, models, rays = scene
    built = ctx.build(tris, models=models)
    bvh = ctx.bvh_from_nodes(changed_nodes(built.nodes(), mode), tris, models=models)
    for flags in (predicate, predicate | crt.TRACE_ANY):
        want = ctx.trace(bvh, rays, flags | crt.PER_RAY_THREADS)
        few = np.concatenate([ctx.trace(bvh, rays[:40000], flags), ctx.trace(bvh, rays[40000:], flags)])
        any_hit = bool(flags & crt.TRACE_ANY)
        _cmp_hits(few, want, any_hit)
        any_hit = any_hit or mode in ("shrunk", "unnested")
        _cmp_hits(ctx.trace(bvh, rays, flags), want, any_hit)
        _cmp_hits(ctx.trace(bvh, rays, flags | crt.SORT_RAYS), want, any_hit)
        _cmp_hits(ctx.trace(bvh, rays[:500], flags | crt.TRACE_COMPRESSED), want[:500], any_hit)
    light = np.array([2.0, 2.0, -2.0], np.float32)
    cam = S.camera_gpu_data((0.5, 0.5, -1.5))
    prim = ctx.raygen(cam, 200, 160)
    want_p = ctx.trace(bvh, prim, predicate | crt.PER_RAY_THREADS)
    want_s = ctx.trace(bvh, ctx.shadow_rays(prim, want_p, light), predicate | crt.TRACE_ANY | crt.PER_RAY_THREADS)
    for _ in range(2):
        got_p, got_s = ctx.trace_frame(bvh, cam, 200, 160, light, predicate)
        _cmp_hits(got_p, want_p)
        _cmp_hits(got_s, want_s, any_hit=True)
    bvh.free()
    built.free()


@pytest.mark.parametrize("mode", MODES)
def test_refit_makes_the_boxes_the_triangles_own(ctx, scene, mode):
    tris, models, rays = scene
    built = ctx.build(tris, models=models)
    bvh = ctx.bvh_from_nodes(changed_nodes(built.nodes(), mode), tris, models=models)
    bvh.refit(tris, models=models)
    for flags in (crt.TRI_REFERENCE, crt.TRI_WATERTIGHT):
        _cmp_hits(ctx.trace(bvh, rays, flags), ctx.trace(built, rays, flags))
    bvh.free()
    built.free()
