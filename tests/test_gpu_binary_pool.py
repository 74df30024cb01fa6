"""Large closest-hit traces of scenes and rays that the walk over the compressed
nodes cannot take: persistent warps over the binary nodes (crt_pool.cuh), chosen
at once (a scene outside the quantised range, imported boxes that are not the
triangles'), after a launch has found that nothing can be quantised (vertices
that are not numbers), or for the rays left over.  Hits against one thread per
ray bit for bit (which other tests hold against the oracle), at trees of 2 to 5
leaves, deeper than the short stack, and at numbers of rays around the pool's
smallest launch."""
import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

from test_gpu_trace import _cmp_hits
from test_gpu_walk4 import mixed_rays, scene

pytestmark = pytest.mark.gpu

SCALE = np.float32(2.0 ** 52)


@pytest.mark.parametrize("flags", [crt.TRI_WATERTIGHT, crt.TRI_REFERENCE])
@pytest.mark.parametrize("n", [65535, 65536, 65536 + 33])
@pytest.mark.parametrize("name", ["n2", "n3", "n5", "n1025", "duplicates"])
def test_scene_outside_the_quantised_range(ctx, name, n, flags):
    tris = scene(name).copy()
    for c in (0, 4, 8):
        tris[:, c:c + 3] *= SCALE
    models = S.identity_models(1)
    rays = mixed_rays(tris, seed=len(name), n=n)
    bvh = ctx.build(tris, models=models)
    want = ctx.trace(bvh, rays, flags | crt.PER_RAY_THREADS)
    for order in (0, crt.SORT_RAYS):
        np.testing.assert_array_equal(ctx.trace(bvh, rays, flags | order).view(np.uint32), want.view(np.uint32))
    bvh.free()


@pytest.mark.parametrize("flags", [crt.TRI_WATERTIGHT, crt.TRI_REFERENCE, crt.TRI_WATERTIGHT | crt.TRACE_ANY])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_refit_to_vertices_that_are_not_finite(ctx, value, flags):
    """The first launch finds it out, the later ones know; the next refit makes the tree ordinary again."""
    tris = S.uniform_soup(30000, seed=71)
    models = S.identity_models(1)
    rays = S.sphere_rays(90001, seed=72)
    bvh = ctx.build(tris, models=models)
    good = ctx.trace(bvh, rays, flags)
    bad = tris.copy()
    bad[17, 0], bad[18, 5] = value, value
    any_hit = bool(flags & crt.TRACE_ANY)
    for _ in range(2):
        bvh.refit(bad, models=models)
        want = ctx.trace(bvh, rays, flags | crt.PER_RAY_THREADS)
        for order in (0, crt.SORT_RAYS, 0):
            _cmp_hits(ctx.trace(bvh, rays, flags | order), want, any_hit)
        bvh.refit(tris, models=models)
        for _ in range(2):
            _cmp_hits(ctx.trace(bvh, rays, flags), good, any_hit)
    bvh.free()
