"""One-launch frames over the compressed nodes: images whose tiles have
remainders, more tiles than resident warps, one row, trees below the walk's
smallest and scenes it cannot quantise, with shadow rays and shaded, against the
separate raygen, per-ray trace, shadow-ray and shade calls bit for bit."""
import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

from test_gpu_trace import _cmp_hits
from test_gpu_walk4 import scene

pytestmark = pytest.mark.gpu

LIGHT = np.array([2.0, 2.0, -2.0], np.float32)


@pytest.mark.parametrize("wt", [crt.TRI_WATERTIGHT, crt.TRI_REFERENCE])
@pytest.mark.parametrize("name,w,h", [("n1", 33, 5), ("n2", 8, 4), ("n5", 1, 1), ("n1025", 129, 1), ("clustered", 67, 43),
                                      ("clustered", 512, 400), ("duplicates", 40, 24), ("huge", 64, 32)])
def test_frame_matches_separate_calls(ctx, name, w, h, wt):
    tris = scene(name)
    models = S.identity_models(1)
    bvh = ctx.build(tris, models=models)
    size = np.float32(2.0 ** 52) if name == "huge" else np.float32(1.0)
    cam = S.camera_gpu_data((0.5, 0.5, -1.5), aspect=w / h)
    cam[[12, 13, 14, 16, 17, 18]] *= size
    light = LIGHT * size
    rays = ctx.raygen(cam, w, h)
    want_p = ctx.trace(bvh, rays, wt | crt.PER_RAY_THREADS)
    want_s = ctx.trace(bvh, ctx.shadow_rays(rays, want_p, light), wt | crt.TRACE_ANY | crt.PER_RAY_THREADS)
    mats = S.materials([[0.75, 0.5, 0.25, 1.0]])
    want_i = ctx.shade(bvh, None, want_p, models=models, materials=mats, shade_flags=crt.SHADE_WIREFRAME)
    for _ in range(3):  # the first frames of a large tree may walk the binary nodes
        got_p, got_s = ctx.trace_frame(bvh, cam, w, h, light, wt)
        _cmp_hits(got_p, want_p)
        _cmp_hits(got_s, want_s, any_hit=True)
        img = ctx.render_frame(bvh, cam, w, h, models=models, materials=mats, shade_flags=crt.SHADE_WIREFRAME, flags=wt)
        np.testing.assert_array_equal(img.view(np.uint32), want_i.view(np.uint32))
    bvh.free()
