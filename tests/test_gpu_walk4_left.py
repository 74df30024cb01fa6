"""Rays and pixels that the walk over the compressed nodes leaves to the binary
walk: their list is reserved with the context or the batch, so a first call
allocates nothing however many rays there are to a triangle; more rays than the
list holds (65,536) are found by their marks, and a launch that leaves most of its
rays gives up and walks all on the binary nodes.  None, one, about as many as fit,
three quarters and all of the rays are left over, in
caller and sorted order, by traces, frames and batches; hits against one thread
per ray on the binary nodes, bit for bit."""
import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

from test_gpu_trace import _cmp_hits

pytestmark = pytest.mark.gpu

N_RAYS = 200003
LISTED = 65536


def far_rays(n, n_far, seed):
    """Sphere rays, n_far of them (spread out) from 30 scene sizes further back: beyond what the walk takes."""
    rays = S.sphere_rays(n, seed=seed)
    k = (np.arange(n_far, dtype=np.int64) * n) // max(n_far, 1)
    rays[k, 0:3] -= 30 * rays[k, 4:7]
    return rays


@pytest.mark.parametrize("flags", [crt.TRI_WATERTIGHT, crt.TRI_REFERENCE, crt.TRI_WATERTIGHT | crt.TRACE_ANY])
@pytest.mark.parametrize("n_far", [0, 1, LISTED - 1, LISTED, LISTED + 1, 150001, N_RAYS])
def test_any_number_left_over(ctx, n_far, flags):
    tris = S.uniform_soup(3000, seed=61)
    bvh = ctx.build(tris, models=S.identity_models(1))
    rays = far_rays(N_RAYS, n_far, seed=62)
    want = ctx.trace(bvh, rays, flags | crt.PER_RAY_THREADS)
    for order in (0, crt.SORT_RAYS, 0):
        _cmp_hits(ctx.trace(bvh, rays, flags | order), want, bool(flags & crt.TRACE_ANY))
    bvh.free()


@pytest.mark.parametrize("z", [-1.5, -12.0])
@pytest.mark.parametrize("w,h", [(100, 80), (640, 409), (1280, 720)])
def test_frames_from_near_and_far(ctx, w, h, z):
    models = S.identity_models(1)
    bvh = ctx.build(S.uniform_soup(3000, seed=63), models=models)
    cam = S.camera_gpu_data((0.5, 0.5, z), fov=45.0 if z > -2 else 6.0, aspect=w / h)
    light = np.array([2.0, 2.0, -2.0], np.float32)
    rays = ctx.raygen(cam, w, h)
    want_p = ctx.trace(bvh, rays, crt.TRI_WATERTIGHT | crt.PER_RAY_THREADS)
    want_s = ctx.trace(bvh, ctx.shadow_rays(rays, want_p, light), crt.TRI_WATERTIGHT | crt.TRACE_ANY | crt.PER_RAY_THREADS)
    for flags in (crt.TRI_WATERTIGHT, crt.TRI_WATERTIGHT | crt.TRACE_STATS, crt.TRI_WATERTIGHT):
        got_p, got_s = ctx.trace_frame(bvh, cam, w, h, light, flags)
        _cmp_hits(got_p, want_p)
        _cmp_hits(got_s, want_s, any_hit=True)
    bvh.free()


@pytest.mark.parametrize("flags", [crt.TRI_WATERTIGHT, crt.TRI_WATERTIGHT | crt.TRACE_ANY])
@pytest.mark.parametrize("n_far", [1, LISTED, LISTED + 1, 150001, N_RAYS])
def test_batches(ctx, n_far, flags):
    torch = pytest.importorskip("torch")
    tris = [S.uniform_soup(n, seed=n) for n in (700, 1, 3001)]
    rays = [far_rays(N_RAYS, n_far, seed=64), S.sphere_rays(10, seed=65), S.sphere_rays(5000, seed=66)]
    batch = crt.Batch(ctx, [len(t) for t in tris], [len(r) for r in rays], models=S.identity_models(1))
    d_tris, d_rays = (torch.from_numpy(np.concatenate(x)).cuda() for x in (tris, rays))
    hits = torch.empty((d_rays.shape[0], 4), dtype=torch.float32, device="cuda")
    for graph in (False, True, True):
        hits.zero_()
        batch.run(d_tris, d_rays, hits, flags, graph=graph)
        got, off = hits.cpu().numpy(), 0
        for t, r in zip(tris, rays):
            bvh = ctx.build(t, models=S.identity_models(1))
            want = ctx.trace(bvh, r, flags | crt.PER_RAY_THREADS)
            _cmp_hits(got[off:off + len(r)], want, bool(flags & crt.TRACE_ANY))
            off += len(r)
            bvh.free()
    batch.free()


@pytest.mark.parametrize("imported", [False, True])
def test_first_calls_allocate_nothing(imported):
    """More than 18 rays and pixels to a triangle, in a context that has built or imported its tree and no more."""
    torch = pytest.importorskip("torch")
    tris, models = S.uniform_soup(2000, seed=67), S.identity_models(1)
    w, h = 1280, 720
    cam = S.camera_gpu_data((0.5, 0.5, -1.5), aspect=w / h)
    rays = torch.from_numpy(S.sphere_rays(1000000, seed=68)).cuda()
    hits = torch.empty((1000000, 4), dtype=torch.float32, device="cuda")
    image = torch.empty((w * h, 4), dtype=torch.float32, device="cuda")
    warm = crt.Context()  # loads the kernels
    nodes = None
    for c in (warm, crt.Context()):
        bvh = c.bvh_from_nodes(nodes, tris, models=models) if imported and nodes is not None else c.build(tris, models=models)
        nodes = bvh.nodes()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        c.trace_frame(bvh, cam, w, h, None, crt.TRI_WATERTIGHT, hits_primary=image)
        c.trace(bvh, rays, crt.TRI_WATERTIGHT, out=hits)
        c.trace(bvh, rays, crt.TRI_WATERTIGHT | crt.TRACE_ANY, out=hits)
        after = torch.cuda.mem_get_info()[0]
        if c is not warm:
            assert after == before, f"{before - after} bytes"
        bvh.free()
    c.close()
    warm.close()
