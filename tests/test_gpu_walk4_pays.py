"""Large traces on both sides of the size at which deriving the compressed nodes
pays (closest hits: 64 triangles a ray, any hits: 16): just above it the first
trace walks the binary nodes and a later one the compressed ones, just below
both walk those, and a change of the tree starts over; one scene and a batch,
against one thread per ray on the binary nodes bit for bit."""
import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

pytestmark = pytest.mark.gpu

N_RAYS = 65536


def same(got, want, any_hit):
    g, w = got.cpu().numpy().view(np.uint32), want.cpu().numpy().view(np.uint32)
    if any_hit:
        g, w = g[:, 0] == crt.MISS, w[:, 0] == crt.MISS
    np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("flags,n", [(crt.TRI_WATERTIGHT, 64 * N_RAYS), (crt.TRI_WATERTIGHT, 64 * N_RAYS + 1),
                                     (crt.TRI_WATERTIGHT | crt.TRACE_ANY, 16 * N_RAYS),
                                     (crt.TRI_WATERTIGHT | crt.TRACE_ANY, 16 * N_RAYS + 1)])
def test_first_and_later_traces(ctx, flags, n):
    torch = pytest.importorskip("torch")
    gen = torch.Generator(device="cuda").manual_seed(81)
    tris, rays = S.device_soup(n, gen), S.device_sphere_rays(N_RAYS, gen)
    bvh = ctx.build(tris, models=S.identity_models(1))
    want, got = (torch.empty((N_RAYS, 4), dtype=torch.float32, device="cuda") for _ in range(2))
    for change in (None, lambda: bvh.refit(tris, models=S.identity_models(1)),
                   lambda: bvh.rebuild(tris, models=S.identity_models(1))):
        if change:
            change()
        ctx.trace(bvh, rays, flags | crt.PER_RAY_THREADS, out=want)
        for order in (0, 0, crt.SORT_RAYS):
            got.zero_()
            ctx.trace(bvh, rays, flags | order, out=got)
            same(got, want, bool(flags & crt.TRACE_ANY))
    bvh.free()


@pytest.mark.parametrize("flags,n", [(crt.TRI_WATERTIGHT, 64 * N_RAYS + 2), (crt.TRI_WATERTIGHT | crt.TRACE_ANY, 16 * N_RAYS + 2),
                                     (crt.TRI_WATERTIGHT | crt.TRACE_ANY, 16 * N_RAYS)])
def test_batches(ctx, flags, n):
    torch = pytest.importorskip("torch")
    gen = torch.Generator(device="cuda").manual_seed(82)
    tris = [S.device_soup(k, gen) for k in (n // 2 + 7, n - n // 2 - 7)]
    rays = [S.device_sphere_rays(N_RAYS // 2, gen) for _ in range(2)]
    want = torch.empty((N_RAYS, 4), dtype=torch.float32, device="cuda")
    for k in range(2):
        bvh = ctx.build(tris[k], models=S.identity_models(1))
        ctx.trace(bvh, rays[k], flags | crt.PER_RAY_THREADS, out=want[k * (N_RAYS // 2):(k + 1) * (N_RAYS // 2)])
        bvh.free()
    batch = crt.Batch(ctx, [len(t) for t in tris], [N_RAYS // 2] * 2, models=S.identity_models(1))
    all_tris, all_rays, got = torch.cat(tris), torch.cat(rays), torch.empty_like(want)
    for graph in (False, True, True):
        got.zero_()
        batch.run(all_tris, all_rays, got, flags, graph=graph)
        same(got, want, bool(flags & crt.TRACE_ANY))
        for _ in range(2):
            got.zero_()
            batch.trace(all_rays, got, flags)
            same(got, want, bool(flags & crt.TRACE_ANY))
    batch.free()
