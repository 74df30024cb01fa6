"""Any-hit rays whose tmax puts the pruning bound on a farther child's entry
distance: the persistent walk over the compressed nodes (traces of at least
65,536 rays, frames' shadow rays) must still visit the nearer children, which
hold the occluder.  Consecutive float values of tmax sweep the bound across the
entry distance, so that some ray meets every relation the two can have.  Every
ray has a hit well before its tmax, so no tolerance is involved."""
import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

pytestmark = pytest.mark.gpu

N_RAYS = 1 << 20  # tmax 2.0 .. 2.25, one float after the other


def occluders_and_far(far_x):
    """Three triangles across the x axis near x = 1 and one behind far_x: the four children of the root record."""
    def across(x, tilt):
        return [[x, -1.0, -1.0], [x, -1.0, 3.0], [x + tilt, 3.0, -1.0]]
    v = np.array([across(1.0, 0.0), across(1.02, 0.01), across(1.04, 0.02), across(far_x, 0.2)], np.float32)
    return S.pack_triangles(v[:, 0], v[:, 1], v[:, 2])


def sweep(n=N_RAYS):
    rays = np.zeros((n, 8), np.float32)
    rays[:, 1:3] = 0.125
    rays[:, 4] = 1.0
    rays[:, 7] = (np.float32(2.0).view(np.uint32) + np.arange(n, dtype=np.uint32)).view(np.float32)
    return rays


@pytest.mark.parametrize("predicate", [crt.TRI_WATERTIGHT, crt.TRI_REFERENCE])
@pytest.mark.parametrize("far_x", [2.04, 2.0625, 2.09, 2.1, 2.125, 2.15, 2.17, 2.2])
def test_occluder_before_a_child_at_the_bound(ctx, far_x, predicate):
    bvh = ctx.build(occluders_and_far(far_x), models=S.identity_models(1))
    rays = sweep()
    for flags in (predicate | crt.TRACE_ANY, predicate | crt.TRACE_ANY | crt.PER_RAY_THREADS):
        missed = ctx.trace(bvh, rays, flags)[:, 0].view(np.uint32) == crt.MISS
        assert not missed.any(), f"{flags:#x}: {int(missed.sum())} of {N_RAYS} rays, tmax {rays[missed][:4, 7]}"
    bvh.free()


def test_batches_too(ctx):
    torch = pytest.importorskip("torch")
    tris = [occluders_and_far(x) for x in (2.06, 2.11, 2.16)]
    rays = sweep()
    batch = crt.Batch(ctx, [len(t) for t in tris], [N_RAYS] * 3, models=S.identity_models(1))
    d_tris = torch.from_numpy(np.concatenate(tris)).cuda()
    d_rays = torch.from_numpy(np.concatenate([rays] * 3)).cuda()
    hits = torch.empty((3 * N_RAYS, 4), dtype=torch.float32, device="cuda")
    batch.run(d_tris, d_rays, hits, crt.TRI_WATERTIGHT | crt.TRACE_ANY)
    assert int((hits.view(torch.int32)[:, 0] == -1).sum()) == 0
    batch.free()
