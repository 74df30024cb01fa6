"""Batches in which some scenes cannot be quantised (too large or too small a
range for the compressed nodes) beside ordinary ones: only those scenes' rays go
to the binary walk, and every scene's hits are those of the scene alone, one
thread per ray on the binary nodes, bit for bit — traced after a build, by a
captured graph, and again once every scene is ordinary."""
import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

from test_gpu_trace import _cmp_hits
from test_gpu_walk4 import mixed_rays, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [crt.TRI_WATERTIGHT, crt.TRI_REFERENCE, crt.TRI_WATERTIGHT | crt.TRACE_ANY])
@pytest.mark.parametrize("bad", [(0,), (1, 3), (4,), (0, 1, 2, 3, 4)])
def test_unquantised_scenes_beside_ordinary_ones(ctx, bad, flags):
    torch = pytest.importorskip("torch")
    models = S.identity_models(1)
    ordinary = [S.uniform_soup(n, seed=n, edge_lo=0.02, edge_hi=0.1) for n in (900, 3000, 2, 1025, 5000)]
    odd = [scene("huge") if k % 2 else scene("tiny") for k in range(5)]
    odd = [o[:len(t)] if len(o) >= len(t) else np.resize(o, t.shape) for o, t in zip(odd, ordinary)]

    def run(batch, tris, graph):
        rays = [mixed_rays(t, seed=k, n=16000 + 7 * k) for k, t in enumerate(tris)]
        d_tris, d_rays = (torch.from_numpy(np.concatenate(x)).cuda() for x in (tris, rays))
        hits = torch.empty((d_rays.shape[0], 4), dtype=torch.float32, device="cuda")
        if graph:
            for _ in range(2):
                hits.zero_()
                batch.run(d_tris, d_rays, hits, flags, graph=True)
        else:
            batch.build(d_tris)
            batch.trace(d_rays, hits, flags)
        got, off = hits.cpu().numpy(), 0
        for t, r in zip(tris, rays):
            bvh = ctx.build(t, models=models)
            _cmp_hits(got[off:off + len(r)], ctx.trace(bvh, r, flags | crt.PER_RAY_THREADS), bool(flags & crt.TRACE_ANY))
            off += len(r)
            bvh.free()

    batch = crt.Batch(ctx, [len(t) for t in ordinary], [16000 + 7 * k for k in range(5)], models=models)
    mixed = [odd[k] if k in bad else ordinary[k] for k in range(5)]
    run(batch, mixed, graph=False)
    run(batch, mixed, graph=True)
    run(batch, ordinary, graph=False)
    batch.free()
