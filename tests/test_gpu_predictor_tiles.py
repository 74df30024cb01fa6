"""Predictor gradients where the persistent training kernel's split can go wrong:
a single sample, a partial and one past a 128-sample tile, one tile on each of the 152
CTAs, one sample past that, and several tiles a CTA with a remainder."""
import numpy as np
import pytest

from oracle import predictor_oracle as PO
from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 129, 152 * 128, 152 * 128 + 1, 2 * 152 * 128 + 37])
def test_gradients_by_tile_count(n):
    """Both sides round to fp16 at the same points and sum in float32, in another
    order: a sum's relative error is a few times 2^-24 and an activation that lands on
    the other side of an fp16 rounding moves a term by 2^-11, rarely, so a block's
    relative error in the 2-norm stays well below 2e-3 at any n."""
    ctx = crt.Context()
    bvh = ctx.build(S.uniform_soup(2000, seed=3), models=S.identity_models(1))
    pred = crt.Predictor(ctx, bvh, seed=3)
    rays = S.sphere_rays(n, seed=n)
    targets = np.random.default_rng(n).integers(0, 128, n).astype(np.uint16)
    g, loss = pred.gradients(rays, targets)
    root = bvh.nodes()[0]
    g_ref, loss_ref, _ = PO.forward_backward(pred.params(), rays, targets, root[0:3], root[4:7])
    assert abs(loss - loss_ref) <= 1e-3 * abs(loss_ref)
    for name, a, b in PO.BLOCKS:
        da, db = g[a:b].astype(np.float64), g_ref[a:b].astype(np.float64)
        rel = np.linalg.norm(da - db) / max(np.linalg.norm(db), 1e-30)
        assert rel < 2e-3, f"gradient block {name}: relative error {rel:.3e}"
    pred.free()
    bvh.free()
    ctx.close()
