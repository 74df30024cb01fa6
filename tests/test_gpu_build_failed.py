"""Builds that cannot end — a vertex that is not finite, whose cluster no merge
takes — return an error, and none of their later kernels follows the records
that the earlier ones did not write, also where a larger build has left its own
there; the context and the batch stay usable.  Sizes: one cluster launch, two
positions more than it holds, and a scene of a batch."""
import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def broken(n, value):
    tris = S.uniform_soup(n, seed=n)
    tris[n // 2, 0] = value
    return tris


@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("n", [2, 50, 2000, 16 * 2016 + 2])
def test_build_that_cannot_end(n, value):
    models = S.identity_models(1)
    good = S.uniform_soup(60000, seed=1)
    c = crt.Context()
    bvh = c.build(good, models=models)
    want = bvh.nodes().view(np.uint32)
    with pytest.raises(crt.CrtError) as e:
        c.build(broken(n, value), models=models)
    assert "PLOC does not end" in str(e.value)
    np.testing.assert_array_equal(c.build(good, models=models).nodes().view(np.uint32), want)
    c.close()


def test_batch_with_a_scene_that_cannot_end():
    torch = pytest.importorskip("torch")
    n = 3000
    good = S.uniform_soup(n, seed=2)
    c = crt.Context()
    batch = crt.Batch(c, [n, n, n], [1] * 3, models=S.identity_models(1))

    def build(second):
        batch.build(torch.from_numpy(np.concatenate([good, second, good])).cuda())
    build(good)
    want = [batch.nodes(k).view(np.uint32) for k in range(3)]
    with pytest.raises(crt.CrtError, match="batch: device error word"):
        build(broken(n, np.inf))
    build(good)
    for k in range(3):
        np.testing.assert_array_equal(batch.nodes(k).view(np.uint32), want[k])
    batch.free()
    c.close()
