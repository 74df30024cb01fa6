"""The PLOC iterations that one thread-block cluster runs in shared memory, at
the sizes where its split can go wrong: one segment exactly full and one past it
(64 positions), sixteen minimal segments (1,024), the largest number of clusters
that fits (16 segments of 2,048 positions less two halos of R) and one past it,
where the whole GPU runs the first iterations.  The tree is the oracle's, bit for
bit, and the per-iteration launches' (srcCommon/scene/geometry/bvh.cpp)."""
import numpy as np
import pytest

from oracle import oracle as O
from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _fits(radius):
    return 16 * (2048 - 2 * radius)


def _check(tris, radius):
    n = tris.shape[0]
    ref = O.build_bvh(tris, n, S.identity_models(1), radius=radius)
    want = ref["nodes"].view(np.uint32)
    for multi in (False, True):
        c = crt.Context(ploc_radius=radius, multi_launch_build=multi)
        got = c.build(tris, models=S.identity_models(1)).nodes().view(np.uint32)
        assert c.last_build_stats()["ploc_iterations"] == ref["iterations"]
        c.close()
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("radius", [16, 8, 32, 5])
@pytest.mark.parametrize("at", [64, 1024, "largest"])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_segment_edges(radius, at, off):
    n = (_fits(radius) if at == "largest" else at) + off
    _check(S.uniform_soup(n, seed=n + radius), radius)


@pytest.mark.parametrize("radius", [16, 32, 7])
def test_equal_boxes(radius):
    """Groups of equal triangles: ties of the surface area go to the lowest
    position, also where the candidates are split over threads."""
    one = S.uniform_soup(40, seed=5)
    _check(np.repeat(one, 37, axis=0), radius)


@pytest.mark.parametrize("n_scenes", [1, 6, 15, 30, 70, 200])
def test_batches_of_scenes(n_scenes):
    """A batch splits the SMs over its scenes' clusters (16 blocks a scene down to
    one), and its layout the grid over their nodes: every scene is the oracle's tree,
    for scenes around what each cluster size holds among tiny ones."""
    torch = pytest.importorskip("torch")
    edges = [b * 2016 + o for b in (1, 2, 4, 8, 16) for o in (0, 1, -1)] + [1, 2, 64, 65, 257]
    sizes = [edges[(7 * k) % len(edges)] if k < len(edges) else 1 + (37 * k) % 90 for k in range(n_scenes)]
    scenes = [S.uniform_soup(n, seed=3 * k + n) for k, n in enumerate(sizes)]
    ctx = crt.Context()
    batch = crt.Batch(ctx, sizes, [1] * n_scenes, models=S.identity_models(1))
    tris = torch.from_numpy(np.concatenate(scenes)).cuda()
    for _ in range(2):  # a second build starts from the first one's scratch
        batch.build(tris)
    for k, t in enumerate(scenes):
        ref = O.build_bvh(t, sizes[k], S.identity_models(1))
        np.testing.assert_array_equal(batch.nodes(k).view(np.uint32), ref["nodes"].view(np.uint32), err_msg=f"scene {k}")
        assert batch.scene_info(k)["iterations"] == ref["iterations"]
    batch.free()
    ctx.close()


@pytest.mark.parametrize("radius,n", [(16, 304 * 976), (16, 304 * 976 + 1), (8, 304 * 1000 + 1), (32, 304 * 928 + 1),
                                      (5, 304 * 1009 + 1), (16, 600_001)])
def test_more_tiles_than_blocks(radius, n):
    """Iterations of more tiles than the one-wave launch has blocks (two an SM) run
    opened and closed a tile apart: the largest size without one, one past it for each
    compiled radius and another, and several tiles a block."""
    _check(S.uniform_soup(n, seed=n + radius), radius)


def test_equal_boxes_over_many_tiles():
    """Equal boxes across tile and warp boundaries: the lowest position wins ties."""
    _check(np.repeat(S.uniform_soup(17_000, seed=8), 21, axis=0), 16)
