"""One tree traced from two contexts at once, a host thread and a stream each.
The first large trace, frame or 4-wide trace of a fresh tree derives the nodes
it walks; the other context must not read them before they are there.  Hits
against one thread per ray on the binary nodes, which every build writes, bit
for bit; the node array read by both after a refit likewise."""
import threading

import numpy as np
import pytest

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

pytestmark = pytest.mark.gpu

N_RAYS = 65536 + 11


def at_once(*calls):
    """Runs the calls on a thread each, started together; their results."""
    out, gate = [None] * len(calls), threading.Barrier(len(calls))

    def run(k):
        gate.wait()
        try:
            out[k] = calls[k]()
        except Exception as e:  # handed to the test's thread
            out[k] = e
    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for o in out:
        if isinstance(o, Exception):
            raise o
    return out


def test_two_contexts_trace_a_fresh_tree(ctx):
    models = S.identity_models(1)
    tris = S.uniform_soup(200000, seed=41)
    rays = S.sphere_rays(N_RAYS, seed=42)
    cam = S.camera_gpu_data((0.5, 0.5, -1.5))
    other = crt.Context()
    bvh = ctx.build(tris, models=models)
    want = ctx.trace(bvh, rays, crt.TRI_WATERTIGHT | crt.PER_RAY_THREADS).view(np.uint32)
    want_frame = ctx.trace(bvh, ctx.raygen(cam, 320, 240), crt.TRI_WATERTIGHT | crt.PER_RAY_THREADS).view(np.uint32)
    nodes = bvh.nodes().view(np.uint32)
    for k in range(12):
        if k % 3 == 2:
            bvh.refit(tris, models=models)
            for got in at_once(lambda: ctx_nodes(ctx, bvh), lambda: ctx_nodes(other, bvh)):
                np.testing.assert_array_equal(got, nodes)
        else:
            bvh.rebuild(tris, models=models)
        flags = crt.TRI_WATERTIGHT | (crt.TRACE_WIDE if k % 2 else 0)
        for got in at_once(lambda: ctx.trace(bvh, rays, flags), lambda: other.trace(bvh, rays, flags)):
            np.testing.assert_array_equal(got.view(np.uint32), want)
        bvh.rebuild(tris, models=models)
        for got, _ in at_once(lambda: ctx.trace_frame(bvh, cam, 320, 240, None, crt.TRI_WATERTIGHT),
                              lambda: other.trace_frame(bvh, cam, 320, 240, None, crt.TRI_WATERTIGHT)):
            np.testing.assert_array_equal(got.view(np.uint32), want_frame)
    bvh.free()
    other.close()


def ctx_nodes(c, bvh):
    out = np.empty((bvh.n_nodes, 12), np.float32)
    crt._check(crt.lib().crt_bvh_copy_nodes(c.handle, bvh.handle, crt._ptr(out)))
    return out.view(np.uint32)
