"""Plain frames recorded by stream capture amid the caller's own work: after a memset on the stream, joined with
another stream, and with a fork behind them.  The library's kernels are dependent launches, whose edges the capture
has to take in each of these places; the recorded frame gives what the same frame launched directly gives, bit for
bit, also as a child of another graph."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
V = C.c_void_p


def runtime():
    import os
    from tressfx_gb300 import build as B
    return C.CDLL(os.path.join(str(B._cuda_home()), "lib64", "libcudart.so"))


@pytest.mark.parametrize("work", ["none", "before", "joined", "behind"])
def test_recorded_frame_equals_direct(ctx, work):
    from tressfx_gb300 import _capi as A
    from tressfx_gb300.headless import FrameInputs, PlainPipeline
    from tressfx_gb300.synthetic import scene_head
    rt = runtime()

    def ok(e):
        assert e == 0, e

    A.lib().tfx_context_stream.restype, A.lib().tfx_context_stream.argtypes = V, [V]
    s = V(A.lib().tfx_context_stream(ctx.handle))
    sc = scene_head(seed=7, num_guides=96, n=16, follows=1, triangles=4500, sdf_cells=32, frames=2)
    recorded, direct = PlainPipeline(ctx, sc), PlainPipeline(ctx, sc)
    direct.step(0)
    direct.step(1)
    buf, other, ev0, ev1, g, x, top, node = (V() for _ in range(8))
    ok(rt.cudaMalloc(C.byref(buf), C.c_size_t(1 << 20)))
    ok(rt.cudaStreamCreateWithFlags(C.byref(other), 1))
    for ev in (ev0, ev1):
        ok(rt.cudaEventCreateWithFlags(C.byref(ev), 2))

    def aside():   # a memset on another stream, from here on
        ok(rt.cudaEventRecord(ev0, s))
        ok(rt.cudaStreamWaitEvent(other, ev0, 0))
        ok(rt.cudaMemsetAsync(buf, 0, C.c_size_t(1 << 20), other))
        ok(rt.cudaEventRecord(ev1, other))

    recorded.step(0)   # a first frame as every later one, so that nothing is allocated in the capture
    fin = FrameInputs(sc, 1)
    recorded.prepare(fin)
    ctx.synchronize()
    ok(rt.cudaStreamBeginCapture(s, 2))
    if work == "before":
        ok(rt.cudaMemsetAsync(buf, 0, C.c_size_t(1 << 20), s))
    if work == "joined":
        aside()
        recorded.meshes[0].skin(fin.mesh_bones[0])
        ok(rt.cudaStreamWaitEvent(s, ev1, 0))
    recorded.run(fin)
    if work == "behind":
        aside()
        ok(rt.cudaStreamWaitEvent(s, ev1, 0))
    ok(rt.cudaStreamEndCapture(s, C.byref(g)))
    ok(rt.cudaGraphCreate(C.byref(top), 0))
    ok(rt.cudaGraphAddChildGraphNode(C.byref(node), top, None, C.c_size_t(0), g))
    ok(rt.cudaGraphInstantiate(C.byref(x), top, C.c_ulonglong(0)))
    ok(rt.cudaGraphLaunch(x, s))
    ctx.synchronize()
    for b in (A.BUF_POSITIONS, A.BUF_POSITIONS_PREV, A.BUF_TANGENTS):
        got, want = recorded.hair[0].read(b), direct.hair[0].read(b)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (work, b)
    ok(rt.cudaGraphExecDestroy(x))
    ok(rt.cudaGraphDestroy(top))
    ok(rt.cudaGraphDestroy(g))
    for ev in (ev0, ev1):
        ok(rt.cudaEventDestroy(ev))
    ok(rt.cudaStreamDestroy(other))
    ok(rt.cudaFree(buf))
    recorded.close()
    direct.close()
