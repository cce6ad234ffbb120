"""Served frames while the host program captures a graph in CUDA's default
(global) mode: the worker's queries neither fail nor end the capture."""
import ctypes as C

import numpy as np
import pytest

import av1pf as A
import oracle as O
from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

if cuda_available():
    import gpu_util as G
    import torch

L = A.lib


def test_serving_during_a_global_capture():
    ctx, sf = G.Ctx(), A.SynthHandle(width=320, height=180, bit_depth=10, enable_grain=1, seed=8)
    _, want = O.chain(sf)
    srv, sid, t = C.c_void_p(), C.c_int32(), C.c_uint64()
    A.check(L().av1pf_serve_open(ctx.p, C.byref(A.ServeConfig(1 << 30, 4, 2, 100)), C.byref(srv)), "serve_open")
    A.check(L().av1pf_serve_open_stream(srv, C.byref(sf.f.info), C.byref(sid)))
    inp = O.HostPlanes.like_synth(sf)
    rq = A.Request()
    rq.info, rq.params, rq.maps = C.pointer(sf.f.info), C.pointer(sf.f.params), C.pointer(sf.f.maps)
    rq.inp = C.cast(inp.c, C.POINTER(A.Plane))
    out = np.zeros(A.frame_bytes(sf.f.info), np.uint8)

    def serve():
        out[:] = 0
        A.check(L().av1pf_serve_submit(srv, sid.value, C.byref(rq), C.byref(t)), "submit")
        A.check(L().av1pf_serve_poll(srv, t, 5000, out.ctypes.data, None), "poll")
        assert np.array_equal(out, want)

    for _ in range(4):  # the stream's staging and both batches' buffers exist
        serve()
    x = torch.zeros(1024, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global"):
        x += 1
        for _ in range(8):
            serve()
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 2048
    serve()
    A.check(L().av1pf_serve_close(srv))
    ctx.close()
