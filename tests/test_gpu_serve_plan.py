"""Served batches that keep the work lists of the batch before them: groups of
the same structure with other frames and parameters, and groups whose structure
changes in between (a filter off, film grain, another stream set, a batch that
outgrows the buffers), on one batch stream. Against the oracle, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import av1pf as A
import oracle as O
from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

if cuda_available():
    import gpu_util as G

L = A.lib
STREAMS = [dict(width=200, height=120, bit_depth=8, sample_bytes=1),
           dict(width=136, height=72, bit_depth=10, enable_grain=1),
           dict(width=256, height=144, bit_depth=12, subsampling_x=0, subsampling_y=0, superres_denom=12)]
# (streams of the group, what is changed in its parameters), in turn
GROUPS = [((0, 1), None), ((0, 1), None), ((0, 1), "no_luma_lf"), ((0, 1), None), ((0, 1), "no_cdef"),
          ((0, 1), "no_grain"), ((0, 1), None), ((0, 1, 2), None), ((0, 1, 2), None), ((2,), None), ((2, 2), None),
          ((0, 1), None), ((0, 1), None)]


def change(p, what):
    if what == "no_luma_lf":
        p.loop_filter_level[0] = p.loop_filter_level[1] = 0
    elif what == "no_cdef":
        p.cdef_enabled = 0
    elif what == "no_grain":
        p.film_grain.apply = 0


@pytest.mark.parametrize("device", [False, True])
def test_groups_in_turn(device):
    ctx = G.Ctx()
    cfg = A.ServeConfig(40 << 30, 32, 1, 100, 4)
    srv = C.c_void_p()
    A.check(L().av1pf_serve_open(ctx.p, C.byref(cfg), C.byref(srv)), "serve_open")
    sids = []
    for st in STREAMS:
        s, sf = C.c_int32(), A.SynthHandle(**st, seed=1)
        A.check(L().av1pf_serve_open_stream(srv, C.byref(sf.f.info), C.byref(s)))
        sids.append(s.value)
    for g, (streams, what) in enumerate(GROUPS):
        n, keep = len(streams), []
        reqs, tickets = (A.Request * n)(), (C.c_uint64 * n)()
        for r, k in zip(reqs, streams):
            sf = A.SynthHandle(**STREAMS[k], seed=500 + 16 * g + len(keep), frame_index=g)
            change(sf.f.params, what)
            src = G.DevFrame(sf) if device else None
            inp = src.inp if device else O.HostPlanes.like_synth(sf)
            out = G.dev_bytes(A.frame_bytes(sf.f.info)) if device else np.zeros(A.frame_bytes(sf.f.info), np.uint8)
            r.info, r.params = C.pointer(sf.f.info), C.pointer(sf.f.params)
            r.maps = C.pointer(src.maps if device else sf.f.maps)
            r.inp = C.cast(inp.c, C.POINTER(A.Plane))
            r.device = int(device)
            if device:
                r.frame_out = out.data_ptr()
            keep.append((sf, src, inp, out))
        ids = (C.c_int32 * n)(*[sids[k] for k in streams])
        A.check(L().av1pf_serve_submit_many(srv, n, ids, reqs, tickets), "submit_many")
        for t, (sf, _, _, out) in zip(tickets, keep):
            A.check(L().av1pf_serve_poll(srv, t, 20000, None if device else out.ctypes.data, None), "poll")
            got = out[:A.frame_bytes(sf.f.info)].cpu().numpy() if device else out
            assert np.array_equal(got, O.chain(sf, threads=0)[1]), (g, streams, what)
    A.check(L().av1pf_serve_close(srv))
    ctx.close()
