"""Chain calls whose input is what a call before them writes, one to three calls
back, queued without a wait in between: stream order holds for them as for any
other work. Also from a batch that runs without a graph, through a captured
pair of calls, and between two contexts. Against the oracle, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import av1pf as A

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import gpu_util as G  # noqa: E402
import oracle as O  # noqa: E402

# multiples of 8: the filters read no sample beyond the visible area that the chain writes
SHAPES = {
    "one_tile": dict(width=64, height=64, bit_depth=8, sample_bytes=1),
    "small": dict(width=200, height=136, bit_depth=10),
    "small_grain": dict(width=200, height=136, bit_depth=10, enable_grain=1),
    "444_12bit": dict(width=328, height=208, bit_depth=12, subsampling_x=0, subsampling_y=0),
    "720p": dict(width=1280, height=720, bit_depth=8, sample_bytes=1),
    "1080p_wide": dict(width=2200, height=1080, bit_depth=10),
}


def buffers(sf, n):
    """n sets of planes in the input's geometry, the first frame in the first set."""
    first = O.HostPlanes.like_synth(sf)
    return [first] + [O.HostPlanes.zeros_like(first) for _ in range(n - 1)]


def oracle_step(sf, src, dst):
    f, fb = sf.f, np.zeros(A.frame_bytes(sf.f.info), np.uint8)
    assert O.lib().oracle_chain(C.byref(f.info), C.byref(f.params), C.byref(f.maps), src.c, dst.c, fb.ctypes.data, 0) == 0
    return fb


def gpu_step(ctx, d, src, dst, fb, stream=None):
    A.check(A.lib().av1pf_chain(ctx.p, C.byref(d.info), C.byref(d.params), C.byref(d.maps), src.c, dst.c, fb.data_ptr(),
                                stream), "av1pf_chain")


def walk(n, back, calls):
    """(source, target) of each call: the source was written `back` calls before, the first ones read set 0."""
    out = []
    for k in range(calls):
        out.append((1 + (k - back) % (n - 1) if k >= back else 0, 1 + k % (n - 1)))
    return out


@pytest.mark.parametrize("back", [1, 2, 3])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_input_written_calls_before(name, back):
    ctx, n, calls = G.Ctx(0), 6, 9
    sf = A.SynthHandle(seed=51, **SHAPES[name])
    d, host = G.DevFrame(sf), buffers(sf, n)
    steps = walk(n, back, calls)
    dev = [G.DevPlanes.from_host(sf.f.info, h) for h in host]
    other, spare = G.DevPlanes.from_host(sf.f.info, host[0]), G.DevPlanes.from_host(sf.f.info, host[1])
    fbs = [G.dev_bytes(A.frame_bytes(sf.f.info)) for _ in range(calls)]
    want = [oracle_step(sf, host[a], host[b]) for a, b in steps]
    for _ in range(4):
        for _ in range(5):  # unrelated calls, which overlap
            gpu_step(ctx, d, other, spare, fbs[0])
        for (a, b), fb in zip(steps, fbs):
            gpu_step(ctx, d, dev[a], dev[b], fb)
        torch.cuda.synchronize()
        for k, (fb, w) in enumerate(zip(fbs, want)):
            assert np.array_equal(fb[: w.size].cpu().numpy(), w), f"call {k}"
            fb.zero_()
    ctx.close()


@pytest.mark.parametrize("name", ["small", "small_grain", "1080p_wide"])
def test_input_written_by_a_batch_without_a_graph(name):
    ctx = G.Ctx(0)
    sf = A.SynthHandle(seed=52, **SHAPES[name])
    d, host = G.DevFrame(sf), buffers(sf, 3)
    dev = [G.DevPlanes.from_host(sf.f.info, h) for h in host]
    fb = [G.dev_bytes(A.frame_bytes(sf.f.info)) for _ in range(2)]
    want = [oracle_step(sf, host[0], host[1]), oracle_step(sf, host[1], host[2])]
    job = (A.Job * 1)()
    job[0].info, job[0].params, job[0].maps = C.pointer(d.info), C.pointer(d.params), C.pointer(d.maps)
    job[0].inp, job[0].ref_out = C.cast(dev[0].c, C.POINTER(A.Plane)), C.cast(dev[1].c, C.POINTER(A.Plane))
    job[0].frame_out = fb[0].data_ptr()
    b = C.c_void_p()
    A.check(A.lib().av1pf_batch_create(ctx.p, job, 1, 1, C.byref(b)), "batch_create")
    for _ in range(4):
        for _ in range(3):
            A.check(A.lib().av1pf_batch_run(b, None), "batch_run")
            gpu_step(ctx, d, dev[1], dev[2], fb[1])
        torch.cuda.synchronize()
        for k in range(2):
            assert np.array_equal(fb[k][: want[k].size].cpu().numpy(), want[k]), k
            fb[k].zero_()
    A.check(A.lib().av1pf_batch_destroy(b))
    ctx.close()


@pytest.mark.parametrize("name", ["small", "small_grain", "1080p_wide"])
def test_input_written_by_a_captured_call(name):
    ctx = G.Ctx(0)
    sf = A.SynthHandle(seed=53, **SHAPES[name])
    d, host = G.DevFrame(sf), buffers(sf, 3)
    dev = [G.DevPlanes.from_host(sf.f.info, h) for h in host]
    fb = [G.dev_bytes(A.frame_bytes(sf.f.info)) for _ in range(2)]
    want = [oracle_step(sf, host[0], host[1]), oracle_step(sf, host[1], host[2])]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s = torch.cuda.current_stream().cuda_stream
        gpu_step(ctx, d, dev[0], dev[1], fb[0], s)
        gpu_step(ctx, d, dev[1], dev[2], fb[1], s)
    for _ in range(4):
        g.replay()
        torch.cuda.synchronize()
        for k in range(2):
            assert np.array_equal(fb[k][: want[k].size].cpu().numpy(), want[k]), k
            fb[k].zero_()
    del g
    ctx.close()


@pytest.mark.parametrize("back", [1, 2])
@pytest.mark.parametrize("name", ["one_tile", "small", "small_grain", "1080p_wide"])
def test_input_written_by_another_context(name, back):
    """Two contexts in turn on one stream, each reading what was written one or two calls before."""
    ctxs, n, calls = [G.Ctx(0), G.Ctx(0)], 6, 9
    sf = A.SynthHandle(seed=54, **SHAPES[name])
    d, host = G.DevFrame(sf), buffers(sf, n)
    steps = walk(n, back, calls)
    dev = [G.DevPlanes.from_host(sf.f.info, h) for h in host]
    other, spare = G.DevPlanes.from_host(sf.f.info, host[0]), G.DevPlanes.from_host(sf.f.info, host[1])
    fbs = [G.dev_bytes(A.frame_bytes(sf.f.info)) for _ in range(calls)]
    want = [oracle_step(sf, host[a], host[b]) for a, b in steps]
    for _ in range(4):
        for k in range(8):
            gpu_step(ctxs[k % 2], d, other, spare, fbs[0])
        for k, ((a, b), fb) in enumerate(zip(steps, fbs)):
            gpu_step(ctxs[k % 2], d, dev[a], dev[b], fb)
        torch.cuda.synchronize()
        for k, (fb, w) in enumerate(zip(fbs, want)):
            assert np.array_equal(fb[: w.size].cpu().numpy(), w), f"call {k}"
            fb.zero_()
    for c in ctxs:
        c.close()
