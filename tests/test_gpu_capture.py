"""Chain calls captured into a graph: replays between direct calls on the same
context (other frames of the structure, other structures), on a context that
holds nothing yet, with the edge-list loop filter, under a memory cap, and what
the context holds once the graph is gone. Against the oracle, bit for bit."""
import ctypes as C
import gc

import numpy as np
import pytest

import av1pf as A

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import gpu_util as G  # noqa: E402
import oracle as O  # noqa: E402

SMALL = dict(width=200, height=136, bit_depth=10)
LARGE = dict(width=1920, height=1080, bit_depth=10)  # grain templates on the side stream


class Call:
    """A frame with outputs of its own and the oracle's result."""

    def __init__(self, seed, **kw):
        self.sf = A.SynthHandle(seed=seed, frame_index=seed, **kw)
        self.d = G.DevFrame(self.sf)
        self.ref, self.fb = G.DevPlanes.visible(self.d.info), G.dev_bytes(A.frame_bytes(self.d.info))
        self.want = O.chain(self.sf)

    def status(self, ctx, stream=None):
        d = self.d
        return A.lib().av1pf_chain(ctx.p, C.byref(d.info), C.byref(d.params), C.byref(d.maps), d.inp.c, self.ref.c,
                                   self.fb.data_ptr(), stream)

    def run(self, ctx, stream=None):
        A.check(self.status(ctx, stream), "av1pf_chain")

    def capture(self, ctx, mode="global"):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, capture_error_mode=mode):
            self.run(ctx, torch.cuda.current_stream().cuda_stream)
        return g

    def check(self):
        torch.cuda.synchronize()
        ref, fb = self.want
        assert np.array_equal(self.fb[: fb.size].cpu().numpy(), fb)
        for p in range(self.d.info.num_planes):
            assert np.array_equal(self.ref.host(p), ref.arrays[p]), f"plane {p}"
        self.fb.zero_()


def held(ctx):
    n = C.c_uint64()
    A.check(A.lib().av1pf_ctx_memory(ctx.p, C.byref(n)))
    return n.value


@pytest.mark.parametrize("warm", [False, True], ids=["cold", "warm"])
@pytest.mark.parametrize("mode", ["global", "relaxed"])
@pytest.mark.parametrize("shape", [dict(SMALL, enable_grain=1), dict(LARGE, enable_grain=1), dict(LARGE, superres_denom=11)],
                         ids=["small_grain", "1080p_grain", "1080p_superres"])
def test_replays_between_direct_calls(shape, mode, warm):
    ctx = G.Ctx(0)
    a, b, c = Call(3, **shape), Call(4, **shape), Call(5, width=2600, height=300, bit_depth=8, sample_bytes=1)
    if warm:
        for _ in range(2):
            b.run(ctx)
        a.run(ctx)
        a.check()
    g = a.capture(ctx, mode)
    for order in ("rb", "br", "rbr", "rbbbr", "crb", "rcr", "cccr", "brc"):
        for _ in range(4):
            for o in order:
                g.replay() if o == "r" else (b if o == "b" else c).run(ctx)
        for o in set(order):
            {"r": a, "b": b, "c": c}[o].check()
    del g
    ctx.close()


@pytest.mark.parametrize("lf_mode", [0, 1, 2])
def test_replays_with_edge_lists(lf_mode):
    ctx = G.Ctx(0)
    A.check(A.lib().av1pf_set_tuning(ctx.p, C.byref(A.Tuning(lf_mode, 64))))
    a, b = Call(11, **SMALL), Call(12, **SMALL)
    g = a.capture(ctx)
    for _ in range(3):
        g.replay()
        b.run(ctx)
        g.replay()
        a.check()
        b.check()
    del g
    ctx.close()


def test_capture_under_a_cap_shares_the_scratch():
    """No room for a second scratch: the captured call uses the context's, which
    then is neither moved nor freed while the graph lives."""
    a, b, big = Call(21, **SMALL), Call(22, **SMALL), Call(23, width=1300, height=700, bit_depth=10)
    probe = G.Ctx(0, 1 << 40)  # (a cap, for the layout that calls under one take)
    b.run(probe)
    b.run(probe)
    torch.cuda.synchronize()
    need = held(probe)
    probe.close()
    ctx = G.Ctx(0, need + (1 << 17))
    b.run(ctx)
    b.run(ctx)
    g = a.capture(ctx)
    for _ in range(3):
        g.replay()
        b.run(ctx)
        g.replay()
        a.check()
        b.check()
        assert big.status(ctx) == A.ERR_ADMISSION
        g.replay()
        a.check()
    del g
    ctx.close()


def test_graph_gives_its_memory_back():
    ctx = G.Ctx(0)
    a, b = Call(31, **SMALL), Call(32, **SMALL)
    for _ in range(2):
        b.run(ctx)
    before = held(ctx)
    for _ in range(3):
        g = a.capture(ctx)
        g.replay()
        a.check()
        assert held(ctx) > before
        del g
        gc.collect()
        torch.cuda.synchronize()
        b.run(ctx)
        b.check()
    assert held(ctx) == before
    ctx.close()
