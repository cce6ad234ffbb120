"""Consecutive chain calls on one context, whose descriptors travel with the
launches: shapes taken in turn (work lists resident and replaced), frames of
one shape whose parameters differ, one output buffer for all of them, and a
captured call replayed."""
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

PLAIN = dict(width=200, height=136, bit_depth=8, sample_bytes=1)
SEQUENCES = {
    "one_shape": [PLAIN] * 6,
    "grain": [dict(PLAIN, enable_grain=1)] * 5,
    "two_shapes": [PLAIN, dict(width=330, height=210, bit_depth=10)] * 3,
    "replaced": [PLAIN, PLAIN, dict(width=330, height=210, bit_depth=10), dict(PLAIN, enable_grain=1),
                 dict(PLAIN, superres_denom=11), PLAIN, dict(PLAIN, bit_depth=12, sample_bytes=2), PLAIN, PLAIN],
    "wide": [dict(width=2200, height=80, bit_depth=10)] * 5,
}


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


def call(ctx, d, ref, fb, stream=None):
    A.check(A.lib().av1pf_chain(ctx.p, C.byref(d.info), C.byref(d.params), C.byref(d.maps), d.inp.c, ref.c,
                                fb.data_ptr(), stream), "av1pf_chain")


@pytest.mark.parametrize("name", sorted(SEQUENCES))
def test_calls_in_a_row(ctx, name):
    sfs = [A.SynthHandle(**c, seed=300 + i, frame_index=i + 1) for i, c in enumerate(SEQUENCES[name])]
    dfs = [G.DevFrame(s) for s in sfs]
    outs = [(G.DevPlanes.visible(d.info), G.dev_bytes(A.frame_bytes(d.info))) for d in dfs]
    for _ in range(3):
        for d, (ref, fb) in zip(dfs, outs):
            call(ctx, d, ref, fb)
    torch.cuda.synchronize()
    for i, (sf, (ref, fb)) in enumerate(zip(sfs, outs)):
        ref_cpu, fb_cpu = O.chain(sf)
        assert np.array_equal(fb[: A.frame_bytes(sf.f.info)].cpu().numpy(), fb_cpu), f"frame {i}"
        for p in range(sf.f.info.num_planes):
            assert np.array_equal(ref.host(p), ref_cpu.arrays[p]), f"frame {i} plane {p}"


@pytest.mark.parametrize("size", [(200, 136), (1280, 720)])
def test_shared_output_holds_the_last_frame(ctx, size):
    """Calls queued back to back into one output buffer: what remains is the last call's frame."""
    sfs = [A.SynthHandle(width=size[0], height=size[1], bit_depth=10, seed=400 + i) for i in range(3)]
    dfs = [G.DevFrame(s) for s in sfs]
    ref, fb = G.DevPlanes.visible(dfs[0].info), G.dev_bytes(A.frame_bytes(dfs[0].info))
    wants = [O.chain(s)[1] for s in sfs]
    for n in range(3, 15):
        for i in range(n):
            call(ctx, dfs[i % 3], ref, fb)
        torch.cuda.synchronize()
        assert np.array_equal(fb[: A.frame_bytes(dfs[0].info)].cpu().numpy(), wants[(n - 1) % 3]), f"after {n} calls"


def test_captured_call_replays(ctx):
    sf = A.SynthHandle(**PLAIN, seed=77)
    d = G.DevFrame(sf)
    ref, fb = G.DevPlanes.visible(d.info), G.dev_bytes(A.frame_bytes(d.info))
    for _ in range(2):  # both descriptor buffers hold the work lists
        call(ctx, d, ref, fb)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        call(ctx, d, ref, fb, torch.cuda.current_stream().cuda_stream)
    _, want = O.chain(sf)
    for _ in range(3):
        fb.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(fb[: A.frame_bytes(d.info)].cpu().numpy(), want)
