"""The encoder's loop-filter level search where its kernel can go wrong: frames
smaller than a tile, one sample past one and cropped inside a 4x4, every chroma
layout and sample width, per-block and per-segment levels, scales that filter
nothing, and errors at the largest a sample can have. Against the oracle, bit
for bit."""
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

SHAPES = {
    "one_block_8bit": dict(width=8, height=8, bit_depth=8, sample_bytes=1),
    "past_a_tile_8bit": dict(width=65, height=65, bit_depth=8, sample_bytes=1),
    "cropped_10bit_deltas": dict(width=197, height=163, bit_depth=10, segmentation=1, delta_lf=2),
    "422_12bit_deltas": dict(width=140, height=70, bit_depth=12, subsampling_x=1, subsampling_y=0, delta_lf=1),
    "444_8bit_u16": dict(width=131, height=99, bit_depth=8, sample_bytes=2, subsampling_x=0, subsampling_y=0),
    "mono_10bit": dict(width=128, height=128, bit_depth=10, mono=1, segmentation=1),
}
# the frame's levels: ordinary, the largest, one pass and one chroma plane only, scales that round to 0
LEVELS = [(30, 22, 17, 9), (63, 63, 63, 63), (0, 12, 0, 5), (1, 0, 1, 0), (0, 0, 8, 8)]


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


def search(ctx, frames):
    """av1pf_lf_search_many on [(sf, params, cur, src)]: per frame (levels, errors)."""
    jobs, keep, out = (A.LfSearchJob * len(frames))(), [], []
    for j, (sf, params, cur, src) in zip(jobs, frames):
        info = sf.f.info
        df, dc, dsr = G.DevFrame(sf), G.DevPlanes.from_host(info, cur), G.DevPlanes.from_host(info, src)
        sse = np.zeros((6, 3), np.uint64)
        j.info, j.params, j.maps = C.pointer(info), C.pointer(params), C.pointer(df.maps)
        j.cur, j.src = C.cast(dc.c, C.POINTER(A.Plane)), C.cast(dsr.c, C.POINTER(A.Plane))
        j.sse_out = sse.ctypes.data
        keep.append((df, dc, dsr))
        out.append(sse)
    A.check(A.lib().av1pf_lf_search_many(ctx.p, len(frames), jobs, None), "lf_search_many")
    return [(list(j.levels_out), s) for j, s in zip(jobs, out)]


def with_levels(sf, levels, sharpness):
    p = A.Params.from_buffer_copy(sf.f.params)
    for k, v in enumerate(levels):
        p.loop_filter_level[k] = v
    p.loop_filter_sharpness = sharpness
    return p


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_levels_and_errors(ctx, name):
    sf = A.SynthHandle(**SHAPES[name], seed=61, frame_index=1)
    cur, src = O.search_inputs(sf, 62)
    for i, levels in enumerate(LEVELS):
        p = with_levels(sf, levels, (0, 3, 7)[i % 3])
        want = O.lf_search(sf, cur, src, params=p)
        (lv, sse), = search(ctx, [(sf, p, cur, src)])
        assert np.array_equal(sse, want[1]), levels
        assert lv == list(want[0]), levels


def test_batch_of_all_shapes(ctx):
    frames = []
    for i, name in enumerate(sorted(SHAPES)):
        sf = A.SynthHandle(**SHAPES[name], seed=63 + i, frame_index=2)
        frames.append((sf, with_levels(sf, LEVELS[i % len(LEVELS)], 0), *O.search_inputs(sf, 64)))
    for (lv, sse), (sf, p, cur, src) in zip(search(ctx, frames), frames):
        want = O.lf_search(sf, cur, src, params=p)
        assert np.array_equal(sse, want[1]) and lv == list(want[0])


def test_largest_errors(ctx):
    """12-bit, the reconstruction at the maximum and the source at 0: every square is 4095^2."""
    sf = A.SynthHandle(width=128, height=96, bit_depth=12, seed=71, frame_index=1)
    cur, src = (O.HostPlanes([np.full_like(a, v) for a in O.HostPlanes.like_synth(sf).arrays]) for v in (4095, 0))
    p = with_levels(sf, (40, 40, 40, 40), 0)
    want = O.lf_search(sf, cur, src, params=p)
    (lv, sse), = search(ctx, [(sf, p, cur, src)])
    assert np.array_equal(sse, want[1]) and lv == list(want[0])
    assert int(sse[0, 0]) == 128 * 96 * 4095**2
