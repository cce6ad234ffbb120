"""The encoder's CDEF search where its packed kernel and its one-kernel greedy
can go wrong: errors at the largest a block can hold (sums past 32 bits), frames
cropped inside a block, blocks cut in half by the frame's edge, every chroma
layout, a batch of 8-, 10- and 12-bit frames, and a table too large for the
greedy's shared memory. Against the oracle, bit for bit."""
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
    "half_block_8bit": dict(width=70, height=90, bit_depth=8, sample_bytes=1),
    "cropped_10bit": dict(width=197, height=163, bit_depth=10),
    "422_10bit": dict(width=140, height=70, bit_depth=10, subsampling_x=1, subsampling_y=0),
    "444_8bit_u16": dict(width=131, height=99, bit_depth=8, sample_bytes=2, subsampling_x=0, subsampling_y=0),
    "mono_10bit": dict(width=130, height=130, bit_depth=10, mono=1),
}


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


def search(ctx, frames, q, lam, thorough):
    """av1pf_cdef_search_many on [(sf, cur, src)]: per frame (result, table, block errors)."""
    jobs, keep, out = (A.CdefSearchJob * len(frames))(), [], []
    for j, (sf, cur, src) in zip(jobs, frames):
        info = sf.f.info
        rows, cols = (info.mi_rows + 15) // 16, (info.mi_cols + 15) // 16
        df, dc, dsr = G.DevFrame(sf), G.DevPlanes.from_host(info, cur), G.DevPlanes.from_host(info, src)
        res, table = A.CdefSearchResult(), np.zeros(rows * df.maps.cdef_stride, np.int8)
        sse = np.zeros((rows * cols, sum(A.CDEF_SEARCH_N[thorough])), np.uint64)
        j.info, j.maps = C.pointer(info), C.pointer(df.maps)
        j.cur, j.src = C.cast(dc.c, C.POINTER(A.Plane)), C.cast(dsr.c, C.POINTER(A.Plane))
        j.base_q_idx, j.lam, j.result = q, lam, C.pointer(res)
        j.cdef_idx_out, j.block_sse = table.ctypes.data, sse.ctypes.data
        keep.append((df, dc, dsr))
        out.append((res, table, sse))
    A.check(A.lib().av1pf_cdef_search_many(ctx.p, len(frames), jobs, int(thorough), None), "cdef_search_many")
    return out


def check(got, frames, q, lam, thorough):
    for i, ((rg, tg, sg), (sf, cur, src)) in enumerate(zip(got, frames)):
        ro, to, so = O.cdef_search(sf, cur, src, q, lam, thorough)
        assert np.array_equal(sg, so), f"frame {i}: block errors differ at {np.argwhere(sg != so)[:5]}"
        assert (rg.damping_minus_3, rg.bits, rg.pairs()) == (ro.damping_minus_3, ro.bits, ro.pairs()), f"frame {i}"
        assert np.array_equal(tg, to), f"frame {i}"


@pytest.mark.parametrize("thorough", [False, True], ids=["fast", "thorough"])
@pytest.mark.parametrize("content", ["noise", "extremes"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_search_matches_oracle(ctx, name, content, thorough):
    sf = A.SynthHandle(**SHAPES[name], seed=17, skip_pct=10)
    cur, src = O.search_inputs(sf, 5, amp=20)
    if content == "extremes":
        rng, top = np.random.default_rng(3), (1 << sf.f.info.bit_depth) - 1
        for a, b in zip(cur.arrays, src.arrays):
            a[...] = rng.choice(np.array([0, 1, top], a.dtype), size=a.shape)
            b[...] = top - a
    frames = [(sf, cur, src)]
    check(search(ctx, frames, 140, 30.0, thorough), frames, 140, 30.0, thorough)


def test_batch_of_all_depths(ctx):
    frames = []
    for i, c in enumerate([dict(bit_depth=8, sample_bytes=1), dict(bit_depth=12), dict(bit_depth=10, width=333)]):
        sf = A.SynthHandle(**dict(dict(width=200, height=136), **c), seed=70 + i)
        frames.append((sf, *O.search_inputs(sf, 80 + i, amp=24)))
    check(search(ctx, frames, 100, 12.0, False), frames, 100, 12.0, False)


def test_large_table(ctx):
    """A 4K frame with the thorough lists: the greedy as a kernel a step."""
    sf = A.SynthHandle(width=3840, height=2160, bit_depth=8, sample_bytes=1, seed=9)
    frames = [(sf, *O.search_inputs(sf, 6, amp=24))]
    check(search(ctx, frames, 120, 40.0, True), frames, 120, 40.0, True)


def test_block_errors_under_a_tight_cap(ctx):
    """A memory cap with room for the search but not for the turned error table: the same result."""
    sf = A.SynthHandle(width=320, height=200, bit_depth=10, seed=3)
    frames = [(sf, *O.search_inputs(sf, 4, amp=20))]
    probe, held = G.Ctx(0), C.c_uint64()
    search(probe, frames, 90, 20.0, False)
    A.check(A.lib().av1pf_ctx_memory(probe.p, C.byref(held)))
    probe.close()
    tight = G.Ctx(0, held.value - 512)
    check(search(tight, frames, 90, 20.0, False), frames, 90, 20.0, False)
    tight.close()


@pytest.mark.parametrize("thorough", [False, True], ids=["fast", "thorough"])
def test_batch_of_single_blocks(ctx, thorough):
    """Many frames of one block: clusters that start apart and stage next to nothing before their first exchange."""
    shapes = [dict(width=16 + 5 * i, height=70 - 6 * i, bit_depth=(8, 10, 12)[i % 3]) for i in range(9)]
    frames = []
    for i in range(45):
        sf = A.SynthHandle(**shapes[i % 9], seed=200 + i)
        frames.append((sf, *O.search_inputs(sf, 90 + i, amp=24)))
    check(search(ctx, frames, 80, 9.0, thorough), frames, 80, 9.0, thorough)
