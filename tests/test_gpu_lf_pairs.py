"""The loop filter's two-lane arithmetic at its limits: samples at 0 and at the
maximum, steps around the filter's thresholds, and flat areas for the wide
filters, at every bit depth, chroma layout and sample width. Whole chains
against the oracle, bit for bit."""
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

FORMATS = {
    "8bit": dict(bit_depth=8, sample_bytes=1),
    "8bit_u16_444": dict(bit_depth=8, sample_bytes=2, subsampling_x=0, subsampling_y=0),
    "10bit_422": dict(bit_depth=10, subsampling_x=1, subsampling_y=0),
    "12bit": dict(bit_depth=12),
}
# how far samples stray from a level that changes every 4x4, as parts of the range, and that level
CONTENT = {"extremes": None, "low": (64, 0.0), "high": (64, 1.0), "flat": (256, 0.5), "steps": (24, 0.5)}


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


def fill(sf, content, rng):
    f, top = sf.f, (1 << sf.f.info.bit_depth) - 1
    for p in range(f.info.num_planes):
        pl = f.planes[p]
        dt = np.uint8 if f.info.sample_bytes == 1 else np.uint16
        n = pl.stride * pl.height
        a = np.frombuffer((C.c_uint8 * (n * dt().itemsize)).from_address(pl.data), dt).reshape(pl.height, pl.stride)
        if CONTENT[content] is None:
            v = rng.integers(0, 2, a.shape) * top
        else:
            part, level = CONTENT[content]
            amp = max(1, (top + 1) // part)
            cells = rng.integers(-amp, amp + 1, ((pl.height + 3) // 4, (pl.stride + 3) // 4))
            v = level * top + np.kron(cells, np.ones((4, 4), np.int64))[:pl.height, :pl.stride]
            v += rng.integers(-1, 2, a.shape) * (amp > 2)
        a[:] = np.clip(v, 0, top).astype(dt)


@pytest.mark.parametrize("content", sorted(CONTENT))
@pytest.mark.parametrize("fmt", sorted(FORMATS))
def test_chain_on_filter_limits(ctx, fmt, content):
    sf = A.SynthHandle(width=203, height=150, seed=91, frame_index=1, **FORMATS[fmt])
    fill(sf, content, np.random.default_rng(92))
    for k, (levels, sharp) in enumerate((((63, 63, 63, 63), 0), ((20, 9, 31, 40), 5))):
        for i, v in enumerate(levels):
            sf.f.params.loop_filter_level[i] = v
        sf.f.params.loop_filter_sharpness = sharp
        want, packed = O.chain(sf, threads=0)
        got, got_packed = G.gpu_chain(ctx, G.DevFrame(sf))
        for p, (g, w) in enumerate(zip(got, want.arrays)):
            assert np.array_equal(g, w), f"plane {p}, levels {levels}: {np.argwhere(g != w)[:4]}"
        assert np.array_equal(got_packed, packed)
