"""Super-resolution on the device against the oracle, bit for bit: every ratio,
widths from a few samples to thousands (odd ones leave a thread one column), row
counts that leave an item short, both sample sizes, samples at the ends of their
range (all 64 phases, the taps of 128 among them), and output planes whose rows
start at odd samples."""
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
    "tiny_d16": dict(width=17, height=9, bit_depth=10, superres_denom=16),
    "tiny_8bit_d9": dict(width=8, height=8, bit_depth=8, sample_bytes=1, superres_denom=9),
    "odd_8bit_d11": dict(width=203, height=37, bit_depth=8, sample_bytes=1, superres_denom=11),
    "odd_d13_422_12bit": dict(width=333, height=66, bit_depth=12, subsampling_x=1, subsampling_y=0, superres_denom=13),
    "d10_444": dict(width=510, height=23, bit_depth=10, subsampling_x=0, subsampling_y=0, superres_denom=10),
    "d12_mono_8bit_u16": dict(width=641, height=18, bit_depth=8, sample_bytes=2, mono=1, superres_denom=12),
    "wide_d15": dict(width=5001, height=8, bit_depth=10, superres_denom=15),
    "widest_d14": dict(width=16384, height=8, bit_depth=12, superres_denom=14),
}


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "odd_rows"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_superres_matches_oracle(ctx, name, shift):
    sf = A.SynthHandle(**SHAPES[name], seed=81)
    info, params = sf.f.info, sf.f.params
    rng, top = np.random.default_rng(82), (1 << info.bit_depth) - 1
    src = O.HostPlanes.like_synth(sf)
    for a in src.arrays:
        a[...] = rng.choice(np.array([0, 1, top // 2, top - 1, top], a.dtype), size=a.shape)
    want = O.HostPlanes.upscaled(info)
    assert O.lib().oracle_superres(C.byref(info), C.byref(params), src.c, want.c) == 0
    dims = [(a.shape[1], a.shape[0]) for a in want.arrays]
    got = G.DevPlanes(info, dims, strides=[(w + 63) // 64 * 64 + shift for w, _ in dims])
    A.check(A.lib().av1pf_superres(ctx.p, C.byref(info), C.byref(params), G.DevPlanes.from_host(info, src).c, got.c, None))
    torch.cuda.synchronize()
    for p in range(info.num_planes):
        w, h = sf.plane_dims(p)
        assert np.array_equal(got.host(p, w, h), want.arrays[p][:h, :w]), f"plane {p}"
        assert not got.host(p)[:h, w:].any(), f"plane {p}: written past the row"
