"""Loop restoration on the device against the oracle, bit for bit: rectangles of
every width class (two columns a lane, two groups a warp, U and V in one CTA),
heights that leave groups without rows, every parameter set, and samples at the
ends of the range, where the packed sums are largest."""
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
    "tiny_8bit": dict(width=9, height=7, bit_depth=8, sample_bytes=1),
    "one_stripe_10bit": dict(width=66, height=57, bit_depth=10),
    "odd_8bit": dict(width=161, height=131, bit_depth=8, sample_bytes=1),
    "odd_8bit_u16": dict(width=97, height=122, bit_depth=8, sample_bytes=2),
    "units_128_10bit": dict(width=330, height=190, bit_depth=10, lr_unit_shift=1),
    "units_64_chroma_64": dict(width=290, height=150, bit_depth=10, lr_uv_shift=0),
    "422_12bit": dict(width=203, height=93, bit_depth=12, subsampling_x=1, subsampling_y=0),
    "444_12bit": dict(width=131, height=121, bit_depth=12, subsampling_x=0, subsampling_y=0),
    "mono_12bit": dict(width=100, height=89, bit_depth=12, mono=1),
}


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


def restore(ctx, sf, cur, cdef):
    """The oracle's and the device's planes, visible area."""
    info, params, maps = sf.f.info, sf.f.params, sf.f.maps
    want, got = O.HostPlanes.zeros_like(cur), G.DevPlanes.visible(info)
    assert O.lib().oracle_loop_restoration(C.byref(info), C.byref(params), C.byref(maps), cur.c, cdef.c, want.c, 0) == 0
    df = G.DevFrame(sf)
    d_cur, d_cdef = G.DevPlanes.from_host(info, cur), G.DevPlanes.from_host(info, cdef)
    A.check(A.lib().av1pf_loop_restoration(ctx.p, C.byref(info), C.byref(params), C.byref(df.maps), d_cur.c, d_cdef.c,
                                           got.c, None))
    torch.cuda.synchronize()
    for p in range(info.num_planes):
        w, h = sf.plane_dims(p)
        yield p, want.arrays[p][:h, :w], got.host(p, w, h)


@pytest.mark.parametrize("cols", [64, 32])
@pytest.mark.parametrize("content", ["field", "extremes", "flat_top"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_restoration_matches_oracle(ctx, name, content, cols):
    sf = A.SynthHandle(**SHAPES[name], seed=23)
    info, params, maps = sf.f.info, sf.f.params, sf.f.maps
    rng = np.random.default_rng(7)
    cur, cdef = O.HostPlanes.like_synth(sf), O.HostPlanes.like_synth(sf)
    top = (1 << info.bit_depth) - 1
    for a, b in zip(cur.arrays, cdef.arrays):
        if content == "extremes":
            a[...] = rng.choice(np.array([0, 1, top - 1, top], a.dtype), size=a.shape)
            b[...] = rng.choice(np.array([0, 1, top - 1, top], a.dtype), size=a.shape)
        elif content == "flat_top":  # the largest sums, with next to no variance
            a[...] = top - rng.integers(0, 2, size=a.shape).astype(a.dtype)
            b[...] = top - rng.integers(0, 2, size=a.shape).astype(a.dtype)
        else:
            b[...] = np.clip(b.astype(np.int64) + rng.integers(-9, 10, size=b.shape), 0, top).astype(b.dtype)
    if content != "field":  # every set in turn, a Wiener filter now and then, weights at their ends
        for p in range(info.num_planes):
            n = params.lr_unit_rows[p] * params.lr_unit_cols[p]
            units = C.cast(maps.lr_units[p], C.POINTER(A.LrUnit))
            for k in range(n):
                u = units[k]
                u.type, u.sgr_set = (1 if k % 5 == 4 else 2), (k + 5 * p) % 16
                u.sgr_xqd[0], u.sgr_xqd[1] = [(-96, -32), (31, 95), (-96, 95), (31, -32)][k % 4]
                for side in range(2):
                    for j, (lo, hi) in enumerate([(-5, 10), (-23, 8), (-17, 46)]):
                        u.wiener[side][j] = 0 if p and j == 0 else int(rng.choice([lo, hi]))
    t = A.Tuning(-1, cols)
    A.check(A.lib().av1pf_set_tuning(ctx.p, C.byref(t)))
    for p, want, got in restore(ctx, sf, cur, cdef):
        assert np.array_equal(got, want), f"plane {p}: {(got != want).sum()} of {want.size} differ"


@pytest.mark.parametrize("width", [8, 31, 32, 33, 63, 64, 65, 95, 96, 97])
def test_widths_and_packing(ctx, width):
    """A whole chain at rectangle widths around the classes' edges: the packed frame's rows are unaligned at odd widths."""
    for depth, sb in ((8, 1), (10, 2)):
        sf = A.SynthHandle(width=width, height=70 + width % 7, bit_depth=depth, sample_bytes=sb, seed=width)
        ref_cpu, fb_cpu = O.chain(sf)
        ref_gpu, fb_gpu = G.gpu_chain(ctx, G.DevFrame(sf))
        assert np.array_equal(fb_gpu, fb_cpu), f"{depth}-bit: {(fb_gpu != fb_cpu).sum()} bytes differ"
        for p, (a, b) in enumerate(zip(ref_gpu, ref_cpu.arrays)):
            assert np.array_equal(a, b), f"{depth}-bit plane {p}"
