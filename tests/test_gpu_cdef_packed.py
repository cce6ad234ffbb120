"""CDEF's two-samples-a-lane kernels (in half precision for bit depths up to 10,
in integers for 12) against the oracle, bit for bit: windows inside the frame and at each of its edges, half and whole
superblock CTAs, every chroma layout, extreme samples and strengths, and a
batch whose frames need both CDEF kernels."""
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
    # fewer than a superblock; one 4-sample chroma column short of a chunk (292 = 4 mod 16)
    "tiny_8bit": dict(width=20, height=12, bit_depth=8, sample_bytes=1),
    "ragged_10bit": dict(width=292, height=196, bit_depth=10),
    "422_10bit": dict(width=296, height=212, bit_depth=10, subsampling_x=1, subsampling_y=0),
    "444_8bit_u16": dict(width=264, height=140, bit_depth=8, sample_bytes=2, subsampling_x=0, subsampling_y=0),
    "mono_10bit": dict(width=328, height=200, bit_depth=10, mono=1),
    "tiny_12bit": dict(width=20, height=12, bit_depth=12),
    "ragged_12bit": dict(width=292, height=196, bit_depth=12),
    "422_12bit": dict(width=296, height=212, bit_depth=12, subsampling_x=1, subsampling_y=0),
    "444_12bit": dict(width=261, height=139, bit_depth=12, subsampling_x=0, subsampling_y=0),
    "mono_12bit": dict(width=328, height=200, bit_depth=12, mono=1),
    "whole_420_12bit": dict(width=2564, height=1044, bit_depth=12),
    # more superblocks than one wave of half superblocks: whole-superblock CTAs
    "whole_420_8bit": dict(width=2564, height=1044, bit_depth=8, sample_bytes=1),
    "whole_444_10bit": dict(width=2564, height=1036, bit_depth=10, subsampling_x=0, subsampling_y=0),
}


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


@pytest.mark.parametrize("content", ["field", "extremes", "noise"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_cdef_stage_matches_oracle(ctx, name, content):
    sf = A.SynthHandle(**SHAPES[name], seed=91, skip_pct=15)
    info, params, maps = sf.f.info, sf.f.params, sf.f.maps
    cur = O.HostPlanes.like_synth(sf)
    if content != "field":  # samples at and next to the range's ends, or anywhere; the strongest and weakest filters
        rng = np.random.default_rng(5)
        top = (1 << info.bit_depth) - 1
        for a in cur.arrays:
            a[...] = (rng.choice(np.array([0, 1, 2, top // 2, top - 1, top], a.dtype), size=a.shape)
                      if content == "extremes" else
                      np.clip(top // 2 + rng.normal(0, top / 24, a.shape), 0, top).astype(a.dtype))
        for k, (yp, ys, up, us) in enumerate([(15, 4, 15, 4), (15, 0, 0, 4), (0, 4, 15, 0), (1, 1, 1, 1),
                                              (0, 0, 0, 0), (8, 2, 7, 1), (3, 4, 2, 4), (0, 1, 1, 0)]):
            params.cdef_y_pri_strength[k], params.cdef_y_sec_strength[k] = yp, ys
            params.cdef_uv_pri_strength[k], params.cdef_uv_sec_strength[k] = up, us
        params.cdef_damping = 6 if content == "extremes" else 4
    want = O.HostPlanes.zeros_like(cur)
    assert O.lib().oracle_cdef(C.byref(info), C.byref(params), C.byref(maps), cur.c, want.c, 0) == 0
    df = G.DevFrame(sf)
    d_cur, d_out = G.DevPlanes.from_host(info, cur), G.DevPlanes.from_host(info, O.HostPlanes.zeros_like(cur))
    A.check(A.lib().av1pf_cdef(ctx.p, C.byref(info), C.byref(params), C.byref(df.maps), d_cur.c, d_out.c, None))
    torch.cuda.synchronize()
    for p in range(info.num_planes):
        w = (info.mi_cols * 4) >> (info.subsampling_x if p else 0)
        h = (info.mi_rows * 4) >> (info.subsampling_y if p else 0)
        got = d_out.host(p, w, h)
        assert np.array_equal(got, want.arrays[p][:h, :w]), f"plane {p}: {(got != want.arrays[p][:h, :w]).sum()} differ"


def test_batch_of_both_depths(ctx):
    """8-, 10- and 12-bit frames in one batch: each CDEF kernel leaves the other's frames alone."""
    sfs = [A.SynthHandle(width=264, height=200, seed=60 + i, frame_index=i, **c) for i, c in enumerate(
        [dict(bit_depth=8, sample_bytes=1), dict(bit_depth=12), dict(bit_depth=10),
         dict(bit_depth=12, subsampling_x=0, subsampling_y=0)])]
    dfs = [G.DevFrame(s) for s in sfs]
    outs = [(G.DevPlanes.visible(d.info), G.dev_bytes(A.frame_bytes(d.info))) for d in dfs]
    jobs = (A.Job * len(dfs))()
    for j, d, (ref, fb) in zip(jobs, dfs, outs):
        j.info, j.params, j.maps = C.pointer(d.info), C.pointer(d.params), C.pointer(d.maps)
        j.inp, j.ref_out = C.cast(d.inp.c, C.POINTER(A.Plane)), C.cast(ref.c, C.POINTER(A.Plane))
        j.frame_out = fb.data_ptr()
    b = C.c_void_p()
    A.check(A.lib().av1pf_batch_create(ctx.p, jobs, len(dfs), 0, C.byref(b)))
    for _ in range(2):
        A.check(A.lib().av1pf_batch_run(b, None))
    torch.cuda.synchronize()
    A.lib().av1pf_batch_destroy(b)
    for i, (sf, (ref, fb)) in enumerate(zip(sfs, outs)):
        ref_cpu, fb_cpu = O.chain(sf)
        assert np.array_equal(fb[: A.frame_bytes(sf.f.info)].cpu().numpy(), fb_cpu), f"frame {i}"
        for p in range(sf.f.info.num_planes):
            assert np.array_equal(ref.host(p), ref_cpu.arrays[p]), f"frame {i} plane {p}"
