"""The encoder's restoration search where its self-guided kernel can go wrong:
units cut into strips with one or a few columns left, stripes of a few rows and
odd heights, units of several stripes, rows that no vector load may take, two
sets of a narrow unit side by side and one set a CTA (few units), and errors at
the largest the sums can hold. Against the oracle, bit for bit."""
import numpy as np
import pytest

import av1pf as A

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import gpu_util as G  # noqa: E402
import oracle as O  # noqa: E402
from test_gpu_search import gpu_lr_search  # noqa: E402

SHAPES = {
    "strip_and_one_column_10bit": dict(width=66, height=64, bit_depth=10, lr_unit_shift=1),
    "odd_8bit": dict(width=193, height=121, bit_depth=8, sample_bytes=1),
    "aligned_8bit": dict(width=256, height=130, bit_depth=8, sample_bytes=1, lr_unit_shift=1),
    "tall_stripes_444_10bit": dict(width=97, height=187, bit_depth=10, subsampling_x=0, subsampling_y=0),
    "422_12bit": dict(width=161, height=59, bit_depth=12, subsampling_x=1, subsampling_y=0),
    "narrow_mono_10bit": dict(width=24, height=75, bit_depth=10, mono=1),
    "256_units_10bit": dict(width=330, height=210, bit_depth=10, lr_unit_shift=2, lr_uv_shift=0),
    "many_units_10bit": dict(width=1600, height=1088, bit_depth=10),
}


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


def planes(like, f):
    return O.HostPlanes([f(p, a).astype(a.dtype) for p, a in enumerate(like.arrays)])


def compare(ctx, sf, cur, cdef, src, lam, effort):
    assert gpu_lr_search(ctx, sf, cur, cdef, src, lam, effort) == O.lr_search(sf, cur, cdef, src, lam, effort)


@pytest.mark.parametrize("effort", [0, 2], ids=["fast", "thorough"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_self_guided_units(ctx, name, effort):
    """Smooth frames under noise of a size that changes from unit to unit: units
    for which the self-guided filters win, with fits that differ between sets."""
    if name == "many_units_10bit":
        effort = min(effort, 1)
    sf = A.SynthHandle(seed=61, enable_lr=1, **SHAPES[name])
    rng = np.random.default_rng(62)
    maxv = (1 << sf.f.info.bit_depth) - 1
    base, _, _ = O.lr_search_inputs(sf, 63)
    yy = [np.add.outer(np.arange(a.shape[0]), np.arange(a.shape[1])) for a in base.arrays]
    src = planes(base, lambda p, a: maxv // 4 + (yy[p] * maxv // 700) % (maxv // 2))
    noise = [rng.normal(0, 1, a.shape) * (1 + (yy[p] // 40) % 5) * maxv / 200 for p, a in enumerate(src.arrays)]
    cdef = planes(src, lambda p, a: np.clip(a + noise[p], 0, maxv))
    cur = planes(cdef, lambda p, a: np.clip(a + rng.integers(-9, 10, a.shape), 0, maxv))
    compare(ctx, sf, cur, cdef, src, 0.0, effort)


@pytest.mark.parametrize("bd,shift", [(8, 0), (10, 0), (10, 2), (12, 0), (12, 2)])
def test_self_guided_extremes(ctx, bd, shift):
    """Samples at both ends of their range: the largest differences, products and
    sums."""
    sf = A.SynthHandle(width=200, height=136, bit_depth=bd, seed=71, enable_lr=1, lr_unit_shift=shift, lr_uv_shift=0)
    rng = np.random.default_rng(72)
    maxv = (1 << bd) - 1
    base, _, _ = O.lr_search_inputs(sf, 73)
    cdef = planes(base, lambda p, a: maxv * (rng.random(a.shape) < 0.5))
    src = planes(cdef, lambda p, a: maxv - a.astype(np.int64))
    compare(ctx, sf, cdef, cdef, src, 0.0, 1)


@pytest.mark.parametrize("height", [25, 41, 49, 52, 56])
def test_one_stripe(ctx, height):
    """Planes of one stripe, whose rows the warps' shares reach past, in wide units."""
    sf = A.SynthHandle(width=330, height=height, bit_depth=10, seed=81, enable_lr=1, lr_unit_shift=2, lr_uv_shift=0)
    cur, cdef, src = O.lr_search_inputs(sf, 82)
    compare(ctx, sf, cur, cdef, src, 10.0, 1)
