"""Film-grain templates on the device at every auto-regression lag, depth and
chroma layout, with extreme coefficients, against the oracle, bit for bit."""
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

LAYOUTS = {"420_8bit": dict(bit_depth=8, sample_bytes=1), "420_10bit": dict(bit_depth=10),
           "422_10bit": dict(bit_depth=10, subsampling_x=1, subsampling_y=0),
           "444_12bit": dict(bit_depth=12, subsampling_x=0, subsampling_y=0), "mono_12bit": dict(bit_depth=12, mono=1)}


@pytest.fixture(scope="module")
def ctx():
    c = G.Ctx(0)
    yield c
    c.close()


@pytest.mark.parametrize("coefs", ["random", "extreme"])
@pytest.mark.parametrize("lag", [0, 1, 2, 3])
@pytest.mark.parametrize("name", sorted(LAYOUTS))
def test_grain_lags_match_oracle(ctx, name, lag, coefs):
    sf = A.SynthHandle(width=200, height=136, enable_grain=1, seed=40 + lag, frame_index=9 + lag, **LAYOUTS[name])
    g = sf.f.params.film_grain
    g.ar_coeff_lag = lag
    if coefs == "extreme":  # the ends of the coefficients' range, the smallest shift: values clip at both ends
        rng = np.random.default_rng(lag)
        for arr, n in ((g.ar_coeffs_y_plus_128, 24), (g.ar_coeffs_cb_plus_128, 25), (g.ar_coeffs_cr_plus_128, 25)):
            for k in range(n):
                arr[k] = int(rng.choice([0, 255]))
        g.ar_coeff_shift_minus_6 = 0
        g.grain_scale_shift = 0
    ref_cpu, fb_cpu = O.chain(sf)
    df = G.DevFrame(sf)
    ref_gpu, fb_gpu = G.gpu_chain(ctx, df)
    for p, (a, b) in enumerate(zip(ref_gpu, ref_cpu.arrays)):
        assert np.array_equal(a, b), f"reference plane {p}"
    assert np.array_equal(fb_gpu, fb_cpu), f"{(fb_gpu != fb_cpu).sum()} bytes differ"


@pytest.mark.parametrize("lag", [0, 1, 2, 3])
@pytest.mark.parametrize("name", ["420_8bit", "422_10bit", "444_12bit", "mono_12bit"])
def test_grain_coefficients_beyond_8_bits(ctx, name, lag):
    """The coefficients' fields are 32 bits wide and are not checked: values that
    no stream codes are multiplied as they are, in one plane or in all."""
    sf = A.SynthHandle(width=200, height=136, enable_grain=1, seed=60 + lag, frame_index=5 + lag, **LAYOUTS[name])
    g = sf.f.params.film_grain
    g.ar_coeff_lag = lag
    g.ar_coeff_shift_minus_6 = 3
    results = []
    for arr in (g.ar_coeffs_y_plus_128, g.ar_coeffs_cb_plus_128, g.ar_coeffs_cr_plus_128):
        arr[0], arr[2 * lag * (lag + 1) - 1 if lag else 0] = 128 + 200, 128 - 700
        results.append((O.chain(sf), G.gpu_chain(ctx, G.DevFrame(sf))))
    for k, ((ref_cpu, fb_cpu), (ref_gpu, fb_gpu)) in enumerate(results):
        for p, (a, b) in enumerate(zip(ref_gpu, ref_cpu.arrays)):
            assert np.array_equal(a, b), f"step {k} reference plane {p}"
        assert np.array_equal(fb_gpu, fb_cpu), f"step {k}: {(fb_gpu != fb_cpu).sum()} bytes differ"
