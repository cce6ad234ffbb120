"""A context made while the legacy stream is busy, and calls on another stream
right away: nothing of the context's set-up may run behind the legacy stream's
work. Against the oracle, bit for bit."""
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


@pytest.mark.parametrize("grain", [0, 1])
def test_calls_beside_a_busy_legacy_stream(grain):
    sf = A.SynthHandle(width=200, height=136, bit_depth=10, enable_grain=grain, seed=5)
    _, want = O.chain(sf)
    G.Ctx(0).close()  # (the module and its tables are loaded)
    d = G.DevFrame(sf)
    outs = [(G.DevPlanes.visible(d.info), G.dev_bytes(A.frame_bytes(d.info))) for _ in range(12)]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)  # about 50 ms of the legacy stream
    ctx = G.Ctx(0)
    for ref, fb in outs:
        A.check(A.lib().av1pf_chain(ctx.p, C.byref(d.info), C.byref(d.params), C.byref(d.maps), d.inp.c, ref.c,
                                    fb.data_ptr(), side.cuda_stream), "av1pf_chain")
    side.synchronize()
    torch.cuda.synchronize()
    for k, (_, fb) in enumerate(outs):
        assert np.array_equal(fb[: want.size].cpu().numpy(), want), f"call {k}"
    ctx.close()
