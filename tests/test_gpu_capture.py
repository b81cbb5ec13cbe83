"""GPU: single transforms captured into a CUDA graph. Plans are made, and
scratch is grown, before the capture, as the library asks for."""
import numpy as np
import pytest

from tests._helpers import rel_l2, tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("shape", [(48, 918), (6, 10, 494)])
def test_first_full_spectrum_of_a_plan_under_capture(prec, shape):
    """Nothing is allocated then: a plan that has run no full spectrum yet can
    be captured, later calls and replays agree."""
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    dt = np.float32 if prec == "f32" else np.float64
    size = int(np.prod(shape))
    name = "Float" if prec == "f32" else "Double"
    # (sizes of this precision and dimension alone: tables of other tests' plans are shared)
    shape = shape[:-1] + (shape[-1] + (0 if prec == "f32" else 34),)
    size = int(np.prod(shape))
    f = getattr(J, "%sFFT_%dD" % (name, len(shape)))(*shape)
    x = np.random.default_rng(size).standard_normal((2,) + shape).astype(dt)
    want = [np.fft.fftn(v.astype(np.float64)) for v in x]
    src = torch.from_numpy(x.reshape(2, -1)).cuda()
    a = torch.zeros(2 * size, dtype=src.dtype, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):  # grows this thread's scratch
        getattr(J, name + "FFT_1D")(100003).complexForward(torch.zeros(2 * 100003, dtype=src.dtype, device="cuda"))
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        f.realForwardFull(a)

    def got():
        torch.cuda.synchronize()
        return a.cpu().numpy().astype(np.float64).view(np.complex128).reshape(shape)

    for i in (0, 1, 0):
        a[:size] = src[i]
        g.replay()
        assert rel_l2(got(), want[i]) <= tol(size, dt)
    a[:size] = src[1]
    f.realForwardFull(a)
    assert rel_l2(got(), want[1]) <= tol(size, dt)
    a[:size] = src[0]
    g.replay()
    assert rel_l2(got(), want[0]) <= tol(size, dt)
