"""GPU: a batch whose tasks need much shared memory still runs after another
with small ones was made, directly and as a graph, in both precisions."""
import numpy as np
import pytest

from tests._helpers import rel_l2, tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mode", ["run", "run_graph"])
def test_an_older_batch_runs_after_a_smaller_one(prec, mode):
    import torch
    from jtransforms_gb300 import _native as N
    dt = np.float32 if prec == "f32" else np.float64
    p = N.FLOAT32 if prec == "f32" else N.FLOAT64
    rng = np.random.default_rng(3)

    def batch(lengths):
        x = [rng.standard_normal(2 * n).astype(dt) for n in lengths]
        dev = [torch.from_numpy(v).cuda() for v in x]
        return lengths, x, dev, N.Batch([(N.Plan(N.FFT, p, [n]), N.COMPLEX_FORWARD, d, False) for n, d in zip(lengths, dev)])

    def check(lengths, x, dev, b):
        getattr(b, mode)()
        torch.cuda.synchronize()
        for n, v, d in zip(lengths, x, dev):
            want = np.fft.fft(v.astype(np.float64).view(np.complex128))
            assert rel_l2(d.cpu().numpy().astype(np.float64).view(np.complex128), want) <= tol(n, dt)

    large = batch([4000, 2000, 1000])
    small = batch([16, 20, 24])
    check(*large)
    check(*small)
