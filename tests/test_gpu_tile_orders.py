"""GPU: lengths with a prime factor of 17 to 61, which run the tile passes in
both precisions, in each of their four pass orders, complex and real."""
import numpy as np
import pytest

from tests._helpers import rel_l2, tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n", [17, 34, 76, 184, 544, 1156, 2014, 2928, 3596])
def test_orders(order, prec, n):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    dt = np.float64 if prec == "f64" else np.float32
    prev = N.set_option(N.OPT_RADIX_ORDER, order)
    try:
        f = (J.FloatFFT_1D if prec == "f32" else J.DoubleFFT_1D)(n)
        assert f.plan.algorithm(0) == 0  # one pass
        batch = 9
        rng = np.random.default_rng(n + order)
        x = rng.uniform(-1, 1, (batch, 2 * n)).astype(dt)
        dev = torch.from_numpy(x.ravel().copy()).cuda()
        f.plan.execute(N.COMPLEX_FORWARD, dev, 0, False, batch=batch, dist=2 * n)
        got = dev.cpu().numpy().astype(np.float64).view(np.complex128).reshape(batch, n)
        assert rel_l2(got, np.fft.fft(x.astype(np.float64).view(np.complex128), axis=1)) <= tol(n, dt)
        dist = n + (n & 1)  # arrays start on pairs
        r = rng.uniform(-1, 1, (batch, dist)).astype(dt)
        rd = torch.from_numpy(r.ravel().copy()).cuda()
        f.plan.execute(N.REAL_FORWARD, rd, 0, False, batch=batch, dist=dist)
        f.plan.execute(N.REAL_INVERSE, rd, 0, True, batch=batch, dist=dist)
        assert rel_l2(rd.cpu().numpy().reshape(batch, dist)[:, :n], r[:, :n]) <= 2 * tol(n, dt)
    finally:
        N.set_option(N.OPT_RADIX_ORDER, prev)
