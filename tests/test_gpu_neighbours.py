"""GPU: a finite double line's result does not depend on the lines beside it.
An infinity or a NaN in one line, or one array of a batch, leaves the bits of
all others as they are; its own line spreads it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(plan, op, scale, x, at, batch, dist, bad):
    """x: batch x dist; number `at` of array 1 becomes bad."""
    import torch
    out = []
    for special in (False, True):
        y = x.copy()
        if special:
            y[1, at] = bad
        dev = torch.from_numpy(y.ravel()).cuda()
        plan.execute(op, dev, 0, scale, batch=batch, dist=dist)
        out.append(dev.cpu().numpy().reshape(batch, dist))
    rest = np.arange(batch) != 1
    assert np.array_equal(out[0][rest].view(np.int64), out[1][rest].view(np.int64))
    own = out[1][1].view(np.complex128) if plan.kind == 0 and op < 2 else out[1][1]
    assert np.isfinite(out[0]).all() and not np.isfinite(own).any()


# one pass of powers of two, of small primes, of larger ones; two passes; a convolution
@pytest.mark.parametrize("n", [16, 32, 64, 256, 512, 1024, 4096, 8192, 24, 96, 100, 1000, 3000, 121, 122, 1331, 1922, 1 << 14, 5000, 131])
@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_complex_lines(n, inverse, bad):
    from jtransforms_gb300 import _native as N
    batch = max(5, 9000 // n)
    x = np.random.default_rng(n).standard_normal((batch, 2 * n))
    _compare(N.Plan(N.FFT, N.FLOAT64, [n]), N.COMPLEX_INVERSE if inverse else N.COMPLEX_FORWARD, inverse, x, n // 3, batch, 2 * n, bad)


@pytest.mark.parametrize("n", [32, 64, 128, 512, 1024, 4096, 8192, 200, 242, 2662])
@pytest.mark.parametrize("kind", ["dct", "dst", "dht", "real"])
@pytest.mark.parametrize("fwd", [True, False])
def test_real_lines(n, kind, fwd):
    from jtransforms_gb300 import _native as N
    batch = max(5, 9000 // n)
    x = np.random.default_rng(n).standard_normal((batch, n))
    plan = N.Plan({"dct": N.DCT, "dst": N.DST, "dht": N.DHT, "real": N.FFT}[kind], N.FLOAT64, [n])
    op = (N.REAL_FORWARD if fwd else N.REAL_INVERSE) if kind == "real" else N.FORWARD if fwd else N.INVERSE
    _compare(plan, op, not fwd, x, n // 3, batch, n, np.inf)


# columns of several arrays share a tile
@pytest.mark.parametrize("dims", [(16, 6), (64, 10), (256, 6), (512, 6), (1024, 10), (4096, 2), (100, 6), (1000, 6), (122, 10)])
@pytest.mark.parametrize("kind", ["fft", "dct", "dht"])
def test_columns(dims, kind):
    from jtransforms_gb300 import _native as N
    batch, size = 7, int(np.prod(dims)) * (2 if kind == "fft" else 1)
    x = np.random.default_rng(size).standard_normal((batch, size))
    plan = N.Plan({"fft": N.FFT, "dct": N.DCT, "dht": N.DHT}[kind], N.FLOAT64, list(dims))
    _compare(plan, N.COMPLEX_FORWARD if kind == "fft" else N.FORWARD, False, x, size // 3, batch, size, np.nan)
