"""GPU: float lines of mixed-radix length (jt_mixed.cuh) in rows, in columns
and in both passes of the two-pass scheme, with partial tiles; each pass
radix 2..16 occurs first, in the middle or last.  Bound: the library's
4 eps log2(n) relative L2 against numpy in FP64.
"""
import numpy as np
import pytest

from tests._helpers import rel_l2, tol

pytestmark = pytest.mark.gpu

# single radices (columns run them in one pass), two, three, four and five
# passes, the longest line, odd and even first radices
LENGTHS = [3, 6, 7, 9, 10, 11, 12, 13, 14, 15, 18, 22, 24, 26, 33, 39, 48, 49, 77, 96, 121, 143, 169, 210, 225, 240, 250, 343, 360,
           500, 729, 1000, 1001, 1080, 1331, 1536, 1920, 2002, 2197, 3000, 3072, 4410, 5005, 6000, 6561, 7168, 7776, 8100]


def _c64(shape, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def _device(z):
    import torch
    return torch.from_numpy(z.view(np.float32).ravel().copy()).cuda()


@pytest.mark.parametrize("n", LENGTHS)
def test_rows(n):
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    f = J.FloatFFT_1D(n)
    for batch in (1, 2, 3, max(5, 30011 // n)):
        z = _c64((batch, n), n)
        dev = _device(z)
        f.plan.execute(N.COMPLEX_FORWARD, dev, 0, False, batch=batch, dist=2 * n)
        got = dev.cpu().numpy().view(np.complex64).reshape(batch, n)
        assert rel_l2(got, np.fft.fft(z.astype(complex), axis=1)) <= tol(n, np.float32)
        f.plan.execute(N.COMPLEX_INVERSE, dev, 0, True, batch=batch, dist=2 * n)
        assert rel_l2(dev.cpu().numpy().view(np.complex64).reshape(batch, n), z) <= 2 * tol(n, np.float32)


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("cols", [2, 33])
def test_columns(n, cols):
    import jtransforms_gb300 as J
    z = _c64((n, cols), n + cols)
    f = J.FloatFFT_2D(n, cols)
    dev = _device(z)
    f.complexForward(dev)
    assert rel_l2(dev.cpu().numpy().view(np.complex64).reshape(n, cols), np.fft.fft2(z.astype(complex))) <= tol(z.size, np.float32)
    f.complexInverse(dev, True)
    assert rel_l2(dev.cpu().numpy().view(np.complex64).reshape(n, cols), z) <= 2 * tol(z.size, np.float32)


@pytest.mark.parametrize("n", [9000, 10080, 12345 * 2, 50000, 65520, 3 ** 10, 7 ** 5 * 2, 13 ** 4, 1000000, 1536 * 1000])
@pytest.mark.parametrize("batch", [1, 3])
def test_two_passes(n, batch):
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    f = J.FloatFFT_1D(n)
    z = _c64((batch, n), n)
    dev = _device(z)
    f.plan.execute(N.COMPLEX_FORWARD, dev, 0, False, batch=batch, dist=2 * n)
    got = dev.cpu().numpy().view(np.complex64).reshape(batch, n)
    assert rel_l2(got, np.fft.fft(z.astype(complex), axis=1)) <= tol(n, np.float32)
    f.plan.execute(N.COMPLEX_INVERSE, dev, 0, True, batch=batch, dist=2 * n)
    assert rel_l2(dev.cpu().numpy().view(np.complex64).reshape(batch, n), z) <= 2 * tol(n, np.float32)


@pytest.mark.parametrize("n", [67, 71, 101, 127, 263, 509, 1021, 2 * 1021, 2039, 3 * 1361, 4093, 4099, 8191, 10007, 2 * 5003, 20011, 65521,
                               131071, 3 * 67 * 1009, 524287])
@pytest.mark.parametrize("batch", [1, 3, 40])
def test_bluestein(n, batch):
    """Lengths with a prime factor above 61: one kernel up to 4096 points
    (jt_bluemix.cuh), three beyond."""
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    if n * batch > 3000000:
        batch = 2
    f = J.FloatFFT_1D(n)
    dist = n + 3
    z = _c64((batch, dist), n)
    dev = _device(z)
    f.plan.execute(N.COMPLEX_FORWARD, dev, 0, False, batch=batch, dist=2 * dist)
    got = dev.cpu().numpy().view(np.complex64).reshape(batch, dist)
    assert np.array_equal(got[:, n:], z[:, n:])  # what lies between the lines is left alone
    assert rel_l2(got[:, :n], np.fft.fft(z[:, :n].astype(complex), axis=1)) <= tol(n, np.float32)
    f.plan.execute(N.COMPLEX_INVERSE, dev, 0, True, batch=batch, dist=2 * dist)
    assert rel_l2(dev.cpu().numpy().view(np.complex64).reshape(batch, dist)[:, :n], z[:, :n]) <= 2 * tol(n, np.float32)
