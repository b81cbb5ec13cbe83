"""GPU: lines of mixed-radix length, floats (jt_mixed.cuh) and doubles
(jt_fixmix.cuh, the fixed-point tile passes of jt_device.cuh), in rows, in
columns and in both passes of the two-pass scheme, with partial tiles; each
pass radix occurs first, in the middle or last.  Bound: the library's
4 eps log2(n) relative L2 against numpy in FP64, for doubles per line.
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


DLENGTHS = [6, 11, 15, 18, 24, 45, 48, 49, 50, 60, 61, 72, 77, 96, 122, 143, 210, 225, 250, 343, 360, 529, 720, 729, 1000, 1001, 1080,
            1331, 1536, 1920, 2025, 2401, 2744, 3000, 3072, 3125, 3600, 3721, 3969, 4050, 4095]


def _lines64(n, batch, seed):
    rng = np.random.default_rng(seed)
    z = rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))
    return z * (10.0 ** np.linspace(-10, 10, batch))[:, None]


@pytest.mark.parametrize("n", DLENGTHS)
@pytest.mark.parametrize("special", [None, np.inf, np.nan])
def test_double_rows(n, special):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    f = J.DoubleFFT_1D(n)
    for batch in (1, 3, max(5, 9001 // n)):
        z = _lines64(n, batch, n)
        if batch > 1:
            z[1] = 0
        bad = batch - 1 if special is not None else -1
        if bad >= 0:
            z[bad, n // 3] = special
        for inverse in (False, True):
            dev = torch.from_numpy(z.view(np.float64).ravel().copy()).cuda()
            f.plan.execute(N.COMPLEX_INVERSE if inverse else N.COMPLEX_FORWARD, dev, 0, inverse, batch=batch, dist=2 * n)
            got = dev.cpu().numpy().view(np.complex128).reshape(batch, n)
            with np.errstate(invalid="ignore"):
                want = np.fft.ifft(z, axis=1) if inverse else np.fft.fft(z, axis=1)
            for b in range(batch):
                if b == bad:
                    assert not np.isfinite(got[b]).any()
                else:
                    assert rel_l2(got[b], want[b]) <= tol(n, np.float64)


@pytest.mark.parametrize("n", DLENGTHS)
@pytest.mark.parametrize("cols", [2, 33])
def test_double_columns(n, cols):
    import torch
    import jtransforms_gb300 as J
    z = _lines64(cols, n, n)[::-1].copy() if n < 100 else _lines64(n, cols, n).T.copy()
    f = J.DoubleFFT_2D(n, cols)
    dev = torch.from_numpy(z.view(np.float64).ravel().copy()).cuda()
    f.complexForward(dev)
    assert rel_l2(dev.cpu().numpy().view(np.complex128).reshape(n, cols), np.fft.fft2(z)) <= tol(z.size, np.float64)
    f.complexInverse(dev, True)
    assert rel_l2(dev.cpu().numpy().view(np.complex128).reshape(n, cols), z) <= 2 * tol(z.size, np.float64)


@pytest.mark.parametrize("n", [9000, 10080, 50000, 65520, 3 ** 10, 7 ** 5 * 2, 13 ** 4, 1000000, 1536 * 1000, 1021, 10007])
@pytest.mark.parametrize("batch", [1, 3])
def test_double_two_passes(n, batch):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    f = J.DoubleFFT_1D(n)
    z = _lines64(n, batch, n)
    dev = torch.from_numpy(z.view(np.float64).ravel().copy()).cuda()
    f.plan.execute(N.COMPLEX_FORWARD, dev, 0, False, batch=batch, dist=2 * n)
    got = dev.cpu().numpy().view(np.complex128).reshape(batch, n)
    want = np.fft.fft(z, axis=1)
    for b in range(batch):
        assert rel_l2(got[b], want[b]) <= tol(n, np.float64)
    f.plan.execute(N.COMPLEX_INVERSE, dev, 0, True, batch=batch, dist=2 * n)
    back = dev.cpu().numpy().view(np.complex128).reshape(batch, n)
    for b in range(batch):
        assert rel_l2(back[b], z[b]) <= 2 * tol(n, np.float64)


@pytest.mark.parametrize("n", [12, 50, 96, 100, 122, 210, 360, 1000, 1331 * 2, 1920, 3000, 4050, 6000])
@pytest.mark.parametrize("kind", ["dct", "dst"])
@pytest.mark.parametrize("fwd", [True, False])
def test_double_r2r_rows(n, kind, fwd):
    import scipy.fft as sfft
    import torch
    from jtransforms_gb300 import _native as N
    batch = max(3, 9001 // n)
    x = _lines64(n, batch, n).real.copy()
    plan = N.Plan(N.DCT if kind == "dct" else N.DST, N.FLOAT64, [n])
    dev = torch.from_numpy(x.ravel().copy()).cuda()
    plan.execute(N.FORWARD if fwd else N.INVERSE, dev, 0, True, batch=batch, dist=n)
    got = dev.cpu().numpy().reshape(batch, n)
    want = (sfft.dct if kind == "dct" else sfft.dst)(x, type=2 if fwd else 3, norm="ortho", axis=1)
    for b in range(batch):
        assert rel_l2(got[b], want[b]) <= tol(n, np.float64)
