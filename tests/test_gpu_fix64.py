"""GPU: power-of-two lines of doubles, which run in 64-bit block-fixed-point
arithmetic (jt_fix64.cuh): every line length in the row, column and
transposing forms, lines whose magnitudes differ, the ends of the double
range, and infinities and NaNs.

The bound is the library's 4 eps log2(n) relative L2 per line, against numpy
in FP64; a line's exponent is its own, so it holds for each line however
large its neighbours are.
"""
import numpy as np
import pytest

from tests._helpers import rel_l2, tol

pytestmark = pytest.mark.gpu


def _lines(n, batch, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))


def _rows(n, z, inverse=False, scale=False):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    f = J.DoubleFFT_1D(n)
    dev = torch.from_numpy(np.ascontiguousarray(z).view(np.float64).ravel().copy()).cuda()
    f.plan.execute(N.COMPLEX_INVERSE if inverse else N.COMPLEX_FORWARD, dev, 0, scale, batch=z.shape[0], dist=2 * n)
    return dev.cpu().numpy().view(np.complex128).reshape(z.shape)


@pytest.mark.parametrize("lg", range(4, 18))
def test_lines_of_any_magnitude(lg):
    n = 1 << lg
    batch = max(3, 5000 // n)
    z = _lines(n, batch, lg)
    # 24 orders of magnitude from line to line, the same kernel tile
    z *= (10.0 ** np.linspace(-12, 12, batch))[:, None]
    z[1] = 0
    got = _rows(n, z)
    want = np.fft.fft(z, axis=1)
    assert np.all(got[1] == 0)
    for b in range(batch):
        assert rel_l2(got[b], want[b]) <= tol(n, np.float64)
    back = _rows(n, want, inverse=True, scale=True)
    for b in range(batch):
        assert rel_l2(back[b], z[b]) <= 2 * tol(n, np.float64)


@pytest.mark.parametrize("n", [16, 64, 1024, 4096])
@pytest.mark.parametrize("size", [1e-315, 1e-307, 1e-290, 1e-270, 1e285, 1e300])
def test_ends_of_the_range(n, size):
    z = _lines(n, 5, n)
    z[2:4] *= size
    got = _rows(n, z)
    for b in range(5):
        s = size if b in (2, 3) else 1.0
        # the inputs themselves are rounded to the subnormal grid
        x = z[b] / s if size > 1e-308 or s == 1.0 else (z[b] * 2.0 ** 600) / (size * 2.0 ** 600)
        g = got[b] / s if size > 1e-308 or s == 1.0 else (got[b] * 2.0 ** 600) / (size * 2.0 ** 600)
        want = np.fft.fft(x)
        # half a subnormal unit, 2^-1075, per output (formed without underflow)
        grid = 2.0 ** -475 / (s * 2.0 ** 600) if s < 1.0 else 0.0
        assert np.linalg.norm(g - want) <= tol(n, np.float64) * np.linalg.norm(want) + 2 * grid * np.sqrt(2 * n)


@pytest.mark.parametrize("n", [16, 256, 2048, 8192])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_infinities_and_nans(n, bad):
    batch = max(3, 4096 // n)
    z = _lines(n, batch, n)
    z[1, n // 3] = bad
    got = _rows(n, z)
    assert not np.isfinite(got[1]).any()
    for b in range(batch):
        if b != 1:
            assert rel_l2(got[b], np.fft.fft(z[b])) <= tol(n, np.float64)


@pytest.mark.parametrize("dims", [(16, 32), (64, 50), (128, 7), (256, 512), (512, 9), (1024, 33), (2048, 6), (4096, 3),
                                  (16, 8, 128), (32, 64, 16)])
def test_columns(dims):
    import torch
    import jtransforms_gb300 as J
    rng = np.random.default_rng(sum(dims))
    z = rng.standard_normal(dims) + 1j * rng.standard_normal(dims)
    f = (J.DoubleFFT_2D if len(dims) == 2 else J.DoubleFFT_3D)(*dims)
    dev = torch.from_numpy(z.view(np.float64).ravel().copy()).cuda()
    f.complexForward(dev)
    got = dev.cpu().numpy().view(np.complex128).reshape(dims)
    assert rel_l2(got, np.fft.fftn(z)) <= tol(z.size, np.float64)
    f.complexInverse(dev, True)
    assert rel_l2(dev.cpu().numpy().view(np.complex128).reshape(dims), z) <= 2 * tol(z.size, np.float64)


@pytest.mark.parametrize("split", [(4, 12, 0), (12, 4, 0), (6, 7, 0), (10, 9, 0), (11, 8, 0), (4, 5, 6), (7, 7, 5)])
@pytest.mark.parametrize("inverse", [False, True])
def test_two_and_three_passes(split, inverse):
    from jtransforms_gb300 import _native as N
    lg = sum(split)
    assert N.load().jt_set_split(N.FLOAT64, lg, *split) == 0
    try:
        z = _lines(1 << lg, 3, lg)
        got = _rows(1 << lg, z, inverse, inverse)
        want = np.fft.ifft(z, axis=1) if inverse else np.fft.fft(z, axis=1)
        for b in range(3):
            assert rel_l2(got[b], want[b]) <= tol(1 << lg, np.float64)
    finally:
        N.load().jt_set_split(N.FLOAT64, lg, -1, 0, 0)


def _r2r_want(kind, fwd, x):
    import scipy.fft as sfft
    if kind == "dht":
        z = np.fft.fft(x, axis=-1)
        return (z.real - z.imag) / (1 if fwd else x.shape[-1])
    return (sfft.dct if kind == "dct" else sfft.dst)(x, type=2 if fwd else 3, norm="ortho", axis=-1)


@pytest.mark.parametrize("lg", range(5, 14))
@pytest.mark.parametrize("kind", ["dct", "dst", "dht"])
@pytest.mark.parametrize("fwd", [True, False])
@pytest.mark.parametrize("off", [0, 1])
def test_r2r_rows(lg, kind, fwd, off):
    """Rows of the half lengths 16..4096, at even and odd offsets, 20 orders
    of magnitude and a row of zeros among them, one row with an infinity."""
    import torch
    from jtransforms_gb300 import _native as N
    n = 1 << lg
    batch = max(4, 9000 // n)
    x = np.random.default_rng(lg).standard_normal((batch, n)) * (10.0 ** np.linspace(-10, 10, batch))[:, None]
    x[2] = 0
    plan = N.Plan({"dct": N.DCT, "dst": N.DST, "dht": N.DHT}[kind], N.FLOAT64, [n])
    for special in (False, True):
        if special:
            x[3, n // 3] = np.inf
        buf = np.full(off + batch * n + 3, 5.0)
        buf[off:off + batch * n] = x.ravel()
        dev = torch.from_numpy(buf).cuda()
        plan.execute(N.FORWARD if fwd else N.INVERSE, dev, off, kind != "dht" or not fwd, batch=batch, dist=n)
        out = dev.cpu().numpy()
        got = out[off:off + batch * n].reshape(batch, n)
        assert np.all(out[:off] == 5.0) and np.all(out[off + batch * n:] == 5.0)
        for b in range(batch):
            if special and b == 3:
                assert not np.isfinite(got[b]).any()
            else:
                assert rel_l2(got[b], _r2r_want(kind, fwd, x[b])) <= tol(n, np.float64)


@pytest.mark.parametrize("n,cols", [(32, 150), (64, 33), (256, 40), (512, 17), (1024, 9), (2048, 6), (4096, 5), (8192, 3)])
@pytest.mark.parametrize("kind", ["dct", "dst", "dht"])
def test_r2r_columns(n, cols, kind):
    import torch
    import jtransforms_gb300 as J
    x = np.random.default_rng(n).standard_normal((n, cols))
    f = getattr(J, "Double%s_2D" % kind.upper())(n, cols)
    dev = torch.from_numpy(x.copy().ravel()).cuda()
    if kind == "dht":
        f.forward(dev)
        z = np.fft.fft2(x)
        want = z.real - z.imag
    else:
        f.forward(dev, True)
        want = _r2r_want(kind, True, _r2r_want(kind, True, x).T).T
    assert rel_l2(dev.cpu().numpy().reshape(n, cols), want) <= tol(x.size, np.float64)
    f.inverse(dev, True)
    assert rel_l2(dev.cpu().numpy().reshape(n, cols), x) <= 2 * tol(x.size, np.float64)


@pytest.mark.parametrize("lg", range(5, 14))
@pytest.mark.parametrize("off", [0, 2])
def test_packed_real_rows(lg, off):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    n = 1 << lg
    batch = max(3, 9000 // n)
    x = np.random.default_rng(lg).standard_normal((batch, n)) * (10.0 ** np.linspace(-10, 10, batch))[:, None]
    f = J.DoubleFFT_1D(n)
    dev = torch.from_numpy(np.concatenate([np.zeros(off), x.ravel()])).cuda()
    f.plan.execute(N.REAL_FORWARD, dev, off, False, batch=batch, dist=n)
    got = dev.cpu().numpy()[off:].reshape(batch, n)
    F = np.fft.rfft(x, axis=1)
    want = np.empty_like(x)
    want[:, 0], want[:, 1] = F[:, 0].real, F[:, n // 2].real
    want[:, 2::2], want[:, 3::2] = F[:, 1:n // 2].real, F[:, 1:n // 2].imag
    for b in range(batch):
        assert rel_l2(got[b], want[b]) <= tol(n, np.float64)
    f.plan.execute(N.REAL_INVERSE, dev, off, True, batch=batch, dist=n)
    back = dev.cpu().numpy()[off:].reshape(batch, n)
    for b in range(batch):
        assert rel_l2(back[b], x[b]) <= 2 * tol(n, np.float64)
