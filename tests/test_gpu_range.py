"""GPU: double lines whose own numbers differ in size. The fixed-point passes
hold a line with one exponent, so its large numbers decide how its small ones
are rounded: a spike above noise, a constant, a decay, a wave packet, numbers
over 15 orders of magnitude. The spikes' mantissas (1.0 and 1.41) are about
the best and the worst for that exponent.

Compared in extended precision (np.longdouble). The bound is what an FP64
transform is known by, an RMS error of about u sqrt(log2 n) (u = 2^-53; W. M.
Gentleman and G. Sande, Fast Fourier Transforms for fun and profit, 1966)."""
import numpy as np
import pytest
import scipy.fft as sfft

pytestmark = pytest.mark.gpu

LD, CLD = np.longdouble, np.clongdouble
LINES = ["normal", "spike 1.0 3", "spike 1.41 3", "spike 1.0 9", "spike 1.41 9", "constant 1.0", "constant 1.41", "decay", "packet", "orders"]
B = 6


def _lines(kind, n, cplx, peak=None):
    rng = np.random.default_rng(n)

    def normal():
        z = rng.standard_normal((B, n))
        return z + 1j * rng.standard_normal((B, n)) if cplx else z

    t = np.arange(n) / n
    word = kind.split()
    if word[0] == "spike":
        z = 10.0 ** -int(word[2]) * normal()
        z[np.arange(B), rng.integers(0, n, B) if peak is None else peak] = float(word[1])
        return z
    if word[0] == "constant":
        return float(word[1]) + 1e-8 * normal()
    if kind == "decay":
        return normal() * np.exp(-30 * t)
    if kind == "packet":
        return normal()[:, :1] * np.exp(-((t - 0.4) / 0.1) ** 2 / 2) * (np.exp(0.22j * np.pi * n * t) if cplx else np.cos(0.22 * np.pi * n * t))
    if kind == "orders":
        return normal() * 10.0 ** rng.uniform(-15, 0, (B, n))
    return normal()


def _check(got, want, n):
    err = [float(np.linalg.norm(g - w) / np.linalg.norm(w)) for g, w in zip(got, want)]
    assert np.sqrt(np.mean(np.square(err))) <= 2.0 ** -53 * np.sqrt(np.log2(n))


# power-of-two lines, register passes of small primes, tile passes with primes of 11 to 61
@pytest.mark.parametrize("n", [16, 64, 512, 1024, 4096, 8192, 100, 1000, 3000, 4000, 122, 1331, 1369, 1922, 2809, 3721])
@pytest.mark.parametrize("kind", LINES)
@pytest.mark.parametrize("inverse", [False, True])
def test_complex(n, kind, inverse):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    z = np.ascontiguousarray(_lines(kind, n, True).astype(np.complex128))
    dev = torch.from_numpy(z.view(np.float64).ravel().copy()).cuda()
    J.DoubleFFT_1D(n).plan.execute(N.COMPLEX_INVERSE if inverse else N.COMPLEX_FORWARD, dev, 0, inverse, batch=B, dist=2 * n)
    got = dev.cpu().numpy().view(np.complex128).reshape(B, n).astype(CLD)
    _check(got, (sfft.ifft if inverse else sfft.fft)(z.astype(CLD), axis=1), n)


@pytest.mark.parametrize("n", [32, 512, 1024, 4096, 8192, 200, 2662])
@pytest.mark.parametrize("kind", LINES)
@pytest.mark.parametrize("op", ["dct", "dst", "dht"])
@pytest.mark.parametrize("fwd", [True, False])
def test_real(n, kind, op, fwd):
    import torch
    from jtransforms_gb300 import _native as N
    # (an inverse cosine or sine transform's large number is its first coefficient or the one that takes its place)
    x = _lines(kind, n, False, None if fwd or op == "dht" else 0 if op == "dct" else n - 1)
    dev = torch.from_numpy(x.ravel().copy()).cuda()
    plan = N.Plan({"dct": N.DCT, "dst": N.DST, "dht": N.DHT}[op], N.FLOAT64, [n])
    plan.execute(N.FORWARD if fwd else N.INVERSE, dev, 0, op != "dht" or not fwd, batch=B, dist=n)
    if op == "dht":
        Z = sfft.fft(x.astype(CLD), axis=1)
        want = (Z.real - Z.imag) / LD(1 if fwd else n)
    else:
        want = (sfft.dct if op == "dct" else sfft.dst)(x.astype(LD), type=2 if fwd else 3, norm="ortho", axis=1)
    _check(dev.cpu().numpy().reshape(B, n).astype(LD), want, n)


@pytest.mark.parametrize("n", [32, 512, 4096, 8192])
@pytest.mark.parametrize("kind", LINES)
def test_packed_real(n, kind):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    x = _lines(kind, n, False)
    f = J.DoubleFFT_1D(n)
    dev = torch.from_numpy(x.ravel().copy()).cuda()
    f.plan.execute(N.REAL_FORWARD, dev, 0, False, batch=B, dist=n)
    F = sfft.rfft(x.astype(LD), axis=1)
    want = np.empty((B, n), LD)
    want[:, 0], want[:, 1] = F[:, 0].real, F[:, n // 2].real
    want[:, 2::2], want[:, 3::2] = F[:, 1:n // 2].real, F[:, 1:n // 2].imag
    _check(dev.cpu().numpy().reshape(B, n).astype(LD), want, n)
    # the inverse of the same numbers taken as a packed spectrum
    dev = torch.from_numpy(x.ravel().copy()).cuda()
    f.plan.execute(N.REAL_INVERSE, dev, 0, True, batch=B, dist=n)
    G = np.zeros((B, n // 2 + 1), CLD)
    G[:, 0], G[:, n // 2] = x[:, 0], x[:, 1]
    G[:, 1:n // 2] = x[:, 2::2] + 1j * x[:, 3::2].astype(CLD)
    _check(dev.cpu().numpy().reshape(B, n).astype(LD), sfft.irfft(G, n, axis=1), n)


# one pass, two passes whose columns' outputs take a four-step factor (of 256,
# 64, 256 and, with mixed radices, 200 points), and three
@pytest.mark.parametrize("n,passes", [(256, 1), (4096, 1), (8192, 1), (1000, 1), (3000, 1), (1331, 1),
                                      (1 << 14, 2), (1 << 15, 2), (1 << 18, 2), (50000, 2), (1 << 23, 3)])
def test_impulses(n, passes):
    """An impulse of 1 at j has the roots e^{-2 pi i jk/n} themselves as its
    spectrum. A pass over memory rounds each part to a double, 2^-54 at most,
    and the passes after it turn that error, which makes it sqrt(2) of that at
    most. All else stays below 2^-55: twiddles are right to 2^-62, butterflies
    round at 2^-58, four-step factors, powers of one, add 15 units of 2^-60."""
    bound = (1 + np.sqrt(2) * (passes - 1)) * 2.0 ** -54 + 2.0 ** -55
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    rows = B if n < 1 << 20 else 1
    j = np.random.default_rng(n).integers(0, n, rows)
    z = np.zeros((rows, n), np.complex128)
    z[np.arange(rows), j] = 1
    dev = torch.from_numpy(z.view(np.float64).ravel()).cuda()
    J.DoubleFFT_1D(n).plan.execute(N.COMPLEX_FORWARD, dev, 0, False, batch=rows, dist=2 * n)
    got = dev.cpu().numpy().view(np.complex128).reshape(rows, n)
    for g, at in zip(got, j):
        # eighths of a turn and a rest, so that the argument is exact
        r = (int(at) * np.arange(n)) % n
        o = (8 * r + n // 2) // n
        t = (8 * r - o * n).astype(LD) / LD(4 * n) * LD("3.14159265358979323846264338327950288")
        c, s, h = np.cos(t), np.sin(t), np.sqrt(LD(0.5))
        co = np.array([1, h, 0, -h, -1, -h, 0, h, 1], LD)[o]
        si = np.array([0, h, 1, h, 0, -h, -1, -h, 0], LD)[o]
        assert np.abs(g.real - (co * c - si * s)).max() <= bound
        assert np.abs(g.imag + (si * c + co * s)).max() <= bound
