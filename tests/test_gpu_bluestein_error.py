"""GPU: float transforms of lengths just above a power of two. Their
convolution could be a little over 2n points instead of the power of two near
4n, but its rounding then falls on the n numbers that are kept alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _error(n, batch):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    rng = np.random.default_rng(n)
    z = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(np.complex64)
    dev = torch.from_numpy(z.view(np.float32).ravel().copy()).cuda()
    J.FloatFFT_1D(n).plan.execute(N.COMPLEX_FORWARD, dev, 0, False, batch=batch, dist=2 * n)
    got = dev.cpu().numpy().view(np.complex64).reshape(batch, n).astype(np.complex128)
    want = np.fft.fft(z.astype(np.complex128), axis=1)
    return np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("n", [2053, 4099, 4493])
def test_error_against_one_power_of_two_transform(n):
    """Two FFTs of N points are sqrt(2) times as far off as one where all N
    numbers are kept, and less where about a quarter of them is."""
    lg = int(np.ceil(np.log2(2 * n - 1)))
    assert _error(n, 64) <= 0.95 * np.sqrt(2) * _error(1 << lg, 16)


def _power_of_two_error(n, batch):
    """Of the same numbers through the convolution of the next power of two, with
    the library's transform of that length and tables from FP64."""
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    rng = np.random.default_rng(n)
    z = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(np.complex64)
    L = 1 << int(np.ceil(np.log2(2 * n - 1)))
    b = np.exp(1j * np.pi * (np.arange(n) ** 2 % (2 * n)) / n)
    wrapped = np.zeros(L, np.complex128)
    wrapped[:n] = b
    wrapped[L - n + 1:] = b[:0:-1]
    chirp = torch.from_numpy(b.conj().astype(np.complex64)).cuda()
    spectrum = torch.from_numpy((np.fft.fft(wrapped) / L).astype(np.complex64)).cuda()
    work = torch.zeros(batch, L, dtype=torch.complex64, device="cuda")
    work[:, :n] = torch.from_numpy(z).cuda() * chirp
    plan = J.FloatFFT_1D(L).plan
    flat = torch.view_as_real(work).reshape(-1)
    plan.execute(N.COMPLEX_FORWARD, flat, 0, False, batch=batch, dist=2 * L)
    work *= spectrum
    plan.execute(N.COMPLEX_INVERSE, flat, 0, False, batch=batch, dist=2 * L)
    got = (work[:, :n] * chirp).cpu().numpy().astype(np.complex128)
    want = np.fft.fft(z.astype(np.complex128), axis=1)
    return np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("n", [79, 107, 263, 461, 1997, 2336])
def test_short_lengths_against_power_of_two_convolution(n):
    """4 % of the variance is what the choice allows, 5 % how well it is fitted."""
    assert _error(n, 512) <= np.sqrt(1.04 * 1.05) * _power_of_two_error(n, 512)
