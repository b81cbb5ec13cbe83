"""GPU: realForwardFull / realInverseFull of several 2D or 3D arrays in one
call. The arrays' reals begin at the distance of their spectra, 2N, and each
is transformed from its own numbers: even rows whose half length runs in one
kernel, in two passes, as a convolution and as a copy, and odd rows."""
import numpy as np
import pytest

from tests._helpers import rel_l2, tol

pytestmark = pytest.mark.gpu

SHAPES = [(4, 6), (16, 32), (64, 50), (33, 34), (5, 2), (71, 134), (3, 32768), (100, 31),
          (3, 4, 6), (16, 8, 32), (71, 5, 8), (7, 71, 6), (2, 3, 2), (5, 3, 134), (3, 4, 5)]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("op", ["forward", "inverse", "inverse scaled"])
@pytest.mark.parametrize("batch,where", [(3, "device"), (3, "host"), (3, "host apart"), (2, "device")])
def test_full_of_several_arrays(prec, shape, op, batch, where):
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    dt = np.float32 if prec == "f32" else np.float64
    f = getattr(J, "%sFFT_%dD" % ("Float" if prec == "f32" else "Double", len(shape)))(*shape)
    size = int(np.prod(shape))
    # each array of its own magnitude: numbers of another would show
    x = np.random.default_rng(sum(shape)).standard_normal((batch,) + shape) * 10.0 ** np.arange(batch).reshape((-1,) + (1,) * len(shape))
    x = x.astype(dt)
    dist = 2 * size + (6 if where == "host apart" else 0)
    a = np.full((batch, dist), 7.0, dt)
    a[:, :size] = x.reshape(batch, -1)
    code = N.REAL_FORWARD_FULL if op == "forward" else N.REAL_INVERSE_FULL
    if where == "device":
        dev = torch.from_numpy(a.ravel()).cuda()
        f.plan.execute(code, dev, 0, op == "inverse scaled", batch=batch, dist=dist)
        out = dev.cpu().numpy().reshape(batch, dist)
    else:
        out = a.ravel().copy()
        f.plan.execute(code, out, 0, op == "inverse scaled", batch=batch, dist=dist)
        out = out.reshape(batch, dist)
    assert np.all(out[:, 2 * size:] == 7.0)
    for b in range(batch):
        z = x[b].astype(np.float64)
        want = np.fft.fftn(z) if op == "forward" else np.fft.ifftn(z) * (1 if op == "inverse scaled" else size)
        got = np.ascontiguousarray(out[b, :2 * size]).astype(np.float64).view(np.complex128).reshape(shape)
        assert rel_l2(got, want) <= tol(size, dt)


def test_slices_of_several_arrays_share_scratch():
    """71 slices run through a transposed copy (0.6 MB an array) and a
    convolution of 256 (2.1 MB an array): beside the reals of all arrays
    (2.3 MB) that is 5 MB for eight arrays as for one, and 24 MB if each array
    had its own."""
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    shape, batch = (71, 8, 64), 8
    size = int(np.prod(shape))
    f = J.DoubleFFT_3D(*shape)
    x = np.random.default_rng(0).standard_normal((batch,) + shape)
    a = np.zeros((batch, 2 * size))
    a[:, :size] = x.reshape(batch, -1)
    dev = torch.from_numpy(a.ravel()).cuda()
    prev = N.set_option(N.OPT_ARENA_LIMIT_MB, 8)
    try:
        f.plan.execute(N.REAL_FORWARD_FULL, dev, 0, False, batch=batch, dist=2 * size)
    finally:
        N.set_option(N.OPT_ARENA_LIMIT_MB, prev)
    got = dev.cpu().numpy().view(np.complex128).reshape((batch,) + shape)
    for b in range(batch):
        assert rel_l2(got[b], np.fft.fftn(x[b])) <= tol(size, np.float64)
