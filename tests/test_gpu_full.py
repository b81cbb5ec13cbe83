"""GPU: realForwardFull / realInverseFull of 2D and 3D arrays. Even rows run
half-length row FFTs, half the columns and the symmetric fill; odd rows the
complex transform. Rows, columns and slices that have a column kernel and such
that go through transposed copies, down to the smallest sizes."""
import numpy as np
import pytest

from tests._helpers import rel_l2, tol

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2), (2, 3), (3, 2), (4, 6), (16, 32), (33, 34), (64, 50), (67, 64), (71, 134), (100, 31), (128, 2048), (1080, 96), (8192, 4),
          (2, 2, 2), (3, 4, 5), (5, 3, 4), (16, 8, 32), (7, 71, 6), (71, 5, 8), (30, 20, 50)]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("op", ["forward", "inverse", "inverse scaled"])
def test_full(prec, shape, op):
    import torch
    import jtransforms_gb300 as J
    dt = np.float32 if prec == "f32" else np.float64
    f = getattr(J, "%sFFT_%dD" % ("Float" if prec == "f32" else "Double", len(shape)))(*shape)
    x = np.random.default_rng(sum(shape)).standard_normal(shape).astype(dt)
    a = np.full(2 * x.size, 7.0, dt)
    a[:x.size] = x.ravel()
    dev = torch.from_numpy(a).cuda()
    if op == "forward":
        f.realForwardFull(dev)
        want = np.fft.fftn(x.astype(np.float64))
    else:
        f.realInverseFull(dev, op == "inverse scaled")
        want = np.fft.ifftn(x.astype(np.float64)) * (1 if op == "inverse scaled" else x.size)
    got = dev.cpu().numpy().astype(np.float64).view(np.complex128).reshape(shape)
    assert rel_l2(got, want) <= tol(x.size, dt)
