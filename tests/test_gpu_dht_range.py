"""GPU: 3D Hartley transforms at the top of the range. An impulse's transform
is its height everywhere; the joining step sums three of four such numbers,
and heights up to a third of the largest number come through it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 4, 7), (4, 6, 8), (16, 32, 64)])
@pytest.mark.parametrize("fwd", [True, False])
@pytest.mark.parametrize("part", [0.2, 0.3, -0.3])
def test_impulses_near_the_largest_number(prec, dims, fwd, part):
    import torch
    import jtransforms_gb300 as J
    dt = np.float32 if prec == "f32" else np.float64
    f = getattr(J, "%sDHT_3D" % ("Float" if prec == "f32" else "Double"))(*dims)
    x = np.zeros(dims, dt)
    x[0, 0, 0] = height = dt(part * float(np.finfo(dt).max))
    dev = torch.from_numpy(x.ravel()).cuda()
    f.forward(dev) if fwd else f.inverse(dev, False)
    got = dev.cpu().numpy()
    assert np.abs(got / height - 1).max() <= 4 * np.finfo(dt).eps * np.log2(x.size)
