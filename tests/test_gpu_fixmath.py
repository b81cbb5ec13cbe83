"""GPU: the 64-bit fixed-point arithmetic of the double lines (jt_fixmath.cuh)
against exact integers. A small kernel around its functions is compiled when
the tests run."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "jt_fixmath.cuh"
using namespace jt;
template <int SIGN> __global__ void mul_kernel(const long long *v, const long long *w, long long *out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Fx r = fx_mul<SIGN>(Fx{v[2 * i], v[2 * i + 1]}, fx_as_factor(Fx{w[2 * i], w[2 * i + 1]}));
    out[2 * i] = r.x;
    out[2 * i + 1] = r.y;
}
extern "C" int mul(int sign, const long long *v, const long long *w, long long *out, int n) {
    if (sign < 0) mul_kernel<-1><<<(n + 255) / 256, 256>>>(v, w, out, n);
    else mul_kernel<1><<<(n + 255) / 256, 256>>>(v, w, out, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import torch  # (the CUDA runtime of the process)
    from jtransforms_gb300 import build as B
    d = tmp_path_factory.mktemp("fixmath")
    src, so = os.path.join(d, "t.cu"), os.path.join(d, "t.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call([B.nvcc(), *B.ARCH, *B.FLAGS, "-I" + B.CSRC, "-shared", src, "-o", so])
    torch.cuda.init()
    return ctypes.CDLL(so)


def _dev(values):
    import torch
    return torch.tensor(values, dtype=torch.int64).cuda()


@pytest.mark.parametrize("sign", [-1, 1])
def test_products_with_factors_formed_at_run_time(lib, sign):
    """v w / 4 and v conj(w) / 4 for factors at 2^62, those among them whose
    low halves are the ends of an int's range. A result is rounded once (half
    a unit), leaves the low halves' products out (two of a quarter at most)
    and may have its factor moved by one (v / 2^64, below half a unit): two
    units cover them."""
    rng = np.random.default_rng(1)
    lows = [0, 1, 0x7fffffff, 0x80000000, 0x80000001, 0xffffffff]
    v, w = [], []
    for lx in lows:
        for ly in lows:
            for _ in range(50):
                v.append([int(x) for x in rng.integers(-(1 << 60), 1 << 60, 2)])
                a = rng.uniform(0, 2 * np.pi)
                h = [int(np.floor(f(a) * 2.0 ** 29.99)) for f in (np.cos, np.sin)]
                w.append([(h[0] << 32) + lx, (h[1] << 32) + ly])
    dv, dw, out = _dev(v), _dev(w), _dev(v)
    assert lib.mul(sign, ctypes.c_void_p(dv.data_ptr()), ctypes.c_void_p(dw.data_ptr()), ctypes.c_void_p(out.data_ptr()), len(v)) == 0
    for (x, y), (c, s), (gx, gy) in zip(v, w, out.cpu().tolist()):
        if sign > 0:
            s = -s
        assert abs((gx << 64) - (x * c - y * s)) <= 2 << 64
        assert abs((gy << 64) - (x * s + y * c)) <= 2 << 64
