"""GPU: rounding of single steps of the float transforms, by small kernels
around the library's functions that are compiled when the tests run."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "jt_mixed.cuh"
using namespace jt;
__global__ void split_kernel(const float2 *in, float2 *out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) real_split_pair(in[3 * i], in[3 * i + 1], in[3 * i + 2], 1.0f, out[2 * i], out[2 * i + 1]);
}
__global__ void nine_kernel(const float2 *in, float2 *out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 v[9];
    for (int k = 0; k < 9; k++) v[k] = in[9 * i + k];
    dft_any<9, -1, float, true>(v);
    for (int k = 0; k < 9; k++) out[9 * i + k] = v[k];
}
extern "C" int split(const float2 *in, float2 *out, int n) {
    split_kernel<<<(n + 255) / 256, 256>>>(in, out, n);
    return (int)cudaDeviceSynchronize();
}
extern "C" int nine(const float2 *in, float2 *out, int n) {
    nine_kernel<<<(n + 255) / 256, 256>>>(in, out, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import torch
    from jtransforms_gb300 import build as B
    d = tmp_path_factory.mktemp("floatmath")
    src, so = os.path.join(d, "t.cu"), os.path.join(d, "t.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call([B.nvcc(), *B.ARCH, *B.FLAGS, "-I" + B.CSRC, "-shared", src, "-o", so])
    torch.cuda.init()
    return ctypes.CDLL(so)


def _run(f, z, shape):
    import torch
    dev = torch.from_numpy(np.ascontiguousarray(z).view(np.float32).ravel().copy()).cuda()
    out = torch.empty(2 * int(np.prod(shape)), dtype=torch.float32, device="cuda")
    assert f(ctypes.c_void_p(dev.data_ptr()), ctypes.c_void_p(out.data_ptr()), shape[0]) == 0
    return out.cpu().numpy().view(np.complex64).reshape(shape).astype(np.complex128)


def _complex(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def test_real_split_rounds_once(lib):
    """X_k = (a - i w d) / 2, X_{h-k} = conj(a + i w d) / 2 in each part: one
    rounding of the result, and 2^-44 of the terms for what the corrections'
    own roundings leave (half of them cancel here all but completely)."""
    rng = np.random.default_rng(0)
    n = 40000
    z = _complex(rng, (n, 3))
    z[:, 2] /= np.abs(z[:, 2])
    z[n // 2:, 1] = np.conj(z[n // 2:, 0]) * (1 + 1e-5 * rng.standard_normal(n - n // 2)).astype(np.float32)
    got = _run(lib.split, z, (n, 2))
    zk, zh, w = z.astype(np.complex128).T
    a, d = zk + np.conj(zh), zk - np.conj(zh)
    for g, want in ((got[:, 0], (a - 1j * w * d) / 2), (got[:, 1], np.conj(a + 1j * w * d) / 2)):
        for part in ("real", "imag"):
            e = np.abs(getattr(g, part) - getattr(want, part))
            assert np.all(e <= 2.0 ** -24 * np.abs(getattr(want, part)) + 2.0 ** -44 * (np.abs(a) + np.abs(d)))


def test_nine_points_of_chirped_data(lib):
    """Root mean square error of numbers even in size: one unit roundoff."""
    z = _complex(np.random.default_rng(1), (40000, 9))
    got, want = _run(lib.nine, z, (40000, 9)), np.fft.fft(z.astype(np.complex128), axis=1)
    assert np.linalg.norm(got - want) <= 2.0 ** -24 * np.linalg.norm(want)
