"""GPU: the transforms' kernels may be placed before the kernel ahead of them
has ended (programmatic stream serialisation), and wait for it. Their results
are those of plain stream order: under capture, with kernels of the caller's
around them that use the same attribute and signal early, and on two streams
that wait for each other by events."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (class, sizes, number of calls' arrays, complex): one kernel and chains of
# kernels, of each family; small ones, where blocks come and go the fastest
CASES = [("DoubleFFT_1D", (1024,), 1), ("DoubleFFT_1D", (1024,), 300), ("DoubleFFT_1D", (1 << 14,), 3), ("DoubleFFT_1D", (1000,), 40),
         ("DoubleFFT_1D", (1331,), 9), ("DoubleFFT_1D", (1009,), 5), ("FloatFFT_1D", (1000,), 60), ("FloatFFT_1D", (4096,), 8),
         ("FloatFFT_1D", (1 << 16,), 4), ("FloatFFT_1D", (10007,), 6), ("FloatFFT_1D", (509,), 20), ("FloatFFT_2D", (128, 256), 1),
         ("DoubleDCT_2D", (128, 96), 1), ("DoubleDHT_3D", (16, 32, 16), 1), ("FloatDST_2D", (64, 100), 1)]

SOURCE = r"""
#include <cuda_runtime.h>
// signals at once that the next kernel may come, then waits for the one before, and writes late
__global__ void put_kernel(float *x, const float *src, int n) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int i = 0; i < 20; i++) __nanosleep(1000);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = src[i];
}
__global__ void take_kernel(float *out, const float *x, int n) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = x[i];
}
template <typename K, typename... A> static int launch(K k, int n, void *s, A... a) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((n + 255) / 256);
    c.blockDim = dim3(256);
    c.stream = (cudaStream_t)s;
    c.attrs = &at;
    c.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&c, k, a...);
}
extern "C" int put(float *x, const float *src, int n, void *s) { return launch(put_kernel, n, s, x, src, n); }
extern "C" int take(float *out, const float *x, int n, void *s) { return launch(take_kernel, n, s, out, (const float *)x, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import torch
    from jtransforms_gb300 import build as B
    d = tmp_path_factory.mktemp("order")
    src, so = os.path.join(d, "t.cu"), os.path.join(d, "t.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call([B.nvcc(), *B.ARCH, *B.FLAGS, "-shared", src, "-o", so])
    torch.cuda.init()
    return ctypes.CDLL(so)


def _setup(case):
    """The plan, its two directions as calls on an array, and a block of numbers."""
    import torch
    import jtransforms_gb300 as J
    from jtransforms_gb300 import _native as N
    name, dims, batch = case
    f = getattr(J, name)(*dims)
    fft = "FFT" in name
    size = int(np.prod(dims)) * (2 if fft else 1)
    fwd, inv = (N.COMPLEX_FORWARD, N.COMPLEX_INVERSE) if fft else (N.FORWARD, N.INVERSE)
    dt = torch.float32 if name.startswith("Float") else torch.float64
    x = torch.randn(batch * size, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(size))

    def both(a, count=2):
        for _ in range(count):
            f.plan.execute(fwd, a, 0, False, batch=batch, dist=size)
            f.plan.execute(inv, a, 0, True, batch=batch, dist=size)
        f.plan.execute(fwd, a, 0, False, batch=batch, dist=size)

    want = x.clone()
    both(want)
    torch.cuda.synchronize()
    return x, both, want


@pytest.mark.parametrize("case", CASES, ids=str)
def test_captured(case):
    import torch
    x, both, want = _setup(case)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    a = x.clone()
    with torch.cuda.stream(s):
        both(a)  # the scratch of this thread, last used on this stream
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        a.copy_(x)
        both(a)
        b = a + 1
    for _ in range(3):
        a.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(a, want) and torch.equal(b, want + 1)


@pytest.mark.parametrize("case", CASES, ids=str)
def test_between_kernels_that_signal_early(lib, case):
    import torch
    x, both, want = _setup(case)
    n = x.numel() * x.element_size() // 4
    a = torch.zeros_like(x)
    outs = [torch.zeros_like(x) for _ in range(4)]
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    for out in outs:  # without a wait on the host between
        assert lib.put(ptr(a), ptr(x), n, s) == 0
        both(a)
        assert lib.take(ptr(out), ptr(a), n, s) == 0
    torch.cuda.synchronize()
    for out in outs:
        assert torch.equal(out, want)


@pytest.mark.parametrize("case", CASES, ids=str)
def test_two_streams_that_wait_for_each_other(case):
    import torch
    x, both, want = _setup(case)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    a, outs = torch.zeros_like(x), [torch.zeros_like(x) for _ in range(6)]
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    done.record()
    for i, out in enumerate(outs):
        s = streams[i % 2]
        s.wait_event(done)
        with torch.cuda.stream(s):
            a.copy_(x)
            both(a)
        mid = torch.cuda.Event()
        mid.record(s)
        other = streams[(i + 1) % 2]
        other.wait_event(mid)
        with torch.cuda.stream(other):
            out.copy_(a)
        done = torch.cuda.Event()
        done.record(other)
    torch.cuda.synchronize()
    for out in outs:
        assert torch.equal(out, want)
