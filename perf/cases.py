"""The work that programs have this library do, as cases that can be timed.

Each case is one of five uses of the public entry points:

rows   many 1D transforms of one length in a device array
       (`plan.execute(op, tensor, 0, scale, batch=, dist=)`); one transform
       goes through the class method, as in the reference's API
nd     one 2D or 3D transform of a device array through its class method
full   realForwardFull: n reals in, the full 2n-slot spectrum out
batch  transforms of mixed lengths and kinds as one launch (`Batch.run_graph`)
host   a transform of a numpy array: copied in, transformed, copied back

A pass of rows, nd and host is one forward transform of one array and one
scaled inverse of another: a program that analyses one block while it
synthesises the next.  The transforms work in place, so a pass leaves a
spectrum where the block was and a block where the spectrum was, and the next
pass takes them the other way round: magnitudes stay put however often it
runs.  full and batch refill their arrays from the inputs first.
"""
import math

import numpy as np
import torch

import jtransforms_gb300 as J
from jtransforms_gb300 import _native as N

_CODES = {"cf": N.COMPLEX_FORWARD, "rf": N.REAL_FORWARD, "dct": N.FORWARD}


def listed():
    return [
        # one short transform at a time: a filter or a solver's inner step, where the call itself counts
        dict(name="one_fft_f64_1024", use="rows", t="fft", prec="f64", n0=1024, n1=0, n2=0, batch=1),
        # the reference's plain method on a few hundred arrays
        dict(name="rows_fft_f64_4096", use="rows", t="fft", prec="f64", n0=4096, n1=0, n2=0, batch=256),
        # long power-of-two lines, far beyond one block's shared memory
        dict(name="rows_fft_f32_2p20", use="rows", t="fft", prec="f32", n0=1 << 20, n1=0, n2=0, batch=64),
        # a length of 2s and 5s, as of frames counted in milliseconds, in a few thousand channels
        dict(name="rows_fft_f32_1000", use="rows", t="fft", prec="f32", n0=1000, n1=0, n2=0, batch=32768),
        # a prime length: whatever the caller's data happens to be
        dict(name="rows_fft_f32_10007", use="rows", t="fft", prec="f32", n0=10007, n1=0, n2=0, batch=1024),
        # a float image's packed real spectrum and back: filtering, registration
        dict(name="real_2d_f32_2048", use="nd", t="real", prec="f32", n0=2048, n1=2048, n2=0, batch=1),
        # a double image's cosine transform: compression, Poisson solvers
        dict(name="dct_2d_f64_1024", use="nd", t="dct", prec="f64", n0=1024, n1=1024, n2=0, batch=1),
        # a complex volume in double: spectral solvers
        dict(name="fft_3d_f64_256", use="nd", t="fft", prec="f64", n0=256, n1=256, n2=256, batch=1),
        # a real volume's Hartley transform, whose axes are joined by one more step
        dict(name="dht_3d_f64_128", use="nd", t="dht", prec="f64", n0=128, n1=128, n2=128, batch=1),
        # a video frame's whole spectrum: sides that are no powers of two
        dict(name="full_2d_f32_1080", use="full", t="real", prec="f32", n0=1080, n1=1920, n2=0, batch=1),
        # a thousand transforms of every kind and length in one launch
        dict(name="batch_mixed_1000", use="batch", t="mixed", prec="both", n0=0, n1=0, n2=0, batch=1000),
        # an image in host memory, as the reference's callers hold it
        dict(name="host_fft_2d_f64_256", use="host", t="fft", prec="f64", n0=256, n1=256, n2=0, batch=1),
    ]


def _smooth(lo, hi):
    return sorted(v for v in {2 ** a * 3 ** b * 5 ** c * 7 ** d for a in range(24) for b in range(12) for c in range(8)
                              for d in range(7)} if lo <= v <= hi)


def _is_prime(n):
    return n > 1 and all(n % p for p in range(2, math.isqrt(n) + 1))


def _length(rng, lo, hi, kinds="psor"):
    """A length spread over the logarithm of [lo, hi]: a power of two, a product of 2, 3, 5 and 7, an odd number or a prime."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    kind = rng.choice(kinds)
    if kind == "p":
        n = 2 ** round(math.log2(x))
    elif kind == "s":
        n = min(_smooth(lo, hi), key=lambda v: abs(math.log(v / x)))
    elif kind == "o":
        n = int(x) | 1
    else:
        n = int(x) | 1
        while not _is_prime(n):
            n += 2
    return max(lo, min(hi, n)) if kind != "r" else n


def draw(rng):
    use = rng.choice(["rows"] * 8 + ["nd"] * 6 + ["full"] * 2 + ["batch"] * 1 + ["host"] * 3)
    prec = rng.choice(["f32", "f64"])
    c = dict(use=use, t="fft", prec=prec, n0=0, n1=0, n2=0, batch=1)
    if use == "rows":
        c["t"] = rng.choice(["fft", "fft", "fft", "real", "dct", "dst", "dht"])
        c["n0"] = _length(rng, 16, 1 << 20, "ppssor")
        # from one transform to an array of 16 million (complex float) numbers
        most = 1 << (24 if prec == "f32" else 23)
        total = math.exp(rng.uniform(math.log(c["n0"]), math.log(most)))
        c["batch"] = max(1, round(total / c["n0"]))
    elif use == "nd":
        c["t"] = rng.choice(["fft", "fft", "real", "dct", "dst", "dht"])
        kinds = "p" if c["t"] == "real" else "pppso"  # packed 2D real transforms take powers of two
        if rng.random() < 0.6 or c["t"] == "real":
            c["n0"], c["n1"] = _length(rng, 32, 2048, kinds), _length(rng, 32, 2048, kinds)
        else:
            c["n0"], c["n1"], c["n2"] = (_length(rng, 16, 256, kinds) for _ in range(3))
    elif use == "full":
        c["t"] = "real"
        c["n0"] = _length(rng, 32, 1500, "pso")
        c["n1"] = _length(rng, 32, 1500, "pso") if rng.random() < 0.7 else 0
        if not c["n1"]:
            c["batch"] = rng.randint(1, 2000)
    elif use == "batch":
        c["t"], c["prec"] = "mixed", "both"
        c["batch"] = round(math.exp(rng.uniform(math.log(50), math.log(1000))))
    else:
        c["t"] = rng.choice(["fft", "dct", "dht"])
        if rng.random() < 0.5:
            c["n0"] = _length(rng, 64, 1 << 18, "pso")
        else:
            c["n0"], c["n1"] = _length(rng, 32, 512, "pso"), _length(rng, 32, 512, "pso")
    return c


def _dims(c):
    return [d for d in (c["n0"], c["n1"], c["n2"]) if d]


def _plan(c):
    kind = {"fft": "FFT", "real": "FFT", "dct": "DCT", "dst": "DST", "dht": "DHT"}[c["t"]]
    dims = _dims(c)
    return getattr(J, "%s%s_%dD" % ("Float" if c["prec"] == "f32" else "Double", kind, len(dims)))(*dims)


def _row(c):
    """(values of one transform, distance from one to the next) in scalars."""
    n = math.prod(_dims(c))
    if c["t"] == "fft" or c["use"] == "full":
        return 2 * n, 2 * n
    return n, n + (n & 1) if c["t"] == "real" and c["batch"] > 1 else n


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _image(dims, g, dtype):
    """A sum of Gaussian blobs and a little noise."""
    rows, cols = dims
    y, x = (torch.arange(d, device="cuda", dtype=torch.float64) for d in (rows, cols))
    p = torch.rand(4, 20, 1, generator=g, device="cuda", dtype=torch.float64)
    s = (0.02 + 0.2 * p[2]) * min(rows, cols)
    img = (p[3] * torch.exp(-((y - p[0] * rows) / s) ** 2 / 2)).T @ torch.exp(-((x - p[1] * cols) / s) ** 2 / 2)
    return (img + 0.01 * torch.randn(rows, cols, generator=g, device="cuda", dtype=torch.float64)).to(dtype).reshape(-1)


def _inputs(c, seed):
    """The block that the forward transform takes and the spectrum that the inverse takes."""
    g = _gen(seed)
    dtype = torch.float32 if c["prec"] == "f32" else torch.float64
    dims, dist = _dims(c), _row(c)[1]
    n = math.prod(dims)
    if len(dims) == 2 and c["t"] != "fft":
        x = _image(dims, g, dtype)
    else:
        x = torch.randn(c["batch"] * (n if c["use"] == "full" else dist), generator=g, device="cuda", dtype=dtype)
    if c["use"] == "full":
        return x, None
    y = torch.randn(c["batch"] * dist, generator=g, device="cuda", dtype=dtype)
    if c["t"] in ("fft", "real", "dht"):
        y *= math.sqrt(n)
    return x, y


def _primes_up_to(hi):
    sieve = np.ones(hi + 1, bool)
    sieve[:2] = False
    for i in range(2, math.isqrt(hi) + 1):
        if sieve[i]:
            sieve[i * i::i] = False
    return np.nonzero(sieve)[0]


def _mixed(count):
    """(kind, n, offset, extent) of a mixed batch: lengths log-uniform in
    [16, 65536], 40% powers of two, 40% of 2, 3, 5 and 7, 20% primes; 50%
    complex float, 25% real float, 25% double cosine transforms.  The lengths
    are the caller's own and stay the same; the data changes with the seed."""
    rng = np.random.default_rng(count)
    smooth, primes = np.array(_smooth(16, 65536)), _primes_up_to(65536)[6:]
    at, got = {"f32": 0, "f64": 0}, []
    for _ in range(count):
        x = math.exp(rng.uniform(math.log(16), math.log(65536)))
        k = rng.uniform()
        n = 2 ** round(math.log2(x)) if k < 0.4 else int(smooth[np.argmin(np.abs(smooth - x))]) if k < 0.8 else int(
            primes[np.argmin(np.abs(primes - x))])
        k = rng.uniform()
        kind = "cf" if k < 0.5 else "rf" if k < 0.75 else "dct"
        prec = "f64" if kind == "dct" else "f32"
        ext = 2 * n if kind == "cf" else n
        got.append((kind, n, at[prec], ext))
        at[prec] += (ext + 3) & ~3  # every array starts on a 16-byte boundary
    return got, at


def _mixed_inputs(at, seed):
    g = _gen(seed)
    return [torch.rand(max(at[p], 1), generator=g, device="cuda", dtype=t) * 2 - 1 for p, t in (("f32", torch.float32), ("f64", torch.float64))]


def prepare(case, seed):
    c = case
    if c["use"] == "batch":
        items, at = _mixed(c["batch"])
        x32, x64 = _mixed_inputs(at, seed)
        b32, b64 = torch.empty_like(x32), torch.empty_like(x64)
        plans = {}
        for kind, n, _, _ in items:
            if (kind, n) not in plans:
                plans[kind, n] = N.Plan(N.DCT, N.FLOAT64, [n]) if kind == "dct" else N.Plan(N.FFT, N.FLOAT32, [n])
        batch = N.Batch([(plans[kind, n], _CODES[kind], (b64 if kind == "dct" else b32)[o:], kind == "dct")
                         for kind, n, o, _ in items])
        return dict(case=c, batch=batch, x=(x32, x64), a=(b32, b64))
    x, y = _inputs(c, seed)
    s = dict(case=c, f=_plan(c), x=x, y=y)
    if c["use"] == "host":
        s["x"], s["y"] = x.cpu().numpy(), y.cpu().numpy()
    if c["use"] == "full":
        s["a"] = torch.empty(2 * x.numel(), dtype=x.dtype, device="cuda")
    return s


def _forward(c, f, a):
    if c["t"] == "fft":
        f.complexForward(a)
    elif c["t"] == "real":
        f.realForward(a)
    elif c["t"] == "dht":
        f.forward(a)
    else:
        f.forward(a, True)


def _inverse(c, f, a):
    if c["t"] == "fft":
        f.complexInverse(a, True)
    elif c["t"] == "real":
        f.realInverse(a, True)
    else:
        f.inverse(a, True)


_OPS = {"fft": (N.COMPLEX_FORWARD, N.COMPLEX_INVERSE), "real": (N.REAL_FORWARD, N.REAL_INVERSE)}


def run(state):
    c, s = state["case"], state
    if c["use"] == "batch":
        for a, x in zip(s["a"], s["x"]):
            a.copy_(x)
        s["batch"].run_graph()
        return s["a"]
    if c["use"] == "full":
        a, x = s["a"], s["x"]
        if c["batch"] > 1:
            n = c["n0"]
            a.view(-1, 2 * n)[:, :n].copy_(x.view(-1, n))
            s["f"].plan.execute(N.REAL_FORWARD_FULL, a, 0, False, batch=c["batch"], dist=2 * n)
        else:
            a[:x.numel()].copy_(x)
            s["f"].realForwardFull(a)
        return a
    x, y = s["x"], s["y"]
    if c["batch"] > 1:
        fwd, inv = _OPS.get(c["t"], (N.FORWARD, N.INVERSE))
        dist = _row(c)[1]
        s["f"].plan.execute(fwd, x, 0, c["t"] in ("dct", "dst"), batch=c["batch"], dist=dist)
        s["f"].plan.execute(inv, y, 0, True, batch=c["batch"], dist=dist)
    else:
        _forward(c, s["f"], x)
        _inverse(c, s["f"], y)
    s["x"], s["y"] = y, x
    return x, y


def work(case):
    c = case
    if c["use"] == "batch":
        items, at = _mixed(c["batch"])
        return {"bytes": 2.0 * (4 * at["f32"] + 8 * at["f64"]),
                "flops": float(sum((5.0 if k == "cf" else 2.5) * n * math.log2(n) for k, n, _, _ in items))}
    n, size = math.prod(_dims(c)), 4 if c["prec"] == "f32" else 8
    flops = (5.0 if c["t"] == "fft" else 2.5) * n * math.log2(n) * c["batch"]
    if c["use"] == "full":
        return {"bytes": float(3 * n * size * c["batch"]), "flops": flops}
    return {"bytes": float(4 * _row(c)[0] * size * c["batch"]), "flops": 2 * flops}


# -- the same transforms in 64 bits ------------------------------------------

def _dct2(x, axis):
    x = np.moveaxis(x, axis, -1)
    n = x.shape[-1]
    k = np.arange(n)
    v = np.concatenate([x[..., ::2], x[..., 1::2][..., ::-1]], axis=-1)
    c = (np.fft.fft(v) * np.exp(-0.5j * np.pi * k / n)).real * math.sqrt(2.0 / n)
    c[..., 0] *= math.sqrt(0.5)
    return np.moveaxis(c, -1, axis)


def _dct3(x, axis):
    d = np.moveaxis(x, axis, -1) * 1.0
    n = d.shape[-1]
    k = np.arange(n)
    d *= math.sqrt(n / 2.0)
    d[..., 0] *= math.sqrt(2.0)
    r = np.zeros_like(d)
    r[..., 1:] = d[..., :0:-1]
    v = np.fft.ifft((d - 1j * r) * np.exp(0.5j * np.pi * k / n)).real
    out = np.empty_like(d)
    h = (n + 1) // 2
    out[..., ::2], out[..., 1::2] = v[..., :h], v[..., h:][..., ::-1]
    return np.moveaxis(out, -1, axis)


def _signs(x, axis):
    s = np.ones(x.shape[axis])
    s[1::2] = -1
    return np.moveaxis(np.moveaxis(x, axis, -1) * s, -1, axis)


def _r2r(t, x, inverse):
    axes = tuple(range(1, x.ndim))
    if t == "dht":
        z = np.fft.fftn(x, axes=axes)
        return (z.real - z.imag) / (math.prod(x.shape[1:]) if inverse else 1)
    for ax in axes:
        if t == "dct":
            x = (_dct3 if inverse else _dct2)(x, ax)
        else:
            x = _signs(_dct3(np.flip(x, ax), ax), ax) if inverse else np.flip(_dct2(_signs(x, ax), ax), ax)
    return x


def _pack1(F, n):
    out = np.empty((F.shape[0], n))
    m = (n + 1) // 2
    out[:, 0] = F[:, 0].real
    if n > 1:
        out[:, 1] = F[:, n // 2].real if n % 2 == 0 else F[:, m - 1].imag
    out[:, 2::2] = F[:, 1:1 + out[:, 2::2].shape[1]].real
    out[:, 3::2] = F[:, 1:1 + out[:, 3::2].shape[1]].imag
    return out


def _unpack1(p, n):
    F = np.zeros((p.shape[0], n // 2 + 1), complex)
    F[:, 0] = p[:, 0]
    re, im = p[:, 2::2], p[:, 3::2]
    F[:, 1:1 + re.shape[1]] = re
    F[:, 1:1 + im.shape[1]] += 1j * im
    if n % 2 == 0:
        F[:, n // 2] = p[:, 1]
    elif n > 1:
        F[:, n // 2] += 1j * p[:, 1]
    return F


def _pack2(F, R, C):
    P, h, k = np.empty((R, C)), C // 2, np.arange(1, R // 2)
    P[:, 2::2], P[:, 3::2] = F[:, 1:h].real, F[:, 1:h].imag
    P[k, 0], P[k, 1] = F[k, 0].real, F[k, 0].imag
    P[R - k, 1], P[R - k, 0] = F[k, h].real, -F[k, h].imag
    P[0, 0], P[0, 1], P[R // 2, 0], P[R // 2, 1] = F[0, 0].real, F[0, h].real, F[R // 2, 0].real, F[R // 2, h].real
    return P


def _unpack2(P, R, C):
    F, h, k = np.zeros((R, C // 2 + 1), complex), C // 2, np.arange(1, R // 2)
    F[:, 1:h] = P[:, 2::2] + 1j * P[:, 3::2]
    F[k, 0] = P[k, 0] + 1j * P[k, 1]
    F[k, h] = P[R - k, 1] - 1j * P[R - k, 0]
    F[R - k, 0], F[R - k, h] = np.conj(F[k, 0]), np.conj(F[k, h])
    F[0, 0], F[0, h], F[R // 2, 0], F[R // 2, h] = P[0, 0], P[0, 1], P[R // 2, 0], P[R // 2, 1]
    return F


def _complex(a):
    return np.ascontiguousarray(a).view(np.complex128)


def _exact_one(t, x, inverse, dims):
    """The transform of each row of x (batch x values), rows laid out as the library lays them out."""
    b = x.shape[0]
    axes = tuple(range(1, len(dims) + 1))
    if t == "fft":
        z = _complex(x).reshape([b] + dims)
        z = np.fft.ifftn(z, axes=axes) if inverse else np.fft.fftn(z, axes=axes)
        return np.ascontiguousarray(z).view(np.float64).reshape(b, -1)
    if t == "real":
        if len(dims) == 1:
            n = dims[0]
            return np.fft.irfft(_unpack1(x, n), n) if inverse else _pack1(np.fft.rfft(x), n)
        r, c = dims
        if inverse:
            return np.fft.irfft2(_unpack2(x.reshape(r, c), r, c), (r, c)).reshape(1, -1)
        return _pack2(np.fft.rfft2(x.reshape(r, c)), r, c).reshape(1, -1)
    return _r2r(t, x.reshape([b] + dims), inverse).reshape(b, -1)


def exact(case, seed):
    c = case
    if c["use"] == "batch":
        items, at = _mixed(c["batch"])
        out = [x.double().cpu().numpy() for x in _mixed_inputs(at, seed)]
        for kind, n, o, ext in items:
            a = out[kind == "dct"]
            t = {"cf": "fft", "rf": "real", "dct": "dct"}[kind]
            a[o:o + ext] = _exact_one(t, a[o:o + ext].reshape(1, -1), False, [n])[0]
        return out
    dims = _dims(c)
    ext, dist = _row(c)
    x, y = (None if a is None else a.double().cpu().numpy() for a in _inputs(c, seed))
    if c["use"] == "full":
        z = np.fft.fftn(x.reshape([c["batch"]] + dims), axes=tuple(range(1, len(dims) + 1)))
        return np.ascontiguousarray(z).view(np.float64).reshape(-1)
    for a, inverse in ((x, False), (y, True)):
        rows = a.reshape(c["batch"], dist)
        rows[:, :ext] = _exact_one(c["t"], rows[:, :ext], inverse, dims)
    return x, y
