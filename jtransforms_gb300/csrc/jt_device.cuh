// jt_device.cuh -- device code of jtransforms_gb300 (sm_103a).
//
// Kernels:
//   fft_tile_kernel     batched complex FFT of one length L held in shared
//                       memory: self-sorting (Stockham) passes of radix
//                       16/8/4/2/3/5/7 and generic odd radices, strided line
//                       layouts so the same kernel serves contiguous rows,
//                       2D/3D column passes and both passes of the large-N
//                       two-pass (four-step) scheme.  Replaces the Ooura
//                       split-radix tree (utils/CommonUtils.java:708-5749),
//                       bitrv2* and the FFTPACK passes (fft/DoubleFFT_1D.java:
//                       6630-7842).  Lines that no register kernel takes
//                       (jt_stockham.cuh, jt_fix64.cuh, jt_mixed.cuh,
//                       jt_fixmix.cuh); doubles of 48 points and more compute in
//                       fixed point (tile_passes_fx).
//   real_*              real-FFT pack/unpack around a half-length complex FFT
//                       (replaces rftfsub/rftbsub, utils/CommonUtils.java:5750-5830).
//   bluestein_*         chirp multiplies (fft/DoubleFFT_1D.java:1920-2107).
//   dct_* / dht_*       DCT-II/III, DST, DHT pre/post passes around a real FFT
//                       (dct/DoubleDCT_1D.java:169-440, dst/DoubleDST_1D.java,
//                       dht/DoubleDHT_1D.java).
//   rdft2d_kernel, ytransform*_kernel   2D real packing fix-up and DHT nD
//                       combine (fft/DoubleFFT_2D.java:2544, dht/DoubleDHT_3D.java:2314).
//   fill_symmetric_kernel   the right half of a real array's full spectrum
//                       (fillSymmetric, fft/DoubleFFT_2D.java, fft/DoubleFFT_3D.java).
//   transpose_kernel    batched tiled transpose for axis passes.
//   table kernels       FP64 twiddle/chirp generation with sincospi.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "jt_fixmath.cuh"
#include "jt_launch.cuh"

namespace jt {

template <typename T> struct V2;
template <> struct V2<float> { typedef float2 t; };
template <> struct V2<double> { typedef double2 t; };

template <typename T> __host__ __device__ __forceinline__ typename V2<T>::t mk(T x, T y) {
    typename V2<T>::t r;
    r.x = x;
    r.y = y;
    return r;
}

#define C2 typename V2<T>::t

template <typename T> __device__ __forceinline__ C2 cadd(C2 a, C2 b) { return mk<T>(a.x + b.x, a.y + b.y); }
template <typename T> __device__ __forceinline__ C2 csub(C2 a, C2 b) { return mk<T>(a.x - b.x, a.y - b.y); }
template <typename T> __device__ __forceinline__ C2 cmul(C2 a, C2 b) {
    return mk<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
template <typename T> __device__ __forceinline__ C2 cmulc(C2 a, C2 b) {
    return mk<T>(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
template <typename T> __device__ __forceinline__ C2 cscale(C2 a, T s) { return mk<T>(a.x * s, a.y * s); }
template <typename T> __device__ __forceinline__ C2 cconj(C2 a) { return mk<T>(a.x, -a.y); }
// a * (SIGN * i)
template <int SIGN, typename T> __device__ __forceinline__ C2 mul_si(C2 a) {
    return SIGN > 0 ? mk<T>(-a.y, a.x) : mk<T>(a.y, -a.x);
}

// Padded shared-memory index: one spare slot every 16 elements keeps the
// strided butterfly writes free of bank conflicts for 8- and 16-byte elements.
__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }
__host__ __device__ __forceinline__ int padded_len(int L) { return L + (L >> 4) + 1; }

// ---------------------------------------------------------------------------
// Small DFTs in registers.  SIGN = -1: sum v_m e^{-2 pi i km/R}; +1: e^{+}.
// ---------------------------------------------------------------------------
template <int SIGN, typename T> __device__ __forceinline__ void dft2(C2 *v) {
    C2 a = v[0], b = v[1];
    v[0] = cadd<T>(a, b);
    v[1] = csub<T>(a, b);
}

template <int SIGN, typename T> __device__ __forceinline__ void dft4(C2 &v0, C2 &v1, C2 &v2, C2 &v3) {
    C2 t0 = cadd<T>(v0, v2), t1 = csub<T>(v0, v2);
    C2 t2 = cadd<T>(v1, v3), t3 = mul_si<SIGN, T>(csub<T>(v1, v3));
    v0 = cadd<T>(t0, t2);
    v2 = csub<T>(t0, t2);
    v1 = cadd<T>(t1, t3);
    v3 = csub<T>(t1, t3);
}

template <int SIGN, typename T> __device__ __forceinline__ void dft4v(C2 *v) { dft4<SIGN, T>(v[0], v[1], v[2], v[3]); }

// multiply by e^{SIGN * 2 pi i k / 8}
template <int SIGN, int K, typename T> __device__ __forceinline__ C2 w8(C2 a) {
    const T h = (T)0.70710678118654752440084436210484903928;
    if (K == 0) return a;
    if (K == 2) return mul_si<SIGN, T>(a);
    if (K == 1) return SIGN > 0 ? mk<T>(h * (a.x - a.y), h * (a.x + a.y)) : mk<T>(h * (a.x + a.y), h * (a.y - a.x));
    // K == 3: e^{SIGN 3 pi i/4} = (-h, SIGN h)
    return SIGN > 0 ? mk<T>(-h * (a.x + a.y), h * (a.x - a.y)) : mk<T>(h * (a.y - a.x), -h * (a.x + a.y));
}

template <int SIGN, typename T> __device__ __forceinline__ void dft8(C2 *v) {
    C2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    C2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4<SIGN, T>(e0, e1, e2, e3);
    dft4<SIGN, T>(o0, o1, o2, o3);
    o1 = w8<SIGN, 1, T>(o1);
    o2 = w8<SIGN, 2, T>(o2);
    o3 = w8<SIGN, 3, T>(o3);
    v[0] = cadd<T>(e0, o0); v[4] = csub<T>(e0, o0);
    v[1] = cadd<T>(e1, o1); v[5] = csub<T>(e1, o1);
    v[2] = cadd<T>(e2, o2); v[6] = csub<T>(e2, o2);
    v[3] = cadd<T>(e3, o3); v[7] = csub<T>(e3, o3);
}

// radix 16 as 4 x 4 with internal twiddles e^{SIGN 2 pi i jk/16}
template <int SIGN, typename T> __device__ __forceinline__ void dft16(C2 *v) {
    const T c1 = (T)0.92387953251128675612818318939678828682;  // cos(pi/8)
    const T h = (T)0.70710678118654752440084436210484903928;
    // columns: DFT4 over v[j], v[j+4], v[j+8], v[j+12]
#pragma unroll
    for (int j = 0; j < 4; j++) dft4<SIGN, T>(v[j], v[j + 4], v[j + 8], v[j + 12]);
    // element (k, j) at v[j + 4k] takes w^{jk}, w = e^{SIGN i pi/8}, then the
    // rows' DFT4 over j (output index k + 4 j')
    const T s = (T)SIGN;
    // Each row's twiddles are factored so that their products fold into the
    // row butterfly's additions as FMAs (w = c1 (1 + s i tau), w^3 = c1 (tau
    // + s i), w^2 = h (1 + s i), w^6 = h (-1 + s i), w^9 = -c1 (1 + s i tau)):
    // 144 floating-point instructions for the 16 points instead of 160.
    const T tau = (T)0.41421356237309504880168872420969807857;  // tan(pi/8)
    dft4<SIGN, T>(v[0], v[1], v[2], v[3]);
    // t0, t1 = x0 +- g u; t2, t3 = f P, f M: outputs t0 +- f P, t1 +- s i f M
    auto row = [&](int o, C2 t0, C2 t1, C2 P, C2 M, T f) {
        v[o] = mk<T>(fma(f, P.x, t0.x), fma(f, P.y, t0.y));
        v[o + 2] = mk<T>(fma(-f, P.x, t0.x), fma(-f, P.y, t0.y));
        v[o + 1] = mk<T>(fma(-s * f, M.y, t1.x), fma(s * f, M.x, t1.y));
        v[o + 3] = mk<T>(fma(s * f, M.y, t1.x), fma(-s * f, M.x, t1.y));
    };
    {  // k = 1: w^2 v6 = h u, w v5 = c1 p, w^3 v7 = c1 q
        const C2 x0 = v[4], a = v[5], b = v[6], d = v[7];
        const C2 u = mk<T>(b.x - s * b.y, b.y + s * b.x);
        const C2 t0 = mk<T>(fma(h, u.x, x0.x), fma(h, u.y, x0.y)), t1 = mk<T>(fma(-h, u.x, x0.x), fma(-h, u.y, x0.y));
        const C2 p = mk<T>(fma(-s * tau, a.y, a.x), fma(s * tau, a.x, a.y));
        const C2 q = mk<T>(fma(tau, d.x, -s * d.y), fma(tau, d.y, s * d.x));
        row(4, t0, t1, cadd<T>(p, q), csub<T>(p, q), c1);
    }
    {  // k = 2: w^4 v10 = s i v10, w^2 v9 = h A, w^6 v11 = h D
        const C2 x0 = v[8], a = v[9], b = v[10], d = v[11];
        const C2 t0 = mk<T>(x0.x - s * b.y, x0.y + s * b.x), t1 = mk<T>(x0.x + s * b.y, x0.y - s * b.x);
        const C2 A = mk<T>(a.x - s * a.y, a.y + s * a.x);
        const C2 D = mk<T>(-d.x - s * d.y, s * d.x - d.y);
        row(8, t0, t1, cadd<T>(A, D), csub<T>(A, D), h);
    }
    {  // k = 3: w^6 v14 = h u, w^3 v13 = c1 p, w^9 v15 = -c1 q
        const C2 x0 = v[12], a = v[13], b = v[14], d = v[15];
        const C2 u = mk<T>(-b.x - s * b.y, s * b.x - b.y);
        const C2 t0 = mk<T>(fma(h, u.x, x0.x), fma(h, u.y, x0.y)), t1 = mk<T>(fma(-h, u.x, x0.x), fma(-h, u.y, x0.y));
        const C2 p = mk<T>(fma(tau, a.x, -s * a.y), fma(tau, a.y, s * a.x));
        const C2 q = mk<T>(fma(-s * tau, d.y, d.x), fma(s * tau, d.x, d.y));
        row(12, t0, t1, csub<T>(p, q), cadd<T>(p, q), c1);
    }
    // transpose 4x4: out[k + 4 j'] = v[4k + j']
    C2 t[16];
#pragma unroll
    for (int i = 0; i < 16; i++) t[i] = v[i];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) v[k + 4 * j] = t[4 * k + j];
}

template <int SIGN, typename T> __device__ __forceinline__ void dft3(C2 *v) {
    const T c = (T)-0.5, sn = (T)SIGN * (T)0.86602540378443864676372317075293618347;
    C2 t = cadd<T>(v[1], v[2]);
    C2 d = csub<T>(v[1], v[2]);
    C2 m = mk<T>(v[0].x + c * t.x, v[0].y + c * t.y);
    C2 r = mk<T>(-sn * d.y, sn * d.x);  // i*sn*d
    v[0] = cadd<T>(v[0], t);
    v[1] = cadd<T>(m, r);
    v[2] = csub<T>(m, r);
}

template <int SIGN, typename T> __device__ __forceinline__ void dft5(C2 *v) {
    const T c1 = (T)0.30901699437494742410229341718281905886, c2 = (T)-0.80901699437494742410229341718281905886;
    const T s1 = (T)SIGN * (T)0.95105651629515357211643933337938214340, s2 = (T)SIGN * (T)0.58778525229247312916870595463907276860;
    C2 a1 = cadd<T>(v[1], v[4]), b1 = csub<T>(v[1], v[4]);
    C2 a2 = cadd<T>(v[2], v[3]), b2 = csub<T>(v[2], v[3]);
    C2 x0 = v[0];
    C2 m1 = mk<T>(x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y);
    C2 m2 = mk<T>(x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y);
    // i*(s1 b1 + s2 b2), i*(s2 b1 - s1 b2)
    C2 n1 = mk<T>(-(s1 * b1.y + s2 * b2.y), s1 * b1.x + s2 * b2.x);
    C2 n2 = mk<T>(-(s2 * b1.y - s1 * b2.y), s2 * b1.x - s1 * b2.x);
    v[0] = mk<T>(x0.x + a1.x + a2.x, x0.y + a1.y + a2.y);
    v[1] = cadd<T>(m1, n1);
    v[4] = csub<T>(m1, n1);
    v[2] = cadd<T>(m2, n2);
    v[3] = csub<T>(m2, n2);
}

template <int SIGN, typename T> __device__ __forceinline__ void dft7(C2 *v) {
    const T c1 = (T)0.62348980185873353052500488400423981063, c2 = (T)-0.22252093395631440428890256449679475947,
            c3 = (T)-0.90096886790241912623610231950744505117;
    const T s1 = (T)SIGN * (T)0.78183148246802980870844452667405775023, s2 = (T)SIGN * (T)0.97492791218182360701813168299393121723,
            s3 = (T)SIGN * (T)0.43388373911755812047576833284835875461;
    C2 a1 = cadd<T>(v[1], v[6]), b1 = csub<T>(v[1], v[6]);
    C2 a2 = cadd<T>(v[2], v[5]), b2 = csub<T>(v[2], v[5]);
    C2 a3 = cadd<T>(v[3], v[4]), b3 = csub<T>(v[3], v[4]);
    C2 x0 = v[0];
    // k=1: c1 c2 c3 / s1 s2 s3; k=2: c2 c3 c1 / s2 -s3 -s1; k=3: c3 c1 c2 / s3 -s1 s2
    C2 m1 = mk<T>(x0.x + c1 * a1.x + c2 * a2.x + c3 * a3.x, x0.y + c1 * a1.y + c2 * a2.y + c3 * a3.y);
    C2 m2 = mk<T>(x0.x + c2 * a1.x + c3 * a2.x + c1 * a3.x, x0.y + c2 * a1.y + c3 * a2.y + c1 * a3.y);
    C2 m3 = mk<T>(x0.x + c3 * a1.x + c1 * a2.x + c2 * a3.x, x0.y + c3 * a1.y + c1 * a2.y + c2 * a3.y);
    T p1r = s1 * b1.x + s2 * b2.x + s3 * b3.x, p1i = s1 * b1.y + s2 * b2.y + s3 * b3.y;
    T p2r = s2 * b1.x - s3 * b2.x - s1 * b3.x, p2i = s2 * b1.y - s3 * b2.y - s1 * b3.y;
    T p3r = s3 * b1.x - s1 * b2.x + s2 * b3.x, p3i = s3 * b1.y - s1 * b2.y + s2 * b3.y;
    v[0] = mk<T>(x0.x + a1.x + a2.x + a3.x, x0.y + a1.y + a2.y + a3.y);
    v[1] = mk<T>(m1.x - p1i, m1.y + p1r);
    v[6] = mk<T>(m1.x + p1i, m1.y - p1r);
    v[2] = mk<T>(m2.x - p2i, m2.y + p2r);
    v[5] = mk<T>(m2.x + p2i, m2.y - p2r);
    v[3] = mk<T>(m3.x - p3i, m3.y + p3r);
    v[4] = mk<T>(m3.x + p3i, m3.y - p3r);
}

// ---------------------------------------------------------------------------
// fft_tile_kernel
// ---------------------------------------------------------------------------
#define JT_MAX_PASSES 24
#define JT_MAX_GENERIC_RADIX 64

// Where the elements of line b live: element i of line b is at
//   (b / inner) * outer + (b % inner) * istride + i * estride
// (complex-element units).
struct Layout {
    int64_t inner, outer, istride, estride;
};

struct TileParams {
    int L;            // line length
    int npass;
    int radix[JT_MAX_PASSES];
    int C;            // lines per tile
    int64_t nlines;
    Layout lin, lout;
    double scale;     // output multiplier (1 = none), double plans
    float scalef;     // the same for float plans (no FP64 work in float kernels)
    int do_scale;
    int64_t tw_n;     // four-step post twiddle w_{tw_n}^{sign*k*(b % tw_inner)}; 0 = none
    int64_t tw_inner;
    int tw_lo_bits;
};

// b / d and b % d for the non-negative line indices of the kernels: shift and
// mask for a power-of-two d (every power-of-two plan's layouts), 32-bit
// division when both fit, 64-bit otherwise.
__device__ __forceinline__ int64_t div_fast(int64_t b, int64_t d, int64_t *rem) {
    if ((d & (d - 1)) == 0) {
        *rem = b & (d - 1);
        return b >> (__ffsll(d) - 1);
    }
    if (b <= 0x7fffffff && d <= 0x7fffffff) {
        const uint32_t q = (uint32_t)b / (uint32_t)d;
        *rem = b - (int64_t)q * d;
        return q;
    }
    const int64_t q = b / d;
    *rem = b - q * d;
    return q;
}

__device__ __forceinline__ int64_t line_off(const Layout &l, int64_t b) {
    if (l.inner == 1) return b * l.outer;
    int64_t r;
    const int64_t q = div_fast(b, l.inner, &r);
    return q * l.outer + r * l.istride;
}

// One Stockham pass of radix R for every butterfly of the tile.
template <int R, int SIGN, typename T>
__device__ __forceinline__ void pass_r(const C2 *__restrict__ src, C2 *__restrict__ dst, int lines, int L, int Lp, int Ns,
                                       const C2 *__restrict__ W) {
    const int nb = L / R;
    const int total = lines * nb;
    const int step = L / (Ns * R);
    for (int q = threadIdx.x; q < total; q += blockDim.x) {
        int c = q / nb;
        int j = q - c * nb;
        const C2 *s = src + c * Lp;
        C2 v[R];
#pragma unroll
        for (int k = 0; k < R; k++) v[k] = s[pad(j + k * nb)];
        int jm = j % Ns;
        if (jm) {
#pragma unroll
            for (int k = 1; k < R; k++) {
                C2 w = __ldg(&W[jm * k * step]);
                v[k] = SIGN < 0 ? cmul<T>(v[k], w) : cmulc<T>(v[k], w);
            }
        }
        if (R == 2) dft2<SIGN, T>(v);
        else if (R == 3) dft3<SIGN, T>(v);
        else if (R == 4) dft4v<SIGN, T>(v);
        else if (R == 5) dft5<SIGN, T>(v);
        else if (R == 7) dft7<SIGN, T>(v);
        else if (R == 8) dft8<SIGN, T>(v);
        else if (R == 16) dft16<SIGN, T>(v);
        int idxD = (j - jm) * R + jm;
        C2 *d = dst + c * Lp;
#pragma unroll
        for (int k = 0; k < R; k++) d[pad(idxD + k * Ns)] = v[k];
    }
}

// Generic odd radix (11..63) with the line's own roots of unity: W[m * L/R].
template <int SIGN, typename T>
__device__ void pass_generic(const C2 *__restrict__ src, C2 *__restrict__ dst, int lines, int L, int Lp, int Ns, int R,
                             const C2 *__restrict__ W) {
    const int nb = L / R;
    const int total = lines * nb;
    const int step = L / (Ns * R);
    const int rstep = L / R;
    if (total < (int)blockDim.x) {
        // fewer butterflies than threads (a prime line is one butterfly): one
        // thread per output k of a butterfly, each forming its own sum in
        // the same order as below
        const int items = total * R;
        for (int idx = threadIdx.x; idx < items; idx += blockDim.x) {
            const int q = idx / R, k = idx - q * R;
            const int c = q / nb, j = q - c * nb;
            const C2 *s = src + c * Lp;
            const int jm = j % Ns;
            T sr = 0, si = 0;
            int e = 0;  // k m mod R
            for (int m = 0; m < R; m++) {
                C2 x = s[pad(j + m * nb)];
                if (jm && m) {
                    const C2 w = __ldg(&W[jm * m * step]);
                    x = SIGN < 0 ? cmul<T>(x, w) : cmulc<T>(x, w);
                }
                if (m == 0) {
                    sr = x.x;
                    si = x.y;
                } else {
                    C2 w = __ldg(&W[e * rstep]);
                    if (SIGN > 0) w.y = -w.y;
                    sr += x.x * w.x - x.y * w.y;
                    si += x.x * w.y + x.y * w.x;
                }
                e += k;
                if (e >= R) e -= R;
            }
            dst[c * Lp + pad((j - jm) * R + jm + k * Ns)] = mk<T>(sr, si);
        }
        return;
    }
    for (int q = threadIdx.x; q < total; q += blockDim.x) {
        int c = q / nb;
        int j = q - c * nb;
        const C2 *s = src + c * Lp;
        C2 v[JT_MAX_GENERIC_RADIX];
        int jm = j % Ns;
        for (int k = 0; k < R; k++) {
            C2 x = s[pad(j + k * nb)];
            if (jm && k) {
                C2 w = __ldg(&W[jm * k * step]);
                x = SIGN < 0 ? cmul<T>(x, w) : cmulc<T>(x, w);
            }
            v[k] = x;
        }
        int idxD = (j - jm) * R + jm;
        C2 *d = dst + c * Lp;
        for (int k = 0; k < R; k++) {
            T sr = v[0].x, si = v[0].y;
            int e = 0;
            for (int m = 1; m < R; m++) {
                e += k;
                if (e >= R) e -= R;
                C2 w = __ldg(&W[e * rstep]);
                if (SIGN > 0) w.y = -w.y;
                sr += v[m].x * w.x - v[m].y * w.y;
                si += v[m].x * w.y + v[m].y * w.x;
            }
            d[pad(idxD + k * Ns)] = mk<T>(sr, si);
        }
    }
}

// The Stockham passes of a tile: `lines` lines of length L at stride Lp in
// `src`, ping-ponging with `dst`; returns the buffer holding the result.
template <int SIGN, typename T>
__device__ C2 *tile_passes_fp(C2 *src, C2 *dst, int lines, int L, int Lp, int npass, const int *radix, const C2 *__restrict__ W) {
    int Ns = 1;
    for (int ps = 0; ps < npass; ps++) {
        const int R = radix[ps];
        switch (R) {
            case 2: pass_r<2, SIGN, T>(src, dst, lines, L, Lp, Ns, W); break;
            case 3: pass_r<3, SIGN, T>(src, dst, lines, L, Lp, Ns, W); break;
            case 4: pass_r<4, SIGN, T>(src, dst, lines, L, Lp, Ns, W); break;
            case 5: pass_r<5, SIGN, T>(src, dst, lines, L, Lp, Ns, W); break;
            case 7: pass_r<7, SIGN, T>(src, dst, lines, L, Lp, Ns, W); break;
            case 8: pass_r<8, SIGN, T>(src, dst, lines, L, Lp, Ns, W); break;
            case 16: pass_r<16, SIGN, T>(src, dst, lines, L, Lp, Ns, W); break;
            default: pass_generic<SIGN, T>(src, dst, lines, L, Lp, Ns, R, W); break;
        }
        __syncthreads();
        C2 *t = src;
        src = dst;
        dst = t;
        Ns *= R;
    }
    return src;
}

// ---------------------------------------------------------------------------
// The same passes of doubles in 64-bit block fixed point (jt_fixmath.cuh): the
// FP64 pipe, at two instructions a clock and SM, was what they waited for.
// Measured (GB300, 2 M points): n = 122 767 us where FP64 took 2602, 1331 471 /
// 929; DCT of n = 1000 90 / 139.
// ---------------------------------------------------------------------------
// Words per line after the two buffers: three rounds of bits, the exponent,
// the scaling of lines at the ends of the double range.
#define JT_FX_WORDS 5
template <typename T> __host__ __device__ constexpr size_t tile_words() { return sizeof(T) == 8 ? JT_FX_WORDS * sizeof(uint32_t) : 0; }

// Joins x (OR, or the largest) of line c into dst[c]; the lanes of a warp
// mostly share a line.
template <bool MAX> __device__ __forceinline__ void fx_join(uint32_t *dst, int c, uint32_t x) {
    const uint32_t mask = __activemask();
    const int first = __ffs(mask) - 1;
    if (__all_sync(mask, c == __shfl_sync(mask, c, first))) {
        x = MAX ? __reduce_max_sync(mask, x) : __reduce_or_sync(mask, x);
        if ((threadIdx.x & 31) != first) return;
    }
    if (MAX) atomicMax(dst + c, x);
    else atomicOr(dst + c, x);
}

// One pass of radix R: line c's numbers are brought to 60 bits by its bits in
// `bin` (the first pass, Ns = 1, takes them as converted) and divided by 4 by
// their twiddles; the outputs' bits go to `bout`.
template <int R, int SIGN>
__device__ __forceinline__ void fx_pass_r(const Fx *src, Fx *dst, int lines, int L, int Lp, int Ns, const int4 *__restrict__ Wq,
                                          const uint32_t *bin, uint32_t *bout) {
    const int nb = L / R, total = lines * nb, step = L / (Ns * R);
    for (int q = threadIdx.x; q < total; q += blockDim.x) {
        const int c = q / nb, j = q - c * nb;
        const Fx *s = src + c * Lp;
        Fx v[R];
#pragma unroll
        for (int k = 0; k < R; k++) v[k] = s[pad(j + k * nb)];
        const int jm = j % Ns;
        if (Ns > 1) {
            int sh = fx_norm_shift(bin[c]);
            if (sh < 0) {
#pragma unroll
                for (int k = 0; k < R; k++) v[k] = Fx{v[k].x << -sh, v[k].y << -sh};
                sh = 0;
            }
            const long long r1 = fx_half(sh);
            v[0] = fx_shr(v[0], sh + 2, fx_half(sh + 2));
#pragma unroll
            for (int k = 1; k < R; k++) v[k] = fx_mul<SIGN>(fx_shr(v[k], sh, r1), __ldg(&Wq[jm * k * step]));
        }
        fx_dft<R, SIGN>(v);
        uint32_t bits = 0;
        const int idxD = (j - jm) * R + jm;
        Fx *d = dst + c * Lp;
#pragma unroll
        for (int k = 0; k < R; k++) {
            bits |= fx_bits(v[k].x) | fx_bits(v[k].y);
            d[pad(idxD + k * Ns)] = v[k];
        }
        fx_join<false>(bout, c, bits);
    }
}

// A generic odd radix (11..63): one thread per output, whose R products by roots
// are summed with 24 bits below the unit, over 4 (after twiddles that divide by
// nothing).  Its numbers have fx_room's bits less than 60, so that the sum fits.
// (Rounded product by product it was 1.4 to 6 times as far off as FP64 on lines
// with one large number.)
__host__ __device__ constexpr bool fx_generic(int R) { return !(R == 2 || R == 3 || R == 4 || R == 5 || R == 7 || R == 8 || R == 16); }
__host__ __device__ constexpr int fx_room(int R) { return R > 32 ? 2 : R > 16 ? 1 : 0; }
template <int SIGN>
__device__ void fx_pass_generic(const Fx *src, Fx *dst, int lines, int L, int Lp, int Ns, int R, const int4 *__restrict__ Wq,
                                const uint32_t *bin, uint32_t *bout) {
    const int nb = L / R, step = L / (Ns * R), rstep = L / R, items = lines * L;
    for (int idx = threadIdx.x; idx < items; idx += blockDim.x) {
        // neighbouring threads take one output of neighbouring butterflies
        const int c = idx / L, e0 = idx - c * L, k = e0 / nb, j = e0 - k * nb;
        const Fx *s = src + c * Lp;
        const int jm = j % Ns;
        int sh = Ns > 1 ? fx_norm_shift(bin[c]) + fx_room(R) : 0;
        const int left = sh < 0 ? -sh : 0;
        sh = sh < 0 ? 0 : sh;
        const long long r1 = fx_half(sh);
        Fx hi{0, 0}, mid{0, 0};  // of weight 4 and 2^-30 (mid: over 2^8)
        int e = 0;  // k m mod R
        for (int m = 0; m < R; m++) {
            Fx x = s[pad(j + m * nb)];
            x = Fx{x.x << left, x.y << left};
            if (Ns > 1) {
                x = fx_shr(x, sh, r1);
                if (m > 0) x = fx_mul_full<SIGN>(x, __ldg(&Wq[jm * m * step]));
            }
            const int4 w = __ldg(&Wq[e * rstep]);
            const int xh = fx_hi(x.x), xl = fx_lo(x.x), yh = fx_hi(x.y), yl = fx_lo(x.y);
            const int ph = SIGN < 0 ? w.z : -w.z, pl = SIGN < 0 ? w.w : -w.w;
            hi.x = fx_madw(yh, -ph, fx_madw(xh, w.x, hi.x));
            hi.y = fx_madw(xh, ph, fx_madw(yh, w.x, hi.y));
            mid.x += fx_madw(yl, -ph, fx_madw(yh, -pl, fx_madw(xl, w.x, fx_madw(xh, w.y, 0)))) >> 8;
            mid.y += fx_madw(xl, ph, fx_madw(xh, pl, fx_madw(yl, w.x, fx_madw(yh, w.y, 0)))) >> 8;
            e += k;
            if (e >= R) e -= R;
        }
        const Fx sum{hi.x + ((mid.x + (1 << 23)) >> 24), hi.y + ((mid.y + (1 << 23)) >> 24)};
        dst[c * Lp + pad((j - jm) * R + jm + k * Ns)] = sum;
        fx_join<false>(bout, c, fx_bits(sum.x) | fx_bits(sum.y));
    }
}

// `lines` finite lines of doubles in `src` to doubles in the returned buffer.
// Wq: the roots in fixed point.  words: each line's largest number, zero and
// three more (JT_FX_WORDS), each `ws` words apart.
template <int SIGN>
__device__ __forceinline__ double2 *tile_lines_fx(double2 *src, double2 *dst, int lines, int L, int Lp, int npass, const int *radix,
                                                  const int4 *__restrict__ Wq, uint32_t *words, int ws) {
    uint32_t *b0 = words, *b1 = words + ws, *b2 = words + 2 * ws;
    int *ex = reinterpret_cast<int *>(words + 3 * ws), *pre = ex + ws;
    const int tid = threadIdx.x, nt = blockDim.x, tot = lines * L;
    const int low = fx_generic(radix[0]) ? fx_room(radix[0]) - 2 : 0;  // against 58 bits
    for (int c = tid; c < lines; c += nt) {
        const FxLine l = fx_line(b0[c]);
        ex[c] = l.ex + low;
        pre[c] = l.pre;
    }
    __syncthreads();
    Fx *s = reinterpret_cast<Fx *>(src), *d = reinterpret_cast<Fx *>(dst);
    for (int i = tid; i < tot; i += nt) {
        const int c = i / L, at = c * Lp + pad(i - c * L);
        const FxLine l{ex[c], pre[c]};
        double2 x = src[at];
        if (__any_sync(__activemask(), l.pre != 0)) x = cscale<double>(x, fx_pre(l.pre));
        s[at] = Fx{fx_from(x.x, l), fx_from(x.y, l)};
    }
    int Ns = 1;
    for (int ps = 0; ps < npass; ps++) {
        __syncthreads();
        const int R = radix[ps];
        const bool gen = fx_generic(R);
        for (int c = tid; c < lines; c += nt) {
            if (Ns > 1) ex[c] += fx_norm_shift(b0[c]) + 2 + (gen ? fx_room(R) : 0);
            else if (gen) ex[c] += 2;
            b2[c] = 0;
        }
        switch (R) {
            case 2: fx_pass_r<2, SIGN>(s, d, lines, L, Lp, Ns, Wq, b0, b1); break;
            case 3: fx_pass_r<3, SIGN>(s, d, lines, L, Lp, Ns, Wq, b0, b1); break;
            case 4: fx_pass_r<4, SIGN>(s, d, lines, L, Lp, Ns, Wq, b0, b1); break;
            case 5: fx_pass_r<5, SIGN>(s, d, lines, L, Lp, Ns, Wq, b0, b1); break;
            case 7: fx_pass_r<7, SIGN>(s, d, lines, L, Lp, Ns, Wq, b0, b1); break;
            case 8: fx_pass_r<8, SIGN>(s, d, lines, L, Lp, Ns, Wq, b0, b1); break;
            case 16: fx_pass_r<16, SIGN>(s, d, lines, L, Lp, Ns, Wq, b0, b1); break;
            default: fx_pass_generic<SIGN>(s, d, lines, L, Lp, Ns, R, Wq, b0, b1); break;
        }
        Fx *t = s;
        s = d;
        d = t;
        uint32_t *w = b0;
        b0 = b1;
        b1 = b2;
        b2 = w;
        Ns *= R;
    }
    __syncthreads();
    double2 *r = reinterpret_cast<double2 *>(s);
    for (int i = tid; i < tot; i += nt) {
        const int c = i / L, at = c * Lp + pad(i - c * L);
        const Fx x = s[at];
        double2 y = make_double2(fx_to(x.x, ex[c]), fx_to(x.y, ex[c]));
        if (__any_sync(__activemask(), pre[c] != 0)) y = cscale<double>(y, fx_pre(-pre[c]));
        r[at] = y;
    }
    __syncthreads();
    return r;
}

// Doubles in `src` to doubles in the returned buffer.  `words`: JT_FX_WORDS
// per line.  A line with an infinity or a NaN runs tile_passes_fp; its tile
// then goes line by line, so that no finite line's result depends on it.
template <int SIGN>
__device__ __noinline__ double2 *tile_passes_fx(double2 *src, double2 *dst, int lines, int L, int Lp, int npass, const int *radix,
                                                const double2 *__restrict__ W, uint32_t *words) {
    const int tid = threadIdx.x, nt = blockDim.x, tot = lines * L;
    for (int c = tid; c < 2 * lines; c += nt) words[c] = 0;
    __syncthreads();
    bool special = false;
    for (int i = tid; i < tot; i += nt) {
        const int c = i / L;
        const double2 d = src[c * Lp + pad(i - c * L)];
        const uint32_t m = max((uint32_t)__double2hiint(d.x) << 1, (uint32_t)__double2hiint(d.y) << 1);
        special |= m >= 0xffe00000u;
        fx_join<true>(words, c, m);
    }
    const bool one = __syncthreads_or(special);
    const int step = one ? 1 : lines;
    double2 *r = src;
    for (int c = 0; c < lines; c += step) {
        double2 *s = src + c * Lp, *d = dst + c * Lp;
        r = one && words[c] >= 0xffe00000u ? tile_passes_fp<SIGN, double>(s, d, 1, L, Lp, npass, radix, W)
                                           : tile_lines_fx<SIGN>(s, d, step, L, Lp, npass, radix, reinterpret_cast<const int4 *>(W + L), words + c, lines);
        r -= c * Lp;
    }
    return r;
}

// words: tile_words<T>() bytes per line (doubles)
template <int SIGN, typename T>
__device__ __forceinline__ C2 *tile_passes(C2 *src, C2 *dst, int lines, int L, int Lp, int npass, const int *radix,
                                           const C2 *__restrict__ W, C2 *words) {
    // (lines of doubles below 48 have too little arithmetic for the conversions:
    // 65,536 points of n = 24 took 18.7 us against 15.3)
    if constexpr (sizeof(T) == 8) if (L >= 48) return tile_passes_fx<SIGN>(src, dst, lines, L, Lp, npass, radix, W, reinterpret_cast<uint32_t *>(words));
    return tile_passes_fp<SIGN, T>(src, dst, lines, L, Lp, npass, radix, W);
}

// W: e^{-2 pi i t/L}, t < L.  Whi/Wlo: two-level table of the four-step post
// twiddle, e^{-2 pi i t/tw_n} = Whi[t >> lo_bits] * Wlo[t & mask].
// Tile `blk` of a generic line pass, run by the calling CTA with its shared
// memory at `smem_raw` (2 * C * padded L elements).
// FP: FP64 passes for doubles.
template <int SIGN, typename T, bool FP = false>
__device__ void tile_fft_body(const C2 *in, C2 *out, const TileParams &p, const C2 *__restrict__ W, const C2 *__restrict__ Whi,
                              const C2 *__restrict__ Wlo, int64_t blk, unsigned char *smem_raw) {
    const int L = p.L, Lp = padded_len(L);
    C2 *bufA = reinterpret_cast<C2 *>(smem_raw);
    C2 *bufB = bufA + p.C * Lp;
    const int64_t b0 = blk * p.C;
    const int lines = (int)min((int64_t)p.C, p.nlines - b0);
    if (lines <= 0) return;
    const int tot = lines * L;

    // load: contiguous lines read element-fastest; strided lines read
    // line-fastest so neighbouring threads touch neighbouring columns.
    if (p.lin.estride == 1) {
        for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
            int c = idx / L, i = idx - c * L;
            bufA[c * Lp + pad(i)] = in[line_off(p.lin, b0 + c) + i];
        }
    } else {
        for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
            int i = idx / lines, c = idx - i * lines;
            bufA[c * Lp + pad(i)] = in[line_off(p.lin, b0 + c) + (int64_t)i * p.lin.estride];
        }
    }
    __syncthreads();

    const C2 *src;
    if constexpr (FP) src = tile_passes_fp<SIGN, T>(bufA, bufB, lines, L, Lp, p.npass, p.radix, W);
    else src = tile_passes<SIGN, T>(bufA, bufB, lines, L, Lp, p.npass, p.radix, W, bufB + p.C * Lp);

    T sc;
    if constexpr (sizeof(T) == 4) sc = p.scalef;
    else sc = (T)p.scale;
    const bool do_scale = p.do_scale != 0;
    const int64_t lo_mask = ((int64_t)1 << p.tw_lo_bits) - 1;
    if (p.lout.estride == 1) {
        for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
            int c = idx / L, i = idx - c * L;
            C2 v = src[c * Lp + pad(i)];
            if (p.tw_n) {
                int64_t j2;
                div_fast(b0 + c, p.tw_inner, &j2);
                const int64_t t = (int64_t)i * j2;  // i < n1, j2 < n2: below tw_n = n1 n2
                C2 w = cmul<T>(__ldg(&Whi[t >> p.tw_lo_bits]), __ldg(&Wlo[t & lo_mask]));
                v = SIGN < 0 ? cmul<T>(v, w) : cmulc<T>(v, w);
            }
            if (do_scale) v = cscale<T>(v, sc);
            out[line_off(p.lout, b0 + c) + i] = v;
        }
    } else {
        for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
            int i = idx / lines, c = idx - i * lines;
            C2 v = src[c * Lp + pad(i)];
            if (p.tw_n) {
                int64_t j2;
                div_fast(b0 + c, p.tw_inner, &j2);
                const int64_t t = (int64_t)i * j2;  // i < n1, j2 < n2: below tw_n = n1 n2
                C2 w = cmul<T>(__ldg(&Whi[t >> p.tw_lo_bits]), __ldg(&Wlo[t & lo_mask]));
                v = SIGN < 0 ? cmul<T>(v, w) : cmulc<T>(v, w);
            }
            if (do_scale) v = cscale<T>(v, sc);
            out[line_off(p.lout, b0 + c) + (int64_t)i * p.lout.estride] = v;
        }
    }
}

template <int SIGN, typename T>
__global__ void __launch_bounds__(512) fft_tile_kernel(const C2 *in, C2 *out, TileParams p, const C2 *__restrict__ W,
                                                        const C2 *__restrict__ Whi, const C2 *__restrict__ Wlo) {
    pdl_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    tile_fft_body<SIGN, T>(in, out, p, W, Whi, Wlo, (int64_t)blockIdx.x, smem_raw);
}

// ---------------------------------------------------------------------------
// Table generation (FP64, sincospi), rounded to T.
// ---------------------------------------------------------------------------
// A root's cosine or sine times 2^62 as two signed halves, high and low (the
// low half is negated in products: never the lowest int).
__device__ __forceinline__ int2 fx_split(long long v) {
    if ((int)v == INT32_MIN) v++;
    return make_int2((int)(v >> 32) + (int)((uint32_t)v >> 31), (int)v);
}
// e^{-2 pi i num / den}, 0 <= num < den < 2^60, right to a unit or two of 2^-62: the
// factors of jt_fixmath.cuh.  (Taken from doubles they were 2^-54 off, which the
// four-step store's powers of one factor multiplied by up to 15: lines of 2^14
// points were half as far off again as in FP64.)  The angle within its octant
// is a fraction of pi/4, cosine and sine are their power series to x^20 and
// x^21, nested, in 64-bit fractions.
__device__ __forceinline__ int4 fx_root(int64_t num, int64_t den) {
    const int oct = (int)(8 * num / den);
    int64_t rem = 8 * num - oct * den;
    if (oct & 1) rem = den - rem;
    const unsigned long long f = rem == den ? ~0ull : (unsigned long long)(((unsigned __int128)rem << 64) / (unsigned long long)den);
    const unsigned long long x = __umul64hi(f, 0xC90FDAA22168C235ull), y = __umul64hi(x, x), one = 1ull << 63;
    unsigned long long c = one, s = one;
#pragma unroll
    for (int k = 10; k >= 1; k--) {
        c = one - __umul64hi(y, c) / (unsigned)((2 * k - 1) * (2 * k));
        s = one - __umul64hi(y, s) / (unsigned)((2 * k) * (2 * k + 1));
    }
    s = __umul64hi(x, s);
    const long long a = (long long)((c + 1) >> 1), b = (long long)((s + 1) >> 1);
    const bool swap = ((oct + 1) >> 1) & 1;  // octants 1, 2, 5, 6
    const long long co = swap ? b : a, si = swap ? a : b;
    const int2 u = fx_split(oct >= 2 && oct < 6 ? -co : co), v = fx_split(oct >= 4 ? si : -si);
    return make_int4(u.x, u.y, v.x, v.y);
}

// out[t] = e^{-2 pi i t * num / den} for t < count; fixed (double): the same
// roots as fx_root's after them
template <typename T> __global__ void roots_kernel(C2 *out, int64_t count, int64_t num, int64_t den, bool fixed) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= count) return;
    // reduce t*num mod den exactly in integers, then angle = 2 * r / den (in half turns)
    int64_t r = (t * num) % den;
    double s, c;
    sincospi(-2.0 * (double)r / (double)den, &s, &c);
    out[t] = mk<T>((T)c, (T)s);
    if (sizeof(T) == 8 && fixed) reinterpret_cast<int4 *>(out + count)[t] = fx_root(r, den);
}

// Bluestein chirp bk1[i] = e^{i pi (i^2 mod 2n) / n} (fft/DoubleFFT_1D.java:1864-1879)
template <typename T> __global__ void chirp_kernel(C2 *bk1, double2 *b64, int64_t n, int64_t nB) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nB) return;
    // symmetric, 1/nB-scaled chirp in FP64 for bk2 (fft/DoubleFFT_1D.java:1880-1889)
    double2 v = make_double2(0.0, 0.0);
    int64_t src = -1;
    if (i < n) src = i;
    else if (nB - i < n) src = nB - i;
    if (src >= 0) {
        int64_t k = (src * src) % (2 * n);
        double s, c;
        sincospi((double)k / (double)n, &s, &c);
        if (i < n) bk1[i] = mk<T>((T)c, (T)s);
        v = make_double2(c / (double)nB, s / (double)nB);
    }
    b64[i] = v;
}

template <typename T> __global__ void d2t_kernel(C2 *out, const double2 *in, int64_t count) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < count) out[i] = mk<T>((T)in[i].x, (T)in[i].y);
}

// ---------------------------------------------------------------------------
// Bluestein multiplies.  SIGN=-1 forward.
// ---------------------------------------------------------------------------
// tmp[b][i] = a[b][i] * conj(bk1[i]) (forward) or * bk1[i] (inverse), zero padded to nB.
template <int SIGN, typename T>
__device__ __forceinline__ void bluestein_pre_body(const C2 *a, int64_t dist, C2 *tmp, const C2 *__restrict__ bk1, int64_t n, int64_t nB,
                                     int64_t batch, int64_t idx) {
    if (idx >= batch * nB) return;
    int64_t b = idx / nB, i = idx - b * nB;
    C2 v = mk<T>(0, 0);
    if (i < n) {
        C2 x = a[b * dist + i], w = __ldg(&bk1[i]);
        v = SIGN < 0 ? cmulc<T>(x, w) : cmul<T>(x, w);
    }
    tmp[idx] = v;
}

template <int SIGN, typename T>
__global__ void bluestein_pre_kernel(const C2 *a, int64_t dist, C2 *tmp, const C2 *__restrict__ bk1, int64_t n, int64_t nB,
                                     int64_t batch) {
    pdl_begin_few();
    bluestein_pre_body<SIGN, T>(a, dist, tmp, bk1, n, nB, batch, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

template <int SIGN, typename T>
__device__ __forceinline__ void bluestein_mul_body(C2 *tmp, const C2 *__restrict__ bk2, int64_t nB, int64_t total, int64_t idx) {
    if (idx >= total) return;
    C2 w = __ldg(&bk2[idx % nB]);
    tmp[idx] = SIGN < 0 ? cmul<T>(tmp[idx], w) : cmulc<T>(tmp[idx], w);
}

template <int SIGN, typename T>
__global__ void bluestein_mul_kernel(C2 *tmp, const C2 *__restrict__ bk2, int64_t nB, int64_t total) {
    pdl_begin_few();
    bluestein_mul_body<SIGN, T>(tmp, bk2, nB, total, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

template <int SIGN, typename T>
__device__ __forceinline__ void bluestein_post_body(C2 *a, int64_t dist, const C2 *tmp, const C2 *__restrict__ bk1, int64_t n, int64_t nB,
                                      int64_t batch, T scale, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, i = idx - b * n;
    C2 x = tmp[b * nB + i], w = __ldg(&bk1[i]);
    C2 v = SIGN < 0 ? cmulc<T>(x, w) : cmul<T>(x, w);
    if (scale != (T)1) v = cscale<T>(v, scale);
    a[b * dist + i] = v;
}

template <int SIGN, typename T>
__global__ void bluestein_post_kernel(C2 *a, int64_t dist, const C2 *tmp, const C2 *__restrict__ bk1, int64_t n, int64_t nB,
                                      int64_t batch, T scale) {
    pdl_begin_few();
    bluestein_post_body<SIGN, T>(a, dist, tmp, bk1, n, nB, batch, scale, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Real FFT pack / unpack (even n, h = n/2 complex points).
// Wr[k] = e^{-2 pi i k / n}, k <= n/4.
// ---------------------------------------------------------------------------
// X_k from Z (the h-point FFT of z_j = x_2j + i x_2j+1):
//   X_k = 0.5 (Z_k + conj Z_{h-k}) - 0.5 i w (Z_k - conj Z_{h-k})
// with w = e^{-2 pi i k/n} for the forward transform.  The same formula with
// w = e^{+2 pi i k/n} turns the e^{+} h-point FFT into the e^{+} n-point real
// transform (realInverseFull); only the twiddle changes.
template <typename T>
__device__ __forceinline__ void real_split(C2 zk, C2 zh, C2 w, C2 &xk) {
    C2 a = mk<T>((T)0.5 * (zk.x + zh.x), (T)0.5 * (zk.y - zh.y));
    C2 d = mk<T>((T)0.5 * (zk.x - zh.x), (T)0.5 * (zk.y + zh.y));
    C2 wd = cmul<T>(w, d);
    xk = mk<T>(a.x + wd.y, a.y - wd.x);  // a - i * wd
}

// x + y and what its rounding left out
__device__ __forceinline__ float2 two_sum(float x, float y) {
    const float s = __fadd_rn(x, y), t = __fsub_rn(s, x);
    return make_float2(s, __fadd_rn(__fsub_rn(x, __fsub_rn(s, t)), __fsub_rn(y, t)));
}
// The split of a pair: X_k and X_{h-k} = conj(a + i w d) of half-length spectra
// (a, d = Z_k +- conj Z_{h-k}), times s / 2.  Floats carry the roundings of the
// sums and products along: rounded one by one they made a full spectrum from
// half-length rows a few percent further off than the complex transform.
__device__ __forceinline__ void real_split_pair(float2 zk, float2 zh, float2 w, float s, float2 &xk, float2 &xh) {
    const float2 ax = two_sum(zk.x, zh.x), ay = two_sum(zk.y, -zh.y), dx = two_sum(zk.x, -zh.x), dy = two_sum(zk.y, zh.y);
    // wd.x = w.x d.x - w.y d.y, wd.y = w.x d.y + w.y d.x as sums of two floats
    auto dot = [](float a, float2 x, float b, float2 y) {
        const float p = __fmul_rn(a, x.x), q = __fmul_rn(b, y.x);
        const float2 t = two_sum(p, q);
        const float e = fmaf(a, x.x, -p) + fmaf(b, y.x, -q) + t.y;
        return make_float2(t.x, fmaf(a, x.y, fmaf(b, y.y, e)));
    };
    const float2 u = dot(w.x, dx, -w.y, dy), v = dot(w.x, dy, w.y, dx);
    auto add = [&](float2 a, float2 b) {
        const float2 t = two_sum(a.x, b.x);
        return 0.5f * s * (t.x + (t.y + (a.y + b.y)));
    };
    auto neg = [](float2 a) { return make_float2(-a.x, -a.y); };
    xk = make_float2(add(ax, v), add(ay, neg(u)));
    xh = make_float2(add(ax, neg(v)), -add(ay, u));
}
__device__ __forceinline__ void real_split_pair(double2 zk, double2 zh, double2 w, double s, double2 &xk, double2 &xh) {
    real_split<double>(zk, zh, w, xk);
    real_split<double>(zh, zk, make_double2(-w.x, w.y), xh);
    xk = cscale<double>(xk, s);
    xh = cscale<double>(xh, s);
}

// In place: a holds Z (h complex); writes the packed realForward layout.
template <typename T>
__device__ __forceinline__ void real_post_packed_body(T *a, int64_t dist, int64_t n, int64_t batch, const C2 *__restrict__ Wr, int64_t idx) {
    const int64_t h = n / 2, q = h / 2 + 1;  // pairs k = 0..h/2
    if (idx >= batch * q) return;
    int64_t b = idx / q, k = idx - b * q;
    C2 *z = reinterpret_cast<C2 *>(a + b * dist);
    if (k == 0) {
        C2 z0 = z[0];
        z[0] = mk<T>(z0.x + z0.y, z0.x - z0.y);  // a[0] = X0, a[1] = X_{n/2}
        return;
    }
    int64_t k2 = h - k;
    C2 zk = z[k], zh = z[k2];
    C2 w = __ldg(&Wr[k]);
    C2 xk, xh;
    real_split<T>(zk, zh, w, xk);
    if (k2 != k) {
        // w_{h-k} = -conj(w_k)
        real_split<T>(zh, zk, mk<T>(-w.x, w.y), xh);
        z[k2] = xh;
    }
    z[k] = xk;
}

template <typename T>
__global__ void real_post_packed_kernel(T *a, int64_t dist, int64_t n, int64_t batch, const C2 *__restrict__ Wr) {
    pdl_begin_few();
    real_post_packed_body<T>(a, dist, n, batch, Wr, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// Out of place: z (h complex) -> full spectrum F (n complex) in out.
// SIGN=+1 writes the e^{+} transform (z must be the e^{+} FFT), times scale.
template <int SIGN, typename T>
__device__ __forceinline__ void real_post_full_body(const T *zin, int64_t zdist, T *out, int64_t odist, int64_t n, int64_t batch,
                                      const C2 *__restrict__ Wr, T scale, int64_t idx) {
    const int64_t h = n / 2, q = h / 2 + 1;
    if (idx >= batch * q) return;
    int64_t b = idx / q, k = idx - b * q;
    const C2 *z = reinterpret_cast<const C2 *>(zin + b * zdist);
    C2 *F = reinterpret_cast<C2 *>(out + b * odist);
    const T s = scale;
    if (k == 0) {
        C2 z0 = z[0];
        F[0] = mk<T>((z0.x + z0.y) * s, 0);
        F[h] = mk<T>((z0.x - z0.y) * s, 0);
        return;
    }
    int64_t k2 = h - k;
    C2 zk = z[k], zh = z[k2];
    C2 w = __ldg(&Wr[k]);
    if (SIGN > 0) w.y = -w.y;
    C2 xk, xh;
    real_split_pair(zk, zh, w, s, xk, xh);
    F[k] = xk;
    F[n - k] = cconj<T>(xk);
    if (k2 != k) {
        F[k2] = xh;
        F[n - k2] = cconj<T>(xh);
    }
}

template <int SIGN, typename T>
__global__ void real_post_full_kernel(const T *zin, int64_t zdist, T *out, int64_t odist, int64_t n, int64_t batch,
                                      const C2 *__restrict__ Wr, T scale) {
    pdl_begin_few();
    real_post_full_body<SIGN, T>(zin, zdist, out, odist, n, batch, Wr, scale, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// In place: packed spectrum -> Z (h complex) whose e^{+} h-point FFT is
// (n/2) * x interleaved; everything times `mult`.
template <typename T>
__device__ __forceinline__ void real_pre_inverse_body(T *a, int64_t dist, int64_t n, int64_t batch, const C2 *__restrict__ Wr, T mult, int64_t idx) {
    const int64_t h = n / 2, q = h / 2 + 1;
    if (idx >= batch * q) return;
    int64_t b = idx / q, k = idx - b * q;
    C2 *z = reinterpret_cast<C2 *>(a + b * dist);
    const T m = mult;
    if (k == 0) {
        C2 x = z[0];  // (X0, X_{n/2})
        z[0] = mk<T>((T)0.5 * (x.x + x.y) * m, (T)0.5 * (x.x - x.y) * m);
        return;
    }
    int64_t k2 = h - k;
    C2 xk = z[k], xh = z[k2];
    C2 w = __ldg(&Wr[k]);
    w.y = -w.y;  // e^{+2 pi i k/n}
    // Z_k = 0.5 (Xk + conj Xh) + 0.5 i w (Xk - conj Xh)
    auto mkz = [&](C2 p, C2 r, C2 ww) {
        C2 sa = mk<T>((T)0.5 * (p.x + r.x), (T)0.5 * (p.y - r.y));
        C2 d = mk<T>((T)0.5 * (p.x - r.x), (T)0.5 * (p.y + r.y));
        C2 wd = cmul<T>(ww, d);
        return mk<T>((sa.x - wd.y) * m, (sa.y + wd.x) * m);
    };
    C2 zk = mkz(xk, xh, w);
    if (k2 != k) {
        // e^{+2 pi i (h-k)/n} = -conj(w)
        C2 zh = mkz(xh, xk, mk<T>(-w.x, w.y));
        z[k2] = zh;
    }
    z[k] = zk;
}

template <typename T>
__global__ void real_pre_inverse_kernel(T *a, int64_t dist, int64_t n, int64_t batch, const C2 *__restrict__ Wr, T mult) {
    pdl_begin_few();
    real_pre_inverse_body<T>(a, dist, n, batch, Wr, mult, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// Odd-n (and general) helpers working through a full complex buffer.
// tmp[b][i] = (a[b][i], 0)
template <typename T>
__device__ __forceinline__ void real_to_complex_body(const T *a, int64_t dist, C2 *tmp, int64_t n, int64_t batch, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, i = idx - b * n;
    tmp[idx] = mk<T>(a[b * dist + i], (T)0);
}

template <typename T>
__global__ void real_to_complex_kernel(const T *a, int64_t dist, C2 *tmp, int64_t n, int64_t batch) {
    pdl_begin_few();
    real_to_complex_body<T>(a, dist, tmp, n, batch, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// full spectrum F (n complex) -> packed realForward layout (fft/DoubleFFT_1D.java:433-451)
template <typename T>
__device__ __forceinline__ void pack_from_full_body(const C2 *F, T *a, int64_t dist, int64_t n, int64_t batch, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, i = idx - b * n;
    const C2 *f = F + b * n;
    T v;
    if (i == 0) v = f[0].x;
    else if (i == 1) v = (n % 2 == 0) ? f[n / 2].x : f[(n - 1) / 2].y;
    else {
        int64_t k = i / 2;
        v = (i & 1) ? f[k].y : f[k].x;
    }
    a[b * dist + i] = v;
}

template <typename T>
__global__ void pack_from_full_kernel(const C2 *F, T *a, int64_t dist, int64_t n, int64_t batch) {
    pdl_begin_few();
    pack_from_full_body<T>(F, a, dist, n, batch, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// packed -> full Hermitian spectrum
template <typename T>
__device__ __forceinline__ void unpack_to_full_body(const T *a, int64_t dist, C2 *F, int64_t n, int64_t batch, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, k = idx - b * n;
    const T *p = a + b * dist;
    C2 v;
    int64_t kk = k <= n / 2 ? k : n - k;
    if (kk == 0) v = mk<T>(p[0], 0);
    else if (n % 2 == 0 && kk == n / 2) v = mk<T>(p[1], 0);
    else if (n % 2 == 1 && kk == (n - 1) / 2) v = mk<T>(p[2 * kk], p[1]);
    else v = mk<T>(p[2 * kk], p[2 * kk + 1]);
    if (k != kk) v.y = -v.y;
    F[idx] = v;
}

template <typename T>
__global__ void unpack_to_full_kernel(const T *a, int64_t dist, C2 *F, int64_t n, int64_t batch) {
    pdl_begin_few();
    unpack_to_full_body<T>(a, dist, F, n, batch, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// a[b][i] = Re(F[b][i]) * mult
template <typename T>
__device__ __forceinline__ void real_part_body(const C2 *F, T *a, int64_t dist, int64_t n, int64_t batch, T mult, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, i = idx - b * n;
    a[b * dist + i] = F[idx].x * mult;
}

template <typename T>
__global__ void real_part_kernel(const C2 *F, T *a, int64_t dist, int64_t n, int64_t batch, T mult) {
    pdl_begin_few();
    real_part_body<T>(F, a, dist, n, batch, mult, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// Copies batch*len complex (strided) with an optional scale and conjugation.
template <typename T>
__device__ __forceinline__ void copy_complex_body(const C2 *src, int64_t sdist, C2 *dst, int64_t ddist, int64_t len, int64_t batch,
                                    T scale, int conj, int64_t idx) {
    if (idx >= batch * len) return;
    int64_t b = idx / len, i = idx - b * len;
    C2 v = src[b * sdist + i];
    if (conj) v.y = -v.y;
    if (scale != (T)1) v = cscale<T>(v, scale);
    dst[b * ddist + i] = v;
}

template <typename T>
__global__ void copy_complex_kernel(const C2 *src, int64_t sdist, C2 *dst, int64_t ddist, int64_t len, int64_t batch,
                                    T scale, int conj) {
    pdl_begin_few();
    copy_complex_body<T>(src, sdist, dst, ddist, len, batch, scale, conj, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// DCT-II / DCT-III / DST / DHT passes around a real FFT of length n.
// Wd[k] = e^{-i pi k / (2n)}, k < n.
// ---------------------------------------------------------------------------
// v_j = x_2j, v_{n-1-j} = x_2j+1 (DST: odd inputs negated)
template <typename T>
__device__ __forceinline__ void dct2_pre_body(const T *a, int64_t dist, T *v, int64_t vdist, int64_t n, int64_t batch, int dst, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, i = idx - b * n;
    T x = a[b * dist + i];
    int64_t j = (i & 1) ? n - 1 - (i >> 1) : (i >> 1);
    if (dst && (i & 1)) x = -x;
    v[b * vdist + j] = x;
}

template <typename T>
__global__ void dct2_pre_kernel(const T *a, int64_t dist, T *v, int64_t vdist, int64_t n, int64_t batch, int dst) {
    pdl_begin_few();
    dct2_pre_body<T>(a, dist, v, vdist, n, batch, dst, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// reads V_k (k <= n/2 packed, conj-mirrored above)
template <typename T> __device__ __forceinline__ C2 packed_get(const T *p, int64_t n, int64_t k) {
    int64_t kk = k <= n / 2 ? k : n - k;
    C2 v;
    if (kk == 0) v = mk<T>(p[0], 0);
    else if (n % 2 == 0 && kk == n / 2) v = mk<T>(p[1], 0);
    else if (n % 2 == 1 && kk == (n - 1) / 2) v = mk<T>(p[2 * kk], p[1]);
    else v = mk<T>(p[2 * kk], p[2 * kk + 1]);
    if (k != kk) v.y = -v.y;
    return v;
}

// C_k = Re(e^{-i pi k/2n} V_k) * mult (k=0: * mult0); DST writes C_k to n-1-k.
template <typename T>
__device__ __forceinline__ void dct2_post_body(const T *v, int64_t vdist, T *a, int64_t dist, int64_t n, int64_t batch,
                                 const C2 *__restrict__ Wd, T mult, T mult0, int dst, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, k = idx - b * n;
    C2 V = packed_get<T>(v + b * vdist, n, k);
    C2 w = __ldg(&Wd[k]);
    T c = (w.x * V.x - w.y * V.y) * (k == 0 ? mult0 : mult);
    a[b * dist + (dst ? n - 1 - k : k)] = c;
}

template <typename T>
__global__ void dct2_post_kernel(const T *v, int64_t vdist, T *a, int64_t dist, int64_t n, int64_t batch,
                                 const C2 *__restrict__ Wd, T mult, T mult0, int dst) {
    pdl_begin_few();
    dct2_post_body<T>(v, vdist, a, dist, n, batch, Wd, mult, mult0, dst, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// DCT-III: from coefficients b_k (DST: read reversed) build the packed
// spectrum of V_k = e^{i pi k/2n} (C_k - i C_{n-k}), C_k = g_k * b_k with
// g_0 = mult0, g_k = mult.  Thread k <= n/2 writes V_k.
template <typename T>
__device__ __forceinline__ void dct3_pre_body(const T *a, int64_t dist, T *v, int64_t vdist, int64_t n, int64_t batch,
                                const C2 *__restrict__ Wd, T mult, T mult0, int dst, int64_t idx) {
    const int64_t q = n / 2 + 1;
    if (idx >= batch * q) return;
    int64_t b = idx / q, k = idx - b * q;
    const T *p = a + b * dist;
    T *o = v + b * vdist;
    auto coef = [&](int64_t kk) -> T {
        if (kk >= n) return (T)0;
        T x = p[dst ? n - 1 - kk : kk];
        return x * (T)(kk == 0 ? mult0 : mult);
    };
    T ck = coef(k), cnk = k == 0 ? (T)0 : coef(n - k);
    C2 w = __ldg(&Wd[k]);
    w.y = -w.y;  // e^{+i pi k/2n}
    C2 V = cmul<T>(w, mk<T>(ck, -cnk));
    if (k == 0) o[0] = V.x;
    else if (n % 2 == 0 && k == n / 2) o[1] = V.x;
    else if (n % 2 == 1 && k == (n - 1) / 2) { o[2 * k] = V.x; o[1] = V.y; }
    else { o[2 * k] = V.x; o[2 * k + 1] = V.y; }
}

template <typename T>
__global__ void dct3_pre_kernel(const T *a, int64_t dist, T *v, int64_t vdist, int64_t n, int64_t batch,
                                const C2 *__restrict__ Wd, T mult, T mult0, int dst) {
    pdl_begin_few();
    dct3_pre_body<T>(a, dist, v, vdist, n, batch, Wd, mult, mult0, dst, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// x_2j = v_j, x_2j+1 = v_{n-1-j}; DST negates the odd outputs.
template <typename T>
__device__ __forceinline__ void dct3_post_body(const T *v, int64_t vdist, T *a, int64_t dist, int64_t n, int64_t batch, int dst, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, i = idx - b * n;
    int64_t j = (i & 1) ? n - 1 - (i >> 1) : (i >> 1);
    T x = v[b * vdist + j];
    if (dst && (i & 1)) x = -x;
    a[b * dist + i] = x;
}

template <typename T>
__global__ void dct3_post_kernel(const T *v, int64_t vdist, T *a, int64_t dist, int64_t n, int64_t batch, int dst) {
    pdl_begin_few();
    dct3_post_body<T>(v, vdist, a, dist, n, batch, dst, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// H_k = Re X_k - Im X_k from the packed spectrum (dht/DoubleDHT_1D.java:94-159)
template <typename T>
__device__ __forceinline__ void dht_post_body(const T *v, int64_t vdist, T *a, int64_t dist, int64_t n, int64_t batch, T mult, int64_t idx) {
    if (idx >= batch * n) return;
    int64_t b = idx / n, k = idx - b * n;
    C2 X = packed_get<T>(v + b * vdist, n, k);
    a[b * dist + k] = (X.x - X.y) * mult;
}

template <typename T>
__global__ void dht_post_kernel(const T *v, int64_t vdist, T *a, int64_t dist, int64_t n, int64_t batch, T mult) {
    pdl_begin_few();
    dht_post_body<T>(v, vdist, a, dist, n, batch, mult, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// 2D / 3D helpers
// ---------------------------------------------------------------------------
// rdft2d_sub (fft/DoubleFFT_2D.java:2544-2575): isgn=+1 after the column
// pass of realForward, -1 before the column pass of realInverse.
template <typename T>
__global__ void rdft2d_kernel(T *a, int64_t dist, int64_t rows, int64_t cols, int64_t batch, int isgn) {
    pdl_begin_few();
    const int64_t n1h = rows >> 1;
    const int64_t q = n1h > 1 ? n1h - 1 : 0;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= batch * q) return;
    int64_t b = idx / q, i = idx - b * q + 1;
    T *p = a + b * dist;
    int64_t j = rows - i, i1 = i * cols, i2 = j * cols;
    if (isgn < 0) {
        T xi = p[i1] - p[i2];
        p[i1] += p[i2];
        p[i2] = xi;
        xi = p[i2 + 1] - p[i1 + 1];
        p[i1 + 1] += p[i2 + 1];
        p[i2 + 1] = xi;
    } else {
        T a2 = (T)0.5 * (p[i1] - p[i2]);
        p[i2] = a2;
        p[i1] -= a2;
        T b2 = (T)0.5 * (p[i1 + 1] + p[i2 + 1]);
        p[i2 + 1] = b2;
        p[i1 + 1] -= b2;
    }
}

// rdft3d_sub (fft/DoubleFFT_3D.java:6909-7021): the packed columns 0/1 of
// mirror (slice, row) pairs.  One thread per pair (x, y), enumerated as
// (ii < slices/2, kk < rows/2, w in {0,1}); ii = kk = 0 has no pair.  The
// pairs are disjoint, so any order gives the reference's result.
template <typename T>
__global__ void rdft3d_kernel(T *a, int64_t dist, int64_t slices, int64_t rows, int64_t cols, int64_t batch, int isgn) {
    pdl_begin_few();
    const int64_t n1h = slices >> 1, n2h = rows >> 1, ss = rows * cols, rs = cols;
    const int64_t per = n1h * n2h * 2;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= batch * per) return;
    const int64_t b = idx / per;
    int64_t r = idx - b * per;
    const int w = (int)(r & 1);
    r >>= 1;
    const int64_t ii = r / n2h, kk = r - ii * n2h;
    int64_t x, y;
    if (ii > 0) {
        const int64_t i = ii, j = slices - i;
        if (kk == 0) {
            x = i * ss + (w ? n2h * rs : 0);
            y = j * ss + (w ? n2h * rs : 0);
        } else {
            const int64_t k = kk, l = rows - k;
            x = (w ? j : i) * ss + k * rs;
            y = (w ? i : j) * ss + l * rs;
        }
    } else {
        if (kk == 0) return;
        const int64_t k = kk, l = rows - k, base = w ? n1h * ss : 0;
        x = base + k * rs;
        y = base + l * rs;
    }
    T *p = a + b * dist;
    if (isgn < 0) {
        T t = p[x] - p[y];
        p[x] += p[y];
        p[y] = t;
        t = p[y + 1] - p[x + 1];
        p[x + 1] += p[y + 1];
        p[y + 1] = t;
    } else {
        const T y0 = (T)0.5 * (p[x] - p[y]);
        p[y] = y0;
        p[x] -= y0;
        const T y1 = (T)0.5 * (p[x + 1] + p[y + 1]);
        p[y + 1] = y1;
        p[x + 1] -= y1;
    }
}

// DHT yTransform, 2D (dht/DoubleDHT_2D.java:1288-1310): each thread owns one
// (r, c) quadruple with r <= rows/2, c <= cols/2.  Quadruples that alias
// (r or c on a symmetry line) are processed by one thread in the reference's
// order; they never share elements with other quadruples.
template <typename T>
__global__ void ytransform2_kernel(T *a, int64_t rows, int64_t cols) {
    pdl_begin_few();
    int64_t nr = rows / 2 + 1, nc = cols / 2 + 1;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nr * nc) return;
    int64_t r = idx / nc, c = idx - r * nc;
    int64_t mRow = (rows - r) % rows, i1 = r * cols, i2 = mRow * cols;
    int64_t mCol = (cols - c) % cols;
    T A = a[i1 + c], B = a[i2 + c], C = a[i1 + mCol], D = a[i2 + mCol];
    T E = ((A + D) - (B + C)) / (T)2;
    a[i1 + c] = A - E;
    a[i2 + c] = B + E;
    a[i1 + mCol] = C + E;
    a[i2 + mCol] = D - E;
}

// DHT yTransform, 3D (dht/DoubleDHT_3D.java:2314-2356)
template <typename T>
__global__ void ytransform3_kernel(T *a, int64_t slices, int64_t rows, int64_t cols) {
    pdl_begin_few();
    int64_t ns = slices / 2 + 1, nr = rows / 2 + 1, nc = cols / 2 + 1;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= ns * nr * nc) return;
    int64_t s = idx / (nr * nc), rem = idx - s * nr * nc;
    int64_t r = rem / nc, c = rem - r * nc;
    int64_t ss = rows * cols, rs = cols;
    int64_t sC = (slices - s) % slices, i9 = s * ss, i10 = sC * ss;
    int64_t rC = (rows - r) % rows, i11 = r * rs, i12 = rC * rs;
    int64_t cC = (cols - c) % cols;
    int64_t x1 = i9 + i12 + c, x2 = i9 + i11 + cC, x3 = i10 + i11 + c, x4 = i10 + i12 + cC;
    int64_t x5 = i10 + i12 + c, x6 = i10 + i11 + cC, x7 = i9 + i11 + c, x8 = i9 + i12 + cC;
    T A = a[x1], B = a[x2], C = a[x3], D = a[x4], E = a[x5], F = a[x6], G = a[x7], H = a[x8];
    // (A + B + C - D) / 2 and its like, the half already in the last axis' lines:
    // four sums and differences each serve two numbers, two operations a number
    // where the sums by themselves take four, which for doubles bound this
    // kernel (128^3: 19.0 us at the FP64 pipe's two a clock and SM). No sum of
    // two halves leaves the range, and an infinity stays one. Same store order
    // as the reference so aliased slots end with its value.
    const T s1 = A + B, d1 = A - B, s2 = C + D, d2 = C - D, s3 = E + F, d3 = E - F, s4 = G + H, d4 = G - H;
    a[x7] = s1 + d2;
    a[x3] = s3 + d4;
    a[x1] = s4 + d3;
    a[x5] = s2 + d1;
    a[x2] = s4 - d3;
    a[x6] = s2 - d1;
    a[x8] = s1 - d2;
    a[x4] = s3 - d4;
}

// The right half of the spectrum of real data: F[-s][-r][C - k] = conj
// F[s][r][k], 0 < k < C / 2 (C even), per array of S x R x C.
template <typename T> __global__ void fill_symmetric_kernel(C2 *a, int64_t S, int64_t R, int64_t C, int64_t batch) {
    pdl_begin_few();
    const int64_t q = C / 2 - 1, idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= batch * S * R * q) return;
    int64_t k, r, s;
    const int64_t line = div_fast(idx, q, &k), sl = div_fast(line, R, &r), b = div_fast(sl, S, &s);
    k++;
    const C2 v = a[line * C + k];
    const int64_t s2 = s ? S - s : 0, r2 = r ? R - r : 0;
    a[((b * S + s2) * R + r2) * C + C - k] = cconj<T>(v);
}

// out[o][c][r] = in[o][r][c] for a batch of R x C matrices of E-byte
// elements (E = 4, 8 or 16), 32x32 tiles through shared memory.
template <typename E>
__global__ void transpose_kernel(const E *in, E *out, int64_t R, int64_t C, int64_t outer) {
    pdl_begin();
    __shared__ E tile[32][33];
    int64_t tilesC = (C + 31) / 32, tilesR = (R + 31) / 32;
    int64_t t = blockIdx.x;
    int64_t o = t / (tilesC * tilesR);
    int64_t rem = t - o * tilesC * tilesR;
    int64_t tr = rem / tilesC, tc = rem - tr * tilesC;
    if (o >= outer) return;
    const E *src = in + o * R * C;
    E *dstp = out + o * R * C;
    int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    for (int k = 0; k < 32; k += 8) {
        int64_t r = tr * 32 + ty + k, c = tc * 32 + tx;
        if (r < R && c < C) tile[ty + k][tx] = src[r * C + c];
    }
    __syncthreads();
    for (int k = 0; k < 32; k += 8) {
        int64_t c = tc * 32 + ty + k, r = tr * 32 + tx;
        if (r < R && c < C) dstp[c * R + r] = tile[tx][ty + k];
    }
}

template <typename T> __device__ __forceinline__ void scale_body(T *a, int64_t dist, int64_t len, int64_t batch, T s, int64_t idx) {
    if (idx >= batch * len) return;
    int64_t b = idx / len, i = idx - b * len;
    a[b * dist + i] *= (T)s;
}

template <typename T> __global__ void scale_kernel(T *a, int64_t dist, int64_t len, int64_t batch, T s) {
    pdl_begin_few();
    scale_body(a, dist, len, batch, s, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

// a[b][i] = src[b][i] (real, strided)
template <typename T> __device__ __forceinline__ void copy_real_body(const T *src, int64_t sdist, T *dst, int64_t ddist, int64_t len, int64_t batch, int64_t idx) {
    if (idx >= batch * len) return;
    int64_t b = idx / len, i = idx - b * len;
    dst[b * ddist + i] = src[b * sdist + i];
}

template <typename T> __global__ void copy_real_kernel(const T *src, int64_t sdist, T *dst, int64_t ddist, int64_t len, int64_t batch) {
    pdl_begin_few();
    copy_real_body(src, sdist, dst, ddist, len, batch, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}

#undef C2

}  // namespace jt
