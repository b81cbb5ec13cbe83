// jt_mixed.cuh -- complex FFT lines of mixed-radix length (prime factors up
// to 13, not a power of two).
//
// A CTA holds C lines.  A length is split into the fewest passes of radix
// 2..16 (1000 = 10 x 10 x 10, where prime factors and powers of two apart take
// 8 x 5 x 5 x 5): composite radices are prime-factor DFTs in registers without
// inner twiddles.  The first pass reads global memory and the last one writes
// it, so a line of P passes crosses shared memory P - 1 times.  Twiddles come
// from a table per length and plan, factor by factor, so that neighbouring
// butterflies read neighbouring entries; indexes are divided by multiplying
// with reciprocals.
//
// Measured (GB300, FloatFFT_1D(1000) x 32768, 262 MB, both directions): 251 us,
// 755 with the tile passes of jt_device.cuh, which crossed shared memory ten
// times, divided by run-time lengths and gathered their twiddles; a
// FloatFFT_2D(1080, 1920).realForwardFull 39 against 128 us (rows of half the
// length and half the columns, since).  Rows move at
// 3.9-5.4 TB/s of 6.8 (one line of 1000 per CTA: 32 warps per SM, waiting for
// their loads a third of the time); lines of 3000 and more, of which one or
// two fit an SM, at 1.9-3.0.
//
// Reference: the FFTPACK passes, fft/DoubleFFT_1D.java:6630-7842.
#pragma once

#include "jt_device.cuh"

namespace jt {

#define JT_MIX_PASSES 8

struct MixParams {
    int L, npass, C;
    int R[JT_MIX_PASSES], Ns[JT_MIX_PASSES], toff[JT_MIX_PASSES];
    uint32_t mNs[JT_MIX_PASSES], mNb[JT_MIX_PASSES];  // floor(2^32 / d) + 1 of Ns and L / R
    uint32_t mC;
    int Lp;                  // line stride in shared memory
    int64_t nlines;
    Layout lin, lout;
    float scale;
    int do_scale;
    int64_t tw_n, tw_inner;  // four-step output twiddle, as StockParams
    int tw_lo_bits;
};

#define C2 typename V2<T>::t

// N1 N2 point DFT, N1 and N2 coprime, by the prime-factor map: inputs N2 n1 +
// N1 n2 (mod N), outputs k with k = k1 (mod N1), k = k2 (mod N2).
template <int N1, int N2, int SIGN, typename T, bool CHIRP> __device__ __forceinline__ void dft_pfa(C2 *v);

// R (9, 11, 13) by sums and differences of mirrored inputs:
// X_k, X_{R-k} = x_0 + sum c_{jk} (x_j + x_{R-j}) +- i sum s_{jk} (x_j - x_{R-j})
template <int R, int SIGN, typename T> __device__ __forceinline__ void dft_mirror(C2 *v) {
    constexpr int H = (R - 1) / 2;
    constexpr double c9[4] = {0.76604444311897803520239265, 0.17364817766693034885171663, -0.5, -0.93969262078590838405410928};
    constexpr double s9[4] = {0.64278760968653932632264341, 0.98480775301220805936674302, 0.86602540378443864676372317,
                              0.34202014332566873304409961};
    constexpr double c11[5] = {0.84125353283118116886181165, 0.41541501300188642552927415, -0.14231483827328514044379267,
                               -0.65486073394528506405692508, -0.95949297361449738989036806};
    constexpr double s11[5] = {0.54064081745559758210763596, 0.90963199535451837141171538, 0.98982144188093273237609204,
                               0.75574957435425828377403584, 0.28173255684142969771141792};
    constexpr double c13[6] = {0.88545602565320989590051945, 0.56806474673115580251180756, 0.12053668025532305334906769,
                               -0.35460488704253562596963789, -0.74851074817110109863463060, -0.97094181742605202715698228};
    constexpr double s13[6] = {0.46472317204376854566001533, 0.82298386589365639457961842, 0.99270887409805399280075165,
                               0.93501624268541482343978459, 0.66312265824079520237678549, 0.23931566428755776714875373};
    C2 a[H], b[H], x0 = v[0];
#pragma unroll
    for (int j = 0; j < H; j++) {
        a[j] = cadd<T>(v[j + 1], v[R - 1 - j]);
        b[j] = csub<T>(v[j + 1], v[R - 1 - j]);
    }
#pragma unroll
    for (int k = 1; k <= H; k++) {
        T mr = x0.x, mi = x0.y, nr = 0, ni = 0;
#pragma unroll
        for (int j = 1; j <= H; j++) {
            const int e = (j * k) % R, f = (e <= H ? e : R - e) - 1;
            if (e == 0) {  // (9: j = k = 3)
                mr += a[j - 1].x;
                mi += a[j - 1].y;
                continue;
            }
            const T c = (T)(R == 9 ? c9[f] : R == 11 ? c11[f] : c13[f]);
            const T s = (T)((e <= H ? 1 : -1) * SIGN * (R == 9 ? s9[f] : R == 11 ? s11[f] : s13[f]));
            mr += c * a[j - 1].x;
            mi += c * a[j - 1].y;
            nr += s * b[j - 1].x;
            ni += s * b[j - 1].y;
        }
        v[k] = mk<T>(mr - ni, mi + nr);
        v[R - k] = mk<T>(mr + ni, mi - nr);
    }
#pragma unroll
    for (int j = 0; j < H; j++) x0 = cadd<T>(x0, a[j]);
    v[0] = x0;
}

// 3 x 3 with the inner twiddles w, w^2, w^4 of e^{SIGN 2 pi i/9}
template <int SIGN, typename T> __device__ __forceinline__ void dft9(C2 *v) {
    const C2 w1 = mk<T>((T)0.76604444311897803520239265, (T)SIGN * (T)0.64278760968653932632264341);
    const C2 w2 = mk<T>((T)0.17364817766693034885171663, (T)SIGN * (T)0.98480775301220805936674302);
    const C2 w4 = mk<T>((T)-0.93969262078590838405410928, (T)SIGN * (T)0.34202014332566873304409961);
    C2 t[3][3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        C2 u[3] = {v[j], v[j + 3], v[j + 6]};
        dft3<SIGN, T>(u);
#pragma unroll
        for (int k = 0; k < 3; k++) t[k][j] = u[k];
    }
    t[1][1] = cmul<T>(t[1][1], w1);
    t[1][2] = cmul<T>(t[1][2], w2);
    t[2][1] = cmul<T>(t[2][1], w2);
    t[2][2] = cmul<T>(t[2][2], w4);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        dft3<SIGN, T>(t[k]);
#pragma unroll
        for (int m = 0; m < 3; m++) v[k + 3 * m] = t[k][m];
    }
}

// CHIRP: nine points by dft_mirror, whose sums have fewer roundings than 3 x 3:
// chirped data is even in size, and a transform of 10007 points around 16 x 9 x
// 16 x 9 came out 2.06e-7 off instead of 2.26e-7 (2.19e-7 around a power of
// two). Lines with a large mean are better off with 3 x 3, where it cancels.
template <int R, int SIGN, typename T, bool CHIRP = false> __device__ __forceinline__ void dft_any(C2 *v) {
    if constexpr (R == 2) dft2<SIGN, T>(v);
    else if constexpr (R == 3) dft3<SIGN, T>(v);
    else if constexpr (R == 4) dft4v<SIGN, T>(v);
    else if constexpr (R == 5) dft5<SIGN, T>(v);
    else if constexpr (R == 6) dft_pfa<2, 3, SIGN, T, CHIRP>(v);
    else if constexpr (R == 7) dft7<SIGN, T>(v);
    else if constexpr (R == 8) dft8<SIGN, T>(v);
    else if constexpr (R == 9 && !CHIRP) dft9<SIGN, T>(v);
    else if constexpr (R == 10) dft_pfa<2, 5, SIGN, T, CHIRP>(v);
    else if constexpr (R == 12) dft_pfa<4, 3, SIGN, T, CHIRP>(v);
    else if constexpr (R == 14) dft_pfa<2, 7, SIGN, T, CHIRP>(v);
    else if constexpr (R == 15) dft_pfa<3, 5, SIGN, T, CHIRP>(v);
    else if constexpr (R == 16) dft16<SIGN, T>(v);
    else dft_mirror<R, SIGN, T>(v);
}

template <int N1, int N2, int SIGN, typename T, bool CHIRP> __device__ __forceinline__ void dft_pfa(C2 *v) {
    constexpr int N = N1 * N2;
    C2 a[N1][N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) {
        C2 t[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) t[n1] = v[(N2 * n1 + N1 * n2) % N];
        dft_any<N1, SIGN, T, CHIRP>(t);
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) a[n1][n2] = t[n1];
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) dft_any<N2, SIGN, T, CHIRP>(a[k1]);
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = a[k % N1][k % N2];
}

// Twiddles of one butterfly: the table of a pass (mix_table_kernel) holds its
// factors in pairs (1, 2), (3, 4), ... of Ns entries each and, for an even
// radix, the last factor's Ns entries after them.
template <int R, int SIGN> __device__ __forceinline__ void mix_twiddle(float2 *v, const float2 *__restrict__ tw, int Ns, int jm) {
    auto mul = [](float2 x, float wx, float wy) {
        const float2 w = make_float2(wx, wy);
        return SIGN < 0 ? cmul<float>(x, w) : cmulc<float>(x, w);
    };
    const float2 *t = tw + 2 * jm;
#pragma unroll
    for (int k = 1; k + 1 < R; k += 2) {
        const float4 w = __ldg(reinterpret_cast<const float4 *>(t));
        v[k] = mul(v[k], w.x, w.y);
        v[k + 1] = mul(v[k + 1], w.z, w.w);
        t += 2 * Ns;
    }
    if (R % 2 == 0) {
        const float2 w = __ldg(t - jm);
        v[R - 1] = mul(v[R - 1], w.x, w.y);
    }
}

// Bluestein transforms of n points around a convolution of N = n1 n2 points
// (jt_bluemix.cuh): the chirp bk1 multiplies input and output (conjugated
// forwards), both of which end at n; columns are c < n2.
struct MixBlue {
    int n, n2, inv;
    int64_t din, dout;  // distance of transforms
    float scale;
    const float2 *bk1;
    const float2 *tw;   // w_N^{k1 c} at [k1 n2 + c]
};
enum { MIX_PLAIN = 0, MIX_BLUE_IN = 1, MIX_BLUE_OUT = 2 };

__device__ __forceinline__ float2 mix_chirp(float2 x, const MixBlue &bl, int i) {
    const float2 w = __ldg(&bl.bk1[i]);
    return bl.inv ? cmul<float>(x, w) : cmulc<float>(x, w);
}

// What the passes of one launch share.  POL: MIX_BLUE_IN loads chirped
// columns of the caller's lines, MIX_BLUE_OUT multiplies its columns with the
// conjugate four-step twiddle on the load and stores chirped lines (both take
// that twiddle from a whole table).
template <int SIGN, int MODE, int POL = MIX_PLAIN> struct MixTile {
    const float2 *in;
    float2 *out;
    const MixParams &p;
    const float2 *tw, *Whi, *Wlo;
    int64_t b0;
    int lines;
    MixBlue bl;

    // The butterflies of pass ps: from global memory (FIRST) or src, to global
    // memory (LAST) or dst.  Strided lines are walked lines first.
    template <int R, bool FIRST, bool LAST> __device__ __forceinline__ void pass(int ps, const float2 *src, float2 *dst) const {
        constexpr bool COLS = MODE == 1 || (MODE == 2 && LAST);
        const int nb = p.L / R, Ns = p.Ns[ps], Lp = p.Lp;
        const uint32_t mNb = p.mNb[ps], mNs = p.mNs[ps];
        const int total = (COLS ? p.C : lines) * nb;
        const float2 *twp = tw + p.toff[ps];
        for (int q = threadIdx.x; q < total; q += blockDim.x) {
            int c, j;
            if (COLS) {
                j = p.C == 1 ? q : (int)__umulhi((uint32_t)q, p.mC);
                c = q - j * p.C;
                if (c >= lines) continue;
            } else {
                c = nb == 1 ? q : (int)__umulhi((uint32_t)q, mNb);
                j = q - c * nb;
            }
            float2 v[R];
            if (FIRST && POL == MIX_BLUE_IN) {
                int64_t col;
                const int64_t tr = div_fast(b0 + c, bl.n2, &col);
                const float2 *g = in + tr * bl.din;
                int i = j * bl.n2 + (int)col;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    v[k] = i < bl.n ? mix_chirp(g[i], bl, i) : make_float2(0, 0);
                    i += nb * bl.n2;
                }
            } else if (FIRST) {
                const int64_t es = MODE == 1 ? p.lin.estride : 1, step = nb * es;
                const float2 *g = in + line_off(p.lin, b0 + c) + j * es;
#pragma unroll
                for (int k = 0; k < R; k++) v[k] = g[k * step];
                if (POL == MIX_BLUE_OUT) {
                    int64_t col;
                    div_fast(b0 + c, bl.n2, &col);
                    const float2 *w = bl.tw + j * bl.n2 + col;
#pragma unroll
                    for (int k = 0; k < R; k++) v[k] = cmulc<float>(v[k], __ldg(w + k * nb * bl.n2));
                }
            } else {
                const float2 *s = src + c * Lp + j;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    v[k] = *s;
                    s += nb;
                }
            }
            int base = j * R;
            if (!FIRST) {
                const int jm = LAST ? j : j - (int)__umulhi((uint32_t)j, mNs) * Ns;  // (the last pass: Ns = L / R)
                base -= jm * (R - 1);
                mix_twiddle<R, SIGN>(v, twp, Ns, jm);
            }
            dft_any<R, SIGN, float, POL != MIX_PLAIN>(v);
            if (LAST && POL == MIX_BLUE_OUT) {
                int64_t col;
                const int64_t tr = div_fast(b0 + c, bl.n2, &col);
                float2 *g = out + tr * bl.dout;
                int i = base * bl.n2 + (int)col;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    if (i < bl.n) g[i] = cscale<float>(mix_chirp(v[k], bl, i), bl.scale);
                    i += Ns * bl.n2;
                }
            } else if (LAST) {
                const int64_t es = MODE != 0 ? p.lout.estride : 1, step = Ns * es;
                float2 *g = out + line_off(p.lout, b0 + c) + base * es;
                if (POL == MIX_BLUE_IN) {
                    int64_t col;
                    div_fast(b0 + c, bl.n2, &col);
                    const float2 *w = bl.tw + base * bl.n2 + col;
#pragma unroll
                    for (int k = 0; k < R; k++) v[k] = cmul<float>(v[k], __ldg(w + k * Ns * bl.n2));
                } else if (p.tw_n) {
                    // i < n1 and the line's column below n2: the products stay below tw_n = n1 n2 < 2^31
                    int64_t j2;
                    div_fast(b0 + c, p.tw_inner, &j2);
                    uint32_t e = (uint32_t)base * (uint32_t)j2;
                    const uint32_t de = (uint32_t)Ns * (uint32_t)j2, mask = (1u << p.tw_lo_bits) - 1u;
#pragma unroll
                    for (int k = 0; k < R; k++) {
                        const float2 w = cmul<float>(__ldg(&Whi[e >> p.tw_lo_bits]), __ldg(&Wlo[e & mask]));
                        v[k] = SIGN < 0 ? cmul<float>(v[k], w) : cmulc<float>(v[k], w);
                        e += de;
                    }
                }
                if (p.do_scale) {
#pragma unroll
                    for (int k = 0; k < R; k++) v[k] = cscale<float>(v[k], p.scale);
                }
#pragma unroll
                for (int k = 0; k < R; k++) g[k * step] = v[k];
            } else {
                float2 *d = dst + c * Lp + base;
                const int step = FIRST ? 1 : Ns;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    *d = v[k];
                    d += step;
                }
            }
        }
    }

    template <bool FIRST, bool LAST> __device__ __forceinline__ void any(int ps, const float2 *src, float2 *dst) const {
        switch (p.R[ps]) {
#define JT_MIX(RR) \
    case RR: pass<RR, FIRST, LAST>(ps, src, dst); break;
            JT_MIX(2) JT_MIX(3) JT_MIX(4) JT_MIX(5) JT_MIX(6) JT_MIX(7) JT_MIX(8) JT_MIX(9) JT_MIX(10) JT_MIX(11) JT_MIX(12)
            JT_MIX(13) JT_MIX(14) JT_MIX(15) JT_MIX(16)
#undef JT_MIX
        }
    }

    // Two passes and more through the buffers A and B (B only for three and
    // more); MODE 1 also one pass, between global memory.
    __device__ __forceinline__ void run(float2 *A, float2 *B) const {
        if (MODE == 1 && p.npass == 1) {
            any<true, true>(0, nullptr, nullptr);
            return;
        }
        any<true, false>(0, nullptr, A);
        __syncthreads();
        for (int ps = 1; ps < p.npass - 1; ps++) {
            any<false, false>(ps, A, B);
            __syncthreads();
            float2 *t = A;
            A = B;
            B = t;
        }
        any<false, true>(p.npass - 1, A, nullptr);
    }
};

// Most threads of a CTA (lines of 2048 and more; 256 for shorter ones), at 64
// registers: four CTAs of 256 or two of 512 share an SM.  At 80 registers and
// three CTAs rows of 1920 ran at 3.86 instead of 4.26 TB/s, the smallest
// radices' passes waiting for memory.
#define JT_MIX_THREADS 512

// MODE 0: rows to rows; 1: columns (strided lines) to columns; 2: rows to columns.
template <int SIGN, int MODE>
__global__ void __launch_bounds__(JT_MIX_THREADS, 2) mix_kernel(const float2 *in, float2 *out, MixParams p, const float2 *__restrict__ tw,
                                                                const float2 *__restrict__ Whi, const float2 *__restrict__ Wlo) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_begin();
    const int64_t b0 = (int64_t)blockIdx.x * p.C;
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    MixTile<SIGN, MODE>{in, out, p, tw, Whi, Wlo, b0, (int)min((int64_t)p.C, p.nlines - b0), MixBlue{}}.run(A, A + p.C * p.Lp);
}

// Pass tables of the radices R[0..npass) (mix_twiddle's layout): pass P >= 1
// starts at toff[P] (even) with w_{Ns R}^{jm k}, k = 1..R-1.
static __global__ void mix_table_kernel(float2 *out, MixParams p, int count) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= count) return;
    int ps = 1;
    while (ps + 1 < p.npass && idx >= p.toff[ps + 1]) ps++;
    const int r = idx - p.toff[ps], Ns = p.Ns[ps], R = p.R[ps], pair = r / (2 * Ns), left = r - pair * 2 * Ns;
    int jm = left >> 1, k = 2 * pair + 1 + (left & 1);
    if (pair == (R - 1) / 2) {  // an even radix's last factor
        jm = left;
        k = R - 1;
    }
    if (k >= R || jm >= Ns) return;  // a spare slot before the next pass
    const int64_t den = (int64_t)Ns * R, num = ((int64_t)jm * k) % den;
    double s, c;
    sincospi(-2.0 * (double)num / (double)den, &s, &c);
    out[idx] = make_float2((float)c, (float)s);
}

#undef C2

}  // namespace jt
