// jt_bluemix.cuh -- Bluestein transforms of floats on the mixed-radix passes
// (jt_mixed.cuh).
//
// y_k = conj(b_k) sum_j (x_j conj(b_j)) b_{k-j}, b_j = e^{i pi j^2 / n}, is a
// cyclic convolution of any length N >= 2n - 1.  N is a product of the
// radices below, no noisier than the power of two that would serve (up to twice
// as long as it need be; blue_split).  One kernel up to N = 8192 (blue_mid_kernel<true>); beyond that
// N = n1 n2 in three:
//   in    n1-point columns of the n1 x n2 view, chirped and zero beyond n as
//         they are read, four-step twiddle on the store
//   mid   rows: n2-point FFT, times the chirp's spectrum, inverse FFT; the
//         spectrum never needs its natural order, so the table holds it in
//         the rows' order
//   out   conjugate twiddle on the load, inverse columns, chirp, scale, n
//         numbers stored
// The turn between the two FFTs of a line happens in registers: the last
// forward pass holds the inputs of the inverse transform's first pass when
// that has the same radix, so the inverse takes the radices in reverse.
//
// Measured (GB300, FloatFFT_1D(10007) x 1024, both directions): 608 us, 1300
// with seven kernels around a power-of-two convolution of 32768 (here 20736 =
// 16 x 1296 points): the columns wait for their loads, the rows (half of the
// time) issue in 64 % of the cycles.
//
// Reference: bluestein_complex, fft/DoubleFFT_1D.java:1864-2107.
#pragma once

#include "jt_mixed.cuh"

namespace jt {

// The middle kernel's two FFTs (f: forward radices, g: the same in reverse,
// both with L, C, Lp), their tables and the chirp's spectrum Bp, a row of L
// for each of n1 line numbers (n1 = 1: all lines share it).
struct BlueMid {
    MixParams f, g;
    const float2 *twf, *twg, *Bp;
    int n1;
    MixBlue bl;
};

#define JT_BLUE_RADICES(X) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(16)

// ONE: whole transforms (chirped loads and stores of the caller's lines), else
// rows of the n1 x n2 view in place.
template <bool ONE> struct BlueTile {
    const float2 *in;
    float2 *out;
    const BlueMid &q;
    int64_t b0;
    int lines;

    // from src (FIRST: global memory) to dst (LAST: global memory); TURN: the
    // last forward pass and the first inverse pass
    template <int R, int SIGN, bool FIRST, bool LAST, bool TURN>
    __device__ __forceinline__ void pass(const MixParams &p, const float2 *tw, int ps, const float2 *src, float2 *dst) const {
        const int L = p.L, nb = L / R, Ns = p.Ns[ps], Lp = p.Lp, total = lines * nb;
        const uint32_t mNb = p.mNb[ps], mNs = p.mNs[ps];
        tw += p.toff[ps];
        for (int i = threadIdx.x; i < total; i += blockDim.x) {
            const int c = (int)__umulhi((uint32_t)i, mNb), j = i - c * nb;
            float2 v[R];
            if (FIRST) {
                const float2 *g = in + (ONE ? (b0 + c) * q.bl.din : (b0 + c) * L);
#pragma unroll
                for (int k = 0; k < R; k++) {
                    const int e = j + k * nb;
                    if (ONE) v[k] = e < q.bl.n ? mix_chirp(g[e], q.bl, e) : make_float2(0, 0);
                    else v[k] = g[e];
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
                const int jm = LAST || TURN ? j : j - (int)__umulhi((uint32_t)j, mNs) * Ns;
                base -= jm * (R - 1);
                mix_twiddle<R, SIGN>(v, tw, Ns, jm);
            }
            dft_any<R, SIGN, float, true>(v);
            if (TURN) {
                // v[k]: spectrum number j + k nb; the inverse's first pass has no twiddles
                int64_t row = 0;
                if (!ONE) div_fast(b0 + c, q.n1, &row);
                const float2 *B = q.Bp + row * L + j;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    const float2 w = __ldg(B + k * nb);
                    v[k] = q.bl.inv ? cmulc<float>(v[k], w) : cmul<float>(v[k], w);
                }
                dft_any<R, 1, float, true>(v);
                base = j * R;
            }
            if (LAST) {
                float2 *g = out + (ONE ? (b0 + c) * q.bl.dout : (b0 + c) * L);
#pragma unroll
                for (int k = 0; k < R; k++) {
                    const int e = base + k * Ns;
                    if (!ONE) g[e] = v[k];
                    else if (e < q.bl.n) g[e] = cscale<float>(mix_chirp(v[k], q.bl, e), q.bl.scale);
                }
            } else {
                float2 *d = dst + c * Lp + base;
                const int step = FIRST || TURN ? 1 : Ns;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    *d = v[k];
                    d += step;
                }
            }
        }
    }
    template <int SIGN, bool FIRST, bool LAST, bool TURN>
    __device__ __forceinline__ void any(const MixParams &p, const float2 *tw, int ps, const float2 *src, float2 *dst) const {
        switch (p.R[ps]) {
#define JT_BLUE_CASE(RR) \
    case RR: pass<RR, SIGN, FIRST, LAST, TURN>(p, tw, ps, src, dst); break;
            JT_BLUE_RADICES(JT_BLUE_CASE)
#undef JT_BLUE_CASE
        }
    }
    __device__ __forceinline__ void run(float2 *A, float2 *B) const {
        const int np = q.f.npass;
        auto next = [&] {
            __syncthreads();
            float2 *t = A;
            A = B;
            B = t;
        };
        any<-1, true, false, false>(q.f, q.twf, 0, nullptr, B);
        next();
        for (int ps = 1; ps < np - 1; ps++) {
            any<-1, false, false, false>(q.f, q.twf, ps, A, B);
            next();
        }
        any<-1, false, false, true>(q.f, q.twf, np - 1, A, B);
        next();
        for (int ps = 1; ps < np - 1; ps++) {
            any<1, false, false, false>(q.g, q.twg, ps, A, B);
            next();
        }
        any<1, false, true, false>(q.g, q.twg, np - 1, A, nullptr);
    }
};

template <bool ONE> __global__ void __launch_bounds__(JT_MIX_THREADS, 2) blue_mid_kernel(const float2 *in, float2 *out, BlueMid q) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_begin();
    const int64_t b0 = (int64_t)blockIdx.x * q.f.C;
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    BlueTile<ONE>{in, out, q, b0, (int)min((int64_t)q.f.C, q.f.nlines - b0)}.run(A, A + q.f.C * q.f.Lp);
}

// The first (POL MIX_BLUE_IN) and last (MIX_BLUE_OUT) kernels of three.
template <int SIGN, int POL>
__global__ void __launch_bounds__(JT_MIX_THREADS, 2) blue_cols_kernel(const float2 *in, float2 *out, MixParams p, MixBlue bl,
                                                                      const float2 *__restrict__ tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_begin();
    const int64_t b0 = (int64_t)blockIdx.x * p.C;
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    MixTile<SIGN, 1, POL>{in, out, p, tw, nullptr, nullptr, b0, (int)min((int64_t)p.C, p.nlines - b0), bl}.run(A, A + p.C * p.Lp);
}

// w_N^{k1 c}, N = n1 n2, at [k1 n2 + c]
static __global__ void blue_twiddle_kernel(float2 *out, int n1, int n2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n1 * n2) return;
    const int k1 = i / n2, c = i - k1 * n2;
    double s, co;
    sincospi(-2.0 * (double)((int64_t)k1 * c) / ((double)n1 * n2), &s, &co);
    out[i] = make_float2((float)co, (float)s);
}

// out[k1 n2 + k2] = in[k1 + n1 k2], rounded to float
static __global__ void blue_spectrum_kernel(float2 *out, const double2 *in, int64_t n1, int64_t n2) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n1 * n2) return;
    const int64_t k1 = i / n2, k2 = i - k1 * n2;
    const double2 v = in[k1 + n1 * k2];
    out[i] = make_float2((float)v.x, (float)v.y);
}

}  // namespace jt
