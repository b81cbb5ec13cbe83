// jt_fixmix.cuh -- complex FFT lines of doubles of mixed-radix length (prime
// factors 2, 3, 5, 7, not a power of two) in 64-bit block fixed point: the
// passes of jt_mixed.cuh with the arithmetic of jt_fixmath.cuh.
//
// The first pass takes one butterfly per thread: its numbers wait in
// registers as doubles until the line's largest exponent is known.  Inverse
// transforms exchange real and imaginary parts on the way in and out, so the
// passes exist once.  Lines with an infinity or a NaN run the FP64 passes of
// jt_device.cuh.
//
// Measured (GB300, one direction, FP64 tile passes before): 2 M points of n =
// 1000 49 us (185), of 96 31 (105), of 3000 65 (228); one transform of n = 1000
// 10.8 us (39.4), of 10^6 67 (375).  Relative L2 error against quad precision:
// at most 1.4e-16 for n = 24..3600, 3.3e-16 before.
//
// Reference: the FFTPACK passes, fft/DoubleFFT_1D.java:6630-7842.
#pragma once

#include "jt_mixed.cuh"

namespace jt {

#define JT_FIXMIX_RADICES(X) X(2) X(3) X(4) X(5) X(7) X(8) X(9) X(10) X(12) X(15) X(16)
#define JT_FIXMIX_THREADS 512
#define JT_FX_SPECIAL (1 << 20)  // in the place of a line's scaling (FxLine::pre): an infinity or a NaN among its numbers

struct FixMixParams {
    MixParams m;          // Lp: line stride; tables: factor k of a pass as Ns entries
    int psh;              // number i of a line at i + (i >> psh)
    int cols_in, cols_out, inv;
    int scale_e2, scale_mul;  // the output multiplier as in StockParams
    double scale;
    const int4 *tw, *Whiq, *Wloq;
    // FP64 passes, for special values
    TileParams fp;
    const double2 *W, *Whi, *Wlo;
};

// N1 N2 points, N1 and N2 coprime (dft_pfa's map)
template <int N1, int N2> __device__ __forceinline__ void fx_pfa(Fx *v) {
    constexpr int N = N1 * N2;
    Fx a[N1][N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) {
        Fx t[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) t[n1] = v[(N2 * n1 + N1 * n2) % N];
        fx_dft<N1, -1>(t);
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) a[n1][n2] = t[n1];
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) fx_dft<N2, -1>(a[k1]);
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = a[k % N1][k % N2];
}

// a e^{-2 pi i j/9} for j = 1, 2, 4, by three shears (fx_rot8's; the tangents of
// 20 and 40 degrees and the sines of 40 and 80; 160 degrees is 180 - 20)
__device__ __forceinline__ Fx fx_shear(Fx a, long long t, int si, long long s) {
    a.x += fx_mulk(a.y, t);
    a.y -= fx_mulc(a.x, si, s);
    a.x += fx_mulk(a.y, t);
    return a;
}
__device__ __forceinline__ Fx fx_w9(Fx a, int j) {
    if (j == 1) return fx_shear(a, 6714065761956745581ll, 1, -6589405544070453923ll);
    // 80 degrees as 90 - 10
    if (j == 2) {
        a = Fx{a.y, -a.x};
        return fx_shear(a, -1613880985413607648ll, 0, -3203243492287910726ll);
    }
    // 160 degrees as 180 - 20
    a = Fx{-a.x, -a.y};
    return fx_shear(a, -3252658686418974684ll, 0, -6309158051982071155ll);
}
__device__ __forceinline__ void fx_dft9(Fx *v) {
    Fx t[3][3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        Fx u[3] = {v[j], v[j + 3], v[j + 6]};
        fx_dft3<-1>(u);
#pragma unroll
        for (int k = 0; k < 3; k++) t[k][j] = u[k];
    }
    t[1][1] = fx_w9(t[1][1], 1);
    t[1][2] = fx_w9(t[1][2], 2);
    t[2][1] = fx_w9(t[2][1], 2);
    t[2][2] = fx_w9(t[2][2], 4);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        fx_dft3<-1>(t[k]);
#pragma unroll
        for (int m = 0; m < 3; m++) v[k + 3 * m] = t[k][m];
    }
}
template <int R> __device__ __forceinline__ void fx_dft_any(Fx *v) {
    if constexpr (R == 9) fx_dft9(v);
    else if constexpr (R == 10) fx_pfa<2, 5>(v);
    else if constexpr (R == 12) fx_pfa<4, 3>(v);
    else if constexpr (R == 15) fx_pfa<3, 5>(v);
    else fx_dft<R, -1>(v);
}

struct FixMixTile {
    const double2 *in;
    double2 *out;
    const FixMixParams &p;
    int64_t b0;
    int lines;
    uint32_t *words;  // JT_FX_WORDS x C

    __device__ __forceinline__ int at(int c, int i) const { return c * p.m.Lp + i + (i >> p.psh); }

    // Pass ps.  bin, bout: the lines' bits before and after it.  FIRST: returns
    // whether a value is not finite; the lines of such values are marked and
    // go through the passes as zeros that are not stored.
    template <int R, bool FIRST, bool LAST>
    __device__ __forceinline__ bool pass(int ps, const Fx *src, Fx *dst, uint32_t *bin, uint32_t *bout) const {
        const MixParams &m = p.m;
        const bool cols = FIRST ? p.cols_in : LAST ? p.cols_out : p.cols_in && p.cols_out;
        const int nb = m.L / R, Ns = m.Ns[ps], C = m.C;
        const int total = (cols ? C : lines) * nb;
        const int4 *tw = p.tw + m.toff[ps];
        int *ex = reinterpret_cast<int *>(words + 3 * C), *pre = ex + C;
        bool found = false;
        for (int q = threadIdx.x; FIRST || q < total; q += blockDim.x) {
            int c, j;
            if (cols) {
                j = C == 1 ? q : (int)__umulhi((uint32_t)q, m.mC);
                c = q - j * C;
            } else {
                c = nb == 1 ? q : (int)__umulhi((uint32_t)q, m.mNb[ps]);
                j = q - c * nb;
            }
            const bool ok = q < total && c < lines;
            Fx v[R];
            if (FIRST) {
                // one butterfly per thread (the launcher's block size)
                double2 d[R];
                const int64_t es = m.lin.estride, step = nb * es;
                const double2 *g = in + (ok ? line_off(m.lin, b0 + c) + j * es : 0);
#pragma unroll
                for (int k = 0; k < R; k++) {
                    d[k] = ok ? g[k * step] : make_double2(0, 0);
                    if (p.inv) d[k] = make_double2(d[k].y, d[k].x);
                }
                uint32_t mx = 0;
#pragma unroll
                for (int k = 0; k < R; k++)
                    mx = max(mx, max((uint32_t)__double2hiint(d[k].x) << 1, (uint32_t)__double2hiint(d[k].y) << 1));
                if (ok) fx_join<true>(bin, c, mx);
                const bool special = __syncthreads_or(mx >= 0xffe00000u);
                if (!ok) return special;
                FxLine l = fx_line(bin[c]);
                if (special && bin[c] >= 0xffe00000u) {
                    l = FxLine{0, JT_FX_SPECIAL};
#pragma unroll
                    for (int k = 0; k < R; k++) d[k] = make_double2(0, 0);
                }
                found = special;
                if (j == 0) {
                    ex[c] = l.ex;
                    pre[c] = l.pre;
                }
                if (__any_sync(__activemask(), l.pre != 0)) {
                    const double f = fx_pre(l.pre);
#pragma unroll
                    for (int k = 0; k < R; k++) d[k] = cscale<double>(d[k], f);
                }
#pragma unroll
                for (int k = 0; k < R; k++) v[k] = Fx{fx_from(d[k].x, l), fx_from(d[k].y, l)};
            } else {
                if (!ok) continue;
#pragma unroll
                for (int k = 0; k < R; k++) v[k] = src[at(c, j + k * nb)];
            }
            int jm = 0, s = 0;
            if (!FIRST) {
                jm = LAST ? j : j - (int)__umulhi((uint32_t)j, m.mNs[ps]) * Ns;
                s = fx_norm_shift(bin[c]);
                int r = s;
                if (r < 0) {
#pragma unroll
                    for (int k = 0; k < R; k++) v[k] = Fx{v[k].x << -r, v[k].y << -r};
                    r = 0;
                }
                const long long h = fx_half(r);
                v[0] = fx_shr(v[0], r + 2, fx_half(r + 2));
                const int4 *t = tw + jm;
#pragma unroll
                for (int k = 1; k < R; k++) {
                    v[k] = fx_mul<-1>(fx_shr(v[k], r, h), __ldg(t));
                    t += Ns;
                }
            }
            fx_dft_any<R>(v);
            const int base = (j - jm) * R + jm;
            if (LAST) {
                // (ex[c] is this line's exponent before the pass)
                const int e = ex[c] + s + 2 + p.scale_e2 + (m.tw_n ? 2 : 0);
                const int64_t es = m.lout.estride, step = Ns * es;
                double2 *g = out + line_off(m.lout, b0 + c) + base * es;
                if (m.tw_n) {
                    int64_t j2;
                    div_fast(b0 + c, m.tw_inner, &j2);
                    uint32_t x = (uint32_t)base * (uint32_t)j2;
                    const uint32_t dx = (uint32_t)Ns * (uint32_t)j2, mask = (1u << m.tw_lo_bits) - 1u;
#pragma unroll
                    for (int k = 0; k < R; k++) {
                        const int4 a = __ldg(&p.Whiq[x >> m.tw_lo_bits]);
                        Fx w = fx_mul<-1>(Fx{((long long)a.x << 32) + a.y, ((long long)a.z << 32) + a.w}, __ldg(&p.Wloq[x & mask]));
                        w = Fx{w.x << 2, w.y << 2};
                        v[k] = fx_mul<-1>(v[k], fx_as_factor(w));
                        x += dx;
                    }
                }
                double2 r[R];
#pragma unroll
                for (int k = 0; k < R; k++) r[k] = make_double2(fx_to(v[k].x, e), fx_to(v[k].y, e));
                if (__any_sync(__activemask(), pre[c] != 0) || p.scale_mul) {
                    const double f = fx_pre(-pre[c]) * (p.scale_mul ? p.scale : 1.0);
#pragma unroll
                    for (int k = 0; k < R; k++) r[k] = cscale<double>(r[k], f);
                }
                if (pre[c] != JT_FX_SPECIAL) {
#pragma unroll
                    for (int k = 0; k < R; k++) g[k * step] = p.inv ? make_double2(r[k].y, r[k].x) : r[k];
                }
            } else {
                uint32_t bits = 0;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    bits |= fx_bits(v[k].x) | fx_bits(v[k].y);
                    dst[at(c, base + k * Ns)] = v[k];
                }
                fx_join<false>(bout, c, bits);
            }
            if (FIRST) return found;
        }
        return false;
    }

    template <bool FIRST, bool LAST> __device__ __forceinline__ bool any(int ps, const Fx *src, Fx *dst, uint32_t *bin, uint32_t *bout) const {
        switch (p.m.R[ps]) {
#define JT_FIXMIX(RR) \
    case RR: return pass<RR, FIRST, LAST>(ps, src, dst, bin, bout);
            JT_FIXMIX_RADICES(JT_FIXMIX)
#undef JT_FIXMIX
        }
        return false;
    }

    // At least two passes, through the buffers A and B (B for three and more).
    // Returns whether lines are left for the FP64 passes.
    __device__ __forceinline__ bool run(Fx *A, Fx *B) const {
        const int C = p.m.C;
        uint32_t *b0w = words, *b1w = words + C, *b2w = words + 2 * C;
        int *ex = reinterpret_cast<int *>(words + 3 * C);
        for (int c = threadIdx.x; c < C; c += blockDim.x) b0w[c] = b1w[c] = 0;
        __syncthreads();
        const bool special = any<true, false>(0, nullptr, A, b0w, b1w);
        auto next = [&] {
            uint32_t *t = b0w;
            b0w = b1w;
            b1w = b2w;
            b2w = t;
        };
        next();
        for (int ps = 1; ps < p.m.npass - 1; ps++) {
            for (int c = threadIdx.x; c < C; c += blockDim.x) b1w[c] = 0;
            __syncthreads();
            any<false, false>(ps, A, B, b0w, b1w);
            for (int c = threadIdx.x; c < lines; c += blockDim.x) ex[c] += fx_norm_shift(b0w[c]) + 2;
            Fx *t = A;
            A = B;
            B = t;
            next();
        }
        __syncthreads();
        any<false, true>(p.m.npass - 1, A, nullptr, b0w, nullptr);
        return special;
    }
};

// The marked lines (pre: their marks, beyond the buffers that this uses)
static __device__ __noinline__ void fixmix_fp64(const double2 *in, double2 *out, const FixMixParams &p, int64_t b0, int lines,
                                                const int *pre, unsigned char *smem) {
    for (int l = 0; l < lines; l++) {
        if (pre[l] != JT_FX_SPECIAL) continue;
        __syncthreads();
        if (p.inv) tile_fft_body<1, double, true>(in, out, p.fp, p.W, p.Whi, p.Wlo, b0 + l, smem);
        else tile_fft_body<-1, double, true>(in, out, p.fp, p.W, p.Whi, p.Wlo, b0 + l, smem);
    }
}

// Tile `blk`, at smem_raw: one or two buffers of C lines (room for one line's
// FP64 passes at least) and their words.
__device__ __forceinline__ void fixmix_body(const double2 *in, double2 *out, const FixMixParams &p, int64_t blk, unsigned char *smem_raw) {
    const int64_t b0 = blk * p.m.C;
    const int lines = (int)min((int64_t)p.m.C, p.m.nlines - b0), nbuf = p.m.npass > 2 ? 2 : 1;
    Fx *A = reinterpret_cast<Fx *>(smem_raw);
    uint32_t *words = reinterpret_cast<uint32_t *>(A + max(nbuf * p.m.C * p.m.Lp, 2 * padded_len(p.m.L)));
    if (FixMixTile{in, out, p, b0, lines, words}.run(A, A + p.m.C * p.m.Lp))
        fixmix_fp64(in, out, p, b0, lines, reinterpret_cast<const int *>(words + 4 * p.m.C), smem_raw);
}

}  // namespace jt
