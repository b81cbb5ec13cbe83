// jt_fix64.cuh -- power-of-two complex FFT lines of doubles in 64-bit
// block-fixed-point arithmetic.
//
// GB300 issues about two FP64 instructions per clock and SM, against some
// 57 64-bit integer additions and 18 32 x 32 -> 64 bit multiply-adds, so an
// FFT in FP64 is bound by the FP64 pipe long before memory.  The lines are
// therefore transformed in integers: every line gets one exponent, its
// doubles become 64-bit fixed-point numbers below 2^58 (a double holds 53
// bits), the radix-16 butterflies are integer additions, twiddles are 62-bit
// fixed-point numbers whose products are rounded to nearest, and between two
// passes the line is shifted so that its largest number again has 60 bits.
// The error of a pass is a fraction of 2^-58 of the line's largest value,
// below that of the same pass in FP64 (2^-54 of each value); the twiddles are
// the FP64 tables' own values.  The result is rounded to double once.
//
// Measured (GB300, DoubleFFT_3D(256^3).complexForward and inverse, 268 MB):
// 888 us where the FP64 passes took 4617; DoubleFFT_1D(4096) x 256, both
// directions: 43 against 183 us; DoubleFFT_1D(1024), one line: 14 against
// 37 us a call (the FP64 pipe's latency).  Relative L2 error against quad
// precision over normal, uniform, tone, smooth, real and log-distributed
// inputs: 0.5-1.0e-16 at n = 16..8192, 1.1-2.3e-16 before.  What bounds a
// pass over 256-point lines now is latency: the ALU is 59 % busy, the FP64
// pipe 41 % (the conversions back to double), memory 51 % of its copy rate,
// with four CTAs of 128 registers a thread per SM.
//
// Range: lines whose largest exponent leaves no room (below 2^-900 or above
// 2^900) are scaled by 2^+-512 around the transform, which is exact; a tile
// with an infinity or a NaN runs the FP64 passes of jt_stockham.cuh, so those
// spread as they always did.
#pragma once

#include "jt_stockham.cuh"

namespace jt {

// Fixed-point complex value (one exponent per line, kept beside it).
struct Fx {
    long long x, y;
};

__device__ __forceinline__ long long fx_madw(int a, int b, long long c) {
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
// v as vh 2^32 + vl with both halves signed
__device__ __forceinline__ int fx_hi(long long v) { return (int)(v >> 32) + (int)((uint32_t)v >> 31); }
__device__ __forceinline__ int fx_lo(long long v) { return (int)v; }

// Fixed-point factors w are fx_twiddle's (x, y: cosine's halves; z, w: sine's).
// v w / 4 (SIGN < 0) or v conj(w) / 4, rounded to nearest.  |v| below 2^62.5:
// the partial sums stay below 2^63.  The low x low product is left out (a
// quarter of a unit at most).
template <int SIGN> __device__ __forceinline__ Fx fx_mul(Fx v, int4 w) {
    const int xh = fx_hi(v.x), xl = fx_lo(v.x), yh = fx_hi(v.y), yl = fx_lo(v.y);
    const int ph = SIGN < 0 ? w.z : -w.z, pl = SIGN < 0 ? w.w : -w.w;  // im += x p
    const int nh = SIGN < 0 ? -w.z : w.z, nl = SIGN < 0 ? -w.w : w.w;  // re += y n
    const long long half = 1ll << 31;
    long long m = fx_madw(yl, nh, fx_madw(yh, nl, fx_madw(xl, w.x, fx_madw(xh, w.y, half))));
    Fx r;
    r.x = fx_madw(yh, nh, fx_madw(xh, w.x, m >> 32));
    m = fx_madw(xl, ph, fx_madw(xh, pl, fx_madw(yl, w.x, fx_madw(yh, w.y, half))));
    r.y = fx_madw(xh, ph, fx_madw(yh, w.x, m >> 32));
    return r;
}

// v k / 2^64 rounded, for a constant |k| < 2^63: v times a factor in (-1/2, 1/2)
__device__ __forceinline__ long long fx_mulk(long long v, long long k) {
    const int vh = fx_hi(v), vl = fx_lo(v), kh = (int)((k + (1ll << 31)) >> 32), kl = (int)k;
    const long long m = fx_madw(vl, kh, fx_madw(vh, kl, 1ll << 31));
    return fx_madw(vh, kh, m >> 32);
}
// round(f 2^64) for -1/2 < f < 1/2: cos(pi/4) - 1, sqrt(2) - 1, tan(pi/16), sin(pi/8)
static constexpr long long kFxHm1 = -5402926248376769404ll;
static constexpr long long kFxR2m1 = 7640891576956012809ll;
static constexpr long long kFxTan16 = 3669285534148243471ll;
static constexpr long long kFxSin8 = 7059263338087549767ll;
__device__ __forceinline__ long long fx_mulh(long long v) { return v + fx_mulk(v, kFxHm1); }  // v cos(pi/4)

__device__ __forceinline__ Fx fx_add(Fx a, Fx b) { return Fx{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ Fx fx_sub(Fx a, Fx b) { return Fx{a.x - b.x, a.y - b.y}; }
template <int SIGN> __device__ __forceinline__ Fx fx_si(Fx a) { return SIGN > 0 ? Fx{-a.y, a.x} : Fx{a.y, -a.x}; }

// a e^{SIGN i pi/8}: three shears of the plane (x -= t y, y += s x, x -= t y
// with t = tan(pi/16), s = sin(pi/8)), nine multiply-adds where four real
// products take twelve
template <int SIGN> __device__ __forceinline__ Fx fx_rot8(Fx a) {
    constexpr long long t = SIGN > 0 ? kFxTan16 : -kFxTan16, s = SIGN > 0 ? kFxSin8 : -kFxSin8;
    a.x -= fx_mulk(a.y, t);
    a.y += fx_mulk(a.x, s);
    a.x -= fx_mulk(a.y, t);
    return a;
}

template <int SIGN> __device__ __forceinline__ void fx_dft4(Fx &v0, Fx &v1, Fx &v2, Fx &v3) {
    const Fx t0 = fx_add(v0, v2), t1 = fx_sub(v0, v2), t2 = fx_add(v1, v3), d = fx_sub(v1, v3);
    v0 = fx_add(t0, t2);
    v2 = fx_sub(t0, t2);
    // t1 +- SIGN i d
    v1 = SIGN > 0 ? Fx{t1.x - d.y, t1.y + d.x} : Fx{t1.x + d.y, t1.y - d.x};
    v3 = SIGN > 0 ? Fx{t1.x + d.y, t1.y - d.x} : Fx{t1.x - d.y, t1.y + d.x};
}

template <int SIGN> __device__ __forceinline__ void fx_dft8(Fx *v) {
    Fx e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    Fx o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    fx_dft4<SIGN>(e0, e1, e2, e3);
    fx_dft4<SIGN>(o0, o1, o2, o3);
    // e^{SIGN i pi/4} and e^{SIGN 3 i pi/4}
    o1 = SIGN > 0 ? Fx{fx_mulh(o1.x - o1.y), fx_mulh(o1.x + o1.y)} : Fx{fx_mulh(o1.x + o1.y), fx_mulh(o1.y - o1.x)};
    o2 = fx_si<SIGN>(o2);
    o3 = SIGN > 0 ? Fx{fx_mulh(-o3.x - o3.y), fx_mulh(o3.x - o3.y)} : Fx{fx_mulh(o3.y - o3.x), fx_mulh(-o3.x - o3.y)};
    v[0] = fx_add(e0, o0); v[4] = fx_sub(e0, o0);
    v[1] = fx_add(e1, o1); v[5] = fx_sub(e1, o1);
    v[2] = fx_add(e2, o2); v[6] = fx_sub(e2, o2);
    v[3] = fx_add(e3, o3); v[7] = fx_sub(e3, o3);
}

// radix 16 as 4 x 4: element (k, j) at v[j + 4k] takes e^{SIGN i pi jk/8}
template <int SIGN> __device__ __forceinline__ void fx_dft16(Fx *v) {
#pragma unroll
    for (int j = 0; j < 4; j++) fx_dft4<SIGN>(v[j], v[j + 4], v[j + 8], v[j + 12]);
    auto w2 = [](Fx a) {  // e^{SIGN i pi/4}
        return SIGN > 0 ? Fx{fx_mulh(a.x - a.y), fx_mulh(a.x + a.y)} : Fx{fx_mulh(a.x + a.y), fx_mulh(a.y - a.x)};
    };
    v[5] = fx_rot8<SIGN>(v[5]);
    v[6] = w2(v[6]);
    v[7] = fx_rot8<-SIGN>(fx_si<SIGN>(v[7]));    // w^3 = SIGN i w^-1
    v[9] = w2(v[9]);
    v[10] = fx_si<SIGN>(v[10]);
    v[11] = w2(fx_si<SIGN>(v[11]));              // w^6
    v[13] = fx_rot8<-SIGN>(fx_si<SIGN>(v[13]));  // w^3
    v[14] = w2(fx_si<SIGN>(v[14]));              // w^6
    v[15] = fx_rot8<SIGN>(v[15]);                // w^9 = -w
    v[15] = Fx{-v[15].x, -v[15].y};
#pragma unroll
    for (int k = 0; k < 4; k++) fx_dft4<SIGN>(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    Fx t[16];
#pragma unroll
    for (int i = 0; i < 16; i++) t[i] = v[i];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) v[k + 4 * j] = t[4 * k + j];
}

template <int R, int SIGN> __device__ __forceinline__ void fx_dft(Fx *v) {
    if (R == 2) {
        const Fx a = v[0], b = v[1];
        v[0] = fx_add(a, b);
        v[1] = fx_sub(a, b);
    } else if (R == 4) {
        fx_dft4<SIGN>(v[0], v[1], v[2], v[3]);
    } else if (R == 8) {
        fx_dft8<SIGN>(v);
    } else if (R == 16) {
        fx_dft16<SIGN>(v);
    }
}

// Bits in use: the OR of these over a line has the bit length of its largest
// magnitude's high word.
__device__ __forceinline__ uint32_t fx_bits(long long v) {
    const int h = (int)(v >> 32);
    return (uint32_t)(h ^ (h >> 31));
}

// A line's exponent and what its doubles are scaled by around the transform.
struct FxLine {
    int ex;    // a value is v 2^ex
    int pre;   // 0, or +-512: the doubles were multiplied by 2^pre first
};

#define JT_FX_BIAS 1080  // a double of the line's largest exponent eb is v 2^(eb - 1080), v < 2^58

// From the line's largest (high word << 1) over all its numbers.
__device__ __forceinline__ FxLine fx_line(uint32_t m) {
    const int eb = (int)(m >> 21);
    FxLine l;
    l.pre = eb < 123 ? 512 : eb > 1923 ? -512 : 0;  // (lines of zeros too: subnormals may have no high word)
    l.ex = max(eb, 1) + l.pre - JT_FX_BIAS;
    return l;
}
// The line's numbers below 2^BITS (l.ex is for 58).
template <int BITS = 58> __device__ __forceinline__ long long fx_from(double d, const FxLine &l) {
    const int hi = __double2hiint(d), lo = __double2loint(d);
    const int e = (hi >> 20) & 0x7ff;
    const uint32_t mh = ((uint32_t)hi & 0xfffffu) | 0x100000u;
    const int r = min(l.ex + JT_FX_BIAS + 63 - BITS - e, 63);  // at least 63 - BITS; zeros (and far smaller numbers) go to 0
    unsigned long long u = (((unsigned long long)mh << 32) | (uint32_t)lo) << 10;
    u >>= r;
    const long long s = (long long)(hi >> 31);
    return ((long long)u ^ s) - s;
}
__device__ __forceinline__ double fx_to(long long v, int ex) {
    const double d = __ll2double_rn(v);
    const int hi = __double2hiint(d);
    return v == 0 ? 0.0 : __hiloint2double(hi + (ex << 20), __double2loint(d));
}
// 2^pre and 2^-pre.  Products with them stand behind one branch per block of
// values: a conditional product is issued to the FP64 pipe for every value,
// needed or not, and six of those per number were most of this kernel's time.
__device__ __forceinline__ double fx_pre(int pre) { return pre > 0 ? 1.3407807929942597e154 : pre < 0 ? 7.458340731200207e-155 : 1.0; }

// Shift that brings a line with these bits to BITS bits: right by s > 0 or left by -s.
template <int BITS = 60> __device__ __forceinline__ int fx_norm_shift(uint32_t bits) { return bits ? 64 - BITS - __clz(bits) : 0; }
// (v + rnd) >> s with rnd = half a unit of the result
__device__ __forceinline__ Fx fx_shr(Fx v, int s, long long rnd) { return Fx{(v.x + rnd) >> s, (v.y + rnd) >> s}; }
__device__ __forceinline__ long long fx_half(int s) { return s > 0 ? 1ll << (s - 1) : 0; }
// N values by the shift s (fx_norm_shift's)
template <int N> __device__ __forceinline__ void fx_norm(Fx *v, int s) {
    if (s < 0) {
#pragma unroll
        for (int m = 0; m < N; m++) v[m] = Fx{v[m].x << -s, v[m].y << -s};
        s = 0;
    }
    const long long r = fx_half(s);
#pragma unroll
    for (int m = 0; m < N; m++) v[m] = fx_shr(v[m], s, r);
}

// Fixed-point pass table of a length-L line: the entries of the double table
// (stock_tw_count, factor k of a pass as NS entries) as int4.
__device__ __forceinline__ const int4 *fx_factor(const int4 *W, int off, int ns, int k, int jm) {
    return W + off + (k - 1) * ns + jm;
}

struct FxCfg {
    // most lines per CTA: 128 threads for short lines; of the column modes'
    // longer ones 8 columns (128-byte segments) up to 512, fewer above
    static constexpr int rows_C(int L) { return L >= 128 * fx_elems(L) ? 1 : 128 * fx_elems(L) / L; }
    static constexpr int cols_C(int L) { return L <= 16 * fx_elems(L) ? 128 * fx_elems(L) / L : L <= 512 ? 8 : 4096 / L < 2 ? 2 : 4096 / L; }
    static constexpr int C(int L, int mode) { return mode == 0 ? rows_C(L) : cols_C(L); }
};

// The passes of a CTA's lines: C lines (at most CM, a power of two) of TL
// threads each; MODE 0 keeps a line's threads together, the column modes
// spread the lines across a warp (c fastest).
template <int L, int MODE, int SIGN, int CM> struct FxStock {
    static constexpr int E = fx_elems(L), TL = L / E, NT = CM * TL, LP = L + L / E + 1;
    typedef Stockham<double, L, MODE, SIGN, E> S;
    // a spare slot per E numbers: the first pass writes in strides of E
    static __device__ __forceinline__ int pad(int i) { return i + i / E; }
    static constexpr int NPASS = S::NPASS;
    static constexpr bool WARP_LINE = MODE == 0 && TL <= 32;  // a line's threads share a warp
    // A line's stride in shared memory.  The column modes' quarter-warps (16-byte
    // accesses) cover C lines at 8 / C neighbouring positions: strides of
    // 8 / C modulo 8 spread them over the banks (L + L/E is a multiple of 8
    // for the lines, of 128 and more, that run with C < 8).
    static __host__ __device__ __forceinline__ int stride(int C) { return MODE == 0 || C >= 8 ? LP : LP - 1 + 8 / C; }
    static constexpr size_t SMEM = (size_t)CM * (MODE == 0 || CM >= 8 ? LP : LP - 1 + 8 / CM) * sizeof(Fx);
    // 128 registers a thread, 64 with 8 numbers
    static constexpr int REGT = E == 16 ? 512 : 1024, MINB = NT >= REGT ? 1 : REGT / NT > 16 ? 16 : REGT / NT;
    static constexpr int RED = WARP_LINE ? 1 : (NPASS + 2) * CM;  // words of `red`

    // fewest lines per CTA: whole warps
    static constexpr int CMIN = TL >= 32 ? 1 : 32 / TL;

    // OR (MAX: largest) of x over the threads of this thread's line that are in its warp
    template <bool MAX> static __device__ __forceinline__ uint32_t warp_red(uint32_t x, int C) {
        auto join = [](uint32_t a, uint32_t b) { return MAX ? max(a, b) : a | b; };
        if constexpr (MODE == 0 && TL >= 32) {
            return MAX ? __reduce_max_sync(0xffffffffu, x) : __reduce_or_sync(0xffffffffu, x);
        } else if constexpr (MODE == 0) {
#pragma unroll
            for (int o = 1; o < TL; o <<= 1) x = join(x, __shfl_xor_sync(0xffffffffu, x, o));
        } else {
            for (int o = C; o < 32; o <<= 1) x = join(x, __shfl_xor_sync(0xffffffffu, x, o));
        }
        return x;
    }
    // The same over the whole line: `slot` of red (CM words each, zeroed), and
    // a barrier of the line's threads in any case
    template <bool MAX> static __device__ __forceinline__ uint32_t line_red(uint32_t x, int slot, int c, int tid, int C, uint32_t *red) {
        x = warp_red<MAX>(x, C);
        if constexpr (WARP_LINE) {
            __syncwarp();
            return x;
        } else {
            if (MODE == 0 ? tid % 32 == 0 : tid % 32 < C) {
                if (MAX) atomicMax(&red[slot * CM + c], x);
                else atomicOr(&red[slot * CM + c], x);
            }
            __syncthreads();
            return red[slot * CM + c];
        }
    }
    static __device__ __forceinline__ void line_sync() {
        if constexpr (WARP_LINE) __syncwarp();
        else __syncthreads();
    }

    // Passes P.. on v (below 2^58 at P = 0); the last one's outputs idxD +
    // k NS, k < R, go to store(idxD, u, q).
    template <int P, typename Store>
    static __device__ __forceinline__ void run(Fx (&v)[E], int t, int c, int tid, int C, Fx *xs, const int4 *__restrict__ W,
                                               uint32_t *red, FxLine &ln, Store &store) {
        typedef typename S::template Pass<P> PP;
        const int base = c * stride(C);
        uint32_t bits = 0;
#pragma unroll
        for (int q = 0; q < PP::NB; q++) {
            Fx u[PP::R];
            const int j = t + q * TL, jm = j & (PP::NS - 1);
#pragma unroll
            for (int k = 0; k < PP::R; k++) u[k] = v[q + k * PP::NB];
            if constexpr (P > 0) {
#pragma unroll
                for (int k = 1; k < PP::R; k++)
                    u[k] = fx_mul<SIGN>(u[k], __ldg(fx_factor(W, S::template twoff<P>(), PP::NS, k, jm)));
            }
            fx_dft<PP::R, SIGN>(u);
            const int idxD = (j - jm) * PP::R + jm;
            if constexpr (PP::LAST) {
                store(idxD, u, q);
            } else {
#pragma unroll
                for (int k = 0; k < PP::R; k++) {
                    bits |= fx_bits(u[k].x) | fx_bits(u[k].y);
                    xs[base + pad(idxD + k * PP::NS)] = u[k];
                }
            }
        }
        if constexpr (!PP::LAST) {
            typedef typename S::template Pass<P + 1> NP;
            bits = line_red<false>(bits, P + 1, c, tid, C, red);
#pragma unroll
            for (int m = 0; m < E; m++) v[m] = xs[base + pad(t + m * TL)];
            if constexpr (P + 2 < NPASS) line_sync();  // the next pass writes the buffer again
            int s = fx_norm_shift(bits);
            ln.ex += s + 2;  // the twiddle products divide by 4
            if (s < 0) {
#pragma unroll
                for (int m = 0; m < E; m++) v[m] = Fx{v[m].x << -s, v[m].y << -s};
                s = 0;
            }
            // the butterflies' first inputs have no twiddle: the division by 4 joins their shift
            const long long r0 = fx_half(s + 2), r1 = fx_half(s);
#pragma unroll
            for (int m = 0; m < E; m++) v[m] = m < NP::NB ? fx_shr(v[m], s + 2, r0) : fx_shr(v[m], s, r1);
            run<P + 1>(v, t, c, tid, C, xs, W, red, ln, store);
        }
    }
};

// One tile of C = blockDim / TL lines per CTA (several CTAs share an SM:
// their loads overlap each other's arithmetic).
template <int L, int MODE, int SIGN, bool TW>
__global__ void __launch_bounds__(FxStock<L, MODE, SIGN, FxCfg::C(L, MODE)>::NT, FxStock<L, MODE, SIGN, FxCfg::C(L, MODE)>::MINB)
    fix_kernel(const double2 *__restrict__ in, double2 *__restrict__ out, StockParams p, const double2 *__restrict__ W,
               const double2 *__restrict__ Whi, const double2 *__restrict__ Wlo, const int4 *__restrict__ Wq,
               const int4 *__restrict__ Whiq, const int4 *__restrict__ Wloq) {
    typedef FxStock<L, MODE, SIGN, FxCfg::C(L, MODE)> F;
    typedef typename F::S S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t red[F::RED];
    Fx *xs = reinterpret_cast<Fx *>(smem_raw);
    const int tid = threadIdx.x, NT = blockDim.x, C = NT / F::TL;
    const int c = MODE == 0 ? tid / F::TL : tid & (C - 1), t = MODE == 0 ? tid % F::TL : tid / C;
    const int64_t ntiles = gridDim.x;
    const int64_t tile = p.reverse ? ntiles - 1 - blockIdx.x : blockIdx.x;
    const int64_t b0 = tile * C, b = b0 + c;
    const bool valid = b < p.nlines;
    if constexpr (!F::WARP_LINE)
        for (int i = tid; i < F::RED; i += NT) red[i] = 0;
    const int stride = F::stride(C), base = c * stride;
    double2 d[F::E];
    if constexpr (MODE == 2) {
        double2 *sd = reinterpret_cast<double2 *>(smem_raw);
        double2 x[F::E];
#pragma unroll
        for (int u = 0; u < F::E; u++) {
            const int i = tid + u * NT, cc = i / L, e = i % L;
            x[u] = b0 + cc < p.nlines ? in[line_off(p.lin, b0 + cc) + e] : make_double2(0, 0);
        }
#pragma unroll
        for (int u = 0; u < F::E; u++) {
            const int i = tid + u * NT, cc = i / L, e = i % L;
            sd[cc * stride + F::pad(e)] = x[u];
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < F::E; m++) d[m] = sd[base + F::pad(t + m * F::TL)];
    } else {
        const double2 *src = in + (valid ? line_off(p.lin, b) : 0);
        const int64_t es = MODE == 0 ? 1 : p.lin.estride;
#pragma unroll
        for (int m = 0; m < F::E; m++) d[m] = valid ? src[(int64_t)(t + m * F::TL) * es] : make_double2(0, 0);
        if constexpr (!F::WARP_LINE) __syncthreads();  // red is zeroed
    }
    uint32_t mx = 0;
#pragma unroll
    for (int m = 0; m < F::E; m++)
        mx = max(mx, max((uint32_t)__double2hiint(d[m].x) << 1, (uint32_t)__double2hiint(d[m].y) << 1));
    const bool special = mx >= 0xffe00000u;  // an infinity or a NaN
    mx = F::template warp_red<true>(mx, C);
    if constexpr (!F::WARP_LINE)
        if (MODE == 0 ? tid % 32 == 0 : tid % 32 < C) atomicMax(&red[c], mx);
    // (MODE 2: this barrier also ends the reads of the staged lines)
    const bool fp = __syncthreads_or(special);
    double2 *dst = out + (valid ? line_off(p.lout, b) : 0);
    const int64_t oes = MODE == 0 ? 1 : p.lout.estride;
    const uint64_t spol = p.stream_out ? policy_evict_first() : policy_evict_normal();
    int64_t j2l = 0;
    if constexpr (TW) div_fast(valid ? b : 0, p.tw_inner, &j2l);
    const uint32_t j2 = (uint32_t)j2l;
    if (fp) {
        auto store = [&](int pos, double2 val, int) {
            if (TW) {
                const double2 w = tw_lookup<double>(Whi, Wlo, (uint32_t)pos * j2, p);
                val = SIGN < 0 ? cmul<double>(val, w) : cmulc<double>(val, w);
            }
            if (p.do_scale) val = cscale<double>(val, p.scale);
            if (valid) st_hint(&dst[(int64_t)pos * oes], val, spol);
        };
        PadIdx xi{c * S::LP};
        S::run_all(d, t, reinterpret_cast<double2 *>(smem_raw), xi, W, store);
        return;
    }
    if constexpr (!F::WARP_LINE) mx = red[c];
    FxLine ln = fx_line(mx);
    if (__any_sync(0xffffffffu, ln.pre != 0)) {
        const double f = fx_pre(ln.pre);
#pragma unroll
        for (int m = 0; m < F::E; m++) d[m] = cscale<double>(d[m], f);
    }
    Fx v[F::E];
#pragma unroll
    for (int m = 0; m < F::E; m++) v[m] = Fx{fx_from(d[m].x, ln), fx_from(d[m].y, ln)};
    // four-step twiddle w^{pos j2} of the last pass's outputs, pos = t + TL m
    // with m = q + k NB in slot q R + k: w^{t j2} g^m, g = w^{TL j2}, formed by
    // successive products (each a unit of 2^-60 off at most)
    auto two_level = [&](uint32_t x) -> Fx {
        x &= p.tw_mask;
        const int4 a = __ldg(&Whiq[x >> p.tw_lo_bits]);
        const Fx f{((long long)a.x << 32) + a.y, ((long long)a.z << 32) + a.w};
        const Fx r = fx_mul<-1>(f, __ldg(&Wloq[x & ((1u << p.tw_lo_bits) - 1u)]));
        return Fx{r.x << 2, r.y << 2};
    };
    auto factor = [](Fx a) { return make_int4(fx_hi(a.x), fx_lo(a.x), fx_hi(a.y), fx_lo(a.y)); };
    typedef typename S::template Pass<F::NPASS - 1> LP_;
    Fx wq{0, 0}, w{0, 0};
    int4 g1 = make_int4(0, 0, 0, 0), gn = g1;
    if constexpr (TW) {
        const uint32_t g = (uint32_t)F::TL * j2;
        wq = two_level((uint32_t)t * j2);
        g1 = factor(two_level(g));
        gn = LP_::NB > 1 ? factor(two_level((uint32_t)LP_::NB * g)) : g1;
    }
    auto times = [](Fx a, int4 b) {
        const Fx r = fx_mul<-1>(a, b);
        return Fx{r.x << 2, r.y << 2};
    };
    const bool mul = __any_sync(0xffffffffu, ln.pre != 0) || p.scale_mul;
    const double f = fx_pre(-ln.pre) * (p.scale_mul ? p.scale : 1.0);
    auto store = [&](int pos, Fx *u, int q) {
        const int ex = ln.ex + p.scale_e2 + (TW ? 2 : 0);
        double2 r[LP_::R];
#pragma unroll
        for (int k = 0; k < LP_::R; k++) {
            if constexpr (TW) {
                if (k == 0) {
                    if (q > 0) wq = times(wq, g1);
                    w = wq;
                } else {
                    w = times(w, gn);
                }
                u[k] = fx_mul<SIGN>(u[k], factor(w));
            }
            r[k] = make_double2(fx_to(u[k].x, ex), fx_to(u[k].y, ex));
        }
        if (mul) {
#pragma unroll
            for (int k = 0; k < LP_::R; k++) r[k] = cscale<double>(r[k], f);
        }
        if (valid) {
#pragma unroll
            for (int k = 0; k < LP_::R; k++) st_hint(&dst[(int64_t)(pos + k * LP_::NS) * oes], r[k], spol);
        }
    };
    F::template run<0>(v, t, c, tid, C, xs, Wq, red, ln, store);
}

// Lines per CTA: the most that fit, halved while the grid has fewer CTAs than
// two per SM (whole warps, and 64-byte segments of the column modes, stay).
inline int fix_lines(int64_t nlines, int most, int least, int sms) {
    int C = most;
    while (C > least && (nlines + C - 1) / C < 2 * (int64_t)sms) C /= 2;
    return C;
}

template <int L> struct FixLaunch {
    template <int MODE, int SIGN, bool TW>
    static void one(const double2 *in, double2 *out, const StockParams &p, const double2 *W, const double2 *Whi, const double2 *Wlo,
                    const int4 *Wq, const int4 *Whiq, const int4 *Wloq, int sms, cudaStream_t s) {
        constexpr int CM = FxCfg::C(L, MODE);
        typedef FxStock<L, MODE, SIGN, CM> F;
        auto kern = fix_kernel<L, MODE, SIGN, TW>;
        static bool attr = false;
        if (!attr) {
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::SMEM);
            attr = true;
        }
        const int C = fix_lines(p.nlines, CM, std::min(CM, std::max(F::CMIN, MODE == 0 ? 1 : 4)), sms);
        const int64_t ntiles = (p.nlines + C - 1) / C;
        kern<<<(unsigned)ntiles, C * F::TL, (size_t)C * F::stride(C) * sizeof(Fx), s>>>(in, out, p, W, Whi, Wlo, Wq, Whiq, Wloq);
    }
    template <int MODE, int SIGN, typename... A> static void tw(const double2 *in, double2 *out, const StockParams &p, A... a) {
        if constexpr (MODE == 1) {
            if (p.tw_n != 0) {
                one<MODE, SIGN, true>(in, out, p, a...);
                return;
            }
        }
        one<MODE, SIGN, false>(in, out, p, a...);
    }
    template <typename... A> static void go(int mode, int sign, A... a) {
        if (mode == 0) {
            sign < 0 ? tw<0, -1>(a...) : tw<0, 1>(a...);
            return;
        }
        if constexpr (L <= 4096) {
            if (mode == 1) sign < 0 ? tw<1, -1>(a...) : tw<1, 1>(a...);
            else sign < 0 ? tw<2, -1>(a...) : tw<2, 1>(a...);
        }
    }
};

}  // namespace jt
