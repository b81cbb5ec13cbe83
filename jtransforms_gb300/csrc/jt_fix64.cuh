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
// right to 2^-62 (fx_root).  The result is rounded to double once.
//
// Measured (GB300, DoubleFFT_3D(256^3).complexForward and inverse, 268 MB):
// 873 us where the FP64 passes took 4617; DoubleFFT_1D(4096) x 256, both
// directions: 40 against 183 us; DoubleFFT_1D(1024), one line: 11 against
// 37 us a call (the FP64 pipe's latency).  Relative L2 error against quad
// precision over normal, uniform, tone, smooth, real, constant and
// log-distributed inputs and a spike: at most 1.3e-16 at n = 16..8192, 2.5e-16
// before; 1.0e-16 at 2^14..2^18, 3.5e-16 before.  What bounds a
// pass over 256-point lines now is latency: the ALU is 62 % busy, the FP64
// pipe 43 % (the conversions back to double), memory 52 % of its copy rate,
// with four CTAs of 128 registers a thread per SM.
//
// Range: lines whose largest exponent leaves no room (below 2^-900 or above
// 2^900) are scaled by 2^+-512 around the transform, which is exact; a line
// with an infinity or a NaN runs the FP64 passes of jt_stockham.cuh, so those
// spread as they always did.
#pragma once

#include "jt_fixmath.cuh"
#include "jt_stockham.cuh"

namespace jt {

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

// The tile's lines with an infinity or a NaN (`bad`: the thread's line b is one)
// by the FP64 passes, after the others: a finite line's result does not depend
// on its neighbours.
template <int L, int MODE, int SIGN, bool TW>
__device__ __noinline__ void fix_fp64_lines(const double2 *in, double2 *out, const StockParams &p, const double2 *W, const double2 *Whi,
                                            const double2 *Wlo, int64_t b, int t, int c, bool bad, unsigned char *smem) {
    typedef FxStock<L, MODE, SIGN, FxCfg::C(L, MODE)> F;
    typedef typename F::S S;
    if (!bad) b = 0;
    const double2 *src = in + line_off(p.lin, b);
    double2 *dst = out + line_off(p.lout, b);
    double2 d[F::E];
#pragma unroll
    for (int m = 0; m < F::E; m++) d[m] = bad ? src[(t + m * F::TL) * p.lin.estride] : make_double2(0, 0);
    int64_t j2 = 0;
    if constexpr (TW) div_fast(b, p.tw_inner, &j2);
    auto store = [&](int pos, double2 val, int) {
        if (TW) {
            const double2 w = tw_lookup<double>(Whi, Wlo, (uint32_t)pos * (uint32_t)j2, p);
            val = SIGN < 0 ? cmul<double>(val, w) : cmulc<double>(val, w);
        }
        if (p.do_scale) val = cscale<double>(val, p.scale);
        if (bad) dst[(int64_t)pos * p.lout.estride] = val;
    };
    PadIdx xi{c * S::LP};
    __syncthreads();  // the exchange buffer
    S::run_all(d, t, reinterpret_cast<double2 *>(smem), xi, W, store);
}

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
    pdl_begin();
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
    if constexpr (!F::WARP_LINE) mx = red[c];
    bool keep = valid;
    if (fp && mx >= 0xffe00000u) {
        // goes through the passes as zeros that are not stored
        mx = 0;
        keep = false;
#pragma unroll
        for (int m = 0; m < F::E; m++) d[m] = make_double2(0, 0);
    }
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
    typedef typename S::template Pass<F::NPASS - 1> LP_;
    Fx wq{0, 0}, w{0, 0};
    int4 g1 = make_int4(0, 0, 0, 0), gn = g1;
    if constexpr (TW) {
        const uint32_t g = (uint32_t)F::TL * j2;
        wq = two_level((uint32_t)t * j2);
        g1 = fx_as_factor(two_level(g));
        gn = LP_::NB > 1 ? fx_as_factor(two_level((uint32_t)LP_::NB * g)) : g1;
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
                u[k] = fx_mul<SIGN>(u[k], fx_as_factor(w));
            }
            r[k] = make_double2(fx_to(u[k].x, ex), fx_to(u[k].y, ex));
        }
        if (mul) {
#pragma unroll
            for (int k = 0; k < LP_::R; k++) r[k] = cscale<double>(r[k], f);
        }
        if (keep) {
#pragma unroll
            for (int k = 0; k < LP_::R; k++) st_hint(&dst[(int64_t)(pos + k * LP_::NS) * oes], r[k], spol);
        }
    };
    F::template run<0>(v, t, c, tid, C, xs, Wq, red, ln, store);
    if (fp) fix_fp64_lines<L, MODE, SIGN, TW>(in, out, p, W, Whi, Wlo, b, t, c, valid && !keep, smem_raw);
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
        pdl_launch(kern, (unsigned)ntiles, C * F::TL, (size_t)C * F::stride(C) * sizeof(Fx), s, in, out, p, W, Whi, Wlo, Wq, Whiq, Wloq);
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
