// jt_fixr2r.cuh -- DCT-II/III, DST-II/III, DHT and packed real lines of doubles
// in one kernel each, in the 64-bit block fixed point of jt_fix64.cuh: the
// line operations of jt_r2r.cuh for power-of-two half lengths H = 16..4096.
//
// A thread holds E (16 or 8) of the line's H complex values, t + m H/E.  Everything
// around the H-point FFT works on pairs (k, H - k) or (j, H - 1 - j): the
// lower half of the line (m < E/2) stays in the thread's registers and only the
// upper half changes hands through shared memory.  Inputs come from global
// memory into registers and outputs go from registers to global memory, in
// runs across t (rows) or across lines (columns); nothing is staged.
//
//   DCT-II / DST-II  the four reals x_4m .. x_4m+3 are z_m = (x_4m, x_4m+2)
//                    and z_{H-1-m} = (x_4m+3, x_4m+1) (DST: odd ones negated);
//                    after the FFT V_k = (a - i w_k d) / 2 and V_{H-k} = (conj a -
//                    i conj(w_k d)) / 2, a, d = Z_k +- conj Z_{H-k}; with u =
//                    e^{-i pi k/2n} V_k: C_k = Re u, C_{n-k} = -Im u
//   DHT              H_k = Re V_k - Im V_k, H_{n-k} = Re V_k + Im V_k
//   realForward      X_k = V_k
//   DCT-III / DST-III  V_k = e^{i pi k/2n} (C_k - i C_{n-k}), Z_k = (s + i w d) / 2
//                    and Z_{H-k} = (conj s + i conj(w d)) / 2 with s, d = V_k +- conj
//                    V_{H-k}, w = e^{2 pi i k/n}; after the FFT the reverse of
//                    DCT-II's reordering
//   realInverse      the same with X in the place of V
//
// What bounded the FP64 form (jt_r2r.cuh) was the FP64 pipe; see jt_fix64.cuh.
// Lines with an infinity or a NaN still run it.  Measured (GB300, both
// directions): DoubleDCT_2D(1024^2) 72 us where the FP64 form took 254,
// DoubleDHT_3D(128^3) 116 where it took 508.  Relative L2 error
// of DCTs of noise and images, 32^2 to 1024^2, against quad precision: 6.4-8.0e-17,
// 2.0-3.7e-16 before.
// At these sizes a kernel is one wave of few warps and bound by their
// latency: of the 10 cycles between two of a warp's instructions 3 to 4 wait
// for its loads and 1.4 for shared memory.
#pragma once

#include "jt_fix64.cuh"
#include "jt_r2r.cuh"

namespace jt {

template <int H, int MODE, int OP> struct FixR2r {
    static constexpr int SIGN = r2r_inverse(OP) ? 1 : -1;
    // most lines per CTA: 128 threads or one line; columns at least four
    // (32-byte runs)
    static constexpr int CM = MODE == 0 ? FxCfg::rows_C(H) : H <= 128 ? 128 * fx_elems(H) / H : H <= 256 ? 16 : H <= 512 ? 8 : 4;
    typedef FxStock<H, MODE, SIGN, CM> F;
};

// The FP64 form of the calling CTA's lines with an infinity or a NaN (marks),
// one at a time, after the others: a finite line's result does not depend on
// its neighbours.
template <int H, int OP>
__device__ __noinline__ void fix_r2r_fp64(const double *in, double *out, const R2rParams &p, const double2 *Wp, const double2 *Wr,
                                          const double2 *Wd, const bool *marks, unsigned char *smem) {
    const int64_t b0 = (int64_t)blockIdx.x * p.C;
    const int lines = (int)min((int64_t)p.C, p.nlines - b0);
    R2rParams q = p;
    q.nlines = b0 + 1;  // one line, in the place of the CTA's first
    __syncthreads();
    for (int l = 0; l < lines; l++) {
        if (!marks[l]) continue;
        r2r_reg_body<double, H, OP, fx_elems(H)>(in + (line_off(p.lin, b0 + l) - line_off(p.lin, b0)),
                                                 out + (line_off(p.lout, b0 + l) - line_off(p.lout, b0)), q, Wp, Wr, Wd, smem);
        __syncthreads();
    }
}

// The finite lines of the calling CTA; returns whether others are left (marks).
template <int H, int MODE, int OP>
__device__ __forceinline__ bool fix_r2r_lines(const double *in, double *out, const R2rParams &p, const FixR2rScale &fs,
                                              const int4 *__restrict__ Wpq, const int4 *__restrict__ Wrq,
                                              const int4 *__restrict__ Wdq, bool *marks, unsigned char *smem_raw) {
    typedef typename FixR2r<H, MODE, OP>::F F;
    typedef typename F::S S;
    constexpr int n = 2 * H, TL = F::TL, E = F::E, EH = E / 2;
    auto pad = [](int i) { return F::pad(i); };
    __shared__ uint32_t red[F::RED];
    Fx *xs = reinterpret_cast<Fx *>(smem_raw);
    double2 *xd = reinterpret_cast<double2 *>(smem_raw);
    const int tid = threadIdx.x, NT = blockDim.x, C = NT / TL;
    const int c = MODE == 0 ? tid / TL : tid & (C - 1), t = MODE == 0 ? tid % TL : tid / C;
    const int64_t b = (int64_t)blockIdx.x * C + c;
    const bool valid = b < p.nlines;
    const int base = c * F::stride(C);
    if constexpr (!F::WARP_LINE)
        for (int i = tid; i < F::RED; i += NT) red[i] = 0;
    const double *src = in + (valid ? line_off(p.lin, b) : 0);
    double *dst = out + (valid ? line_off(p.lout, b) : 0);
    const int64_t es = MODE == 0 ? 1 : p.lin.estride, os = MODE == 0 ? 1 : p.lout.estride;
    const bool vec = MODE == 0 && p.vec_in, vec_out = MODE == 0 && p.vec_out;
    // scalars i, i + 1 of the line (i even)
    auto pair_in = [&](int i) -> double2 {
        if (!valid) return make_double2(0, 0);
        if (vec) return *reinterpret_cast<const double2 *>(src + i);
        return make_double2(src[(int64_t)i * es], src[(int64_t)(i + 1) * es]);
    };
    auto one_in = [&](int i) -> double { return valid ? src[(int64_t)i * es] : 0.0; };
    // partner of pair k = t + m TL (m < 8): H - k; k = 0 stands alone and
    // takes H / 2, its own partner, along
    auto partner = [&](int m) -> int { return m == 0 && t == 0 ? H / 2 : H - (t + m * TL); };

    // ---- load -----------------------------------------------------------
    double2 d[E];
    if constexpr (OP == R2R_DCT2) {
#pragma unroll
        for (int m = 0; m < EH; m++) {
            const int k = t + m * TL;
            const double2 u = pair_in(4 * k), w = pair_in(4 * k + 2);
            d[m] = make_double2(u.x, w.x);
            d[EH + m] = make_double2(w.y, u.y);  // z_{H-1-k}, for another thread
        }
        if (p.dst) {
#pragma unroll
            for (int m = EH; m < E; m++) d[m] = make_double2(-d[m].x, -d[m].y);
        }
#pragma unroll
        for (int m = 0; m < EH; m++) xd[base + pad(H - 1 - t - m * TL)] = d[EH + m];
    } else if constexpr (OP == R2R_DCT3) {
        // d[m] = (C_k, C_{n-k}), d[EH + m] = (C_{H-k}, C_{H+k}); k = 0: (C_0, 0)
        // and d[EH] = (C_H, 0) go with H / 2's pair (C_{H/2}, C_{3H/2}), below
        auto coef = [&](int k) { return one_in(p.dst ? n - 1 - k : k); };
#pragma unroll
        for (int m = 0; m < EH; m++) {
            const int k = t + m * TL;
            const bool z = m == 0 && t == 0;
            d[m] = make_double2(coef(k), coef(z ? 3 * H / 2 : n - k));
            d[EH + m] = make_double2(coef(z ? H / 2 : H - k), coef(H + k));
        }
    } else if constexpr (OP == R2R_RINV) {
        // d[m] = X_k, d[EH + m] = X_{H-k}; k = 0: (X_0, X_H), X_{H/2}
#pragma unroll
        for (int m = 0; m < EH; m++) {
            d[m] = pair_in(2 * (t + m * TL));
            d[EH + m] = pair_in(2 * partner(m));
        }
    } else {
#pragma unroll
        for (int m = 0; m < E; m++) d[m] = pair_in(2 * (t + m * TL));
    }
    uint32_t mx = 0;
#pragma unroll
    for (int m = 0; m < E; m++)
        mx = max(mx, max((uint32_t)__double2hiint(d[m].x) << 1, (uint32_t)__double2hiint(d[m].y) << 1));
    const bool special = mx >= 0xffe00000u;  // an infinity or a NaN
    mx = F::template warp_red<true>(mx, C);
    if constexpr (!F::WARP_LINE) {
        __syncthreads();  // red is zeroed
        if (MODE == 0 ? tid % 32 == 0 : tid % 32 < C) atomicMax(&red[c], mx);
    }
    const bool fp = __syncthreads_or(special);
    if constexpr (!F::WARP_LINE) mx = red[c];
    if constexpr (OP == R2R_DCT2) {
#pragma unroll
        for (int m = EH; m < E; m++) d[m] = xd[base + pad(t + m * TL)];
    }
    bool keep = valid;
    if (fp) {
        if (t == 0) marks[c] = mx >= 0xffe00000u;
        if (mx >= 0xffe00000u) {
            // goes through the passes as zeros that are not stored
            mx = 0;
            keep = false;
#pragma unroll
            for (int m = 0; m < E; m++) d[m] = make_double2(0, 0);
        }
    }
    FxLine ln = fx_line(mx);
    const bool scaled = __any_sync(0xffffffffu, ln.pre != 0);
    if (scaled) {
        const double f = fx_pre(ln.pre);
#pragma unroll
        for (int m = 0; m < E; m++) d[m] = cscale<double>(d[m], f);
    }
    Fx v[E];
    if constexpr (r2r_inverse(OP)) {
        // ---- Z of the inverse FFT ---------------------------------------
        uint32_t bits = 0;
#pragma unroll
        for (int m = 0; m < EH; m++) {
            const int k = t + m * TL;
            const bool z = m == 0 && t == 0;
            constexpr int BITS = OP == R2R_DCT3 ? 61 : 59;
            Fx X{fx_from<BITS>(d[m].x, ln), fx_from<BITS>(d[m].y, ln)}, Y{fx_from<BITS>(d[EH + m].x, ln), fx_from<BITS>(d[EH + m].y, ln)};
            Fx X0{0, 0};  // k = 0: (X_0, X_H)
            if (OP == R2R_DCT3) {
                // V = e^{+i pi k/2n} (C_k - i C_{n-k}) / 4
                if (z) {
                    // V_0 = C_0, V_H = e^{i pi/4} (1 - i) C_H = sqrt(2) C_H
                    const long long ch = Y.y;
                    if (fs.c0 == 1) X.x += fx_mulk(X.x, kFxR2m1);
                    X0 = fx_shr(Fx{X.x << (fs.c0 == 2), ch + fx_mulk(ch, kFxR2m1)}, 2, 2);
                    X = Fx{Y.x, X.y};  // the pair of H / 2
                    X = fx_mul<1>(Fx{X.x, -X.y}, __ldg(&Wdq[H / 2]));
                    Y = X;
                } else {
                    X = fx_mul<1>(Fx{X.x, -X.y}, __ldg(&Wdq[k]));
                    Y = fx_mul<1>(Fx{Y.x, -Y.y}, __ldg(&Wdq[H - k]));
                }
            } else if (z) {
                X0 = X;
                X = Y;
            }
            // (59 bits here and sums of four numbers: no division until all are known)
            const Fx s{X.x + Y.x, X.y - Y.y}, dd{X.x - Y.x, X.y + Y.y};
            const Fx w = fx_mul_full<1>(dd, __ldg(&Wrq[z ? H / 2 : k]));  // e^{+2 pi i k/n} d
            v[m] = Fx{s.x - w.y, s.y + w.x};
            Fx u{s.x + w.y, w.x - s.y};
            if (z) {
                u = v[m];
                v[m] = Fx{X0.x + X0.y, X0.x - X0.y};
            }
            bits |= fx_bits(v[m].x) | fx_bits(v[m].y) | fx_bits(u.x) | fx_bits(u.y);
            xs[base + pad(partner(m))] = u;
        }
        bits = F::template line_red<false>(bits, F::NPASS + 1, c, tid, C, red);
#pragma unroll
        for (int m = EH; m < E; m++) v[m] = xs[base + pad(t + m * TL)];
        F::line_sync();
        const int s = fx_norm_shift<58>(bits);
        fx_norm<E>(v, s);
        // from 59 bits (the DCT's from 61, over 4), and the half of Z
        ln.ex += -1 - 1 + s;
    } else {
#pragma unroll
        for (int m = 0; m < E; m++) v[m] = Fx{fx_from(d[m].x, ln), fx_from(d[m].y, ln)};
        if constexpr (OP == R2R_DCT2) F::line_sync();  // the staged inputs are read
    }
    // ---- the H-point FFT: v[m] ends as Z_{t + m TL} ----------------------
    {
        typedef typename S::template Pass<F::NPASS - 1> LP_;
        Fx z[E];
        auto store = [&](int, Fx *u, int q) {
#pragma unroll
            for (int k = 0; k < LP_::R; k++) z[q + k * LP_::NB] = u[k];
        };
        F::template run<0>(v, t, c, tid, C, xs, Wpq, red, ln, store);
#pragma unroll
        for (int m = 0; m < E; m++) v[m] = z[m];
    }
    const int nk = fs.k != 0;
    auto real_out = [&](long long x) -> long long { return nk ? fx_mulk_full(x, fs.k) : x; };
    const bool mul = scaled;
    const double f = fx_pre(-ln.pre);
    // ---- output ---------------------------------------------------------
    if constexpr (OP == R2R_RINV) {
        const int ex = ln.ex + fs.e2;
        double2 r[E];
#pragma unroll
        for (int m = 0; m < E; m++) r[m] = make_double2(fx_to(real_out(v[m].x), ex), fx_to(real_out(v[m].y), ex));
        if (mul) {
#pragma unroll
            for (int m = 0; m < E; m++) r[m] = cscale<double>(r[m], f);
        }
        if (keep) {
#pragma unroll
            for (int m = 0; m < E; m++) {
                const int i = 2 * (t + m * TL);
                if (vec_out) {
                    *reinterpret_cast<double2 *>(dst + i) = r[m];
                } else {
                    dst[(int64_t)i * os] = r[m].x;
                    dst[(int64_t)(i + 1) * os] = r[m].y;
                }
            }
        }
        return fp;
    }
    if constexpr (F::NPASS > 1) F::line_sync();  // the last exchange is read
    if constexpr (OP == R2R_DCT3) {
        const int ex = ln.ex + fs.e2;
#pragma unroll
        for (int m = EH; m < E; m++) xs[base + pad(t + m * TL)] = v[m];
        F::line_sync();
#pragma unroll
        for (int m = 0; m < EH; m++) {
            const int k = t + m * TL;
            const Fx u = xs[base + pad(H - 1 - k)];
            double r0 = fx_to(real_out(v[m].x), ex), r1 = fx_to(real_out(u.y), ex), r2 = fx_to(real_out(v[m].y), ex),
                   r3 = fx_to(real_out(u.x), ex);
            if (p.dst) {
                r1 = -r1;
                r3 = -r3;
            }
            if (mul) {
                r0 *= f;
                r1 *= f;
                r2 *= f;
                r3 *= f;
            }
            if (keep) {
                if (vec_out) {
                    *reinterpret_cast<double2 *>(dst + 4 * k) = make_double2(r0, r1);
                    *reinterpret_cast<double2 *>(dst + 4 * k + 2) = make_double2(r2, r3);
                } else {
                    double *o = dst + (int64_t)(4 * k) * os;
                    o[0] = r0;
                    o[os] = r1;
                    o[2 * os] = r2;
                    o[3 * os] = r3;
                }
            }
        }
        return fp;
    }
    uint32_t bits = 0;
#pragma unroll
    for (int m = 0; m < E; m++) bits |= fx_bits(v[m].x) | fx_bits(v[m].y);
#pragma unroll
    for (int m = EH; m < E; m++) xs[base + pad(t + m * TL)] = v[m];
    bits = F::template line_red<false>(bits, F::NPASS, c, tid, C, red);
    const int s = fx_norm_shift(bits);
    // V doubled, below 2^62 (60 bits before, |A|, |B| below sqrt(2) 2^60): no
    // division by the last products either.  (Each one's 2 bits made a line with
    // one large coefficient, as an image's, up to 5 times as far off as FP64.)
    const int ex0 = ln.ex + s - 1, ex = ex0 + fs.e2;
#pragma unroll
    for (int m = 0; m < EH; m++) {
        const int k = t + m * TL;
        const bool z = m == 0 && t == 0;
        Fx zz[2] = {v[m], xs[base + pad(partner(m))]};
        fx_norm<2>(zz, s);
        Fx A = zz[0], B = zz[1];
        if (z) A = B;  // Z_{H/2}; Z_0 below
        const Fx a{A.x + B.x, A.y - B.y}, dd{A.x - B.x, A.y + B.y};
        const Fx wd = fx_mul_full<-1>(dd, __ldg(&Wrq[z ? H / 2 : k]));
        Fx V{a.x + wd.y, a.y - wd.x};     // V_k (doubled), k = 0: V_{H/2}
        Fx U{a.x - wd.y, -a.y - wd.x};    // V_{H-k}
        if (z) {
            U = V;
            // V_0 = Z_0.x + Z_0.y, V_H = Z_0.x - Z_0.y (doubled)
            V = Fx{(zz[0].x + zz[0].y) << 1, (zz[0].x - zz[0].y) << 1};
        }
        long long q0, q1, q2, q3;  // of k, n - k, H - k, H + k (k = 0: 0, 3H/2, H/2, H)
        if constexpr (OP == R2R_DHT) {
            q0 = z ? V.x : V.x - V.y;
            q1 = V.x + V.y;
            q2 = U.x - U.y;
            q3 = U.x + U.y;
            if (z) {
                q1 = q3;
                q3 = V.y;
            }
        } else if constexpr (OP == R2R_RFWD) {
            q0 = V.x;
            q1 = V.y;
            q2 = U.x;
            q3 = U.y;
        } else {
            const Fx y = fx_mul_full<-1>(U, __ldg(&Wdq[z ? H / 2 : H - k]));
            q2 = y.x;
            q3 = -y.y;
            if (z) {
                q0 = V.x;
                q1 = -y.y;
                q3 = fx_mulh(V.y);  // C_H = cos(pi/4) V_H
            } else {
                const Fx x = fx_mul_full<-1>(V, __ldg(&Wdq[k]));
                q0 = x.x;
                q1 = -x.y;
            }
        }
        double r0 = fx_to(real_out(q0), ex), r1 = fx_to(real_out(q1), ex), r2 = fx_to(real_out(q2), ex), r3 = fx_to(real_out(q3), ex);
        if (OP == R2R_DCT2 && z) r0 = fx_to(fs.k0 ? fx_mulk_full(q0, fs.k0) : q0, ex0 + fs.e20);
        if (mul) {
            r0 *= f;
            r1 *= f;
            r2 *= f;
            r3 *= f;
        }
        if (!keep) continue;
        if constexpr (OP == R2R_RFWD) {
            const int i = 2 * k, j = 2 * partner(m);
            if (vec_out) {
                *reinterpret_cast<double2 *>(dst + i) = make_double2(r0, r1);
                *reinterpret_cast<double2 *>(dst + j) = make_double2(r2, r3);
            } else {
                dst[(int64_t)i * os] = r0;
                dst[(int64_t)(i + 1) * os] = r1;
                dst[(int64_t)j * os] = r2;
                dst[(int64_t)(j + 1) * os] = r3;
            }
        } else {
            const bool rev = OP == R2R_DCT2 && p.dst;
            auto put = [&](int i, double x) { dst[(int64_t)(rev ? n - 1 - i : i) * os] = x; };
            put(k, r0);
            put(z ? 3 * H / 2 : n - k, r1);
            put(z ? H / 2 : H - k, r2);
            put(H + k, r3);
        }
    }
    return fp;
}

template <int H, int MODE, int OP>
__global__ void __launch_bounds__(FixR2r<H, MODE, OP>::F::NT, FixR2r<H, MODE, OP>::F::MINB)
    fix_r2r_kernel(const double *in, double *out, R2rParams p, FixR2rScale fs, const double2 *__restrict__ Wp,
                   const double2 *__restrict__ Wr, const double2 *__restrict__ Wd, const int4 *__restrict__ Wpq,
                   const int4 *__restrict__ Wrq, const int4 *__restrict__ Wdq) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ bool marks[FixR2r<H, MODE, OP>::CM];
    pdl_begin();
    if (fix_r2r_lines<H, MODE, OP>(in, out, p, fs, Wpq, Wrq, Wdq, marks, smem_raw))
        fix_r2r_fp64<H, OP>(in, out, p, Wp, Wr, Wd, marks, smem_raw);
}

// Launches one (H, op); strided lines up to H = 2048 (longer ones would move
// in runs under 32 bytes).
template <int H> struct FixR2rLaunch {
    template <int MODE, int OP>
    static void one(const double *in, double *out, R2rParams p, const FixR2rScale &fs, const double2 *Wp, const double2 *Wr,
                    const double2 *Wd, const int4 *Wpq, const int4 *Wrq, const int4 *Wdq, int sms, cudaStream_t s) {
        typedef FixR2r<H, MODE, OP> G;
        typedef typename G::F F;
        static bool attr = false;
        if (!attr) {
            cudaFuncSetAttribute(fix_r2r_kernel<H, MODE, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::SMEM);
            attr = true;
        }
        p.C = fix_lines(p.nlines, G::CM, std::min(G::CM, std::max(F::CMIN, MODE == 0 ? 1 : 4)), sms);
        const int64_t grid = (p.nlines + p.C - 1) / p.C;
        pdl_launch(fix_r2r_kernel<H, MODE, OP>, (unsigned)grid, p.C * F::TL, (size_t)p.C * F::stride(p.C) * sizeof(Fx), s, in, out, p, fs,
                   Wp, Wr, Wd, Wpq, Wrq, Wdq);
    }
    template <int MODE, typename... A> static void op(int op, A... a) {
        if (op == R2R_DCT2) one<MODE, R2R_DCT2>(a...);
        else if (op == R2R_DCT3) one<MODE, R2R_DCT3>(a...);
        else if (op == R2R_DHT) one<MODE, R2R_DHT>(a...);
        else if constexpr (MODE == 0) {  // packed real lines are rows
            if (op == R2R_RFWD) one<MODE, R2R_RFWD>(a...);
            else one<MODE, R2R_RINV>(a...);
        }
    }
    template <typename... A> static bool go(int o, bool strided, A... a) {
        if (strided) {
            if (H > 2048 || o == R2R_RFWD || o == R2R_RINV) return false;
            if constexpr (H <= 2048) op<1>(o, a...);
        } else {
            op<0>(o, a...);
        }
        return true;
    }
};

}  // namespace jt
