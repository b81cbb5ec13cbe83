// jt_fixmath.cuh -- the 64-bit block-fixed-point arithmetic of the double
// lines (jt_fix64.cuh says why and how): conversions, twiddle products, small
// DFTs.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

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

// Fixed-point factors w are fx_root's (x, y: cosine's halves; z, w: sine's).
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

// The same without the division, for what no butterfly follows: |v| below 2^62,
// results below 2^63.  (Two units off at most.)
template <int SIGN> __device__ __forceinline__ Fx fx_mul_full(Fx v, int4 w) {
    const int xh = fx_hi(v.x), xl = fx_lo(v.x), yh = fx_hi(v.y), yl = fx_lo(v.y);
    const int ph = SIGN < 0 ? w.z : -w.z, pl = SIGN < 0 ? w.w : -w.w;
    const int nh = SIGN < 0 ? -w.z : w.z, nl = SIGN < 0 ? -w.w : w.w;
    const long long half = 1ll << 29;
    long long m = fx_madw(yl, nh, fx_madw(yh, nl, fx_madw(xl, w.x, fx_madw(xh, w.y, half))));
    Fx r;
    r.x = (fx_madw(yh, nh, fx_madw(xh, w.x, 0)) << 2) + (m >> 30);
    m = fx_madw(xl, ph, fx_madw(xh, pl, fx_madw(yl, w.x, fx_madw(yh, w.y, half))));
    r.y = (fx_madw(xh, ph, fx_madw(yh, w.x, 0)) << 2) + (m >> 30);
    return r;
}

// A factor formed at run time (a product of two), with values at 2^62.  fx_mul
// negates the sine's low half, which the lowest int does not survive: it is
// moved by one, as in the tables (fx_split).
__device__ __forceinline__ int4 fx_as_factor(Fx a) {
    if ((int)a.y == INT32_MIN) a.y++;
    return make_int4(fx_hi(a.x), fx_lo(a.x), fx_hi(a.y), fx_lo(a.y));
}

// v k / 2^64 rounded, for a constant |k| < 2^63: v times a factor in (-1/2, 1/2)
__device__ __forceinline__ long long fx_mulk(long long v, long long k) {
    const int vh = fx_hi(v), vl = fx_lo(v), kh = (int)((k + (1ll << 31)) >> 32), kl = (int)k;
    const long long m = fx_madw(vl, kh, fx_madw(vh, kl, 1ll << 31));
    return fx_madw(vh, kh, m >> 32);
}
// v k / 2^62, rounded, for 0 < k < 2^62
__device__ __forceinline__ long long fx_mulk_full(long long v, long long k) {
    const int vh = fx_hi(v), vl = fx_lo(v), kh = fx_hi(k), kl = fx_lo(k);
    const long long m = fx_madw(vl, kh, fx_madw(vh, kl, 1ll << 29));
    return (fx_madw(vh, kh, 0) << 2) + (m >> 30);
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

// v times i + k / 2^64
__device__ __forceinline__ long long fx_mulc(long long v, int i, long long k) {
    return (i > 0 ? v : i < 0 ? -v : 0) + fx_mulk(v, k);
}

template <int SIGN> __device__ __forceinline__ void fx_dft3(Fx *v) {
    const Fx t = fx_add(v[1], v[2]), d = fx_sub(v[1], v[2]);
    const Fx m{v[0].x - ((t.x + 1) >> 1), v[0].y - ((t.y + 1) >> 1)};
    long long sx = fx_mulc(d.x, 1, -2471395088767036514ll), sy = fx_mulc(d.y, 1, -2471395088767036514ll);  // sin(pi/3)
    if (SIGN < 0) {
        sx = -sx;
        sy = -sy;
    }
    v[0] = fx_add(v[0], t);
    v[1] = Fx{m.x - sy, m.y + sx};
    v[2] = Fx{m.x + sy, m.y - sx};
}

// Factors of the 5- and 7-point transforms: cosines and sines of 2 pi j / R
// as i + k / 2^64
template <int SIGN> __device__ __forceinline__ void fx_dft5(Fx *v) {
    auto c1 = [](long long x) { return fx_mulk(x, 5700357409661599243ll); };
    auto c2 = [](long long x) { return fx_mulc(x, -1, 3523014627193176565ll); };
    auto s1 = [](long long x) { return fx_mulc(x, 1, -902847917979075853ll); };
    auto s2 = [](long long x) { return fx_mulc(x, 1, -7604019954369499282ll); };
    const Fx a1 = fx_add(v[1], v[4]), a2 = fx_add(v[2], v[3]), x0 = v[0];
    Fx b1 = fx_sub(v[1], v[4]), b2 = fx_sub(v[2], v[3]);
    if (SIGN < 0) {
        b1 = Fx{-b1.x, -b1.y};
        b2 = Fx{-b2.x, -b2.y};
    }
    const Fx m1{x0.x + c1(a1.x) + c2(a2.x), x0.y + c1(a1.y) + c2(a2.y)};
    const Fx m2{x0.x + c2(a1.x) + c1(a2.x), x0.y + c2(a1.y) + c1(a2.y)};
    const Fx n1{-(s1(b1.y) + s2(b2.y)), s1(b1.x) + s2(b2.x)};
    const Fx n2{-(s2(b1.y) - s1(b2.y)), s2(b1.x) - s1(b2.x)};
    v[0] = fx_add(x0, fx_add(a1, a2));
    v[1] = fx_add(m1, n1);
    v[4] = fx_sub(m1, n1);
    v[2] = fx_add(m2, n2);
    v[3] = fx_sub(m2, n2);
}

template <int SIGN> __device__ __forceinline__ void fx_dft7(Fx *v) {
    auto c1 = [](long long x) { return fx_mulc(x, 1, -6945387266253616282ll); };
    auto c2 = [](long long x) { return fx_mulk(x, -4104786719734957267ll); };
    auto c3 = [](long long x) { return fx_mulc(x, -1, 1826801949133797741ll); };
    auto s1 = [](long long x) { return fx_mulc(x, 1, -4024498807852869538ll); };
    auto s2 = [](long long x) { return fx_mulc(x, 1, -462498387375470819ll); };
    auto s3 = [](long long x) { return fx_mulk(x, 8003742293245756417ll); };
    const Fx x0 = v[0], a1 = fx_add(v[1], v[6]), a2 = fx_add(v[2], v[5]), a3 = fx_add(v[3], v[4]);
    Fx b1 = fx_sub(v[1], v[6]), b2 = fx_sub(v[2], v[5]), b3 = fx_sub(v[3], v[4]);
    if (SIGN < 0) {
        b1 = Fx{-b1.x, -b1.y};
        b2 = Fx{-b2.x, -b2.y};
        b3 = Fx{-b3.x, -b3.y};
    }
    const Fx m1{x0.x + c1(a1.x) + c2(a2.x) + c3(a3.x), x0.y + c1(a1.y) + c2(a2.y) + c3(a3.y)};
    const Fx m2{x0.x + c2(a1.x) + c3(a2.x) + c1(a3.x), x0.y + c2(a1.y) + c3(a2.y) + c1(a3.y)};
    const Fx m3{x0.x + c3(a1.x) + c1(a2.x) + c2(a3.x), x0.y + c3(a1.y) + c1(a2.y) + c2(a3.y)};
    const Fx p1{s1(b1.x) + s2(b2.x) + s3(b3.x), s1(b1.y) + s2(b2.y) + s3(b3.y)};
    const Fx p2{s2(b1.x) - s3(b2.x) - s1(b3.x), s2(b1.y) - s3(b2.y) - s1(b3.y)};
    const Fx p3{s3(b1.x) - s1(b2.x) + s2(b3.x), s3(b1.y) - s1(b2.y) + s2(b3.y)};
    v[0] = fx_add(fx_add(x0, a1), fx_add(a2, a3));
    v[1] = Fx{m1.x - p1.y, m1.y + p1.x};
    v[6] = Fx{m1.x + p1.y, m1.y - p1.x};
    v[2] = Fx{m2.x - p2.y, m2.y + p2.x};
    v[5] = Fx{m2.x + p2.y, m2.y - p2.x};
    v[3] = Fx{m3.x - p3.y, m3.y + p3.x};
    v[4] = Fx{m3.x + p3.y, m3.y - p3.x};
}

template <int R, int SIGN> __device__ __forceinline__ void fx_dft(Fx *v) {
    if (R == 3) {
        fx_dft3<SIGN>(v);
    } else if (R == 5) {
        fx_dft5<SIGN>(v);
    } else if (R == 7) {
        fx_dft7<SIGN>(v);
    } else if (R == 2) {
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

// From the line's largest (high word << 1) over all its numbers: v below 1.4 x
// 2^58 and the largest at least 1.4 x 2^57.  A 16-point DFT of such components
// stays below 16 sqrt(2) 1.4 x 2^58 = 1.98 x 2^62; exponents alone would leave
// lines whose largest is 1.0 (normalised images, constants) a bit less.
#define JT_FX_BIAS 1081
__device__ __forceinline__ FxLine fx_line(uint32_t m) {
    const int eb = (int)((m + 1258291u) >> 21);  // mantissas of 1.4 and more (0.6 2^21) count as the next exponent
    FxLine l;
    l.pre = eb < 123 ? 512 : eb > 1923 ? -512 : 0;  // (lines of zeros too: subnormals may have no high word)
    l.ex = max(eb, 1) + l.pre - JT_FX_BIAS;
    return l;
}
// The line's numbers below 1.4 x 2^BITS (l.ex is for 58), rounded to nearest
// (cut off, they were more than FP64's rounding off in lines of 4096 and more
// with one large number).
template <int BITS = 58> __device__ __forceinline__ long long fx_from(double d, const FxLine &l) {
    const int hi = __double2hiint(d), lo = __double2loint(d);
    const int e = (hi >> 20) & 0x7ff;
    const uint32_t mh = ((uint32_t)hi & 0xfffffu) | 0x100000u;
    const int r = min(l.ex + JT_FX_BIAS + 61 - BITS - e, 63);  // at least 61 - BITS; zeros (and far smaller numbers) go to 0
    const unsigned long long u = (((unsigned long long)mh << 32) | (uint32_t)lo) << 10;
    // (negative: -u - 1, a last place of the double's off, before the shift; one
    // more of the result's halves after it, which rounds)
    return (((long long)(u ^ (long long)(hi >> 31)) >> r) + 1) >> 1;
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

}  // namespace jt
