// jt_batchmix.cuh -- the float steps of a mixed batch (jt_batch.cuh): line
// passes of any layout and Bluestein's convolutions, on the register passes of
// jt_mixed.cuh.  One body serves all of them: the forms of jt_mixed.cuh and
// jt_bluemix.cuh are flags of the step here, and inverse transforms exchange
// real and imaginary parts on the way in and out.
#pragma once

#include "jt_batchmix_params.cuh"

namespace jt {

enum { BM_FIRST = 0, BM_MID = 1, BM_TURN = 2, BM_LAST = 3, BM_ONE = 4 };  // BM_ONE: first and last

__device__ __forceinline__ float2 bm_swap(float2 v) { return make_float2(v.y, v.x); }

struct BatchMixTile {
    const float2 *in;
    float2 *out;
    const BatchMix &q;
    const float2 *Whi, *Wlo;
    int64_t b0;
    int lines;

    template <int R, int KIND>
    __device__ __forceinline__ void pass(const MixParams &p, const float2 *tw, int ps, const float2 *src, float2 *dst) const {
        constexpr bool FIRST = KIND == BM_FIRST || KIND == BM_ONE, LAST = KIND == BM_LAST || KIND == BM_ONE;
        const bool cols = KIND == BM_FIRST ? q.cols_in : KIND == BM_LAST ? q.cols_out : q.cols_in && q.cols_out;
        const int nb = p.L / R, Ns = p.Ns[ps], C = p.C, total = (cols ? C : lines) * nb;
        tw += p.toff[ps];
        for (int i = threadIdx.x; i < total; i += blockDim.x) {
            int c, j;
            if (cols) {
                j = C == 1 ? i : (int)__umulhi((uint32_t)i, p.mC);
                c = i - j * C;
                if (c >= lines) continue;
            } else {
                c = nb == 1 ? i : (int)__umulhi((uint32_t)i, p.mNb[ps]);
                j = i - c * nb;
            }
            float2 v[R];
            int64_t col = 0, tr = b0 + c;
            if ((FIRST && q.chirp_in == 2) || (LAST && q.chirp_out == 2)) tr = div_fast(b0 + c, q.bl.n2, &col);
            if (FIRST && q.chirp_in) {
                const int st = q.chirp_in == 2 ? q.bl.n2 : 1;
                const float2 *g = in + tr * q.bl.din;
                int e = j * st + (int)col;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    v[k] = e < q.bl.n ? mix_chirp(g[e], q.bl, e) : make_float2(0, 0);
                    e += nb * st;
                }
            } else if (FIRST) {
                const int64_t es = p.lin.estride, step = nb * es;
                const float2 *g = in + line_off(p.lin, b0 + c) + j * es;
#pragma unroll
                for (int k = 0; k < R; k++) v[k] = g[k * step];
                if (q.chirp_out == 2) {
                    int64_t c2;
                    div_fast(b0 + c, q.bl.n2, &c2);
                    const float2 *w = q.bl.tw + j * q.bl.n2 + c2;
#pragma unroll
                    for (int k = 0; k < R; k++) v[k] = cmulc<float>(v[k], __ldg(w + k * nb * q.bl.n2));
                }
                if (q.inv) {
#pragma unroll
                    for (int k = 0; k < R; k++) v[k] = bm_swap(v[k]);
                }
            } else {
                const float2 *s = src + c * p.Lp + j;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    v[k] = *s;
                    s += nb;
                }
            }
            int base = j * R;
            if (!FIRST) {
                const int jm = KIND != BM_MID ? j : j - (int)__umulhi((uint32_t)j, p.mNs[ps]) * Ns;
                base -= jm * (R - 1);
                mix_twiddle<R, -1>(v, tw, Ns, jm);
            }
            dft_any<R, -1, float>(v);
            if (KIND == BM_TURN) {
                int64_t row = 0;
                if (q.n1 > 1) div_fast(b0 + c, q.n1, &row);
                const float2 *B = q.Bp + row * p.L + j;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    const float2 w = __ldg(B + k * nb);
                    v[k] = bm_swap(q.bl.inv ? cmulc<float>(v[k], w) : cmul<float>(v[k], w));
                }
                dft_any<R, -1, float>(v);
                base = j * R;
            }
            if (LAST) {
                if (q.chirp_in == 2) {
                    const float2 *w = q.bl.tw;
                    int64_t c2;
                    div_fast(b0 + c, q.bl.n2, &c2);
                    w += base * q.bl.n2 + c2;
#pragma unroll
                    for (int k = 0; k < R; k++) v[k] = cmul<float>(v[k], __ldg(w + k * Ns * q.bl.n2));
                } else if (p.tw_n) {
                    int64_t j2;
                    div_fast(b0 + c, p.tw_inner, &j2);
                    uint32_t e = (uint32_t)base * (uint32_t)j2;
                    const uint32_t de = (uint32_t)Ns * (uint32_t)j2, mask = (1u << p.tw_lo_bits) - 1u;
#pragma unroll
                    for (int k = 0; k < R; k++) {
                        v[k] = cmul<float>(v[k], cmul<float>(__ldg(&Whi[e >> p.tw_lo_bits]), __ldg(&Wlo[e & mask])));
                        e += de;
                    }
                }
                if (q.inv || q.turn) {
#pragma unroll
                    for (int k = 0; k < R; k++) v[k] = bm_swap(v[k]);
                }
                if (q.chirp_out) {
                    const int st = q.chirp_out == 2 ? q.bl.n2 : 1;
                    float2 *g = out + tr * q.bl.dout;
                    int e = base * st + (int)col;
#pragma unroll
                    for (int k = 0; k < R; k++) {
                        if (e < q.bl.n) g[e] = cscale<float>(mix_chirp(v[k], q.bl, e), q.bl.scale);
                        e += Ns * st;
                    }
                } else {
                    const int64_t es = p.lout.estride, step = Ns * es;
                    float2 *g = out + line_off(p.lout, b0 + c) + base * es;
#pragma unroll
                    for (int k = 0; k < R; k++) g[k * step] = p.do_scale ? cscale<float>(v[k], p.scale) : v[k];
                }
            } else {
                float2 *d = dst + c * p.Lp + base;
                const int step = KIND == BM_MID ? Ns : 1;
#pragma unroll
                for (int k = 0; k < R; k++) {
                    *d = v[k];
                    d += step;
                }
            }
        }
    }
    template <int KIND> __device__ __noinline__ void any(const MixParams &p, const float2 *tw, int ps, const float2 *src, float2 *dst) const {
        switch (p.R[ps]) {
#define JT_BM(RR) \
    case RR: pass<RR, KIND>(p, tw, ps, src, dst); break;
            JT_BM(4) JT_BM(5) JT_BM(6) JT_BM(7) JT_BM(8) JT_BM(9) JT_BM(10) JT_BM(12) JT_BM(16)
            default:
                if constexpr (KIND != BM_TURN) {
                    switch (p.R[ps]) {
                        JT_BM(2) JT_BM(3) JT_BM(11) JT_BM(13) JT_BM(14) JT_BM(15)
                    }
                }
#undef JT_BM
        }
    }
    __device__ __forceinline__ void run(float2 *A, float2 *B) const {
        const int np = q.f.npass;
        if (np == 1) {
            any<BM_ONE>(q.f, q.twf, 0, nullptr, nullptr);
            return;
        }
        auto next = [&] {
            __syncthreads();
            float2 *t = A;
            A = B;
            B = t;
        };
        any<BM_FIRST>(q.f, q.twf, 0, nullptr, B);
        next();
        for (int ps = 1; ps < np - 1; ps++) {
            any<BM_MID>(q.f, q.twf, ps, A, B);
            next();
        }
        if (!q.turn) {
            any<BM_LAST>(q.f, q.twf, np - 1, A, nullptr);
            return;
        }
        any<BM_TURN>(q.f, q.twf, np - 1, A, B);
        next();
        for (int ps = 1; ps < np - 1; ps++) {
            any<BM_MID>(q.g, q.twg, ps, A, B);
            next();
        }
        any<BM_LAST>(q.g, q.twg, np - 1, A, nullptr);
    }
};

// Task `blk` of a step; two buffers of C lines at smem_raw.
__device__ __noinline__ void batch_mix_body(const float2 *in, float2 *out, const BatchMix &q, const float2 *Whi, const float2 *Wlo,
                                            int64_t blk, unsigned char *smem_raw) {
    const int64_t b0 = blk * q.f.C;
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    BatchMixTile{in, out, q, Whi, Wlo, b0, (int)min((int64_t)q.f.C, q.f.nlines - b0)}.run(A, A + q.f.C * q.f.Lp);
}

}  // namespace jt
