// jt_pow2_f64.cu -- instantiations of the power-of-two line kernels for
// double (jt_fix64.cuh).
#include "jt_fix64.cuh"

namespace jt {

// Launches the kernel for line length L; returns false when (L, mode) has no
// instantiation (row mode: 16..8192, column modes: 16..4096).  Whiq, Wloq: the
// fixed-point forms of the two-level four-step tables Whi, Wlo; W's follow W.
bool fix_launch(int L, int mode, int sign, const double2 *in, double2 *out, const StockParams &p, const double2 *W,
                const double2 *Whi, const double2 *Wlo, const int4 *Whiq, const int4 *Wloq, int sms, cudaStream_t s) {
    const int4 *Wq = reinterpret_cast<const int4 *>(W + stock_tw_count(L, fx_elems(L)));
#define JT_CASE(LL)                                                                          \
    case LL:                                                                                 \
        FixLaunch<LL>::go(mode, sign, in, out, p, W, Whi, Wlo, Wq, Whiq, Wloq, sms, s);           \
        return true;
    switch (L) {
        JT_CASE(16) JT_CASE(32) JT_CASE(64) JT_CASE(128) JT_CASE(256) JT_CASE(512) JT_CASE(1024)
        JT_CASE(2048) JT_CASE(4096)
        case 8192:
            if (mode != 0) return false;
            FixLaunch<8192>::go(mode, sign, in, out, p, W, Whi, Wlo, Wq, Whiq, Wloq, sms, s);
            return true;
        default: return false;
    }
#undef JT_CASE
}

}  // namespace jt
