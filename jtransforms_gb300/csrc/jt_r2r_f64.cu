// jt_r2r_f64.cu -- instantiations of the DCT/DST/DHT and packed real line
// kernels for double (jt_fixr2r.cuh), half lengths 16..128.
#include "jt_fixr2r.cuh"

namespace jt {

bool fix_r2r_launch(int H, int op, bool strided, const double *in, double *out, const R2rParams &p, const FixR2rScale &fs,
                    const double2 *Wp, const double2 *Wr, const double2 *Wd, const int4 *Wpq, const int4 *Wrq, const int4 *Wdq,
                    int sms, cudaStream_t s) {
#define JT_RCASE(HH) \
    case HH: return FixR2rLaunch<HH>::go(op, strided, in, out, p, fs, Wp, Wr, Wd, Wpq, Wrq, Wdq, sms, s);
    switch (H) {
        JT_RCASE(16)
        JT_RCASE(32)
        JT_RCASE(64)
        JT_RCASE(128)
        default: return false;
    }
#undef JT_RCASE
}

}  // namespace jt
