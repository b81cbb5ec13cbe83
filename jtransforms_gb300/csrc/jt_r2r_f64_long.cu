// jt_r2r_f64_long.cu -- instantiations of the DCT/DST/DHT and packed real line
// kernels for double (jt_fixr2r.cuh), half lengths 256..4096.
#include "jt_fixr2r.cuh"

namespace jt {

bool fix_r2r_launch_long(int H, int op, bool strided, const double *in, double *out, const R2rParams &p, const FixR2rScale &fs,
                    const double2 *Wp, const double2 *Wr, const double2 *Wd, const int4 *Wpq, const int4 *Wrq, const int4 *Wdq,
                    int sms, cudaStream_t s) {
#define JT_RCASE(HH) \
    case HH: return FixR2rLaunch<HH>::go(op, strided, in, out, p, fs, Wp, Wr, Wd, Wpq, Wrq, Wdq, sms, s);
    switch (H) {
        JT_RCASE(256)
        JT_RCASE(512)
        JT_RCASE(1024)
        JT_RCASE(2048)
        JT_RCASE(4096)
        default: return false;
    }
#undef JT_RCASE
}

}  // namespace jt
