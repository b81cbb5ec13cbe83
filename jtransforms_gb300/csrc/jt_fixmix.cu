// jt_fixmix.cu -- the mixed-radix kernel for double (jt_fixmix.cuh).
#include "jt_fixmix.cuh"

namespace jt {

__global__ void __launch_bounds__(JT_FIXMIX_THREADS, 1) fixmix_kernel(const double2 *in, double2 *out, FixMixParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_begin();
    fixmix_body(in, out, p, (int64_t)blockIdx.x, smem_raw);
}

// Pass P >= 1: factor k (1..R-1) as Ns entries w_{Ns R}^{jm k} from toff[P] on.
__global__ void fixmix_table_kernel(int4 *out, MixParams p, int count) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= count) return;
    int ps = 1;
    while (ps + 1 < p.npass && idx >= p.toff[ps + 1]) ps++;
    const int r = idx - p.toff[ps], Ns = p.Ns[ps], jm = r % Ns, k = r / Ns + 1;
    const int64_t den = (int64_t)Ns * p.R[ps], num = ((int64_t)jm * k) % den;
    out[idx] = fx_root(num, den);
}

void fixmix_setup(int smem_optin) {
    cudaFuncSetAttribute(fixmix_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
}

void fixmix_table(int4 *out, const MixParams &p, int count, cudaStream_t s) {
    fixmix_table_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(out, p, count);
}

void fixmix_launch(const double2 *in, double2 *out, const FixMixParams &p, unsigned grid, int threads, size_t smem, cudaStream_t s) {
    pdl_launch(fixmix_kernel, grid, threads, smem, s, in, out, p);
}

}  // namespace jt
