// jt_bluemix.cu -- launchers of the float Bluestein kernels (jt_bluemix.cuh).
#include "jt_bluemix.cuh"

namespace jt {

void blue_setup(int smem_optin) {
    cudaFuncSetAttribute(blue_mid_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
    cudaFuncSetAttribute(blue_mid_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
    cudaFuncSetAttribute(blue_cols_kernel<-1, MIX_BLUE_IN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
    cudaFuncSetAttribute(blue_cols_kernel<1, MIX_BLUE_OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
}

void blue_mid(bool one, const float2 *in, float2 *out, const BlueMid &q, unsigned grid, int threads, size_t smem, cudaStream_t s) {
    if (one) pdl_launch(blue_mid_kernel<true>, grid, threads, smem, s, in, out, q);
    else pdl_launch(blue_mid_kernel<false>, grid, threads, smem, s, in, out, q);
}

void blue_cols(bool first, const float2 *in, float2 *out, const MixParams &p, const MixBlue &bl, const float2 *tw, unsigned grid,
               int threads, size_t smem, cudaStream_t s) {
    if (first) pdl_launch(blue_cols_kernel<-1, MIX_BLUE_IN>, grid, threads, smem, s, in, out, p, bl, tw);
    else pdl_launch(blue_cols_kernel<1, MIX_BLUE_OUT>, grid, threads, smem, s, in, out, p, bl, tw);
}

void blue_twiddle(float2 *out, int n1, int n2, cudaStream_t s) {
    blue_twiddle_kernel<<<(unsigned)((n1 * n2 + 255) / 256), 256, 0, s>>>(out, n1, n2);
}

void blue_spectrum(float2 *out, const double2 *in, int64_t n1, int64_t n2, cudaStream_t s) {
    blue_spectrum_kernel<<<(unsigned)((n1 * n2 + 255) / 256), 256, 0, s>>>(out, in, n1, n2);
}

}  // namespace jt
