// jt_mixed_inv.cu -- the mixed-radix line kernel (jt_mixed.cuh) for float,
// inverse.
#include "jt_mixed.cuh"

namespace jt {

void mix_launch_inv(int mode, const float2 *in, float2 *out, const MixParams &p, const float2 *tw, const float2 *Whi,
                     const float2 *Wlo, unsigned grid, int threads, size_t smem, cudaStream_t s) {
    if (mode == 0) pdl_launch(mix_kernel<1, 0>, grid, threads, smem, s, in, out, p, tw, Whi, Wlo);
    else if (mode == 1) pdl_launch(mix_kernel<1, 1>, grid, threads, smem, s, in, out, p, tw, Whi, Wlo);
    else pdl_launch(mix_kernel<1, 2>, grid, threads, smem, s, in, out, p, tw, Whi, Wlo);
}

void mix_setup_inv(int smem_optin) {
    cudaFuncSetAttribute(mix_kernel<1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
    cudaFuncSetAttribute(mix_kernel<1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
    cudaFuncSetAttribute(mix_kernel<1, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
}

}  // namespace jt
