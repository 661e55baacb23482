// adjoint_inst.cu -- explicit instantiations of k_gloc_ad (adjoint.cuh), one translation unit for all lane groups.
#include "adjoint.cuh"

namespace dg {
AdKernel ad_kernel(int D, int mode, int *lanes) {
    const int lw = D <= 7 ? 4 : (D <= 10 ? 8 : (D <= 14 ? 16 : 32));
    *lanes = lw;
    if (D > 20) return nullptr;
    if (lw == 4) return mode == AD_VJP ? k_gloc_ad<4, AD_VJP> : k_gloc_ad<4, AD_JVP>;
    if (lw == 8) return mode == AD_VJP ? k_gloc_ad<8, AD_VJP> : k_gloc_ad<8, AD_JVP>;
    if (lw == 16) return mode == AD_VJP ? k_gloc_ad<16, AD_VJP> : k_gloc_ad<16, AD_JVP>;
    return mode == AD_VJP ? k_gloc_ad<32, AD_VJP> : k_gloc_ad<32, AD_JVP>;
}
}  // namespace dg
