// adjoint_inst.cu -- explicit instantiations of k_gloc_ad (adjoint.cuh), one translation unit for all lane groups.
#include "adjoint.cuh"

namespace dg {
template <int LW>
static AdKernel pick(int mode) {
    switch (mode) {
        case AD_VJP: return k_gloc_ad<LW, AD_VJP>;
        case AD_JVP: return k_gloc_ad<LW, AD_JVP>;
        case AD_BLOCK: return k_gloc_ad<LW, AD_BLOCK>;
        default: return k_gloc_ad<LW, AD_TRACE>;
    }
}
AdKernel ad_kernel(int D, int mode, int *lanes) {
    *lanes = D <= 7 ? 4 : (D <= 10 ? 8 : (D <= 14 ? 16 : 32));
    if (D > 20) return nullptr;
    return *lanes == 4 ? pick<4>(mode) : (*lanes == 8 ? pick<8>(mode) : (*lanes == 16 ? pick<16>(mode) : pick<32>(mode)));
}
}  // namespace dg
