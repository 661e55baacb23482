// schur_tpi.cu -- instantiations of the thread-per-frequency BLOCK kernel k_schur_tpi (schur.cuh), D = 1 .. 3.
#include "schur.cuh"

namespace dg {
template <class Ops, int D>
static SchurKernel pick(int mode) {
    if (mode == S_BLOCK) return k_schur_tpi<Ops, D>;
    if (mode == S_TRACE) return k_trace_tpi<Ops, D, false>;
    if (mode == (S_TRACE | S_DERIV)) return k_trace_tpi<Ops, D, true>;
    return nullptr;
}
SchurKernel schur_tpi_kernel(int D, int mode, bool mixed) {
    switch (D) {
        case 1: return mixed ? pick<OpsP, 1>(mode) : pick<OpsD, 1>(mode);
        case 2: return mixed ? pick<OpsP, 2>(mode) : pick<OpsD, 2>(mode);
        case 3: return mixed ? pick<OpsP, 3>(mode) : pick<OpsD, 3>(mode);
    }
    return nullptr;
}
}  // namespace dg
