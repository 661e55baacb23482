// impurity.h -- device-level building blocks of the impurity stage (impurity.cu), shared with the
// solver drivers (solvers.cu).  All pointers are device pointers; functions only enqueue work.
#pragma once
#include "linalg.cuh"

// getStimp's lists over distinct minors (impurity.cu), all device pointers
struct S2Lists {
    int d = 0, np1 = 0, np2 = 0, nslot = 0, ne1 = 0;
    const int *i = nullptr;      // off1[d+1], offs[d+1], offb[nslot+1], pairs1[np1][2], pairs2[np2][2],
                                 // e1[ne1][2] = (P1, q), sP2[nslot], bp[nb]
    const double2 *c = nullptr;  // c1[ne1], cb[nb]
};

// U_{ijkl} list (gen_Uijkl, src/gen_Uijkl.cpp:9-87) on the device, with getStimp's lists: over distinct minors, or,
// where those do not fit in shared memory (byI != nullptr), the entries grouped by their first index (byI) and by
// their last index (byJ)
struct DgUList {
    int nu = 0;
    const int *byI = nullptr, *byIoff = nullptr, *byJ = nullptr, *byJoff = nullptr, *uidx = nullptr;
    const double2 *ut = nullptr;
    S2Lists s2;
};

// complex slots of one set of tail data (impurity.cu: 2 d pole energies, then a product per pole and element pair)
__host__ __device__ inline size_t dg_tail_elems(int d) { return (size_t)d + (size_t)d * d * (d + 1); }

int dg_ulist(dmftgpu_ctx *ctx, int d, int nu, const int *uidx_host, const double *ut_host, DgUList &U);
int dg_phase_table(dmftgpu_ctx *ctx, int ntau, double2 **ph);
int dg_w2tau_dev(dmftgpu_ctx *ctx, int d, int nfreq, int ntau, double beta, const double2 *fw, const double2 *mom,
                 double2 *ft);
int dg_fourier_dev(dmftgpu_ctx *ctx, int d, int nfreq, int ntau, double beta, const double2 *fw, int green,
                   const double2 *m1, double2 *ft);
int dg_tau2w_dev(dmftgpu_ctx *ctx, int d, int nfreq, int ntau, double beta, const double2 *ft, double2 *fw, bool check);
int dg_sigma2_dev(dmftgpu_ctx *ctx, int d, int ntau, double beta, const DgUList &U, const double2 *gt, double2 *st);
int dg_fock_dev(dmftgpu_ctx *ctx, int d, const DgUList &U, const double2 *occ, double2 *fock);
int dg_dyson_dev(dmftgpu_ctx *ctx, int d, int nfreq, double beta, double mu, const double2 *himp,
                 const double2 *delta, const double2 *fock, const double2 *s2, double2 *gw, bool check);
int dg_estimate_asymto_dev(dmftgpu_ctx *ctx, int d, int nfreq, double beta, double2 *f, int order);
int dg_occ_dev(dmftgpu_ctx *ctx, int d, int nfreq, double beta, const double2 *gw, double2 *occ);
// the shared parts of getoccMat and FourierTransform: T = tail data (dg_tail_elems), Dw = F - tail
int dg_green_tail_dev(dmftgpu_ctx *ctx, int d, int nfreq, double beta, const double2 *gw, double2 *T, double2 *Dw);
int dg_occ_tail_dev(dmftgpu_ctx *ctx, int d, int nfreq, double beta, const double2 *T, const double2 *Dw,
                    double2 *occ);
int dg_w2tau_tail_dev(dmftgpu_ctx *ctx, int d, int nfreq, int ntau, double beta, const double2 *T, const double2 *Dw,
                      double2 *ft);
int dg_ipt_kk_dev(dmftgpu_ctx *ctx, int nfreq, const double *a, const double *b, const double *c, double2 *s2);
