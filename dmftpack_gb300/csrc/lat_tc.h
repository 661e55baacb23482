// lat_tc.h -- arguments of the tensor-core lattice passes (lat_tc.cu) and their host entries.
#pragma once
#include <cuda_runtime.h>

struct dmftgpu_ctx;

struct LatTcArgs {
    const double2 *H;      // [nk][n][n] column-major, correlated orbitals first
    const double2 *B;      // [nk][m][D]  b_l(a)
    const double *epsQ;    // [nk][m]     eigenvalues of H_QQ
    const double2 *sig;    // [nf2][D][D] Sigma(iw) with its moment tail beyond N_freq
    const double *eps0;    // [nk][n]     eigenvalues of H + m0
    const double2 *UP;     // [nk][n][D]  correlated rows of their eigenvectors (block pass)
    const double2 *m0;     // [D][D]      static moment of Sigma (block pass)
    cudaEvent_t static_ready;  // eps0 and UP are there
    int n, m, nk, nf2, D, wgrid;
    double beta, mu;
};

// true when the N(mu) pass, its derivative, the block pass are the faster form for this lattice (see lat_tc.cu)
bool dg_lat_tc_supported(int n, int D);
bool dg_lat_tc_deriv_supported(int n, int D);
bool dg_lat_tc_block_supported(int n, int D);
// room for the operand images of a supported pass (block: dg_lat_tc_block); false, with nothing held, where the call's share
// (ctx->image_left) or the device has no room for them: the caller takes run_schur, which has no images
bool dg_lat_tc_reserve(dmftgpu_ctx *ctx, int n, int D, int nk, bool block);
// prepare the per-k operand images once (*ready tracks it for the caller's prepared lattice), then run one pass:
// tr[f] = sum_k Re[Tr G(k, iw_f) - Tr G0(k, iw_f)] for f < nf2, and with dtr its derivative by mu (device)
int dg_lat_tc_trace(dmftgpu_ctx *ctx, const LatTcArgs &a, bool *ready, double *tr, double *dtr);
// blk[f] = sum_k G_PP, blk0[f] = sum_k G0_PP (device, [nf2][D][D])
int dg_lat_tc_block(dmftgpu_ctx *ctx, const LatTcArgs &a, double2 *blk, double2 *blk0);
