// common.cuh -- shared device helpers of libdmftgpu (complex FP64 arithmetic, status codes, launch checks).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "dmftgpu.h"
#include "internal.h"

#define DG_PI 3.1415926535897932384626  // src/dmft_common.h:43

// ---------------------------------------------------------------------------------------------------
// complex double as double2 (x = re, y = im)
// ---------------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ double2 cmk(double r, double i) { return make_double2(r, i); }
__host__ __device__ __forceinline__ double2 cadd(double2 a, double2 b) { return cmk(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ double2 csub(double2 a, double2 b) { return cmk(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ double2 cneg(double2 a) { return cmk(-a.x, -a.y); }
__host__ __device__ __forceinline__ double2 cconj(double2 a) { return cmk(a.x, -a.y); }
__host__ __device__ __forceinline__ double2 cscale(double2 a, double s) { return cmk(a.x * s, a.y * s); }
__host__ __device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return cmk(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__host__ __device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
    return cmk(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
// acc + a*b
__host__ __device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 acc) {
    return cmk(fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y)));
}
// acc - a*b
__host__ __device__ __forceinline__ double2 cfms(double2 a, double2 b, double2 acc) {
    return cmk(fma(-a.x, b.x, fma(a.y, b.y, acc.x)), fma(-a.x, b.y, fma(-a.y, b.x, acc.y)));
}
__host__ __device__ __forceinline__ double cabs2(double2 a) { return fma(a.x, a.x, a.y * a.y); }
// 1/a = conj(a)/|a|^2 with a single division (FP64 division is a multi-instruction sequence on this GPU).
// |a| stays within 1e-150..1e150 for every caller (shifted Matsubara frequencies, pivots of well-scaled
// matrices); a zero pivot gives inf/nan, as the reference's division would.
__host__ __device__ __forceinline__ double2 crcp(double2 a) {
    const double r = 1.0 / fma(a.x, a.x, a.y * a.y);
    return cmk(a.x * r, -a.y * r);
}
__host__ __device__ __forceinline__ double2 cdiv(double2 a, double2 b) { return cmul(a, crcp(b)); }
__host__ __device__ __forceinline__ double2 cexpi(double ang) {  // exp(i ang)
    double s, c;
    sincos(ang, &s, &c);
    return cmk(c, s);
}

__device__ __forceinline__ double2 shfl2(double2 v, int src, int width) {
    return cmk(__shfl_sync(0xffffffffu, v.x, src, width), __shfl_sync(0xffffffffu, v.y, src, width));
}
__device__ __forceinline__ void atomic_add_c(double2 *p, double2 v) {
    atomicAdd(&p->x, v.x);
    atomicAdd(&p->y, v.y);
}

// Sum of at(0) + .. + at(n - 1) in a fixed order: up to 16 terms one after the other, else eight running sums over 64 terms,
// added as a tree, then the next 64.  n - 1 additions like one running sum, whose rounding errors grow with the root of n when
// the terms are alike (k chunks of a lattice sum: G_loc in FP64 at 1,200 k in 150 chunks 3.5e-16 off by one running sum,
// 1.6e-16 in 19 longer chunks).
template <class F>
__device__ __forceinline__ double2 chunk_sum(int n, F at) {
    double2 total = at(0);
    if (n <= 16) {
#pragma unroll 4
        for (int q = 1; q < n; q++) total = cadd(total, at(q));
        return total;
    }
    for (int q0 = 0; q0 < n; q0 += 64) {
        const int end = min(n, q0 + 64);
        double2 s;
        int q = q0;
        if (end - q0 >= 8) {
            double2 a[8];
#pragma unroll
            for (int j = 0; j < 8; j++) a[j] = at(q0 + j);
            for (q = q0 + 8; q + 8 <= end; q += 8)
#pragma unroll
                for (int j = 0; j < 8; j++) a[j] = cadd(a[j], at(q + j));
#pragma unroll
            for (int h = 4; h > 0; h >>= 1)
#pragma unroll
                for (int j = 0; j < h; j++) a[j] = cadd(a[j], a[j + h]);
            s = a[0];
        } else {
            s = at(q++);
        }
        for (; q < end; q++) s = cadd(s, at(q));
        total = q0 ? cadd(total, s) : s;
    }
    return total;
}

// status word written by kernels (never a trap): the host reads it after the launch sequence.
__device__ __forceinline__ void dg_flag(int *status, int code) {
    if (status) atomicMax(status, code);
}

#define DG_CUDA(call)                                                   \
    do {                                                                \
        cudaError_t e_ = (call);                                        \
        if (e_ != cudaSuccess) return dg_set_cuda_error(ctx, e_, #call); \
    } while (0)

static inline int dg_ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// `bytes` of dynamic shared memory for a kernel that shares SMs with kernels of another stream (the static eigen-decomposition
// runs beside the Schur data and the lattice kernels), with the same carve-out, the largest, for all of them: an SM changes
// its split between L1 and shared memory only when it is empty, so kernels of different splits wait for one another or run with
// the blocks that fit the other's.  Left to the driver, the same call took 0.90 or 2.03 ms (G_loc in FP64, 4 + 8 orbitals,
// 216 k x 512 points), 0.80 or 1.86 (densities, 3 + 8), 6.6 or 11.4 (G_loc, 6 + 36), whichever kernel came first.
// tight: the smallest carve-out that holds the block, for the tensor-core kernels, whose block fills an SM and which read
// z - Sigma of their frequencies through L1 (in the largest one G_loc at D = 10, 216 k x 512 points, takes 0.56 ms, not 0.51).
template <class K>
inline cudaError_t dg_smem_attr(K kernel, size_t bytes, bool tight = false) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    const int sm = 228 * 1024, percent = tight ? (int)((bytes + 1024) * 100 / sm) : (int)cudaSharedmemCarveoutMaxShared;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, percent);
}
