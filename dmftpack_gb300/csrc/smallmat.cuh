// smallmat.cuh -- block- and thread-level routines for the few small (n <= 32) Hermitian matrices of the
// impurity stage, all working in SHARED memory (the thread_* routines of linalg.cuh work in global scratch
// and are latency-bound there).
//
//  * block_heig: Hermitian eigen-decomposition by one thread block.  Like thread_heig (and
//    Eigen::SelfAdjointEigenSolver) it reads only the lower triangle, takes the diagonal real and returns
//    ascending eigenvalues, with the same complex Jacobi rotation and the same stopping rule
//    (off-diagonal mass <= 1e-28 of the total); the rotations (jacobi_rotation) of one sweep are applied in round-robin
//    ("tournament") order, n/2 disjoint (p, q) pairs at a time, so a sweep takes n - 1 parallel steps.
//  * block_matmul: C = A B, one thread per element.
//  * posdef_lower: is the Hermitian matrix s * (lower triangle of M) - shift * I positive definite (strict)
//    or positive semidefinite?  A Cholesky factorisation answers the eigenvalue-sign questions of the
//    reference (min eigenvalue >= 0 in the positivity fix-up, max eigenvalue < 0 in the causality checks,
//    min eigenvalue > 1 in the moment gate) with ~n^3/6 operations instead of a full eigensolve.  The
//    semidefinite variant accepts an exactly zero pivot when the rest of its column is exactly zero.
#pragma once
#include "linalg.cuh"

struct DgRot {
    int p, q, on;
    double c, s;
    double2 ph;
};

__host__ __device__ __forceinline__ float fast_div(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fdividef(a, b);
#else
    return a / b;
#endif
}
// The tangent of the rotation that removes a_pq: the root |t| <= 1 of r t^2 + d t - r = 0 with r = |a_pq| in [1, 3) and d = a_qq -
// a_pp in the same units.  Found in FP32 and refined by two Newton steps with the residual in FP64 and the slope,
// +-sqrt(d^2 + 4 r^2), in FP32; each leaves some 1e-7 of the error: 1e-7, 1e-14, rounding.  0 where d is beyond 1e30 r (or not
// a number).
__host__ __device__ __forceinline__ double jacobi_tan(double r, double d) {
    const float x = (float)d, rf = (float)r, ax = fabsf(x);
    if (!(ax <= 1e30f)) return 0.0;
    const float slope = ax > 1e9f ? ax : sqrtf(fmaf(x, x, 4.f * rf * rf));
    const double step = copysignf(fast_div(1.f, slope), x);
    double t = copysignf(fast_div(2.f * rf, ax + slope), x);
    t = fma(-step, fma(fma(r, t, d), t, -r), t);
    return fma(-step, fma(fma(r, t, d), t, -r), t);
}
// The rotation of the (p, q) plane: c = (1 + t^2)^-1/2 and ph = a_pq / |a_pq| from one reciprocal-square-root refinement each.  A
// lone warp's FP64 instruction takes 64 cycles, so the square roots and divisions of the plain formulas (seven, ~10
// dependent instructions each) were two thirds of a round; this is 32 instructions.  (24 with the angle left at FP32: every
// rotation then leaves 1e-7 of a_pq, sweeps end up to 1e-14 of the total away in place of rounding, and one in four
// matrices of 8 x 8 takes another sweep.)
__device__ __forceinline__ double fast_rsqrt(double x) {  // x in [0.25, 1e30]
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);                  // y (1 - e)^-1/2 = y (1 + e/2 + 3/8 e^2 + O(e^3))
    return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ DgRot jacobi_rotation(int p, int q, double2 apq, double app, double aqq) {
    DgRot R;
    R.p = p;
    R.q = q;
    R.on = 0;
    R.c = 1.0;
    R.s = 0.0;
    R.ph = cmk(1, 0);
    // a_pq scaled by a power of two to modulus [1, 2) or a little above; zero and denormal entries are left alone
    const int ex = max(__double2hiint(fabs(apq.x)), __double2hiint(fabs(apq.y))) & 0x7ff00000;
    if (ex == 0) return R;
    const double sc = __hiloint2double(0x7fe00000 - ex, 0);
    const double2 z = cscale(apq, sc);
    const double r2 = cabs2(z), inv = fast_rsqrt(r2);
    const double t = jacobi_tan(r2 * inv, (aqq - app) * sc);
    R.c = fast_rsqrt(fma(t, t, 1.0));
    R.s = t * R.c;
    R.ph = cscale(z, inv);
    R.on = 1;
    return R;
}

// all threads of the block call it; a, u: n*n shared, w: n shared doubles, order: n shared ints,
// rot: n/2+1 shared DgRot, red: blockDim.x shared doubles.  Returns DG_OK or DG_NONCONV (block-uniform).
__device__ inline int block_heig(int n, const double2 *A0, double2 *a, double2 *u, double *w, int *order, DgRot *rot,
                                 double *red) {
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int e = tid; e < n * n; e += nt) {
        const int i = e % n, j = e / n;
        double2 v;
        if (i > j) v = DG_AT(A0, n, i, j);
        else if (i < j) v = cconj(DG_AT(A0, n, j, i));
        else v = cmk(DG_AT(A0, n, i, i).x, 0.0);
        a[e] = v;
        if (u) u[e] = cmk(i == j ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();
    const int m = n + (n & 1), half = m / 2;
    __shared__ int conv;
    int st = DG_NONCONV;
    for (int sweep = 0; sweep < 100; sweep++) {
        // off-diagonal and total mass
        double off = 0, tot = 0;
        for (int e = tid; e < n * n; e += nt) {
            const double v = cabs2(a[e]);
            tot += v;
            if (e % n != e / n) off += v;
        }
        red[tid] = off;
        __syncthreads();
        for (int h = nt / 2; h > 0; h >>= 1) {
            if (tid < h) red[tid] += red[tid + h];
            __syncthreads();
        }
        const double offs = red[0];
        __syncthreads();
        red[tid] = tot;
        __syncthreads();
        for (int h = nt / 2; h > 0; h >>= 1) {
            if (tid < h) red[tid] += red[tid + h];
            __syncthreads();
        }
        if (tid == 0) conv = (offs == 0.0 || offs <= 1e-28 * red[0]);
        __syncthreads();
        if (conv) {
            st = DG_OK;
            break;
        }
        for (int r = 0; r < m - 1; r++) {
            // pairs of round r: (r, m-1) and ((r+k) mod (m-1), (r-k) mod (m-1)), k = 1 .. half-1
            if (tid < half) {
                int p, q;
                if (tid == 0) {
                    p = r;
                    q = m - 1;
                } else {
                    p = (r + tid) % (m - 1);
                    q = (r - tid + (m - 1)) % (m - 1);
                }
                if (p > q) {
                    const int t = p;
                    p = q;
                    q = t;
                }
                DgRot R;
                if (q < n) R = jacobi_rotation(p, q, DG_AT(a, n, p, q), DG_AT(a, n, p, p).x, DG_AT(a, n, q, q).x);
                else R.on = 0;
                rot[tid] = R;
            }
            __syncthreads();
            // columns p, q of a (and u): a(:,p) = c a(:,p) - s conj(ph) a(:,q); a(:,q) = s a(:,p) + c conj(ph) a(:,q)
            for (int x = tid; x < (u ? 2 : 1) * half * n; x += nt) {
                double2 *M = x < half * n ? a : u;  // different threads take a's and u's columns
                const int y = x < half * n ? x : x - half * n;
                const DgRot R = rot[y / n];
                if (!R.on) continue;
                const int k = y % n;
                const double2 akp = DG_AT(M, n, k, R.p), z = cmul(cconj(R.ph), DG_AT(M, n, k, R.q));
                DG_AT(M, n, k, R.p) = csub(cscale(akp, R.c), cscale(z, R.s));
                DG_AT(M, n, k, R.q) = cadd(cscale(akp, R.s), cscale(z, R.c));
            }
            __syncthreads();
            // rows p, q: a(p,:) = c a(p,:) - s ph a(q,:); a(q,:) = s a(p,:) + c ph a(q,:)
            for (int x = tid; x < half * n; x += nt) {
                const DgRot R = rot[x / n];
                if (!R.on) continue;
                const int k = x % n;
                const double2 apk = DG_AT(a, n, R.p, k), aqk = DG_AT(a, n, R.q, k);
                DG_AT(a, n, R.p, k) = csub(cscale(apk, R.c), cscale(cmul(R.ph, aqk), R.s));
                DG_AT(a, n, R.q, k) = cadd(cscale(apk, R.s), cscale(cmul(R.ph, aqk), R.c));
            }
            __syncthreads();
            if (tid < half && rot[tid].on) {
                DG_AT(a, n, rot[tid].p, rot[tid].p).y = 0.0;
                DG_AT(a, n, rot[tid].q, rot[tid].q).y = 0.0;
            }
            __syncthreads();
        }
    }
    if (tid == 0) {
        for (int i = 0; i < n; i++) order[i] = i;
        for (int i = 1; i < n; i++) {
            const int v = order[i];
            const double key = DG_AT(a, n, v, v).x;
            int j = i - 1;
            while (j >= 0 && DG_AT(a, n, order[j], order[j]).x > key) {
                order[j + 1] = order[j];
                j--;
            }
            order[j + 1] = v;
        }
        for (int i = 0; i < n; i++) w[i] = DG_AT(a, n, order[i], order[i]).x;
    }
    __syncthreads();
    if (u) {
        for (int e = tid; e < n * n; e += nt) a[e] = u[e];
        __syncthreads();
        for (int e = tid; e < n * n; e += nt) {
            const int k = e % n, i = e / n;
            DG_AT(u, n, k, i) = DG_AT(a, n, k, order[i]);
        }
        __syncthreads();
    }
    return st;
}

// C = A B (n x n, all shared or global, C distinct from A and B); all threads call it; ends with a barrier
__device__ inline void block_matmul(int n, const double2 *A, const double2 *B, double2 *C) {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e % n, j = e / n;
        double2 s = cmk(0, 0);
        for (int k = 0; k < n; k++) s = cfma(DG_AT(A, n, i, k), DG_AT(B, n, k, j), s);
        C[e] = s;
    }
    __syncthreads();
}

// Is the Hermitian matrix whose lower triangle is in A (n x n, column-major, shared or global, this warp's) positive
// definite?  Cholesky by one warp, L left in the lower triangle; all 32 lanes call it, the answer is warp-uniform.
__device__ inline bool warp_cholesky(int n, double2 *A) {
    const int lane = threadIdx.x & 31;
    for (int j = 0; j < n; j++) {
        const double p = DG_AT(A, n, j, j).x;
        if (!(p > 0.0)) return false;
        const double r = 1.0 / sqrt(p);
        __syncwarp();
        if (lane == 0) DG_AT(A, n, j, j) = cmk(p * r, 0.0);
        for (int i = j + 1 + lane; i < n; i += 32) DG_AT(A, n, i, j) = cscale(DG_AT(A, n, i, j), r);
        __syncwarp();
        const int c = n - j - 1;
        for (int e = lane; e < c * c; e += 32) {
            const int i = j + 1 + e % c, k = j + 1 + e / c;
            if (i < k) continue;
            double2 v = csub(DG_AT(A, n, i, k), cmul(DG_AT(A, n, i, j), cconj(DG_AT(A, n, k, j))));
            if (i == k) v.y = 0.0;
            DG_AT(A, n, i, k) = v;
        }
        __syncwarp();
    }
    return true;
}

// Cholesky test of one n x n Hermitian matrix held as its lower triangle in t[idx(i, j)] (i >= j), with
// t[idx] = tri[(idx) * stride] (stride = threads sharing the interleaved shared array).  Destroys t.
// strict: positive definite; else positive semidefinite (an exactly zero pivot with an exactly zero
// remaining column is skipped).
__host__ __device__ inline bool posdef_tri(int n, double2 *t, int stride, bool strict) {
#define DG_TRI(i, j) t[(size_t)(((i) * ((i) + 1)) / 2 + (j)) * stride]
    for (int j = 0; j < n; j++) {
        const double p = DG_TRI(j, j).x;
        if (strict ? !(p > 0.0) : !(p >= 0.0)) return false;
        if (p == 0.0) {
            for (int i = j + 1; i < n; i++)
                if (DG_TRI(i, j).x != 0.0 || DG_TRI(i, j).y != 0.0) return false;
            continue;
        }
        const double r = 1.0 / sqrt(p);
        for (int i = j + 1; i < n; i++) DG_TRI(i, j) = cscale(DG_TRI(i, j), r);
        for (int k = j + 1; k < n; k++) {
            const double2 lkj = DG_TRI(k, j);
            for (int i = k; i < n; i++) DG_TRI(i, k) = csub(DG_TRI(i, k), cmul(DG_TRI(i, j), cconj(lkj)));
            DG_TRI(k, k).y = 0.0;
        }
    }
    return true;
#undef DG_TRI
}

// threads per block for one-matrix-per-thread Cholesky tests on d x d matrices, their lower triangles
// interleaved in shared memory (<= 96 KiB per block)
inline int posdef_threads(int d) {
    const size_t tri = (size_t)d * (d + 1) / 2 * sizeof(double2);
    int t = 64;
    while (t > 1 && (size_t)t * tri > 96 * 1024) t >>= 1;
    return t;
}
