// moments.cu -- getAsymto_moments (src/FourierTransform.cpp:184-465) on the device.
//
// The reference fits F(iw) ~ m0 + m1/iw + m2/(iw)^2 + m3/(iw)^3 by least squares on every suffix window
// [w, N_freq) of the Matsubara axis, with (K^T K)^-1 K^T G per window.  K has two non-zeros per row, so
// K^T G and K^T K are suffix sums of four (resp. six) weighted series: the device forms those sums with one
// backward scan per series (O(N_freq) instead of the reference's O(N_freq^2)), inverts each K^T K (two 2 x 2
// blocks, partial pivoting), and then reproduces the reference's window averaging (2Nv+1 windows, Nv = N_freq/20),
// the variance of the trace of each moment, the positivity gates on the averaged moments, the first-minimum
// window choice (sequential argmin started at the last window) and the final Hermitisation.
//
// What bounds it: the work is ~1e7 FP64 operations, so on this chip (two FP64 lanes per SM and clock) it is the
// spread over SMs and the length of the dependent chains that count, not memory.  Hence one CTA per series with the
// terms formed by all its threads and only the ordered sums left to one warp, Hermitian pairs (a <= b) computed
// once, windows along the lanes so that every load is coalesced, and the gates by Cholesky, one warp per window
// (the eigenvalue signs asked for are those of m1 and of its Schur complement).  One call, measured with the host's
// wait: D = 1, N_freq = 400: 255 -> 234 us; D = 10, N_freq = 4096: 3.5 -> 0.48 ms (green 1.04 -> 0.33 ms); D = 20,
// N_freq = 400, dense F: 148 -> 0.28 ms (one thread per window ran Jacobi eigensolvers in global scratch before).
#include "smallmat.cuh"

namespace {

struct MomArgs {
    int D, Nf, R, C, Nv, ncol, P;  // P = D (D + 1) / 2 element pairs a <= b
    double beta;
    int green;
    const double2 *fw;  // [Nf][D][D]
    double *wt;         // [3][Nf]        series weights -1/z, -1/z^2, 1/z^3
    double2 *S;         // [P][ncol][R]   suffix sums K^T G
    double *KS;         // [6][R]         suffix sums for K^T K
    double2 *mt;        // [P][ncol][R]   fitted moments per window ("momentstest")
    double *tr;         // [ncol][R]
    double2 *avg;       // [ncol][C][D*D]
    double *var;        // [ncol][C]
    int *ok;            // [C]
    double2 *work;      // [C][3][D*D], gates of matrices too large for shared memory
    double2 *mom;       // [4][D][D]
    int *status;
};

__device__ __forceinline__ double zof(int wn, double beta) { return (2 * wn + 1) * DG_PI / beta; }

// the pair q of the row-major upper triangle (a <= b) of a D x D matrix
__device__ __forceinline__ void pair_of(int q, int D, int &a, int &b) {
    a = 0;
    while (q >= D - a) {
        q -= D - a;
        a++;
    }
    b = a + q;
}
__device__ __forceinline__ int pair_at(int a, int b, int D) { return a * D - a * (a - 1) / 2 + (b - a); }

__global__ void k_mom_weights(MomArgs g) {
    const int wn = blockIdx.x * blockDim.x + threadIdx.x;
    if (wn >= g.Nf) return;
    const double z = zof(wn, g.beta), z2 = z * z, z3 = z2 * z;
    g.wt[wn] = -1. / z;
    g.wt[g.Nf + wn] = -1. / z2;
    g.wt[2 * g.Nf + wn] = 1. / z3;
}

// Term wn of a series as (value, weight): the sum adds value * weight.  Series q < P ncol: column c of K^T G for a
// pair; the last six: K^T K.
__device__ __forceinline__ double2 mom_value(const MomArgs &g, int a, int b, int c, int wn) {
    const int DD = g.D * g.D;
    const double2 fab = g.fw[(size_t)wn * DD + a + b * g.D], fba = g.fw[(size_t)wn * DD + b + a * g.D];
    if (g.green ? c == 0 : (c == 0 || c == 2))
        return cmk((fab.x + fba.x) / 2, (fab.y - fba.y) / 2);               // (F_ab + conj F_ba)/2
    double2 im = cmk((fab.y + fba.y) * 0.5, -(fab.x - fba.x) * 0.5);        // (F_ab - conj F_ba)/(2i)
    if (g.green && a == b) im.x -= g.wt[wn];                                 // + 1/z
    return im;
}

// One CTA per series: suffix sums S(w) = sum_{wn >= w} term(wn).  All threads form the terms in shared memory; one
// warp sums them, lane l owning the l-th of 32 contiguous ranges (first the range totals, a suffix scan of them over
// the lanes, then the running sums), and all threads write the sums out.  STAGED = false (N_freq beyond the shared
// memory): the same sums with the terms formed where they are added.
constexpr int SUF_THREADS = 256;
inline size_t suffix_smem(int Nf) { return (size_t)(Nf + 32) * (sizeof(double2) + sizeof(double)); }
template <bool STAGED>
__global__ void __launch_bounds__(SUF_THREADS) k_mom_suffix(MomArgs g) {
    extern __shared__ double2 ssm[];
    const int series = blockIdx.x, nG = g.P * g.ncol;
    const int chunk = (g.Nf + 31) / 32;
    double2 *sv = ssm;                                         // value of term wn at wn + wn / chunk (bank spread)
    double *sw = reinterpret_cast<double *>(ssm + g.Nf + 32);  // its weight
    int a = 0, b = 0;
    const int c = series < nG ? series % g.ncol : series - nG;
    if (series < nG) pair_of(series / g.ncol, g.D, a, b);
    auto term = [&](int wn, double2 &v, double &w) {
        if (series < nG) {
            v = mom_value(g, a, b, c, wn);
            const int p = g.green ? 1 + c : c - 1;             // weight series; c = 0 of the general fit has none
            w = p < 0 ? 1.0 : g.wt[(size_t)p * g.Nf + wn];
        } else {
            const double i1 = g.wt[wn], i2 = g.wt[g.Nf + wn], i3 = g.wt[2 * g.Nf + wn];
            if (c == 0) v = cmk(1.0, 0.0), w = 1.0;
            else if (c == 1) v = cmk(1.0, 0.0), w = i2;        // K(.,0) K(.,2) on Re rows
            else if (c == 2) v = cmk(i2, 0.0), w = i2;
            else if (c == 3) v = cmk(i1, 0.0), w = i1;
            else if (c == 4) v = cmk(i1, 0.0), w = i3;
            else v = cmk(i3, 0.0), w = i3;
        }
    };
    if (STAGED) {
        for (int wn = threadIdx.x; wn < g.Nf; wn += blockDim.x) {
            const int o = wn + wn / chunk;
            term(wn, sv[o], sw[o]);
        }
        __syncthreads();
    }
    double2 *So = g.S + (size_t)series * g.R;
    double *Ko = g.KS + (size_t)(series - nG) * g.R;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const int lo = min(g.Nf, lane * chunk), hi = min(g.Nf, lo + chunk);
        double2 part = cmk(0, 0);
        auto add = [&](double2 s, int wn) {
            double2 v;
            double w;
            if (STAGED) {
                v = sv[wn + lane];
                w = sw[wn + lane];
            } else {
                term(wn, v, w);
            }
            return cmk(fma(v.x, w, s.x), fma(v.y, w, s.y));
        };
#pragma unroll 4
        for (int wn = hi - 1; wn >= lo; wn--) part = add(part, wn);
        // carry = sum of the ranges of all higher lanes (inclusive suffix scan, then shift)
        double2 incl = part;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const double2 v = shfl2(incl, min(31, lane + off), 32);
            if (lane + off < 32) incl = cadd(incl, v);
        }
        double2 run = csub(incl, part);
#pragma unroll 4
        for (int wn = hi - 1; wn >= lo; wn--) {
            run = add(run, wn);
            if (STAGED) sv[wn + lane] = run;
            else if (wn < g.R) {
                if (series < nG) So[wn] = run;
                else Ko[wn] = run.x;
            }
        }
    }
    if (!STAGED) return;
    __syncthreads();
    for (int wn = threadIdx.x; wn < g.R; wn += blockDim.x) {
        const double2 v = sv[wn + wn / chunk];
        if (series < nG) So[wn] = v;
        else Ko[wn] = v.x;
    }
}

// inverse of [[A, B], [B, C]] by Gauss-Jordan with partial pivoting; false for a zero pivot
__device__ __forceinline__ bool inv2(double A, double B, double C, double (&k)[4]) {
    const bool sw = B * B > A * A;
    double r00 = sw ? B : A, r01 = sw ? C : B, r10 = sw ? A : B, r11 = sw ? B : C;
    const double m0 = r00 * r00, i0 = r00 * (1.0 / m0);
    r01 *= i0;
    r11 = fma(-r10, r01, r11);
    r10 = -(r10 * i0);
    r00 = i0;
    const double m1 = r11 * r11, i1 = r11 * (1.0 / m1);
    r10 *= i1;
    r00 = fma(-r01, r10, r00);
    r01 = -(r01 * i1);
    r11 = i1;
    k[0] = sw ? r01 : r00;
    k[1] = sw ? r00 : r01;
    k[2] = sw ? r11 : r10;
    k[3] = sw ? r10 : r11;
    return m0 > 0.0 && m1 > 0.0;
}

// One CTA per 32 windows (lane = window): (K^T K)^-1 per window, the moments m_i = sum_c inv(i, c) (K^T G)_c of every
// pair, and the traces of the moments
constexpr int SOLVE_THREADS = 128;
__global__ void __launch_bounds__(SOLVE_THREADS) k_mom_solve(MomArgs g) {
    __shared__ double ki[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = blockIdx.x * 32 + lane;
    const int wc = min(w, g.R - 1), n = g.ncol;
    if (warp == 0) {
        const double *K = g.KS + wc;
        const size_t R = g.R;
        bool good = true;
        if (!g.green) {
            double e[4], o[4];
            good = inv2(K[0], K[R], K[2 * R], e);
            good &= inv2(K[3 * R], K[4 * R], K[5 * R], o);
            for (int q = 0; q < 4; q++) {
                ki[q][lane] = e[q];
                ki[4 + q][lane] = o[q];
            }
        } else {
            const double x = K[2 * R], y = K[5 * R];
            ki[0][lane] = x * (1.0 / (x * x));
            ki[1][lane] = y * (1.0 / (y * y));
            good = x * x > 0.0 && y * y > 0.0;
        }
        if (!good) dg_flag(g.status, DG_SINGULAR);
    }
    __syncthreads();
    auto dot = [&](double2 x, double kx, double2 y, double ky) {
        return cmk(fma(y.x, ky, x.x * kx), fma(y.y, ky, x.y * kx));
    };
    for (int pr = warp; pr < g.P; pr += SOLVE_THREADS / 32) {
        const double2 *s = g.S + (size_t)pr * n * g.R + wc;
        double2 *m = g.mt + (size_t)pr * n * g.R + w;
        if (w < g.R) {
            if (!g.green) {
                const double2 s0 = s[0], s1 = s[g.R], s2 = s[2 * (size_t)g.R], s3 = s[3 * (size_t)g.R];
                m[0] = dot(s0, ki[0][lane], s2, ki[1][lane]);
                m[g.R] = dot(s1, ki[4][lane], s3, ki[5][lane]);
                m[2 * (size_t)g.R] = dot(s0, ki[2][lane], s2, ki[3][lane]);
                m[3 * (size_t)g.R] = dot(s1, ki[6][lane], s3, ki[7][lane]);
            } else {
                m[0] = cscale(s[0], ki[0][lane]);
                m[g.R] = cscale(s[g.R], ki[1][lane]);
            }
        }
    }
    __syncthreads();  // the diagonal pairs of these windows are written by this CTA
    if (warp < n && w < g.R) {
        double t = 0;
        for (int a = 0; a < g.D; a++) t += g.mt[((size_t)pair_at(a, a, g.D) * n + warp) * g.R + w].x;
        g.tr[(size_t)warp * g.R + w] = t;
    }
}

// Over 2 Nv + 1 consecutive windows: variances of the traces (the first nvar CTAs, one centre per thread, the traces
// staged in shared memory) and averages of the moments for the gates (one thread per run of AVG_RUN centres of one
// series: the first range summed directly, the next ones by sliding)
constexpr int AVG_RUN = 64;
constexpr int AVG_THREADS = 128;
__global__ void __launch_bounds__(AVG_THREADS) k_mom_avg(MomArgs g, int nvar, int staged) {
    extern __shared__ double2 ssm[];
    const int L = 2 * g.Nv + 1;
    if ((int)blockIdx.x < nvar) {
        const int ncb = (g.C + AVG_THREADS - 1) / AVG_THREADS;
        const int i = blockIdx.x / ncb, c0 = (blockIdx.x % ncb) * AVG_THREADS, ci = c0 + threadIdx.x;
        const double *tr = g.tr + (size_t)i * g.R + c0;
        if (staged) {
            double *st = reinterpret_cast<double *>(ssm);
            const int len = min(g.C - c0, AVG_THREADS) + L - 1;
            for (int t = threadIdx.x; t < len; t += AVG_THREADS) st[t] = tr[t];
            __syncthreads();
            tr = st;
        }
        if (ci >= g.C) return;
        tr += threadIdx.x;
        double mean = 0;
#pragma unroll 8
        for (int j = 0; j < L; j++) mean += tr[j];
        mean /= L;
        double ss = 0;
#pragma unroll 8
        for (int j = 0; j < L; j++) ss += (tr[j] - mean) * (tr[j] - mean);
        g.var[(size_t)i * g.C + ci] = sqrt(ss / L);
        return;
    }
    const int DD = g.D * g.D, nrun = (g.C + AVG_RUN - 1) / AVG_RUN;
    const long long t = (long long)(blockIdx.x - nvar) * AVG_THREADS + threadIdx.x;
    if (t >= (long long)nrun * g.P * g.ncol) return;
    const int run = (int)(t % nrun);
    const long long r = t / nrun;
    const int i = (int)(r % g.ncol), pr = (int)(r / g.ncol);
    int a, b;
    pair_of(pr, g.D, a, b);
    const double2 *x = g.mt + ((size_t)pr * g.ncol + i) * g.R;
    const int c0 = run * AVG_RUN, c1 = min(g.C, c0 + AVG_RUN);
    double2 s = cmk(0, 0);
#pragma unroll 8
    for (int iw = c0; iw < c0 + L; iw++) s = cadd(s, x[iw]);
    for (int ci = c0; ci < c1; ci++) {
        if (ci > c0) s = csub(cadd(s, x[ci + L - 1]), x[ci - 1]);
        double2 *o = g.avg + ((size_t)i * g.C + ci) * DD;
        const double2 v = cmk(s.x / L, s.y / L);
        o[a + b * g.D] = v;
        if (a != b) o[b + a * g.D] = cconj(v);
    }
}

// The positivity gates of the window search, one warp per centre.  General fit: min eig(m1) > 0 and, with V =
// sqrt(m1), min eig(V^-1 m3 V^-1 - (V^-1 m2 V^-1)^2) > 0; the second matrix is congruent (by V) to
// m3 - m2 m1^-1 m2, so with m1 = L L^H both signs are Cholesky questions: m1 and m3 - (L^-1 m2)^H (L^-1 m2).
// Green fit (m0 = 0, m1 = I): min eig(avg1 - avg0^2) > 1.  Matrices in shared memory when they fit (SHM), in `work`
// otherwise.  A centre that no moment's argmin can choose (no variance below the last centre's) is not tested.
template <bool SHM>
__global__ void __launch_bounds__(128) k_mom_gate(MomArgs g) {
    extern __shared__ double2 ssm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ci = blockIdx.x * nw + warp;
    if (ci >= g.C) return;
    const int D = g.D, DD = D * D;
    bool cand = false;
    for (int i = 0; i < g.ncol; i++) cand |= g.var[(size_t)i * g.C + ci] < g.var[(size_t)i * g.C + g.C - 1];
    if (!cand) {
        if (lane == 0) g.ok[ci] = 0;
        return;
    }
    double2 *A = SHM ? ssm + (size_t)warp * 3 * DD : g.work + (size_t)ci * 3 * DD;
    double2 *W = A + DD, *X = W + DD;
    bool ok = true;
    if (!g.green) {
        const double2 *m1 = g.avg + ((size_t)1 * g.C + ci) * DD, *m2 = g.avg + ((size_t)2 * g.C + ci) * DD;
        const double2 *m3 = g.avg + ((size_t)3 * g.C + ci) * DD;
        for (int e = lane; e < DD; e += 32) {
            A[e] = m1[e];
            W[e] = m2[e];
            X[e] = m3[e];
        }
        __syncwarp();
        ok = warp_cholesky(D, A);
        if (ok) {
            // W = L^-1 m2, one column per lane
            for (int c = lane; c < D; c += 32)
                for (int i = 0; i < D; i++) {
                    double2 s = DG_AT(W, D, i, c);
                    for (int k = 0; k < i; k++) s = cfms(DG_AT(A, D, i, k), DG_AT(W, D, k, c), s);
                    DG_AT(W, D, i, c) = cscale(s, 1.0 / DG_AT(A, D, i, i).x);
                }
            __syncwarp();
            for (int e = lane; e < DD; e += 32) {
                const int i = e % D, j = e / D;
                if (i < j) continue;
                double2 s = X[e];
                for (int k = 0; k < D; k++) s = cfms(cconj(DG_AT(W, D, k, i)), DG_AT(W, D, k, j), s);
                X[e] = s;
            }
            __syncwarp();
            ok = warp_cholesky(D, X);
        }
    } else {
        const double2 *m0 = g.avg + (size_t)ci * DD, *m1 = g.avg + ((size_t)g.C + ci) * DD;
        for (int e = lane; e < DD; e += 32) W[e] = m0[e];
        __syncwarp();
        for (int e = lane; e < DD; e += 32) {
            const int i = e % D, j = e / D;
            if (i < j) continue;
            double2 s = m1[e];
            for (int k = 0; k < D; k++) s = csub(s, cmul(DG_AT(W, D, i, k), DG_AT(W, D, k, j)));
            if (i == j) s = cmk(s.x - 1.0, 0.0);
            X[e] = s;
        }
        __syncwarp();
        ok = warp_cholesky(D, X);
    }
    if (lane == 0) g.ok[ci] = ok ? 1 : 0;
}

// One CTA per (element pair, moment): window choice of the moment and the average of its fits over the chosen range.
// The sequential argmin of the reference (minPos = C-1; minPos = i when ok[i] and var[i] < var[minPos]) as a
// block reduction: the first index of the smallest var[i] among ok candidates with var[i] < var[C-1], else C-1.
// The fits are Hermitian, so the reference's (m + m^H)/2 takes the pair's conjugate for the other element.
constexpr int FIN_THREADS = 256;
__global__ void __launch_bounds__(FIN_THREADS) k_mom_final(MomArgs g, int staged) {
    extern __shared__ double2 ssm[];
    __shared__ double rv[FIN_THREADS];
    __shared__ int ri[FIN_THREADS];
    const int D = g.D, DD = D * D, mom = blockIdx.y, tid = threadIdx.x, L = 2 * g.Nv + 1;
    int a, b;
    pair_of(blockIdx.x, D, a, b);
    double2 *o = g.mom + (size_t)mom * DD;
    const int src = g.green ? mom - 2 : mom;
    if (src < 0) {  // the fixed moments of the green fit: m0 = 0, m1 = I
        if (tid == 0) {
            o[a + b * D] = cmk(mom == 1 && a == b ? 1.0 : 0.0, 0.0);
            if (a != b) o[b + a * D] = cmk(0, 0);
        }
        return;
    }
    const double *var = g.var + (size_t)src * g.C;
    const double vlast = var[g.C - 1];
    double bv = 0;
    int bi = -1;
#pragma unroll 4
    for (int i = tid; i < g.C; i += FIN_THREADS) {
        const double v = var[i];
        if (g.ok[i] && v < vlast && (bi < 0 || v < bv)) {
            bv = v;
            bi = i;
        }
    }
    rv[tid] = bv;
    ri[tid] = bi;
    __syncthreads();
    for (int h = FIN_THREADS / 2; h > 0; h >>= 1) {
        if (tid < h) {
            const int oi = ri[tid + h], mi = ri[tid];
            const double ov = rv[tid + h];
            if (oi >= 0 && (mi < 0 || ov < rv[tid] || (ov == rv[tid] && oi < mi))) {
                rv[tid] = ov;
                ri[tid] = oi;
            }
        }
        __syncthreads();
    }
    const int w0 = ri[0] >= 0 ? ri[0] : g.C - 1;  // windows w0 .. w0 + 2 Nv
    const double2 *x = g.mt + ((size_t)blockIdx.x * g.ncol + src) * g.R + w0;
    if (staged) {
        for (int t = tid; t < L; t += FIN_THREADS) ssm[t] = x[t];
        __syncthreads();
        x = ssm;
    }
    if (tid != 0) return;
    double2 s = cmk(0, 0);
#pragma unroll 8
    for (int w = 0; w < L; w++) s = cadd(s, x[w]);
    const double2 v = a == b ? cmk(s.x / L, 0.0) : cmk(s.x / L, s.y / L);
    o[a + b * D] = v;
    if (a != b) o[b + a * D] = cconj(v);
}

}  // namespace

int dg_moments_dev(dmftgpu_ctx *ctx, int dim, int nfreq, double beta, const double2 *fw, int green,
                   double2 *mom) {
    MomArgs g;
    g.D = dim;
    g.Nf = nfreq;
    g.green = green ? 1 : 0;
    g.ncol = green ? 2 : 4;
    g.R = green ? nfreq - 1 : nfreq - 3;
    g.Nv = nfreq / 20;
    if (g.Nv == 0) g.Nv = 1;
    g.C = g.R - 2 * g.Nv;
    g.P = dim * (dim + 1) / 2;
    g.beta = beta;
    if (dim < 1 || g.R < 1 || g.C < 1) return dg_fail(ctx, DMFTGPU_BADARG, "moments: N_freq too small");
    const size_t DD = (size_t)dim * dim, P = g.P, L = 2 * (size_t)g.Nv + 1;
    // gates in shared memory for up to 4 warps per CTA within 96 KB, in global scratch for larger matrices
    const size_t gate_warp = 3 * DD * sizeof(double2);
    int gw = 4;
    while (gw > 1 && gw * gate_warp > 96 * 1024) gw >>= 1;
    const bool gate_shm = gw * gate_warp <= 96 * 1024;
    size_t off = 0;
    auto carve = [&](size_t bytes) {
        size_t o = off;
        off += (bytes + 255) & ~(size_t)255;
        return o;
    };
    size_t oWt = carve(3 * (size_t)nfreq * sizeof(double)), oS = carve(P * g.ncol * g.R * sizeof(double2)),
           oKS = carve(6 * (size_t)g.R * sizeof(double)), oMt = carve(P * g.R * g.ncol * sizeof(double2)),
           oTr = carve((size_t)g.ncol * g.R * sizeof(double)), oAvg = carve((size_t)g.ncol * g.C * DD * sizeof(double2)),
           oVar = carve((size_t)g.ncol * g.C * sizeof(double)), oOk = carve((size_t)g.C * sizeof(int)),
           oW = carve(gate_shm ? 0 : (size_t)g.C * gate_warp);
    char *base = (char *)dg_buf(ctx, "moments.work", off);
    if (!base) return DMFTGPU_NOMEM;
    g.fw = fw;
    g.wt = (double *)(base + oWt);
    g.S = (double2 *)(base + oS);
    g.KS = (double *)(base + oKS);
    g.mt = (double2 *)(base + oMt);
    g.tr = (double *)(base + oTr);
    g.avg = (double2 *)(base + oAvg);
    g.var = (double *)(base + oVar);
    g.ok = (int *)(base + oOk);
    g.work = (double2 *)(base + oW);
    g.mom = mom;
    g.status = ctx->d_status;
    cudaStream_t s = ctx->stream;
    k_mom_weights<<<dg_ceil_div(nfreq, 128), 128, 0, s>>>(g);
    DG_LAUNCH(ctx, "k_mom_weights");
    const int nseries = g.P * g.ncol + 6;
    const size_t sms = suffix_smem(nfreq);
    if (sms <= 200 * 1024) {
        DG_CUDA(cudaFuncSetAttribute(k_mom_suffix<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sms));
        k_mom_suffix<true><<<nseries, SUF_THREADS, sms, s>>>(g);
    } else {
        k_mom_suffix<false><<<nseries, 32, 0, s>>>(g);
    }
    DG_LAUNCH(ctx, "k_mom_suffix");
    k_mom_solve<<<dg_ceil_div(g.R, 32), SOLVE_THREADS, 0, s>>>(g);
    DG_LAUNCH(ctx, "k_mom_solve");
    const int nvar = g.ncol * dg_ceil_div(g.C, AVG_THREADS);
    const long long navg = (long long)dg_ceil_div(g.C, AVG_RUN) * g.P * g.ncol;
    const size_t sma = (AVG_THREADS + L) * sizeof(double), smf = L * sizeof(double2);
    const int sta = sma <= 48 * 1024, stf = smf <= 40 * 1024;
    k_mom_avg<<<nvar + dg_ceil_div(navg, AVG_THREADS), AVG_THREADS, sta ? sma : 0, s>>>(g, nvar, sta);
    DG_LAUNCH(ctx, "k_mom_avg");
    if (gate_shm) {
        const size_t smg = gw * gate_warp;
        DG_CUDA(cudaFuncSetAttribute(k_mom_gate<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smg));
        k_mom_gate<true><<<dg_ceil_div(g.C, gw), 32 * gw, smg, s>>>(g);
    } else {
        k_mom_gate<false><<<g.C, 32, 0, s>>>(g);
    }
    DG_LAUNCH(ctx, "k_mom_gate");
    k_mom_final<<<dim3(g.P, 4), FIN_THREADS, stf ? smf : 0, s>>>(g, stf);
    DG_LAUNCH(ctx, "k_mom_final");
    return DMFTGPU_OK;
}

extern "C" int dmftgpu_moments(dmftgpu_ctx *ctx, int dim, int nfreq, double beta, const double *fw, int green_asym,
                               double *mom, int flags) {
    if (!ctx || !fw || !mom || dim < 1 || nfreq < 1) return DMFTGPU_BADARG;
    cudaSetDevice(ctx->device);
    int st;
    size_t DD = (size_t)dim * dim;
    const double2 *dfw = (const double2 *)dg_in(ctx, fw, nfreq * DD * sizeof(double2), flags, "io.fw", &st);
    if (st) return st;
    double2 *dmom = (double2 *)dg_out(ctx, mom, 4 * DD * sizeof(double2), flags, "io.mom", &st);
    if (st) return st;
    DG_TRY(dg_status_reset(ctx));
    DG_TRY(dg_moments_dev(ctx, dim, nfreq, beta, dfw, green_asym, dmom));
    DG_TRY(dg_out_done(ctx, mom, dmom, 4 * DD * sizeof(double2), flags));
    int code = 0;
    DG_TRY(dg_status_read(ctx, &code));
    return code ? code : DMFTGPU_OK;
}
