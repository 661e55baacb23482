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
// terms formed by all its threads and only the ordered sums left to two warps, Hermitian pairs (a <= b) computed
// once, windows along the lanes so that every load is coalesced, and the gates by Cholesky, one warp per window
// (the eigenvalue signs asked for are those of m1 and of its Schur complement).  One call, measured with the host's
// wait: D = 1, N_freq = 400: 255 -> 111 us; D = 10, N_freq = 4096: 3.55 -> 0.30 ms, with a dense F 15.8 -> 0.42 ms
// (green fit 1.04 -> 0.24 ms); D = 20, N_freq = 400, dense F: 148 ms before (one thread per window ran Jacobi
// eigensolvers in global scratch).
#include <algorithm>

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
    double2 *avg;       // [ncol][C][P]   window sums (not yet divided by 2 Nv + 1)
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

// element (a, b) of the data in the form column c of K^T G weighs
__device__ __forceinline__ double2 mom_value(const MomArgs &g, int a, int b, int c, int wn) {
    const int DD = g.D * g.D;
    const double2 fab = g.fw[(size_t)wn * DD + a + b * g.D], fba = g.fw[(size_t)wn * DD + b + a * g.D];
    if (g.green ? c == 0 : (c == 0 || c == 2))
        return cmk((fab.x + fba.x) / 2, (fab.y - fba.y) / 2);               // (F_ab + conj F_ba)/2
    double2 im = cmk((fab.y + fba.y) * 0.5, -(fab.x - fba.x) * 0.5);        // (F_ab - conj F_ba)/(2i)
    if (g.green && a == b) im.x -= g.wt[wn];                                 // + 1/z
    return im;
}

// One CTA per series: suffix sums S(w) = sum_{wn >= w} term(wn).  All threads form the terms in shared memory; two
// warps sum them, one the real and one the imaginary parts (an FP64 instruction holds its quarter of the SM for 64
// cycles whatever lanes are active), lane l owning the l-th of 32 contiguous ranges (first the range totals, a suffix
// scan of them over the lanes, then the running sums), and all threads write the sums out.  Terms are rounded before they are added (the
// window choice compares variances down to their rounding, so it must not depend on which sums are fused).
// STAGED = false (N_freq beyond the shared memory): the same sums with the terms formed where they are added.
constexpr int SUF_THREADS = 256;
inline size_t suffix_smem(int Nf) { return (size_t)(Nf + 32) * sizeof(double2); }
template <bool STAGED>
__global__ void __launch_bounds__(SUF_THREADS) k_mom_suffix(MomArgs g) {
    extern __shared__ double2 ssm[];
    const int series = blockIdx.x, nG = g.P * g.ncol;
    const int chunk = (g.Nf + 31) / 32;
    double2 *sv = ssm;  // term wn at wn + wn / chunk (bank spread)
    int a = 0, b = 0;
    const int c = series < nG ? series % g.ncol : series - nG;
    if (series < nG) pair_of(series / g.ncol, g.D, a, b);
    auto term = [&](int wn) {
        const double *wt = g.wt + wn;
        const int Nf = g.Nf;
        if (series < nG) {
            const double2 v = mom_value(g, a, b, c, wn);
            const int p = g.green ? 1 + c : c - 1;  // the weight series; column 0 of the general fit has none
            if (p < 0) return v;
            const double w = wt[(size_t)p * Nf];
            return cmk(__dmul_rn(v.x, w), __dmul_rn(v.y, w));
        }
        if (c == 0) return cmk(1.0, 0.0);
        if (c == 1) return cmk(wt[Nf], 0.0);  // K(.,0) K(.,2) on Re rows
        const double x = c == 2 ? wt[Nf] : (c == 5 ? wt[2 * Nf] : wt[0]);
        const double y = c == 2 ? wt[Nf] : (c == 3 ? wt[0] : wt[2 * Nf]);
        return cmk(__dmul_rn(x, y), 0.0);
    };
    if (STAGED) {
        for (int wn = threadIdx.x; wn < g.Nf; wn += blockDim.x) sv[wn + wn / chunk] = term(wn);
        __syncthreads();
    }
    double2 *So = g.S + (size_t)series * g.R;
    double *Ko = g.KS + (size_t)(series - nG) * g.R;
    if (threadIdx.x < 64) {
        const int lane = threadIdx.x & 31, im = threadIdx.x >> 5;
        const int lo = min(g.Nf, lane * chunk), hi = min(g.Nf, lo + chunk);
        double *sc = reinterpret_cast<double *>(sv) + im;  // this warp's component
        auto at = [&](int wn) {
            if (STAGED) return sc[2 * (wn + lane)];
            const double2 v = term(wn);
            return im ? v.y : v.x;
        };
        double part = 0;
#pragma unroll 4
        for (int wn = hi - 1; wn >= lo; wn--) part += at(wn);
        // carry = sum of the ranges of all higher lanes (inclusive suffix scan, then shift)
        double incl = part;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const double v = __shfl_sync(0xffffffffu, incl, min(31, lane + off), 32);
            if (lane + off < 32) incl += v;
        }
        double run = incl - part;
#pragma unroll 4
        for (int wn = hi - 1; wn >= lo; wn--) {
            run += at(wn);
            if (STAGED) sc[2 * (wn + lane)] = run;
            else if (wn < g.R) {
                if (series < nG) (im ? So[wn].y : So[wn].x) = run;
                else if (!im) Ko[wn] = run;
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
// staged in shared memory) and sums of the moments for the gates (the other CTAs, one series and a tile of centres
// each: staged, then one thread per component and run of AVG_RUN centres, the first range summed directly and the next
// ones by sliding).  Bound by the FP64 adds, (2 Nv + 1)/AVG_RUN + 2 per centre and component: longer runs mean fewer
// adds but a longer chain; with 64 the green fit takes 68 us at D = 10, N_freq = 4096 (one thread per run of 32 centres
// reading the fits at a stride: 148 us).
constexpr int AVG_RUN = 64;
constexpr int AVG_THREADS = 128;
constexpr int AVG_TILE = AVG_RUN * AVG_THREADS / 2;  // centres per tile
__host__ __device__ constexpr int avg_pad(int i) { return i + i / AVG_RUN; }
__global__ void __launch_bounds__(AVG_THREADS) k_mom_avg(MomArgs g, int nvar, int vstaged, int astaged) {
    extern __shared__ double2 ssm[];
    const int L = 2 * g.Nv + 1;
    if ((int)blockIdx.x < nvar) {
        const int ncb = (g.C + AVG_THREADS - 1) / AVG_THREADS;
        const int i = blockIdx.x / ncb, c0 = (blockIdx.x % ncb) * AVG_THREADS, ci = c0 + threadIdx.x;
        const double *tr = g.tr + (size_t)i * g.R + c0;
        if (vstaged) {
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
    const int ntile = (g.C + AVG_TILE - 1) / AVG_TILE, q = blockIdx.x - nvar;
    const int series = q / ntile, tile0 = (q % ntile) * AVG_TILE;
    const int pr = series / g.ncol, i = series % g.ncol, nc = min(AVG_TILE, g.C - tile0);
    const double2 *x = g.mt + (size_t)series * g.R + tile0;
    if (astaged) {
        for (int t = threadIdx.x; t < nc + L - 1; t += AVG_THREADS) ssm[avg_pad(t)] = x[t];
        __syncthreads();
    }
    const int im = threadIdx.x & 1, c0 = (threadIdx.x >> 1) * AVG_RUN, c1 = min(nc, c0 + AVG_RUN);
    const double *xs = reinterpret_cast<const double *>(astaged ? ssm : x) + im;
    auto at = [&](int t) { return xs[2 * (astaged ? avg_pad(t) : t)]; };
    double *o = reinterpret_cast<double *>(g.avg + ((size_t)i * g.C + tile0) * g.P + pr) + im;
    if (c0 >= nc) return;
    double s = 0;
#pragma unroll 8
    for (int t = c0; t < c0 + L; t++) s += at(t);
    for (int ci = c0; ci < c1; ci++) {
        if (ci > c0) s = (s + at(ci + L - 1)) - at(ci - 1);
        o[2 * (size_t)ci * g.P] = s;
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
    const int P = g.P;
    const double L = 2 * g.Nv + 1;
    // the averaged moment `col` into M
    auto load = [&](int col, double2 *M) {
        const double2 *sum = g.avg + ((size_t)col * g.C + ci) * P;
        for (int q = lane; q < P; q += 32) {
            int a, b;
            pair_of(q, D, a, b);
            const double2 v = cmk(sum[q].x / L, sum[q].y / L);
            M[a + b * D] = v;
            if (a != b) M[b + a * D] = cconj(v);
        }
    };
    if (!g.green) {
        load(1, A);
        load(2, W);
        load(3, X);
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
        load(0, W);
        load(1, X);
        __syncwarp();
        for (int e = lane; e < DD; e += 32) {
            const int i = e % D, j = e / D;
            if (i < j) continue;
            double2 s = X[e];
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
    if (tid > 1) return;
    const double *xs = reinterpret_cast<const double *>(x) + tid;  // thread 0: real parts, thread 1: imaginary parts
    double s = 0;
#pragma unroll 8
    for (int w = 0; w < L; w++) s += xs[2 * w];
    s /= L;
    if (a == b && tid == 1) s = 0.0;
    reinterpret_cast<double *>(o + a + b * D)[tid] = s;
    if (a != b) reinterpret_cast<double *>(o + b + a * D)[tid] = tid ? -s : s;
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
           oTr = carve((size_t)g.ncol * g.R * sizeof(double)), oAvg = carve((size_t)g.ncol * g.C * P * sizeof(double2)),
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
        k_mom_suffix<false><<<nseries, 64, 0, s>>>(g);
    }
    DG_LAUNCH(ctx, "k_mom_suffix");
    k_mom_solve<<<dg_ceil_div(g.R, 32), SOLVE_THREADS, 0, s>>>(g);
    DG_LAUNCH(ctx, "k_mom_solve");
    const int nvar = g.ncol * dg_ceil_div(g.C, AVG_THREADS);
    const int navg = g.P * g.ncol * dg_ceil_div(g.C, AVG_TILE);
    const size_t smv = (AVG_THREADS + L) * sizeof(double), smf = L * sizeof(double2);
    const size_t sma = (size_t)(avg_pad(std::min(g.C, AVG_TILE) + (int)L) + 1) * sizeof(double2);
    const int stv = smv <= 48 * 1024, sta = sma <= 160 * 1024, stf = smf <= 40 * 1024;
    const size_t smavg = std::max(stv ? smv : 0, sta ? sma : 0);
    DG_CUDA(cudaFuncSetAttribute(k_mom_avg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smavg));
    k_mom_avg<<<nvar + navg, AVG_THREADS, smavg, s>>>(g, nvar, stv, sta);
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
