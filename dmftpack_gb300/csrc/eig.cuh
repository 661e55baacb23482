// eig.cuh -- Hermitian eigen-decompositions of the lattice's per-k matrices (n <= 64) in shared memory by groups of T threads
// (one warp or four per matrix): cyclic Jacobi in round-robin order, n/2 disjoint pairs (p, q) per round, in FP64
// (Ops = OpsD) or packed double-float on the FP32 pipe (OpsP, the DMFTGPU_MIXED passes).  The lower triangle is read and the
// diagonal taken real; the rotation is jacobi_rotation's (an FP32 angle refined); it stops when the
// off-diagonal mass is <= tol of the total.
//
// A round is two steps: the rotations (one per thread), then A' = J^H A J by the 2 x 2 blocks of pairs i <= j -- rows and
// columns of a block in one thread, the lower triangle only -- and the columns of U.  A rotation is applied as
// y = conj(ph) x_q, x_p' = c x_p - s y, x_q' = s x_p + c y: 12 real multiply-adds.
//
// What bounds it is latency when the k points are few (the rounds of a 28 x 28 matrix, some 200, follow one another) and
// arithmetic when they are many.  So larger matrices get four warps (eig_one_warp, lattice.cu).  One warp per matrix that
// rotated all columns, then all rows, with c ph and s ph formed per element took 2.8 ms for a single 28 x 28 matrix in
// double-float and 3.85 ms for 1,000, with 0.8 ms for their 18 x 18 blocks before it; the G_loc pass of the d + p model
// at 1,000 k went from 25.7 to 22.5 ms, at two k points and 32 frequencies from 2.8 to 0.66 ms.
#pragma once
#include "df.cuh"
#include "smallmat.cuh"
#include "smallmat_df.cuh"

constexpr int EIG_NMAX = 64;

// c a + s b with real c, s
__device__ __forceinline__ double2 eig_lin(double2 a, double c, double2 b, double s) {
    return cmk(fma(c, a.x, s * b.x), fma(c, a.y, s * b.y));
}
__device__ __forceinline__ pdf eig_lin(pdf a, dfl c, pdf b, dfl s) { return pdf_dot2(a, pdf_both(c), b, pdf_both(s)); }

template <class Ops>
struct JRot {
    int p, q, on;
    typename Ops::R c, s;
    typename Ops::C ph;
};
__device__ __forceinline__ void eig_rotation(JRot<OpsD> &R, double2 apq, double2 app, double2 aqq) {
    const DgRot r = jacobi_rotation(0, 0, apq, app.x, aqq.x);
    R.on = r.on;
    R.c = r.c;
    R.s = r.s;
    R.ph = r.ph;
}
// jacobi_tan in double-float, r in [0.5, 1.5): the FP32 root and one Newton step
__host__ __device__ __forceinline__ dfl jacobi_tan(dfl r, dfl d) {
    const float ax = fabsf(d.h);
    if (!(ax <= 1e30f)) return {0.f, 0.f};
    const float slope = ax > 1e9f ? ax : sqrtf(fmaf(d.h, d.h, 4.f * r.h * r.h));
    const float t = copysignf(fast_div(2.f * r.h, ax + slope), d.h);
    const dfl g = df_sub(df_mul(df_add(df_mul(r, {t, 0.f}), d), {t, 0.f}), r);
    return fast_two_sum(t, -g.h * copysignf(fast_div(1.f, slope), d.h));
}
__device__ __forceinline__ void eig_rotation(JRot<OpsP> &R, pdf apq, pdf app, pdf aqq) {
    R.on = 0;
    R.c = {1.f, 0.f};
    R.s = {0.f, 0.f};
    R.ph = OpsP::one();
    const float mx = fmaxf(fabsf(apq.h.x), fabsf(apq.h.y));
    if (!(mx > 1e-37f)) return;
    // |a_pq| and its phase from the entry scaled by a power of two to [0.5, 1): the squares of a small entry would
    // otherwise lose their low parts to FP32 underflow, and a phase that is not unit breaks the rotation's unitarity
    const float sc = __int_as_float(max(253 - (__float_as_int(mx) >> 23), 1) << 23);
    const dfl ar = {apq.h.x * sc, apq.l.x * sc}, ai = {apq.h.y * sc, apq.l.y * sc};
    const dfl r2 = df_fma(ai, ai, df_mul(ar, ar));
    const dfl ir = df_rsqrt(r2);
    const dfl r = df_mul(r2, ir);  // |a_pq| sc
    const dfl d = df_sub(OpsP::cre(aqq), OpsP::cre(app)), t = jacobi_tan(r, {d.h * sc, d.l * sc});
    R.c = df_rsqrt(df_fma(t, t, {1.f, 0.f}));
    R.s = df_mul(t, R.c);
    R.ph = OpsP::mk(df_mul(ar, ir), df_mul(ai, ir));
    R.on = 1;
}

__device__ __forceinline__ double eig_abs2(double2 v) { return cabs2(v); }
__device__ __forceinline__ float eig_abs2(pdf v) { return __fmaf_rn(v.h.x, v.h.x, __fmul_rn(v.h.y, v.h.y)); }

// shared memory of one matrix: A and U [n][n], eigenvalues, their order, rotations, a reduction's slots
template <class Ops>
struct EigMem {
    typename Ops::C *a, *u;
    double *w;
    int *order;
    JRot<Ops> *rot;
    typename Ops::M *red;  // [8]
    __device__ EigMem(unsigned char *base, int n) {
        a = reinterpret_cast<typename Ops::C *>(base);
        u = a + n * n;
        w = reinterpret_cast<double *>(u + n * n);
        order = reinterpret_cast<int *>(w + EIG_NMAX);
        rot = reinterpret_cast<JRot<Ops> *>(order + EIG_NMAX);
        red = reinterpret_cast<typename Ops::M *>(rot + EIG_NMAX / 2);
    }
};
template <class Ops>
__host__ __device__ constexpr size_t eig_bytes(int n) {
    return ((size_t)2 * n * n * 16 + EIG_NMAX * 12 + EIG_NMAX / 2 * sizeof(JRot<Ops>) + 64 + 15) & ~(size_t)15;
}
// The place of value i in ascending order, equal values by their index and NaN after every number (NaN, as it is in an input,
// fails every plain comparison): over i always a permutation, whatever is in w, for the vectors are addressed through it.
__host__ __device__ inline int eig_rank(const double *w, int n, int i) {
    const double wi = w[i];
    const bool nan = wi != wi;
    int rank = 0;
    for (int j = 0; j < n; j++) {
        const double wj = w[j];
        rank += nan ? (wj == wj || j < i) : (wj < wi || (wj == wi && j < i));
    }
    return rank;
}
template <int T>
__device__ __forceinline__ void eig_sync() {
    if constexpr (T == 32) __syncwarp();
    else __syncthreads();
}

// All T threads of the group (tid 0 .. T - 1; a whole warp, or the whole block) call it with A's lower triangle in e.a.
// Eigenvectors in e.u (columns), eigenvalues in e.w, both unsorted; e.order[l]: the column of the l-th lowest.
template <class Ops, int T>
__device__ int group_heig(int n, const EigMem<Ops> &e, typename Ops::M tol, int tid) {
    typedef typename Ops::C C;
    typedef typename Ops::M M;
    C *a = e.a, *u = e.u;
    for (int x = tid; x < n * n; x += T) u[x] = x % n == x / n ? Ops::one() : Ops::zero();
    eig_sync<T>();
    const int m = n + (n & 1), half = m / 2, nb = half * (half + 1) / 2, inv = (1 << 20) / n + 1;
    const int u0 = (tid + T - nb % T) % T;  // the threads that have a block less begin with the columns of U
    int st = DG_NONCONV;
    for (int sweep = 0; sweep < 100; sweep++) {
        M off = 0, tot = 0;
        for (int x = tid; x < n * n; x += T) {
            const int j = (x * inv) >> 20, i = x - j * n;
            if (i < j) continue;
            const M v = eig_abs2(a[x]);
            tot += i > j ? 2 * v : v;
            if (i > j) off += 2 * v;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if constexpr (T > 32) {
            if ((tid & 31) == 0) {
                e.red[tid / 32] = off;
                e.red[4 + tid / 32] = tot;
            }
            __syncthreads();
            off = tot = 0;
            for (int i = 0; i < T / 32; i++) {
                off += e.red[i];
                tot += e.red[4 + i];
            }
        }
        if (off == M(0) || off <= tol * tot) {  // the same sums in every thread
            st = DG_OK;
            break;
        }
        for (int r = 0; r < m - 1; r++) {
            if (tid < half) {
                int p = r + tid, q = r - tid;
                if (p >= m - 1) p -= m - 1;
                if (q < 0) q += m - 1;
                if (tid == 0) q = m - 1;
                if (p > q) {
                    const int t = p;
                    p = q;
                    q = t;
                }
                JRot<Ops> R;
                R.on = 0;
                if (q < n) eig_rotation(R, Ops::conj(a[q + p * n]), a[p + p * n], a[q + q * n]);
                if (!R.on) {
                    R.c = Ops::cre(Ops::one());
                    R.s = Ops::cre(Ops::zero());
                    R.ph = Ops::one();
                }
                R.p = p;
                R.q = q;
                e.rot[tid] = R;
            }
            eig_sync<T>();
            for (int x = tid; x < nb; x += T) {
                int j = (int)((sqrtf(8.f * x + 1.f) - 1.f) * 0.5f);
                if (j * (j + 1) / 2 > x) j--;
                if ((j + 1) * (j + 2) / 2 <= x) j++;
                const JRot<Ops> R1 = e.rot[x - j * (j + 1) / 2], R2 = e.rot[j];
                if (!(R1.on | R2.on)) continue;
                // rows (p1, q1), columns (p2, q2); an index n (n odd) stands for a row and column of zeros
                auto get = [&](int r_, int c_) {
                    if (r_ >= n || c_ >= n) return Ops::zero();
                    return r_ >= c_ ? a[r_ + c_ * n] : Ops::conj(a[c_ + r_ * n]);
                };
                auto put = [&](int r_, int c_, C v) {
                    if (r_ >= n || c_ >= n) return;
                    if (r_ >= c_) a[r_ + c_ * n] = v;
                    else a[c_ + r_ * n] = Ops::conj(v);
                };
                const bool diag = R1.p == R2.p;
                C pp = get(R1.p, R2.p), pq = get(R1.p, R2.q), qp = get(R1.q, R2.p), qq = get(R1.q, R2.q);
                const auto s1 = Ops::rneg(R1.s), s2 = Ops::rneg(R2.s);
                C y = Ops::mulc(pq, R2.ph), z = Ops::mulc(qq, R2.ph);
                pq = eig_lin(pp, R2.s, y, R2.c);
                pp = eig_lin(pp, R2.c, y, s2);
                qq = eig_lin(qp, R2.s, z, R2.c);
                qp = eig_lin(qp, R2.c, z, s2);
                y = Ops::mul(qp, R1.ph);
                z = Ops::mul(qq, R1.ph);
                qp = eig_lin(pp, R1.s, y, R1.c);
                pp = eig_lin(pp, R1.c, y, s1);
                qq = eig_lin(pq, R1.s, z, R1.c);
                pq = eig_lin(pq, R1.c, z, s1);
                if (diag) {
                    pp = Ops::mk(Ops::cre(pp), Ops::cre(Ops::zero()));
                    qq = Ops::mk(Ops::cre(qq), Ops::cre(Ops::zero()));
                } else {
                    put(R1.p, R2.q, pq);
                }
                put(R1.p, R2.p, pp);
                put(R1.q, R2.p, qp);
                put(R1.q, R2.q, qq);
            }
            for (int x = u0; x < half * n; x += T) {
                const int i = (x * inv) >> 20, k = x - i * n;
                const JRot<Ops> R = e.rot[i];
                if (!R.on) continue;
                const C up = u[k + R.p * n], y = Ops::mulc(u[k + R.q * n], R.ph);
                u[k + R.p * n] = eig_lin(up, R.c, y, Ops::rneg(R.s));
                u[k + R.q * n] = eig_lin(up, R.s, y, R.c);
            }
            eig_sync<T>();
        }
    }
    for (int i = tid; i < n; i += T) e.w[i] = Ops::re(a[i + i * n]);
    eig_sync<T>();
    for (int i = tid; i < n; i += T) e.order[eig_rank(e.w, n, i)] = i;
    eig_sync<T>();
    return st;
}
