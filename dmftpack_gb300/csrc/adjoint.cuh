// adjoint.cuh -- reverse- and forward-mode derivatives of the lattice sum G_loc(iw) = (1/N_k) sum_k G_PP(k, iw)
// with respect to the self-energy and the chemical potential, k_gloc_ad<LW, MODE> (LW lanes per matrix).
//
// With G = (z - H - Sigma)^-1 on the full orbital space and Sigma acting on the correlated block P:
//   dG_PP = G_PP dSigma G_PP                      (dSigma lives on P, so only the P block of G enters)
//   dG_PP = -(G^2)_PP dmu = -G_PP S' G_PP dmu    (S' = I + sum_l w_l^2 b_l b_l^H, the Schur form's dS/dz)
// so for one frequency
//   JVP:  dG_loc = (1/N_k) sum_k G_PP (dSigma - dmu S') G_PP
//   VJP:  Sigma_bar = (1/N_k) sum_k G_PP^H Gbar G_PP^H,   mu_bar = -(1/N_k) sum_k Re Tr[(G_PP S' G_PP)^H Gbar]
// (the adjoint of the holomorphic map in the convention of torch's complex autograd: x_bar = J^H y_bar).  G_PP
// is recomputed for every (k, iw) from the per-k Schur data, as the forward pass does, and never stored: the
// memory is O(N_freq D^2) whatever N_k, N_freq and n are.
//
// What bounds the pass is FP64 instructions: a warp's FP64 instruction holds its SM sub-partition's pipe for 64 cycles
// whatever its lanes do, so lanes have to be full and everything else (shared memory, index arithmetic) is free beside it.
//   - One matrix per group of LW lanes, its D^2 elements dealt over the lanes (at most 13 each): 12.5 of 13 slots carry an
//     element at D = 20 with 32 lanes, 12.5 of 13 at D = 10 with 8.  One column per lane left 12 of 32 lanes idle at D = 20.
//   - S and S' as sums of real weights times the Hermitian products b_l b_l^H: a thread takes a pair (a <= c) and four or
//     eight frequencies and forms the product once for them: 4 FMA per pole, pair and sum where rank-one updates of both
//     triangles take 8 (and a complex product each for their weights).
//   - VJP: Re Tr[(G S' G)^H Gbar] = Re Tr[S'^H Z] with the Z = G^H Gbar G^H that Sigma_bar sums, which leaves two D^3
//     products of four.  S' is formed after Z, so two tiles per matrix serve and two CTAs fit an SM.
// 56 orbitals, D = 20, 125 k x 512 frequencies: 61.8 -> 23.9 ms (JVP) and 72.6 -> 23.9 (VJP),
// the eigensolvers of the preparation (3.5 ms) included; 10 + 18 orbitals 9.4 -> 4.6 and 10.8 -> 4.7, 4 + 12 2.4 -> 0.9 and 2.7 -> 1.0.
// CTA = F frequencies x one chunk of k points; per-chunk sums are reduced in fixed order.
//
// The forward passes in FP64 run in the same way from some 5 orbitals on (run_schur): AD_BLOCK, G_loc and GwHF (the inverse of M and of
// z - m0 - H_PP - S in its second tile), and AD_TRACE, N(mu) (Re[Tr G - Tr G0] of k_schur's TRACE form, the second tile
// I + R).  343 k x 400 frequencies of 10 + 18 orbitals: G_loc 17.3 -> 12.5 ms, N(mu) 18.0 -> 11.7 against the columns of k_schur.
#pragma once
#include "internal.h"
#include "schur.cuh"

namespace dg {

enum { AD_VJP = 1, AD_JVP = 2, AD_BLOCK = 3, AD_TRACE = 4 };
constexpr int AD_EL = 13;        // matrix elements per lane at most
constexpr int AD_THREADS = 256;  // at most; two CTAs per SM

struct AdArgs {
    const double2 *H, *B;  // [nk][n][n]; [nk][m][D] b_l(a)
    const double *epsQ;    // [nk][m]
    const double2 *sig;    // [nf][D][D] Sigma(iw_n), n < nf
    const double2 *m0;     // BLOCK: [D][D] the static moment
    const double *eps0;    // TRACE: [nk][n] eigenvalues of H + m0
    int wgrid;             // TRACE: the N(mu) frequency grid
    const double2 *gin;    // VJP: Gbar [nf][D][D]; JVP: Sigma_dot [nf][D][D]
    double mu_dot;         // JVP
    int n, m, nk, nf, D, kchunk, F;
    double beta, mu;
    double2 *pout;         // [nchunk][nf][D][D] per-chunk sums (Sigma_bar or G_loc_dot, before the 1/N_k)
    double *pmu;           // [nchunk][nf] VJP: per-chunk Re Tr[(G S' G)^H Gbar]
    double2 *pout0;        // BLOCK: the sums of G0_PP; TRACE: [nchunk][nf] (Re[Tr G - Tr G0], 0)
    int *status;
};

// shared memory of one frequency, in double2: two tiles, the weights (w_l, w_l^2), and the inversion's row, column and
// pivot buffers, which lie over the second tile (VJP) or over the weights (else), both free then
__host__ __device__ inline int ad_bufs(int D) { return 2 * D + (D + 3) / 4; }
__host__ __device__ inline int ad_tile1(int D, int mode) {
    return mode == AD_VJP && ad_bufs(D) > D * D ? ad_bufs(D) : D * D;
}
__host__ __device__ inline int ad_weights(int D, int m, int mode) {
    return mode != AD_VJP && ad_bufs(D) > 2 * m ? ad_bufs(D) : 2 * m;
}
inline size_t ad_smem(int F, int D, int m, int mode) {
    return (size_t)F * (D * D + ad_tile1(D, mode) + ad_weights(D, m, mode)) * 16 + (size_t)(D * (D + 1) / 2) * 4;
}

// In-place inverse of the D x D tile A (column-major) by LW lanes; every group of the warp calls it together.  Gauss-Jordan
// with partial pivoting by max(|re|, |im|) compared on the high words (no FP64 work): every element is updated alike as
// A - col(r) row(c), with row k and column k read as zero, row = the scaled pivot row with 1/pivot at k and col(k) = -1.
template <int LW>
__device__ __forceinline__ bool tile_inverse(double2 *A, int D, double2 *rowb, double2 *colb, int *perm, int g) {
    bool sing = false, moved = false;
    const int DD = D * D;
#pragma unroll 1
    for (int k = 0; k < D; k++) {
        unsigned best = 0;
        int p = k;
        for (int r = k + g; r < D; r += LW) {
            const double2 v = A[r + k * D];
            const unsigned key = max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu);
            if (key > best) {
                best = key;
                p = r;
            }
        }
#pragma unroll
        for (int o = LW / 2; o > 0; o >>= 1) {
            const unsigned ob = __shfl_xor_sync(0xffffffffu, best, o, LW);
            const int op = __shfl_xor_sync(0xffffffffu, p, o, LW);
            if (ob > best || (ob == best && op < p)) {
                best = ob;
                p = op;
            }
        }
        if (g == 0) perm[k] = p;
        if (__any_sync(0xffffffffu, p != k)) {
            moved = true;
            for (int c = g; c < D; c += LW) {
                const double2 t = A[k + c * D];
                A[k + c * D] = A[p + c * D];
                A[p + c * D] = t;
            }
            __syncwarp();
        }
        const double2 piv = A[k + k * D];
        const double den = fma(piv.x, piv.x, piv.y * piv.y);
        sing |= (unsigned)__double2hiint(den) - 1u >= 0x7fefffffu;  // zero, infinite or NaN
        const double q = 1.0 / den;
        const double2 ip = cmk(piv.x * q, -piv.y * q);
        for (int c = g; c < D; c += LW) {
            rowb[c] = c == k ? ip : cmul(A[k + c * D], ip);
            colb[c] = c == k ? cmk(-1.0, 0.0) : A[c + k * D];
        }
        __syncwarp();
        int r = g % D, c = g / D;
#pragma unroll 4
        for (int e = g; e < DD; e += LW) {
            const bool z = r == k || c == k;
            A[e] = cfms(colb[r], rowb[c], z ? cmk(0.0, 0.0) : A[e]);
            r += LW;
            while (r >= D) {
                r -= D;
                c++;
            }
        }
        __syncwarp();
    }
    if (!moved) return sing;
#pragma unroll 1
    for (int k = D - 1; k >= 0; k--) {  // undo the row interchanges as column interchanges, last first
        const int p = perm[k];
        for (int r = g; r < D; r += LW) {
            const double2 t = A[r + k * D];
            A[r + k * D] = A[r + p * D];
            A[r + p * D] = t;
        }
        __syncwarp();
    }
    return sing;
}

// sums over the poles of one pair (a, c) and SUB frequencies: s[i] = sum_l (Re, Im of the weight) x (p, q), with
// b_a conj(b_c) = p + iq; slot: the weights' slot (0: w, 1: w^2)
struct PairSum {
    double up, uq, vp, vq;
    __device__ __forceinline__ void add(double2 w, double p, double q) {
        up = fma(w.x, p, up);
        uq = fma(w.x, q, uq);
        vp = fma(w.y, p, vp);
        vq = fma(w.y, q, vq);
    }
    // sum_l w_l b_a conj(b_c) and sum_l w_l b_c conj(b_a)
    __device__ __forceinline__ double2 ac() const { return cmk(up - vq, uq + vp); }
    __device__ __forceinline__ double2 ca() const { return cmk(up + vq, vp - uq); }
};

template <int LW, int MODE>
__global__ void __launch_bounds__(AD_THREADS, 2) k_gloc_ad(AdArgs g) {
    typedef double2 C;
    constexpr bool TWO = MODE == AD_JVP || MODE == AD_TRACE;  // S and S' at once
    constexpr int SUB = TWO ? 4 : 8;
    extern __shared__ double2 sm[];
    const int D = g.D, DD = D * D, m = g.m, F = g.F, npair = D * (D + 1) / 2;
    const int t1 = ad_tile1(D, MODE), ws = ad_weights(D, m, MODE);
    C *T0 = sm, *T1 = T0 + (size_t)F * DD, *sW = T1 + (size_t)F * t1;
    ushort2 *sPair = reinterpret_cast<ushort2 *>(sW + (size_t)F * ws);
    const int lane = threadIdx.x % LW, grp = threadIdx.x / LW, f0 = blockIdx.x * F;
    const bool fvalid = f0 + grp < g.nf;
    const int f = min(f0 + grp, g.nf - 1);
    const int chunk = blockIdx.y, kbeg = chunk * g.kchunk, kend = min(g.nk, kbeg + g.kchunk);
    C *A = T0 + (size_t)grp * DD, *V = T1 + (size_t)grp * t1;
    C *buf = MODE == AD_VJP ? V : sW + (size_t)grp * ws;
    for (int t = threadIdx.x; t < npair; t += blockDim.x) {  // t = a + c (c + 1) / 2, a <= c
        int c = 0;
        while ((c + 1) * (c + 2) / 2 <= t) c++;
        sPair[t] = make_ushort2((unsigned short)(t - c * (c + 1) / 2), (unsigned short)c);
    }
    auto wfreq = [&](int ff) {
        return MODE == AD_TRACE && g.wgrid ? (DG_PI / g.beta + ff * ((2 * DG_PI) / g.beta)) : (DG_PI * (2. * ff + 1.) / g.beta);
    };
    constexpr int NACC = MODE == AD_TRACE ? 1 : AD_EL;
    C acc[NACC], acc0[MODE == AD_BLOCK ? AD_EL : 1];
#pragma unroll
    for (int i = 0; i < NACC; i++) acc[i] = cmk(0, 0);
#pragma unroll
    for (int i = 0; i < (MODE == AD_BLOCK ? AD_EL : 1); i++) acc0[i] = cmk(0, 0);
    FracSum<OpsD> fr;
    double accmu = 0.0;
    bool sing = false;
    const int nsub = (F + SUB - 1) / SUB;
    for (int k = kbeg; k < kend; k++) {
        const C *__restrict__ Bk = g.B + (size_t)k * m * D, *__restrict__ Hk = g.H + (size_t)k * g.n * g.n;
        __syncthreads();
        for (int t = threadIdx.x; t < F * m; t += blockDim.x) {
            const int fl = t / m, l = t - fl * m;
            const double w = wfreq(min(f0 + fl, g.nf - 1));
            const C wl = crcp(cmk(g.mu - g.epsQ[(size_t)k * m + l], w));
            sW[(size_t)fl * ws + 2 * l] = wl;
            if (MODE != AD_BLOCK) sW[(size_t)fl * ws + 2 * l + 1] = cmul(wl, wl);
        }
        if (MODE == AD_TRACE) {  // - Tr G0
            const double w = wfreq(f), w2 = w * w;
            for (int j = lane; j < g.n; j += LW) {
                const double x = g.mu - g.eps0[(size_t)k * g.n + j];
                fr.add(-x, fma(x, x, w2));
            }
        }
        __syncthreads();
        double tk = 0.0;  // this k point's terms of accmu
        if (MODE == AD_TRACE)
            for (int l = lane; l < m; l += LW) tk += sW[(size_t)grp * ws + 2 * l].x;
        // M = z - H_PP - Sigma - S into the first tile; into the second JVP: Sigma_dot - mu_dot S', BLOCK: M with m0 in the place of
        // Sigma, TRACE: S', transposed
        for (int t = threadIdx.x; t < npair * nsub; t += blockDim.x) {
            const int s = t / npair;
            const ushort2 pr = sPair[t - s * npair];
            const int a = pr.x, c = pr.y;
            PairSum x[SUB], y[TWO ? SUB : 1];
#pragma unroll
            for (int i = 0; i < SUB; i++) {
                x[i] = {0, 0, 0, 0};
                if (TWO) y[i] = {0, 0, 0, 0};
            }
            for (int l = 0; l < m; l++) {
                const C pq = cmulc(Bk[l * D + a], Bk[l * D + c]);
#pragma unroll
                for (int i = 0; i < SUB; i++) {
                    const C *w = sW + (size_t)min(s * SUB + i, F - 1) * ws + 2 * l;
                    x[i].add(w[0], pq.x, pq.y);
                    if (TWO) y[i].add(w[1], pq.x, pq.y);
                }
            }
            const C h = Hk[a + c * g.n], ht = Hk[c + a * g.n];
#pragma unroll
            for (int i = 0; i < SUB; i++) {
                const int fl = s * SUB + i;
                if (fl >= F) break;
                const int ff = min(f0 + fl, g.nf - 1);
                const C *sg = g.sig + (size_t)ff * DD;
                C hs = cneg(cadd(h, x[i].ac())), hst = cneg(cadd(ht, x[i].ca()));
                if (a == c) hs = hst = cadd(hs, cmk(g.mu, wfreq(ff)));
                T0[(size_t)fl * DD + a + c * D] = csub(hs, sg[a + c * D]);
                T0[(size_t)fl * DD + c + a * D] = csub(hst, sg[c + a * D]);
                if (MODE == AD_BLOCK) {
                    // m0 as it is below 8 orbitals, from 8 on its lower triangle, as the static spectrum reads it
                    C mt = g.m0[c + a * D], mu_ = g.m0[a + c * D];
                    if (D >= 8) {
                        if (a == c) mt.y = 0.0;
                        mu_ = cconj(mt);
                    }
                    T1[(size_t)fl * DD + a + c * D] = csub(hs, mu_);
                    T1[(size_t)fl * DD + c + a * D] = csub(hst, mt);
                }
                if (MODE == AD_TRACE) {
                    const double one = a == c ? 1.0 : 0.0;
                    const C u = y[i].ac(), v = y[i].ca();
                    T1[(size_t)fl * DD + c + a * D] = cmk(one + u.x, u.y);
                    T1[(size_t)fl * DD + a + c * D] = cmk(one + v.x, v.y);
                }
                if (MODE == AD_JVP) {
                    const C *sd = g.gin + (size_t)ff * DD;
                    const double one = a == c ? 1.0 : 0.0;
                    const C u = y[i].ac(), v = y[i].ca();
                    T1[(size_t)fl * DD + a + c * D] = csub(sd[a + c * D], cscale(cmk(one + u.x, u.y), g.mu_dot));
                    T1[(size_t)fl * DD + c + a * D] = csub(sd[c + a * D], cscale(cmk(one + v.x, v.y), g.mu_dot));
                }
            }
        }
        __syncthreads();
        sing |= tile_inverse<LW>(A, D, buf, buf + D, reinterpret_cast<int *>(buf + 2 * D), lane) && fvalid;
        if (MODE == AD_BLOCK) {
            sing |= tile_inverse<LW>(V, D, buf, buf + D, reinterpret_cast<int *>(buf + 2 * D), lane) && fvalid;
#pragma unroll
            for (int i = 0; i < AD_EL; i++) {
                const int e = lane + i * LW;
                if (e < DD) {
                    acc[MODE == AD_BLOCK ? i : 0] = cadd(acc[MODE == AD_BLOCK ? i : 0], A[e]);
                    acc0[MODE == AD_BLOCK ? i : 0] = cadd(acc0[MODE == AD_BLOCK ? i : 0], V[e]);
                }
            }
        } else if (MODE == AD_TRACE) {
            for (int e = lane; e < DD; e += LW) tk = fma(A[e].x, V[e].x, fma(-A[e].y, V[e].y, tk));  // G(r,c) S'(c,r)
            accmu += tk;
        } else if constexpr (MODE == AD_JVP) {
            // elements e = r + D c: X G, then G (X G)
            C v[AD_EL];
#pragma unroll
            for (int i = 0; i < AD_EL; i++) {
                const int e = lane + i * LW;
                v[i] = cmk(0, 0);
                if (e < DD) {
                    const int c = e / D, r = e - c * D;
#pragma unroll 4
                    for (int b = 0; b < D; b++) v[i] = cfma(V[r + b * D], A[b + c * D], v[i]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < AD_EL; i++)
                if (lane + i * LW < DD) V[lane + i * LW] = v[i];
            __syncwarp();
#pragma unroll
            for (int i = 0; i < AD_EL; i++) {
                const int e = lane + i * LW;
                if (e < DD) {
                    const int c = e / D, r = e - c * D;
                    C x = cmk(0, 0);
#pragma unroll 4
                    for (int b = 0; b < D; b++) x = cfma(A[r + b * D], V[b + c * D], x);
                    acc[i] = cadd(acc[i], x);
                }
            }
        } else if constexpr (MODE == AD_VJP) {
            // elements e = c + D r, so that lanes read along columns of G: Gbar G^H, then Z = G^H (Gbar G^H), transposed
            const C *gb = g.gin + (size_t)f * DD;
#pragma unroll 1
            for (int e = lane; e < DD; e += LW) {
                const int r = e / D, c = e - r * D;
                C x = cmk(0, 0);
#pragma unroll 4
                for (int b = 0; b < D; b++) x = cfma(gb[r + b * D], cconj(A[c + b * D]), x);
                V[e] = x;
            }
            __syncwarp();
            C z[AD_EL];
#pragma unroll
            for (int i = 0; i < AD_EL; i++) {
                const int e = lane + i * LW;
                z[i] = cmk(0, 0);
                if (e < DD) {
                    const int r = e / D, c = e - r * D;
#pragma unroll 4
                    for (int b = 0; b < D; b++) z[i] = cfma(cconj(A[b + r * D]), V[c + b * D], z[i]);
                    acc[i] = cadd(acc[i], z[i]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < AD_EL; i++)
                if (lane + i * LW < DD) V[lane + i * LW] = z[i];
            __syncthreads();
            // S' over G, transposed as Z is
            for (int t = threadIdx.x; t < npair * nsub; t += blockDim.x) {
                const int s = t / npair;
                const ushort2 pr = sPair[t - s * npair];
                const int a = pr.x, c = pr.y;
                PairSum y[SUB];
#pragma unroll
                for (int i = 0; i < SUB; i++) y[i] = {0, 0, 0, 0};
                for (int l = 0; l < m; l++) {
                    const C pq = cmulc(Bk[l * D + a], Bk[l * D + c]);
#pragma unroll
                    for (int i = 0; i < SUB; i++)
                        y[i].add(sW[(size_t)min(s * SUB + i, F - 1) * ws + 2 * l + 1], pq.x, pq.y);
                }
#pragma unroll
                for (int i = 0; i < SUB; i++) {
                    const int fl = s * SUB + i;
                    if (fl >= F) break;
                    const double one = a == c ? 1.0 : 0.0;
                    const C u = y[i].ac(), v = y[i].ca();
                    T0[(size_t)fl * DD + c + a * D] = cmk(one + u.x, u.y);
                    T0[(size_t)fl * DD + a + c * D] = cmk(one + v.x, v.y);
                }
            }
            __syncthreads();
            for (int e = lane; e < DD; e += LW) tk = fma(A[e].x, V[e].x, fma(A[e].y, V[e].y, tk));
            accmu += tk;
        }
    }
    if (sing) dg_flag(g.status, DG_SINGULAR);
    if (MODE == AD_VJP || MODE == AD_TRACE) {
        if (MODE == AD_TRACE) accmu += fr.value();
#pragma unroll
        for (int o = LW / 2; o > 0; o >>= 1) accmu += __shfl_xor_sync(0xffffffffu, accmu, o, LW);
    }
    if (!fvalid) return;
    if (MODE == AD_TRACE) {
        if (lane == 0) g.pout0[(size_t)chunk * g.nf + f] = cmk(accmu, 0.0);
        return;
    }
    C *o = g.pout + ((size_t)chunk * g.nf + f) * DD;
#pragma unroll
    for (int i = 0; i < NACC; i++) {
        const int e = lane + i * LW;
        if (e < DD) {
            o[MODE != AD_VJP ? e : e / D + (e % D) * D] = acc[i];
            if (MODE == AD_BLOCK) g.pout0[((size_t)chunk * g.nf + f) * DD + e] = acc0[MODE == AD_BLOCK ? i : 0];
        }
    }
    if (MODE == AD_VJP && lane == 0) g.pmu[(size_t)chunk * g.nf + f] = accmu;
}

typedef void (*AdKernel)(AdArgs);
// the kernel and its lanes per matrix: the fewest that hold D^2 elements at 13 a lane
AdKernel ad_kernel(int D, int mode, int *lanes);

}  // namespace dg
