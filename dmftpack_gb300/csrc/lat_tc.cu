// lat_tc.cu -- mixed-precision (DMFTGPU_MIXED) lattice passes with the pole sums on the tensor cores: the N(mu) and dN/dmu
// passes of the mu search (GiwToNele, src/GreenFtn.cpp:513-635, in the trace form) of correlated blocks of 4 .. 10 orbitals
// and the G_loc / GwHF pass (GreenFtn_w, src/GreenFtn.cpp:142-422) of 5 .. 10.
//
// Per (k, iw_f), with w_l = 1/(z - e_l), P_l = b_l b_l^H and M = z - H_PP - Sigma(iw_f) - S (schur.cuh):
//     S = sum_l w_l P_l,   R = sum_l w_l^2 P_l,   T = sum_l w_l^3 P_l
//     G_PP = M^-1,   Tr G = Tr[M^-1 (I + R)] + sum_l w_l                                            (I + R = dM/dz)
//     d/dz Tr G = -(Tr X^2 + 2 Tr[M^-1 T] + sum_l w_l^2),   X = M^-1 (I + R).
// S, R and T are sums of a complex weight times Hermitian matrices: S = A + iB with A = sum_l Re(w_l) P_l and
// B = sum_l Im(w_l) P_l both Hermitian, so each is a real GEMM over the D^2 real degrees of freedom ("dofs") of the P_l:
// Re and Im of b_a conj(b_c) for a < c, then the diagonal |b_a|^2.  For one k and a tile of 32 frequencies the GEMM has
// 128 rows (32 frequencies x 4 channels Re w, Im w, Re w^2, Im w^2), K = the m poles (padded to 32) and N = the dofs
// (padded to a multiple of 16): 128 x NP x 32 per k, on tcgen05 with the accumulators in TMEM.  GwHF's k sum,
// blocks of 7 .. 10: sum_k sum_j U_j U_j^H / (z - e0_j) (U, e0: the static eigen-decomposition) needs no inversion between,
// it is one such GEMM with K running over all k and j (k_g0_tc).  Blocks of 5 and 6 invert z - m0 - H_PP - S as well, from
// the same S: as k_schur does at these widths, and ten times closer than the eigenvectors (1e-14 against 1e-13).
//
// Double-float-level accuracy from bf16: each row is scaled by a power of two to |x| <= 1 and split into slices, balanced
// digits of 9 bits after a first one of 8: x = sum_s v_s 2^{-(8 + 9 s)}, integers |v_s| <= 256, each exact in bf16 and
// stored with its weight; the dof columns likewise.  Products of slices (i, j) carry their true weight; those of one level
// i + j accumulate exactly in an FP32 accumulator of their own (sums of at most 64 poles stay below 2^24 in their units),
// and the highest levels share one.
//   N(mu) passes: 5 slices, levels 0, 1, 2 exact, 3 and 4 shared: values below 2^-19 of the row x column scale, so the
//     accumulator's rounding adds ~2^-44 of it, as much as the slices leave.  Four accumulators x NP columns fit TMEM's
//     512, and all 128 lanes carry rows.  (Blocks of 4, whose 16 columns leave room, take six: N(mu) is then as close as
//     k_schur's, 1e-15, where five leave 1e-14.)
//   dN/dmu: 6 slices, levels 0 .. 3 exact, 4 and 5 shared (rounding ~2^-52).  Five accumulators of 112 columns (D > 8) do
//     not fit: the columns are then multiplied and drained in two parts, 64 and NP - 64.
//   G_loc / GwHF: 6 slices likewise, but only 64 rows are needed (32 frequencies x Re w, Im w): the lower columns
//     accumulate in lanes 0 .. 63 and the upper ones in lanes 64 .. 127 of the same accumulators, so that five fit and all
//     four lane quarters drain alike.  In the A image every block of 64 rows stands between 64 rows of zeros; an MMA that
//     starts at the block fills lanes 0 .. 63, one that starts at the zeros before it lanes 64 .. 127.
// (5 slices of 8 bits left 2^-41: five to ten times the error of double-float sums in G_loc, and
// 5 of 9 twenty times in dN/dmu.)
//
// Work split: what bounds the passes is the double-float D x D inversions on the FP32 pipe, so they run on warps of their
// own, one frequency per group of DP lanes (32/DP groups per warp, group_gj_inverse in packed arithmetic), and four
// producer warps prepare the next k beside them: pole weights and slices (A image), MMAs, and the drain of TMEM, which
// leaves the dofs of A and B in shared memory as they are; the inversion warps form S = A + iB and I + R from them and add
// H_PP.  The hand-over is by named barriers: FULL (the tiles of k are there), EMPTY (every inversion warp has its columns
// in registers).
// On the d + p model (n = 28, D = 10, 1,000 k x 2,048 frequencies; 512 k for the search for mu) G_loc took 66.8 ms end to
// end by k_schur, 30.2 with the complex entries formed and H_PP added in the drain and the shared levels of G_loc in a
// fifth sum passed through shared memory, and 25.7 without; the search 119.8 (derivatives by k_schur), 69.6, and 60.8.  They
// take 20.8 and 56.7 now, by the eigensolver, the k chunks and the carve-out.
// The producers were the longer chain then (38,000 cycles per k of which 19,000 the drain, 7,000 the MMAs issued by a
// rolled loop); now it is the inversions: 36,000 cycles per k and CTA, of which the FP32 pipe is busy 24,000.  Without the
// producers' work the pass takes as long; searching the next pivot and forming its reciprocal beside the update, or
// hand-overs by mbarriers (no rendezvous of the inversion warps), gain nothing for G_loc and lose 5 - 8 % for N(mu).
#include <algorithm>

#include <cuda_bf16.h>

#include "df.cuh"
#include "internal.h"
#include "lat_tc.h"
#include "linalg.cuh"
#include "tc.cuh"

namespace {

constexpr int FT = 32;        // Matsubara frequencies per CTA
constexpr int ROWS = 128;     // MMA M: row = 4 * frequency + channel, so that a TMEM lane quarter holds whole frequencies
constexpr int KP = 32;        // poles per k, padded: the GEMM's K
constexpr int KSTEPS = KP / 16;
constexpr int NSB = 6;        // prepared slices of the dof side (the N(mu) passes read five)
constexpr int BLK = 64;       // rows of a two-channel image block, and of the zeros between blocks
constexpr int NE0 = 64;       // static-spectrum entries staged per k (n <= 64)
constexpr int PT = 128;       // producer threads
constexpr uint32_t WAIT_LIMIT = 1u << 22;
enum { TC_TRACE = 0, TC_DERIV = 1, TC_BLOCK = 2 };
// named barriers (0 is __syncthreads')
enum { BAR_FULL = 1, BAR_EMPTY = 2, BAR_FULLT = 3, BAR_DONE = 4, BAR_PROD = 5 };

__host__ __device__ constexpr int np_of(int DP) { return ((DP * DP + 15) / 16) * 16; }
__host__ __device__ constexpr int pow2_at_least(int x) { return x <= 32 ? 32 : (x <= 64 ? 64 : (x <= 128 ? 128 : (x <= 256 ? 256 : 512))); }

// element offset in an operand image of R rows x KP: [slice][k step][row group][k group][8 rows][8 elements]
// (the canonical no-swizzle K-major layout of tc.cuh: LBO 128 B, SBO 256 B)
__host__ __device__ __forceinline__ int img_off(int R, int s, int kk, int r) {
    const int q = kk >> 4, k16 = kk & 15;
    return s * KSTEPS * R * 16 + q * R * 16 + (r >> 3) * 128 + (k16 >> 3) * 64 + (r & 7) * 8 + (k16 & 7);
}
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

template <int DP, int MODE>
struct TT {
    static constexpr bool TWO = MODE == TC_BLOCK;        // two channels (rows 2 f, 2 f + 1), else four (4 f ..)
    static constexpr bool G0I = TWO && DP < 8;           // GwHF by a second inversion (else k_g0_tc)
    static constexpr int NS = MODE == TC_TRACE && DP > 4 ? 5 : 6;  // slices
    static constexpr int NP = np_of(DP);                 // MMA N: dofs padded to a multiple of 16
    static constexpr int DD = DP * DP;
    static constexpr int GPW = 32 / DP;                  // frequency groups per inversion warp
    static constexpr int NGW = (FT + GPW - 1) / GPW;     // inversion warps
    static constexpr int NT = PT + NGW * 32;
    static constexpr int A_EL = (NS * KSTEPS * ROWS + (TWO ? BLK : 0)) * 16;
    static constexpr int B_EL = NSB * KSTEPS * NP * 16;  // stored per k
    static constexpr int B_USED = NS * KSTEPS * NP * 16; // copied to shared memory
    static constexpr int NACC = NS - 1;                    // TMEM accumulators, the last of the shared levels
    static constexpr int LO = NP / 32 * 16;                // TWO: columns in lanes 0 .. 63
    static constexpr int NA = TWO ? NP - LO : (NACC * NP > 512 ? 64 : NP);  // columns of an accumulator
    static constexpr bool PARTS = !TWO && NA < NP;         // the columns in two parts, one after the other
    static constexpr int TMEM = pow2_at_least(NACC * NA);
    // shared memory layout (bytes)
    static constexpr int O_A = 0;
    static constexpr int O_B = O_A + A_EL * 2;
    // drained sums: [FT][TILE] pdf, per frequency the D^2 dofs of A, then (RS on, an odd row: no bank conflicts) of B
    static constexpr int RS = DD / 2 + 1 - (DD / 2) % 2, TILE = 2 * RS > DD ? 2 * RS : DD;
    static constexpr int O_S = O_B + B_USED * 2;                 // S (DERIV: then T)
    static constexpr int O_R = O_S + FT * TILE * 16;             // R, not TWO (DERIV: then G and X as [r][c])
    static constexpr int O_H = O_R + (TWO ? 0 : FT * TILE * 16); // [3][r][c] pdf: H_PP (slot k mod 3)
    static constexpr int O_COL = O_H + 3 * DD * 16;                  // NP floats: dof column scales of k
    static constexpr int O_ROW = O_COL + NP * 4;                 // ROWS floats: row scales
    static constexpr int O_E0 = O_ROW + ROWS * 4;                // [3][NE0] dfl: mu - e0_j (slot k mod 3)
    static constexpr int O_SW = O_E0 + 3 * NE0 * 8;              // [3][FT] two dfl: Re sum_l w_l, Re sum_l w_l^2
    static constexpr int O_EQ = O_SW + 3 * FT * 16;              // KP dfl: mu - e_l
    static constexpr int O_BAR = (O_EQ + KP * 8 + 15) / 16 * 16;  // 2 mbarriers, TMEM slot, error flag
    static constexpr int SMEM = O_BAR + 32;
    static_assert(NACC * NA <= 512 && NP <= 2 * NA, "accumulators exceed TMEM");
    static_assert(NP <= 256 && NP % 16 == 0, "MMA N");
    static_assert(SMEM <= 227 * 1024, "shared memory");
    static_assert(O_B % 128 == 0 && O_COL % 16 == 0 && O_E0 % 16 == 0 && O_SW % 16 == 0, "alignment");
};

// pair (a < c) number idx = c (c - 1) / 2 + a
__host__ __device__ __forceinline__ void pair_of(int idx, int &a, int &c) {
    c = 1;
    while (idx >= c) idx -= c++;
    a = idx;
}

// x = h + l in [-1, 1] -> NS weighted slices, both halves of a pair at once: slice s is x rounded to a multiple of
// 2^{-(8 + 9 s)} (adding and subtracting 1.5 2^{23 - (8 + 9 s)} rounds to it), then removed.  Slices 1 and 2 are chosen
// from h + l but taken from h, which stays exact; what is left after them is small enough for h + l to be exact too.
struct Slicer {
    float2 h, l;
    __device__ __forceinline__ float2 next(int s) {
        if (s == 3) h = p2_add(h, l);
        const float2 t = s == 1 || s == 2 ? p2_add(h, l) : h;
        const float2 m = p2(__int_as_float(((127 + 23 - (8 + 9 * s)) << 23) | 0x400000));
        const float2 r = p2_sub(p2_add(t, m), m);
        h = p2_sub(h, r);
        return r;
    }
};
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}
// the power of two that takes |x| <= mx to [0, 1]; at least 2^-125, for its reciprocal is taken (rows of w^3 at energies of 1e12)
__device__ __forceinline__ float scale_of(float mx) {
    int ex = 0;
    frexpf(mx, &ex);
    return mx > 0.f ? ldexpf(1.f, max(ex, -125)) : 1.f;
}

// per k: the B operand image (dofs of the poles b_l b_l^H, sliced per dof column) and the column scales (unit: 1 for every
// column, for sums over several k).  Built once per prepared lattice and reused by every pass over it.  One thread per
// (k, dof); FP64 products, sliced as double-float
template <int DP>
__global__ void k_tc_prep(int nk, int m, int D, int unit, const double2 *__restrict__ B, __nv_bfloat16 *__restrict__ img,
                          float *__restrict__ colscale) {
    using T = TT<DP, TC_TRACE>;
    const long long total = (long long)nk * T::NP;
    const int npair = D * (D - 1) / 2;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t / T::NP), p = (int)(t % T::NP);
        int a = 0, c = 0;
        const bool pair = p < 2 * npair, live = p < D * D;
        if (pair) pair_of(p >> 1, a, c);
        else if (live) a = c = p - 2 * npair;
        const double2 *b = B + (size_t)k * m * D;
        double v[KP], mx = 0.0;
#pragma unroll
        for (int l = 0; l < KP; l++) {
            v[l] = 0.0;
            if (l < m && live) {
                const double2 x = b[(size_t)l * D + a], y = b[(size_t)l * D + c];
                v[l] = (pair && (p & 1)) ? fma(x.y, y.x, -x.x * y.y) : fma(x.x, y.x, x.y * y.y);
            }
            mx = fmax(mx, fabs(v[l]));
        }
        int ex = 0;
        frexp(mx, &ex);
        const double g = (mx > 0.0 && !unit) ? ldexp(1.0, ex) : 1.0, ig = 1.0 / g;
        colscale[t] = (float)g;
        __nv_bfloat16 *base = img + (size_t)k * T::B_EL + img_off(T::NP, 0, 0, p);
#pragma unroll
        for (int l8 = 0; l8 < KP; l8 += 8) {
            Slicer sl[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const dfl x = df_make(v[l8 + 2 * i] * ig), y = df_make(v[l8 + 2 * i + 1] * ig);
                sl[i] = {p2(x.h, y.h), p2(x.l, y.l)};
            }
#pragma unroll
            for (int s = 0; s < NSB; s++) {
                uint4 o;
                uint32_t *w = reinterpret_cast<uint32_t *>(&o);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float2 r = sl[i].next(s);
                    w[i] = bf16x2(r.x, r.y);
                }
                *reinterpret_cast<uint4 *>(base + s * KSTEPS * T::NP * 16 + img_off(T::NP, 0, l8, 0)) = o;
            }
        }
    }
}

// z - Sigma(iw_f) as double-float, [f][r][c], padded with the identity to DP x DP; stride 0 in f for a static Sigma
template <int DP>
__global__ void k_tc_zsig(int nf2, int D, int wgrid, double beta, double mu, const double2 *__restrict__ sig,
                          int stride, pdf *zs) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nf2 * DP * DP) return;
    const int f = (int)(t / (DP * DP)), e = (int)(t % (DP * DP)), r = e / DP, c = e % DP;
    if (r >= D || c >= D) {
        zs[t] = r == c ? OpsP::one() : OpsP::zero();
        return;
    }
    const double w = wgrid ? (DG_PI / beta + f * ((2 * DG_PI) / beta)) : (DG_PI * (2. * f + 1.) / beta);
    const pdf s = OpsP::from(sig[(size_t)f * stride + r + (size_t)c * D]);
    zs[t] = r == c ? OpsP::sub(OpsP::from(cmk(mu, w)), s) : OpsP::neg(s);
}

struct TcKArgs {
    LatTcArgs a;
    const __nv_bfloat16 *Bimg;  // [nk][B_EL]
    const float *colscale;      // [nk][NP]
    const pdf *zs, *zs0;        // [nf2][DP][DP] z - Sigma, z - m0 (G0I)
    int kchunk;
    double2 *ptr;               // TRACE: [nchunk][nf2] sums of Re[Tr G - Tr G0] and of its derivative
    double2 *pblk, *pblk0;      // BLOCK: [nchunk][nf2][D][D] sums of G_PP, of G0_PP (G0I)
    int *status;
};

// the real part of sum_r x_r y_r, as the lazy pair (sum Re Re, sum Im Im)
__device__ __forceinline__ pdf re_dot(pdf x, pdf y, pdf acc) { return pdf_fma_lazy(x, y, acc); }
__device__ __forceinline__ dfl re_val(pdf acc) {
    acc = pdf_fast_two_sum(acc.h, acc.l);
    return df_sub({acc.h.x, acc.l.x}, {acc.h.y, acc.l.y});
}

// 16 columns of the first four accumulators (levels 0, 1, 2 and, with five slices, 3 and up) of this thread's TMEM lane, one wait
// for all
__device__ __forceinline__ void tmem_ld16x4(uint32_t addr, uint32_t stride, uint32_t (&v)[4][16]) {
#pragma unroll
    for (int i = 0; i < 4; i++)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
            "%15}, [%16];"
            : "=r"(v[i][0]), "=r"(v[i][1]), "=r"(v[i][2]), "=r"(v[i][3]), "=r"(v[i][4]), "=r"(v[i][5]), "=r"(v[i][6]),
              "=r"(v[i][7]), "=r"(v[i][8]), "=r"(v[i][9]), "=r"(v[i][10]), "=r"(v[i][11]), "=r"(v[i][12]), "=r"(v[i][13]),
              "=r"(v[i][14]), "=r"(v[i][15])
            : "r"(addr + i * stride)
            : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    // the values exist from here on: tie every use to the wait
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 16; j++) asm volatile("" : "+r"(v[i][j]));
}
// columns 2j, 2j+1 of the drained sums; SIX: `top` has the shared levels'.  Level L is an integer multiple of 2^{-(16 + 9 L)}
// and level L + 1 below 2^{-2 - 9 L}, so every partial sum is a multiple of the next level's last place, for which the
// three-operation sum is exact whatever the order of magnitudes
template <bool SIX>
__device__ __forceinline__ pdf drained(const uint32_t (&v)[4][16], int j, const float *top) {
    float2 x[4];
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = p2(__uint_as_float(v[i][2 * j]), __uint_as_float(v[i][2 * j + 1]));
    const pdf s = pdf_fast_two_sum(x[0], x[1]), t = pdf_fast_two_sum(s.h, x[2]);
    if (SIX) {
        const pdf u = pdf_fast_two_sum(t.h, x[3]);
        return pdf_fast_two_sum(u.h, p2_add(p2_add(u.l, p2_add(t.l, s.l)), p2(top[2 * j], top[2 * j + 1])));
    }
    return pdf_fast_two_sum(t.h, p2_add(p2_add(t.l, s.l), x[3]));
}
// 16 columns of one accumulator
__device__ __forceinline__ void tmem_ld16_tied(uint32_t addr, float (&f)[16]) {
    tc::tmem_ld16(addr, f);
#pragma unroll
    for (int j = 0; j < 16; j++) asm volatile("" : "+f"(f[j]));
}
__device__ __forceinline__ pdf shfl_xor1(pdf v) {
    return {p2(__shfl_xor_sync(0xffffffffu, v.h.x, 1), __shfl_xor_sync(0xffffffffu, v.h.y, 1)),
            p2(__shfl_xor_sync(0xffffffffu, v.l.x, 1), __shfl_xor_sync(0xffffffffu, v.l.y, 1))};
}
// from a lane pair's A_ac (even lane) and B_ac (odd lane): the even lane's A + iB = (a, c), the odd lane's
// conj(A) + i conj(B) = (c, a)
__device__ __forceinline__ pdf combine(pdf own, pdf oth, bool odd) {
    const pdf A = odd ? oth : own, B = odd ? own : oth;
    const float s = odd ? -1.f : 1.f;
    return pdf_add({p2(A.h.x, s * A.h.y), p2(A.l.x, s * A.l.y)}, {p2(-s * B.h.y, B.h.x), p2(-s * B.l.y, B.l.x)});
}

// The MMAs of N columns of one K = 32 image pair, slice level i + j in accumulator min(i + j, NACC - 1), accumulators NA
// columns apart (b0: the first column's image row); FRESH: the accumulators start from zero.  Two channels: the
// upper columns, which are no fewer, go first, to lanes 64 .. 127, and their zero rows clear the other lanes; the lower
// columns then add to lanes 0 .. 63.
template <class T, int N, bool FRESH>
__device__ __forceinline__ void issue_mmas(uint32_t tbase, uint32_t a0, uint32_t b0) {
    constexpr uint32_t IDESC = tc::idesc_bf16_f32(ROWS, N), IDLO = tc::idesc_bf16_f32(ROWS, T::TWO ? T::LO : N);
    constexpr int UP = T::TWO ? T::LO * 16 * 2 : 0;
    // unrolled: one thread issues them all while four warps wait, and the descriptors are a base and constants
    const uint64_t ad = tc::smem_desc(a0, 128, 256), bd = tc::smem_desc(b0, 128, 256);
#pragma unroll
    for (int q = 0; q < KSTEPS; q++)
#pragma unroll
        for (int i = 0; i < T::NS; i++)
#pragma unroll
            for (int j = 0; j < T::NS - i; j++) {
                const int L = i + j < T::NACC - 1 ? i + j : T::NACC - 1;
                const uint32_t d = tbase + (uint32_t)(L * T::NA);
                const uint64_t ab = ad + (uint64_t)((i * KSTEPS + q) * ROWS * 16 * 2 / 16),
                               bb = bd + (uint64_t)((j * KSTEPS + q) * T::NP * 16 * 2 / 16);
                tc::mma_bf16(d, ab, bb + UP / 16, IDESC, !(FRESH && q == 0 && i == 0 && j <= T::NACC - 1));
                if (T::TWO) tc::mma_bf16(d, ab + BLK * 16 * 2 / 16, bb, IDLO, 1);
            }
}

// slices of 8 poles of one complex channel pair (image rows row, row + 1) into the A image
template <int NS, bool TWO>
__device__ __forceinline__ void store_slices(__nv_bfloat16 *sA, int row, int l8, const pdf (&v)[8], float isr, float isi) {
    Slicer sl[8];
    const float2 is = p2(isr, isi);
#pragma unroll
    for (int i = 0; i < 8; i++) sl[i] = {p2_mul(v[i].h, is), p2_mul(v[i].l, is)};
    if (TWO) row += BLK;
#pragma unroll
    for (int s = 0; s < NS; s++) {
        uint4 re, im;
        uint32_t *wr = reinterpret_cast<uint32_t *>(&re), *wi = reinterpret_cast<uint32_t *>(&im);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 x = sl[2 * i].next(s), y = sl[2 * i + 1].next(s);
            wr[i] = bf16x2(x.x, y.x);
            wi[i] = bf16x2(x.y, y.y);
        }
        *reinterpret_cast<uint4 *>(sA + img_off(ROWS, s, l8, row)) = re;
        *reinterpret_cast<uint4 *>(sA + img_off(ROWS, s, l8, row + 1)) = im;
    }
}
// max over the four threads of a frequency (adjacent lanes) of |re| and |im| of 8 values each
__device__ __forceinline__ void row_max(const pdf (&v)[8], float &mr, float &mi) {
    mr = mi = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        mr = fmaxf(mr, fabsf(v[i].h.x));
        mi = fmaxf(mi, fabsf(v[i].h.y));
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        mr = fmaxf(mr, __shfl_xor_sync(0xffffffffu, mr, o));
        mi = fmaxf(mi, __shfl_xor_sync(0xffffffffu, mi, o));
    }
}

// CTA = 32 Matsubara frequencies x one chunk of k points
template <int DP, int MODE>
__global__ void __launch_bounds__(TT<DP, MODE>::NT, 1) k_lat_tc(TcKArgs g) {
    using T = TT<DP, MODE>;
    constexpr bool TWO = T::TWO;
    typedef OpsP Ops;
    constexpr int DD = T::DD, NT = T::NT;
    extern __shared__ __align__(1024) unsigned char sm[];
    __nv_bfloat16 *sA = reinterpret_cast<__nv_bfloat16 *>(sm + T::O_A);
    __nv_bfloat16 *sB = reinterpret_cast<__nv_bfloat16 *>(sm + T::O_B);
    pdf *sS = reinterpret_cast<pdf *>(sm + T::O_S), *sR = reinterpret_cast<pdf *>(sm + T::O_R);
    pdf *sH = reinterpret_cast<pdf *>(sm + T::O_H);
    float *sCol = reinterpret_cast<float *>(sm + T::O_COL), *rowsc = reinterpret_cast<float *>(sm + T::O_ROW);
    dfl *sE0 = reinterpret_cast<dfl *>(sm + T::O_E0), *sSw = reinterpret_cast<dfl *>(sm + T::O_SW);
    dfl *sEq = reinterpret_cast<dfl *>(sm + T::O_EQ);
    uint64_t *barB = reinterpret_cast<uint64_t *>(sm + T::O_BAR), *barM = barB + 1;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(barB + 2);
    volatile int *err = reinterpret_cast<volatile int *>(tslot + 1);
    const LatTcArgs &a = g.a;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int D = a.D, m = a.m, n = a.n, npair = D * (D - 1) / 2;
    const int chunk = blockIdx.y, kbeg = chunk * g.kchunk, kend = min(a.nk, kbeg + g.kchunk), f0 = blockIdx.x * FT;
    auto wfreq = [&](int ff) {
        return a.wgrid ? (DG_PI / a.beta + ff * ((2 * DG_PI) / a.beta)) : (DG_PI * (2. * ff + 1.) / a.beta);
    };
    if (warp == 0) {
        tc::tmem_alloc(tslot, T::TMEM);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        tc::mbar_init(barB, 1);
        tc::mbar_init(barM, 1);
        *err = 0;
    }
    for (int t = tid; t < (TWO ? 1 : 2) * FT * T::TILE; t += NT) sS[t] = Ops::zero();  // S and R are adjacent
    if (TWO)  // the zero rows of the A image stay
        for (int t = tid; t < T::A_EL / 8; t += NT) reinterpret_cast<uint4 *>(sA)[t] = make_uint4(0, 0, 0, 0);
    for (int t = tid; t < 3 * DD; t += NT) sH[t] = Ops::zero();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = *tslot;

    if (warp < PT / 32) {
        // ---------------- producers: thread = (frequency, eight poles) for the weights, (TMEM lane) for the drain
        const int fq = tid >> 2, l8 = 8 * (tid & 3), ch = lane & 3;
        const dfl wr = df_make(wfreq(min(f0 + fq, a.nf2 - 1))), w2f = df_mul(wr, wr);
        double2 hpre = cmk(0, 0);
        double epre = 0.0;
        const bool q_thread = tid >= NE0 && tid - NE0 < m, e_thread = MODE != TC_BLOCK && tid < n;
        auto prefetch = [&](int k) {
            if (tid < D * D) hpre = a.H[(size_t)k * n * n + tid % D + (size_t)(tid / D) * n];
            if (e_thread) epre = a.eps0[(size_t)k * n + tid];
            else if (q_thread) epre = a.epsQ[(size_t)k * m + tid - NE0];
        };
        // e0 has up to 64 entries, the poles up to 32: different threads
        auto copy_b = [&](int k) {
            if (tid == 0) {
                tc::mbar_arrive_expect_tx(barB, (uint32_t)(T::B_USED * 2 + T::NP * 4));
                tc::bulk_g2s(sB, g.Bimg + (size_t)k * T::B_EL, (uint32_t)(T::B_USED * 2), barB);
                tc::bulk_g2s(sCol, g.colscale + (size_t)k * T::NP, (uint32_t)(T::NP * 4), barB);
            }
        };
        auto weight = [&](int l) {
            if (l >= m) return Ops::zero();
            const dfl x = sEq[l];
            return Ops::pscale(Ops::mk(x, df_neg(wr)), df_rcp(df_fma(x, x, w2f)));
        };
        int mphase = 0;
        // A image written -> MMAs -> accumulators complete; false when a bounded wait ran out
        int bphase = 0;
        auto multiply = [&](bool first, int part) {
            tc::fence_proxy_async_smem();
            tc::fence_before_sync();
            bar_sync(BAR_PROD, PT);
            if (tid == 0) {
                tc::fence_after_sync();
                if (!first || tc::mbar_wait(barB, bphase, WAIT_LIMIT)) {
                    if (part == 0) issue_mmas<T, T::NA, true>(tbase, tc::smem_u32(sA), tc::smem_u32(sB));
                    if constexpr (T::PARTS) {
                        if (part) issue_mmas<T, T::NP - T::NA, true>(tbase, tc::smem_u32(sA), tc::smem_u32(sB + T::NA * 16));
                    }
                    tc::mma_commit(barM);
                } else {
                    *err = 1;
                }
                if (first) bphase ^= 1;
            }
            __syncwarp();
            if (!tc::mbar_wait(barM, mphase, WAIT_LIMIT)) *err = 1;
            mphase ^= 1;
            bar_sync(BAR_PROD, PT);
            tc::fence_after_sync();
            return *err == 0;
        };
        // TMEM -> shared memory, the dofs of A or B of this lane's frequency and sum as they are: the inversion warps put the
        // complex entries together, for these four warps were the longer chain.  third: the T round of DERIV (rows Re w^3,
        // Im w^3); part: of the columns.  Two channels: warps 0 and 1 have the lower columns, 2 and 3 the upper
        auto drain = [&](bool third, int part) {
            const int f = TWO ? (warp & 1) * 16 + (lane >> 1) : warp * 8 + (lane >> 2);
            const float rs = rowsc[(TWO ? warp & 1 : warp) * 32 + lane];
            const bool second = !TWO && ch >= 2;
            pdf *row = (second ? sR : sS) + (size_t)f * T::TILE + (lane & 1) * T::RS;
            const uint32_t la = tbase + ((uint32_t)(warp * 32) << 16);
            const int first = TWO ? (warp < 2 ? 0 : T::LO) : part * T::NA;  // columns first .. last - 1
            const int last = min(D * D, TWO && warp < 2 ? T::LO : first + T::NA);
#pragma unroll 1
            for (int c0 = first; c0 < last; c0 += 16) {
                uint32_t v[4][16];
                float top[16];
                const uint32_t at = la + (uint32_t)(c0 - first);
                __syncwarp();
                if (T::NACC == 5) tmem_ld16_tied(at + 4 * T::NA, top);
                tmem_ld16x4(at, (uint32_t)T::NA, v);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const pdf own = drained<T::NS == 6>(v, j, top);
                    const float2 sc = p2_mul(*reinterpret_cast<const float2 *>(sCol + c0 + 2 * j), p2(rs));
                    if (c0 + 2 * j < DD && !(third && second)) row[c0 / 2 + j] = {p2_mul(own.h, sc), p2_mul(own.l, sc)};
                }
            }
            tc::fence_before_sync();
        };

        copy_b(kbeg);
        prefetch(kbeg);
        for (int k = kbeg, it = 0; k < kend; k++, it++) {
            const int slot = it % 3;  // inversion warps may still read the slot of k - 1 while k + 1 is staged
            if (tid < D * D) sH[slot * DD + (tid % D) * DP + tid / D] = Ops::from(hpre);
            if (e_thread) sE0[slot * NE0 + tid] = df_make(a.mu - epre);
            else if (q_thread) sEq[tid - NE0] = df_make(a.mu - epre);
            if (k + 1 < kend) prefetch(k + 1);
            bar_sync(BAR_PROD, PT);
            {
                pdf w[8];
                float mr, mi;
#pragma unroll
                for (int i = 0; i < 8; i++) w[i] = weight(l8 + i);
                row_max(w, mr, mi);
                const float s0 = scale_of(mr), s1 = scale_of(mi);
                store_slices<T::NS, TWO>(sA, (TWO ? 2 : 4) * fq, l8, w, 1.f / s0, 1.f / s1);
                float s2 = 1.f, s3 = 1.f;
                if (MODE != TC_BLOCK) {
                    pdf sw = Ops::zero(), sw2 = Ops::zero();
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        sw = Ops::add(sw, w[i]);
                        w[i] = Ops::mul(w[i], w[i]);
                        if (MODE == TC_DERIV) sw2 = Ops::add(sw2, w[i]);
                    }
                    row_max(w, mr, mi);
                    s2 = scale_of(mr);
                    s3 = scale_of(mi);
                    store_slices<T::NS, false>(sA, 4 * fq + 2, l8, w, 1.f / s2, 1.f / s3);
#pragma unroll
                    for (int o = 1; o <= 2; o <<= 1) {
                        sw = Ops::add(sw, Ops::shfl(sw, lane ^ o, 32));
                        if (MODE == TC_DERIV) sw2 = Ops::add(sw2, Ops::shfl(sw2, lane ^ o, 32));
                    }
                    if (ch == 0) {
                        sSw[(slot * FT + fq) * 2] = Ops::cre(sw);
                        if (MODE == TC_DERIV) sSw[(slot * FT + fq) * 2 + 1] = Ops::cre(sw2);
                    }
                }
                if (!TWO) rowsc[tid] = ch == 0 ? s0 : (ch == 1 ? s1 : (ch == 2 ? s2 : s3));
                else if (ch < 2) rowsc[2 * fq + ch] = ch ? s1 : s0;
            }
            bool ok = multiply(true, 0);
            if (ok && it > 0) bar_sync(MODE == TC_DERIV ? BAR_DONE : BAR_EMPTY, NT);
            if (ok) drain(false, 0);
            if (T::PARTS && ok) {
                ok = multiply(false, 1);
                if (ok) drain(false, 1);
            }
            bar_arrive(BAR_FULL, NT);
            if (!ok) break;
            if (MODE == TC_DERIV) {
                bar_sync(BAR_PROD, PT);  // every lane has drained before the row scales change
                pdf w[8];
                float mr, mi;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const pdf x = weight(l8 + i);
                    w[i] = Ops::mul(Ops::mul(x, x), x);
                }
                row_max(w, mr, mi);
                const float s0 = scale_of(mr), s1 = scale_of(mi);
                store_slices<T::NS, false>(sA, 4 * fq, l8, w, 1.f / s0, 1.f / s1);
                rowsc[tid] = ch == 0 ? s0 : (ch == 1 ? s1 : 1.f);
                ok = multiply(false, 0);
                if (ok) {
                    bar_sync(BAR_EMPTY, NT);
                    drain(true, 0);
                }
                if (T::PARTS && ok) {
                    ok = multiply(false, 1);
                    if (ok) drain(true, 1);
                }
                bar_arrive(BAR_FULLT, NT);
                if (!ok) break;
            }
            // the MMAs are done with B and, once all have drained, so are H and the scales
            bar_sync(BAR_PROD, PT);
            if (k + 1 < kend) copy_b(k + 1);
        }
        // the inversion warps' last hand-back
        if (!*err) bar_sync(MODE == TC_DERIV ? BAR_DONE : BAR_EMPTY, NT);
        // a copy that timed out is given the chance to land before the CTA's shared memory goes away
        if (*err && tid == 0) tc::mbar_wait(barB, bphase ^ 1, WAIT_LIMIT);
    } else {
        // ---------------- inversions: lanes base .. base+DP-1 of the warp hold the columns of one frequency's matrix
        const int gw = lane / DP, c = lane % DP, base = gw * DP;
        const int gidx = (warp - PT / 32) * T::GPW + gw;
        const bool grp_lane = gw < T::GPW && gidx < FT;
        const int fl = grp_lane ? gidx : FT - 1, f = f0 + fl;
        const bool fvalid = grp_lane && f < a.nf2;
        const int fc = min(f, a.nf2 - 1);
        const dfl wr = df_make(wfreq(fc)), w2f = df_mul(wr, wr);
        const pdf *zs = g.zs + (size_t)fc * DD + c;
        pdf *tS = sS + (size_t)fl * T::TILE, *tR = sR + (size_t)fl * T::TILE;
        // entry (r, c), or (c, r) with tr, of A + iB from the dofs at t; dg: the diagonal entry of this lane's column.  In the
        // lanes of the padding (c >= D) it is some finite number: their columns only ever change themselves
        auto diagonal = [&](const pdf *t) {
            const int i = npair + (min(c, D - 1) >> 1);
            const pdf A = t[i], B = t[T::RS + i];
            return c & 1 ? pdf{p2(A.h.y, B.h.y), p2(A.l.y, B.l.y)} : pdf{p2(A.h.x, B.h.x), p2(A.l.x, B.l.x)};
        };
        auto entry = [&](const pdf *t, const pdf &dg, int r, bool tr) {
            if (r >= D) return Ops::zero();
            const int i = r < c ? c * (c - 1) / 2 + r : r * (r - 1) / 2 + min(c, r);
            const pdf A = t[i], B = t[T::RS + i];
            const float s = (r < c) != tr ? 1.f : -1.f;
            const pdf x = pdf_add({p2(A.h.x, s * A.h.y), p2(A.l.x, s * A.l.y)}, {p2(-s * B.h.y, B.h.x), p2(-s * B.l.y, B.l.x)});
            return r == c ? dg : x;
        };
        const pdf *zs0 = T::G0I ? g.zs0 + (size_t)fc * DD + c : nullptr;
        pdf accG[MODE == TC_BLOCK ? DP : 1], accG0[T::G0I ? DP : 1];
#pragma unroll
        for (int r = 0; r < (MODE == TC_BLOCK ? DP : 1); r++) accG[r] = Ops::zero();
#pragma unroll
        for (int r = 0; r < (T::G0I ? DP : 1); r++) accG0[r] = Ops::zero();
        double acc = 0.0, acc2 = 0.0;
        bool sing = false, ok = true;
        for (int k = kbeg, it = 0; k < kend; k++, it++) {
            pdf col[DP], R[MODE == TC_BLOCK ? 1 : DP], col0[T::G0I ? DP : 1];
            const pdf *hk = sH + (it % 3) * DD + c;
#pragma unroll
            for (int r = 0; r < DP; r++) col[r] = zs[r * DP];
            bar_sync(BAR_FULL, NT);
            if (*err) {
                ok = false;
                break;
            }
            {
                const pdf dg = diagonal(tS);
#pragma unroll
                for (int r = 0; r < DP; r++) {
                    const pdf x = entry(tS, dg, r, false);
                    if (T::G0I) col0[T::G0I ? r : 0] = Ops::sub(zs0[r * DP], x);
                    col[r] = Ops::sub(col[r], x);
                }
            }
            if (MODE != TC_BLOCK) {  // I + R, TRACE: transposed
                const pdf dg = Ops::add(Ops::one(), diagonal(tR));
#pragma unroll
                for (int r = 0; r < DP; r++) R[MODE == TC_BLOCK ? 0 : r] = entry(tR, dg, r, MODE == TC_TRACE);
            }
            bar_arrive(BAR_EMPTY, NT);
#pragma unroll
            for (int r = 0; r < DP; r++) {  // H_PP, in its own slot: the tiles are free before this
                const pdf h = hk[r * DP];
                col[r] = Ops::sub(col[r], h);
                if (T::G0I) col0[T::G0I ? r : 0] = Ops::sub(col0[T::G0I ? r : 0], h);
            }
            sing |= group_gj_inverse<Ops, DP>(col, c, base) && fvalid && c < D;
            if (MODE == TC_BLOCK) {
#pragma unroll
                for (int r = 0; r < DP; r++) accG[MODE == TC_BLOCK ? r : 0] = Ops::add(accG[MODE == TC_BLOCK ? r : 0], col[r]);
                if constexpr (T::G0I) {
                    sing |= group_gj_inverse<Ops, DP>(col0, c, base) && fvalid && c < D;
#pragma unroll
                    for (int r = 0; r < DP; r++) accG0[r] = Ops::add(accG0[r], col0[r]);
                }
                continue;
            }
            const int slot = it % 3;
            const dfl *sw = sSw + (slot * FT + fl) * 2;
            dfl t = {0.f, 0.f}, t2 = {0.f, 0.f};
            if (MODE == TC_TRACE) {
                pdf d = Ops::zero();
                if (c < D) {
#pragma unroll
                    for (int r = 0; r < DP; r++)
                        if (r < D) d = re_dot(col[r], R[MODE == TC_BLOCK ? 0 : r], d);  // G(r, c) (I + R)(c, r)
                }
                t = re_val(d);
            } else {
                // X = G (I + R), row by row: lane s puts G(r, s) into the tile, every lane forms X(r, c) from row r (its
                // column of I + R in registers) and puts it where row r of G was
                __syncwarp();
                if (grp_lane) {
#pragma unroll
                    for (int r = 0; r < DP; r++) tR[r * DP + c] = col[r];
                }
                __syncwarp();
#pragma unroll 1
                for (int r = 0; r < D; r++) {
                    pdf x1 = Ops::zero(), x2 = Ops::zero();
#pragma unroll
                    for (int s = 0; s < DP; s++) {
                        const pdf gv = tR[r * DP + s], rv = R[MODE == TC_BLOCK ? 0 : s];
                        x1 = Ops::pacc(rv, Ops::cre(gv), x1);
                        x2 = Ops::pacc(rv, Ops::cim(gv), x2);
                    }
                    const pdf x = Ops::add(Ops::pnorm(x1), Ops::times_i(Ops::pnorm(x2)));
                    __syncwarp();
                    if (grp_lane) tR[r * DP + c] = x;
                    __syncwarp();
                }
                pdf d = Ops::zero();
                if (c < D) {
                    t = Ops::cre(tR[c * DP + c]);
                    for (int r = 0; r < D; r++) d = re_dot(tR[r * DP + c], tR[c * DP + r], d);
                }
                t2 = df_neg(re_val(d));
                bar_sync(BAR_FULLT, NT);
                if (*err) {
                    ok = false;
                    break;
                }
                d = Ops::zero();
                if (c < D) {
                    const pdf dg = diagonal(tS);
#pragma unroll
                    for (int r = 0; r < DP; r++)
                        if (r < D) d = re_dot(col[r], entry(tS, dg, r, true), d);  // G(r, c) T(c, r)
                }
                const dfl gt = re_val(d);
                t2 = df_sub(t2, df_add(gt, gt));
                if (c == 0) t2 = df_sub(t2, sw[1]);
            }
            for (int j = c; j < n; j += DP) {
                const dfl x = sE0[slot * NE0 + j], r = df_rcp(df_fma(x, x, w2f));
                t = df_sub(t, df_mul(x, r));
                if (MODE == TC_DERIV) {  // Re 1/(x + iw)^2 = (x^2 - w^2) r^2
                    const dfl xr = df_mul(x, r), yr = df_mul(wr, r);
                    t2 = df_add(t2, df_sub(df_mul(xr, xr), df_mul(yr, yr)));
                }
            }
            if (c == 0) t = df_add(t, sw[0]);
            if (fvalid) {
                acc += df_val(t);
                if (MODE == TC_DERIV) acc2 += df_val(t2);
            }
            if (MODE == TC_DERIV) bar_arrive(BAR_DONE, NT);
        }
        if (sing) dg_flag(g.status, DG_SINGULAR);
        if (MODE == TC_BLOCK) {
            if (ok && fvalid && c < D) {
                const size_t o = ((size_t)chunk * a.nf2 + f) * D * D + (size_t)c * D;
#pragma unroll
                for (int r = 0; r < DP; r++)
                    if (r < D) {
                        g.pblk[o + r] = Ops::to(accG[MODE == TC_BLOCK ? r : 0]);
                        if (T::G0I) g.pblk0[o + r] = Ops::to(accG0[T::G0I ? r : 0]);
                    }
            }
        } else {
            // group sum over the DP lanes of each frequency (full-warp shuffles from absolute lanes)
            double s = 0.0, s2 = 0.0;
#pragma unroll
            for (int j = 0; j < DP; j++) {
                s += __shfl_sync(0xffffffffu, acc, (base + j) & 31, 32);
                if (MODE == TC_DERIV) s2 += __shfl_sync(0xffffffffu, acc2, (base + j) & 31, 32);
            }
            if (ok && fvalid && c == 0) g.ptr[(size_t)chunk * a.nf2 + f] = cmk(s, s2);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0 && *err) atomicMax(g.status, (int)DMFTGPU_TIMEOUT);
    if (warp == 0) tc::tmem_dealloc(tbase, T::TMEM);
}

// ---------------------------------------------------------------------------------------------------------------------
// GwHF's k sum: sum_k sum_j U_j U_j^H / (z_f - e0_j), U_j the correlated rows of the eigenvectors of H + m0.  One GEMM over
// all (k, j): CTA = 32 frequencies (rows 2 f, 2 f + 1 = Re, Im of 1/(z - e0)) x one chunk of k.  Two k points share row
// scales and accumulate in TMEM (K = 64, exact levels) before a drain into double-float registers; each half of the
// threads builds the image of one of them.  ~6,000 FP32 lane operations per (k, iw) at D = 10 in place of 28 x 100
// complex multiply-adds (280,000).
// ---------------------------------------------------------------------------------------------------------------------
constexpr int G0T = 256, G0K = 2;
template <int DP>
struct T0 {
    using T = TT<DP, TC_BLOCK>;
    static constexpr int NGH = (T::NA / 16 + 1) / 2;           // column groups per warp: two warps share a TMEM quarter
    static constexpr int O_A = 0;
    static constexpr int O_B = O_A + G0K * T::A_EL * 2;
    static constexpr int O_E = O_B + G0K * T::B_EL * 2;        // [2][G0K][KP] dfl: mu - e0_j
    static constexpr int O_ROW = O_E + 2 * G0K * KP * 8;
    static constexpr int O_BAR = O_ROW + BLK * 4;              // barB[G0K], barM, TMEM slot, error flag
    static constexpr int SMEM = O_BAR + 48;
    static_assert(SMEM <= 227 * 1024, "shared memory");
    static_assert(O_B % 128 == 0 && O_E % 16 == 0 && O_BAR % 16 == 0, "alignment");
};
struct G0Args {
    const double *eps0;         // [nk][n]
    const __nv_bfloat16 *Uimg;  // [nk][B_EL], unit column scales
    int n, nk, nf2, D, wgrid, kchunk;
    double beta, mu;
    double2 *pblk0;             // [nchunk][nf2][D][D]
    int *status;
};
template <int DP>
__global__ void __launch_bounds__(G0T, 1) k_g0_tc(G0Args g) {
    using T = TT<DP, TC_BLOCK>;
    using S = T0<DP>;
    typedef OpsP Ops;
    extern __shared__ __align__(1024) unsigned char sm[];
    __nv_bfloat16 *sA = reinterpret_cast<__nv_bfloat16 *>(sm + S::O_A), *sB = reinterpret_cast<__nv_bfloat16 *>(sm + S::O_B);
    dfl *sE = reinterpret_cast<dfl *>(sm + S::O_E);
    float *rowsc = reinterpret_cast<float *>(sm + S::O_ROW);
    uint64_t *barB = reinterpret_cast<uint64_t *>(sm + S::O_BAR), *barM = barB + G0K;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(barM + 1);
    volatile int *err = reinterpret_cast<volatile int *>(tslot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, n = g.n, D = g.D;
    const int chunk = blockIdx.y, kbeg = chunk * g.kchunk, kend = min(g.nk, kbeg + g.kchunk), nk = kend - kbeg;
    const int f0 = blockIdx.x * FT;
    if (warp == 0) {
        tc::tmem_alloc(tslot, T::TMEM);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < G0K; i++) tc::mbar_init(barB + i, 1);
        tc::mbar_init(barM, 1);
        *err = 0;
    }
    for (int t = tid; t < G0K * T::A_EL / 8; t += G0T) reinterpret_cast<uint4 *>(sA)[t] = make_uint4(0, 0, 0, 0);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = *tslot;
    const int mine = tid >> 7, fq = (tid & 127) >> 2, l8 = 8 * (tid & 3), fw = min(f0 + fq, g.nf2 - 1);
    const double wd = g.wgrid ? (DG_PI / g.beta + fw * ((2 * DG_PI) / g.beta)) : (DG_PI * (2. * fw + 1.) / g.beta);
    const dfl wr = df_make(wd), w2f = df_mul(wr, wr);
    auto copy_b = [&](int i0) {  // the images of the group from i0, each on its own barrier
        if (tid == 0)
            for (int kk = 0; kk < G0K && i0 + kk < nk; kk++) {
                tc::mbar_arrive_expect_tx(barB + kk, (uint32_t)(T::B_EL * 2));
                tc::bulk_g2s(sB + (size_t)kk * T::B_EL, g.Uimg + (size_t)(kbeg + i0 + kk) * T::B_EL, (uint32_t)(T::B_EL * 2),
                             barB + kk);
            }
    };
    copy_b(0);
    pdf acc[S::NGH][8];
#pragma unroll
    for (int q = 0; q < S::NGH; q++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[q][j] = Ops::zero();
    const int quarter = warp & 3, half = warp >> 2;
    const int first = quarter < 2 ? 0 : T::LO, last = min(D * D, quarter < 2 ? T::LO : T::NP);  // this quarter's columns
    const uint32_t la = tbase + ((uint32_t)(quarter * 32) << 16);
    const int row = (quarter & 1) * 32 + lane;
    bool ok = true;
    for (int i0 = 0, gi = 0; i0 < nk; i0 += G0K, gi ^= 1) {
        const int cnt = min(G0K, nk - i0);
        dfl *e = sE + gi * G0K * KP;
        for (int t = tid; t < cnt * n; t += G0T)
            e[(t / n) * KP + t % n] = df_make(g.mu - g.eps0[(size_t)(kbeg + i0) * n + t]);
        __syncthreads();
        // row scales of the group: bounds on |Re 1/(x + iw)| and |Im| from FP32
        float mr = 0.f, mi = 0.f;
        for (int kk = 0; kk < cnt; kk++)
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (l8 + i < n) {
                    const float x = e[kk * KP + l8 + i].h, r = __fdividef(1.f, fmaf(x, x, w2f.h));
                    mr = fmaxf(mr, fabsf(x) * r);
                    mi = fmaxf(mi, wr.h * r);
                }
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            mr = fmaxf(mr, __shfl_xor_sync(0xffffffffu, mr, o));
            mi = fmaxf(mi, __shfl_xor_sync(0xffffffffu, mi, o));
        }
        const float s0 = scale_of(mr * 1.0001f), s1 = scale_of(mi * 1.0001f);
        if (mine == 0 && (tid & 3) < 2) rowsc[2 * fq + (tid & 3)] = (tid & 3) ? s1 : s0;
        if (mine < cnt) {
            pdf w[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                w[j] = Ops::zero();
                if (l8 + j < n) {
                    const dfl x = e[mine * KP + l8 + j];
                    w[j] = Ops::pscale(Ops::mk(x, df_neg(wr)), df_rcp(df_fma(x, x, w2f)));
                }
            }
            store_slices<T::NS, true>(sA + (size_t)mine * T::A_EL, 2 * fq, l8, w, 1.f / s0, 1.f / s1);
        }
        tc::fence_proxy_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            bool there = true;
            for (int kk = 0; kk < cnt && there; kk++) {
                there = tc::mbar_wait(barB + kk, gi, WAIT_LIMIT);
                const uint32_t a0 = tc::smem_u32(sA + (size_t)kk * T::A_EL), b0 = tc::smem_u32(sB + (size_t)kk * T::B_EL);
                if (there && kk == 0) issue_mmas<T, T::NA, true>(tbase, a0, b0);
                else if (there) issue_mmas<T, T::NA, false>(tbase, a0, b0);
            }
            tc::mma_commit(barM);
            if (!there) *err = 1;
        }
        __syncwarp();
        if (!tc::mbar_wait(barM, gi, WAIT_LIMIT)) *err = 1;
        __syncthreads();
        ok = *err == 0;
        if (!ok) break;
        tc::fence_after_sync();
        if (i0 + G0K < nk) copy_b(i0 + G0K);  // the MMAs are done with B
        const float rs = rowsc[row];
#pragma unroll
        for (int q = 0; q < S::NGH; q++) {
            const int c0 = first + (2 * q + half) * 16;
            if (c0 >= last) break;
            uint32_t v[4][16];
            float top[16];
            __syncwarp();
            tmem_ld16_tied(la + (uint32_t)(c0 - first + 4 * T::NA), top);
            tmem_ld16x4(la + (uint32_t)(c0 - first), (uint32_t)T::NA, v);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const pdf x = drained<true>(v, j, top);
                acc[q][j] = Ops::add(acc[q][j], {p2_mul(x.h, p2(rs)), p2_mul(x.l, p2(rs))});
            }
        }
        tc::fence_before_sync();
        __syncthreads();  // the next group's MMAs overwrite the accumulators, its builds the images and scales
        tc::fence_after_sync();
    }
    {
        // A and B of this lane pair's frequency -> the complex entries
        const int npair = D * (D - 1) / 2, f = f0 + (row >> 1);
        const bool odd = lane & 1, put = ok && f < g.nf2;
        double2 *o = g.pblk0 + ((size_t)chunk * g.nf2 + min(f, g.nf2 - 1)) * D * D;
#pragma unroll
        for (int q = 0; q < S::NGH; q++) {
            const int c0 = first + (2 * q + half) * 16;
            if (c0 >= last) break;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int p = c0 + 2 * j;
                if (p >= last) break;
                const pdf own = acc[q][j], oth = shfl_xor1(own);
                if (p < 2 * npair) {
                    int a, c;
                    pair_of(p >> 1, a, c);
                    const pdf x = combine(own, oth, odd);
                    if (put) o[odd ? c + a * D : a + c * D] = Ops::to(x);
                } else {
                    const int di = p - 2 * npair + (odd ? 1 : 0);
                    const pdf x = odd ? pdf{p2(oth.h.y, own.h.y), p2(oth.l.y, own.l.y)}
                                      : pdf{p2(own.h.x, oth.h.x), p2(own.l.x, oth.l.x)};
                    if (put && di < D) o[di + di * D] = Ops::to(x);
                }
            }
        }
    }
    if (!ok && tid == 64) {
        // copies still in flight land before the CTA's shared memory goes away
        for (int kk = 0; kk < G0K; kk++)
            for (int ph = 0; ph < 2; ph++) tc::mbar_wait(barB + kk, ph, WAIT_LIMIT);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0 && *err) atomicMax(g.status, (int)DMFTGPU_TIMEOUT);
    if (warp == 0) tc::tmem_dealloc(tbase, T::TMEM);
}

// fixed-order sums over the k chunks
__global__ void k_tc_reduce_trace(int nchunk, int nf2, const double2 *__restrict__ ptr, double *__restrict__ tr,
                                  double *__restrict__ dtr) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf2) return;
    const double2 s = chunk_sum(nchunk, [&](int q) { return ptr[(size_t)q * nf2 + f]; });
    tr[f] = s.x;
    if (dtr) dtr[f] = s.y;
}
__global__ void k_tc_reduce_block(int n1, int n0, long long len, const double2 *__restrict__ p1,
                                  const double2 *__restrict__ p0, double2 *__restrict__ blk, double2 *__restrict__ blk0) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= len) return;
    const double2 *p = blockIdx.y ? p0 : p1;
    (blockIdx.y ? blk0 : blk)[t] = chunk_sum(blockIdx.y ? n0 : n1, [&](int q) { return p[(size_t)q * len + t]; });
}

int sm_count(dmftgpu_ctx *ctx) {
    int nsm = 152;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device);
    return nsm;
}
// k points per CTA, one CTA per SM: the fewest rounds of CTAs x (their k points and some 0.6 for filling the pipeline), at
// most 16 rounds, and chunks of at least 8; returns the chunks.  (A fixed eight or four rounds left the last one 40 % full at
// 128 tiles and 1,000 k: G_loc 22.5 -> 21.2 ms.)
int chunks_of(int nk, int fblocks, int nsm, int *kchunk) {
    double best = 1e300;
    *kchunk = nk;
    for (int r = 1; r <= 16; r++) {
        const int nc = std::max(1, std::min(dg_ceil_div(nk, 8), (int)((long long)r * nsm / fblocks))), kch = dg_ceil_div(nk, nc);
        const double cost = dg_ceil_div((long long)fblocks * dg_ceil_div(nk, kch), nsm) * (kch + 0.6);
        if (cost < best) {
            best = cost;
            *kchunk = kch;
        }
    }
    return dg_ceil_div(nk, *kchunk);
}

// k images of the poles, z - Sigma, and one pass of the mode
template <int DP, int MODE>
int launch_lat(dmftgpu_ctx *ctx, const LatTcArgs &a, bool *ready, double *tr, double *dtr, double2 *pblk, double2 *pblk0,
               int *nchunk_out) {
    using T = TT<DP, MODE>;
    const int nsm = sm_count(ctx), fblocks = dg_ceil_div(a.nf2, FT);
    TcKArgs g;
    const int nchunk = chunks_of(a.nk, fblocks, nsm, &g.kchunk);
    *nchunk_out = nchunk;
    if (!pblk && MODE == TC_BLOCK) return DMFTGPU_OK;  // the caller asks for the number of chunks first
    __nv_bfloat16 *Bimg = (__nv_bfloat16 *)dg_buf(ctx, "tc.B", (size_t)a.nk * T::B_EL * 2);
    float *col = (float *)dg_buf(ctx, "tc.col", (size_t)a.nk * T::NP * 4);
    pdf *zs = (pdf *)dg_buf(ctx, "tc.zs", (size_t)a.nf2 * T::DD * sizeof(pdf));
    double2 *ptr = MODE == TC_BLOCK ? nullptr : (double2 *)dg_buf(ctx, "tc.ptr", (size_t)nchunk * a.nf2 * sizeof(double2));
    pdf *zs0 = T::G0I ? (pdf *)dg_buf(ctx, "tc.zs0", (size_t)a.nf2 * T::DD * sizeof(pdf)) : nullptr;
    if (!Bimg || !col || !zs || (MODE != TC_BLOCK && !ptr) || (T::G0I && !zs0)) return DMFTGPU_NOMEM;
    if (!*ready) {
        k_tc_prep<DP><<<nsm * 8, 128, 0, ctx->stream>>>(a.nk, a.m, a.D, 0, a.B, Bimg, col);
        DG_LAUNCH(ctx, "k_tc_prep");
        *ready = true;
    }
    const int zblocks = dg_ceil_div((long long)a.nf2 * T::DD, 256);
    k_tc_zsig<DP><<<zblocks, 256, 0, ctx->stream>>>(a.nf2, a.D, a.wgrid, a.beta, a.mu, a.sig, a.D * a.D, zs);
    DG_LAUNCH(ctx, "k_tc_zsig");
    if (T::G0I) {
        k_tc_zsig<DP><<<zblocks, 256, 0, ctx->stream>>>(a.nf2, a.D, a.wgrid, a.beta, a.mu, a.m0, 0, zs0);
        DG_LAUNCH(ctx, "k_tc_zsig");
    }
    DG_CUDA((dg_smem_attr(k_lat_tc<DP, MODE>, T::SMEM, true)));
    g.a = a;
    g.Bimg = Bimg;
    g.colscale = col;
    g.zs = zs;
    g.zs0 = zs0;
    g.ptr = ptr;
    g.pblk = pblk;
    g.pblk0 = pblk0;
    g.status = ctx->d_status;
    {
        DgTimer tm(ctx, "k_lat_tc");
        k_lat_tc<DP, MODE><<<dim3(fblocks, nchunk), T::NT, T::SMEM, ctx->stream>>>(g);
    }
    DG_LAUNCH(ctx, "k_lat_tc");
    if (MODE != TC_BLOCK) {
        k_tc_reduce_trace<<<dg_ceil_div(a.nf2, 256), 256, 0, ctx->stream>>>(nchunk, a.nf2, ptr, tr, dtr);
        DG_LAUNCH(ctx, "k_tc_reduce_trace");
    }
    return DMFTGPU_OK;
}

template <int DP>
int launch_block(dmftgpu_ctx *ctx, const LatTcArgs &a, double2 *blk, double2 *blk0) {
    using T = TT<DP, TC_BLOCK>;
    const int nsm = sm_count(ctx), fblocks0 = dg_ceil_div(a.nf2, FT);
    const long long len = (long long)a.nf2 * a.D * a.D;
    bool ready = false;
    int n1 = 0, n0 = 0;
    DG_TRY((launch_lat<DP, TC_BLOCK>(ctx, a, &ready, nullptr, nullptr, nullptr, nullptr, &n1)));
    G0Args g;
    if (T::G0I) n0 = n1;
    else n0 = chunks_of(a.nk, fblocks0, nsm, &g.kchunk);
    double2 *p1 = (double2 *)dg_buf(ctx, "tc.pblk", (size_t)n1 * len * sizeof(double2));
    double2 *p0 = (double2 *)dg_buf(ctx, "tc.pblk0", (size_t)n0 * len * sizeof(double2));
    if (!p1 || !p0) return DMFTGPU_NOMEM;
    DG_TRY((launch_lat<DP, TC_BLOCK>(ctx, a, &ready, nullptr, nullptr, p1, p0, &n1)));
    const int rblocks = dg_ceil_div(len, 256);
    if constexpr (!T::G0I) {
        __nv_bfloat16 *Uimg = (__nv_bfloat16 *)dg_buf(ctx, "tc.U", (size_t)a.nk * T::B_EL * 2);
        float *col = (float *)dg_buf(ctx, "tc.ucol", (size_t)a.nk * T::NP * 4);
        if (!Uimg || !col) return DMFTGPU_NOMEM;
        DG_CUDA(cudaStreamWaitEvent(ctx->stream, a.static_ready, 0));
        k_tc_prep<DP><<<nsm * 8, 128, 0, ctx->stream>>>(a.nk, a.n, a.D, 1, a.UP, Uimg, col);
        DG_LAUNCH(ctx, "k_tc_prep");
        g.eps0 = a.eps0;
        g.Uimg = Uimg;
        g.n = a.n;
        g.nk = a.nk;
        g.nf2 = a.nf2;
        g.D = a.D;
        g.wgrid = a.wgrid;
        g.beta = a.beta;
        g.mu = a.mu;
        g.pblk0 = p0;
        g.status = ctx->d_status;
        using S = T0<DP>;
        DG_CUDA(dg_smem_attr(k_g0_tc<DP>, S::SMEM, true));
        {
            DgTimer tm(ctx, "k_g0_tc");
            k_g0_tc<DP><<<dim3(fblocks0, n0), G0T, S::SMEM, ctx->stream>>>(g);
        }
        DG_LAUNCH(ctx, "k_g0_tc");
    }
    k_tc_reduce_block<<<dim3(rblocks, 2), 256, 0, ctx->stream>>>(n1, n0, len, p1, p0, blk, blk0);
    DG_LAUNCH(ctx, "k_tc_reduce_block");
    return DMFTGPU_OK;
}

template <int DP>
int launch_trace(dmftgpu_ctx *ctx, const LatTcArgs &a, bool *ready, double *tr, double *dtr) {
    int nchunk;
    return dtr ? launch_lat<DP, TC_DERIV>(ctx, a, ready, tr, dtr, nullptr, nullptr, &nchunk)
               : launch_lat<DP, TC_TRACE>(ctx, a, ready, tr, nullptr, nullptr, nullptr, &nchunk);
}

}  // namespace

// Which pass comes here rather than to the lane groups of k_schur: k_schur's time grows with the poles (S, R and T are m
// rank-one updates each), this one's hardly does.  512 k points x 768 frequencies, eigensolver included, ms k_schur / here:
//              m = 0        m = 2        m = 4        m = 6
//   G_loc   D = 6   1.63 / 1.93  1.84 / 1.97  2.05 / 1.99  2.25 / 2.03
//           D = 8   2.38 / 2.66  2.88 / 2.70  3.33 / 2.75  3.81 / 2.81
//           D = 10  4.75 / 4.36  5.71 / 4.47  6.64 / 4.60  7.62 / 4.66
//   N(mu)   D = 6   0.92 / 1.53  1.33 / 1.62  1.74 / 1.68
//           D = 10  2.61 / 3.99  3.48 / 4.07  4.28 / 4.13
//   dN/dmu  D = 6   1.98 / 2.46  2.82 / 2.54
//           D = 10  6.46 / 7.24  10.1 / 7.30
// The lines below are where these cross.  At D = 4 (512 k x 4,096 frequencies)
//              m = 8        m = 12       m = 16       m = 20       m = 28
//   N(mu)                   3.30 / 3.14  4.12 / 3.24  5.11 / 3.40  8.02 / 3.99
//   dN/dmu     4.74 / 4.59  6.52 / 4.76  8.15 / 4.86  9.93 / 5.05  14.0 / 5.64
// G_loc of four orbitals stays with k_schur (without poles 1.34 / 1.84).
static bool covered(int n, int D, int least) { return D <= 10 && n - D >= least && n - D <= KP && n <= NE0; }
bool dg_lat_tc_supported(int n, int D) { return D >= 4 && covered(n, D, D == 4 ? 12 : 4); }
bool dg_lat_tc_deriv_supported(int n, int D) { return D >= 4 && covered(n, D, D == 4 ? 8 : 2); }
bool dg_lat_tc_block_supported(int n, int D) {
    return D >= 5 && covered(n, D, D <= 6 ? 4 : (D <= 8 ? 2 : 0)) && (D <= 6 || n <= KP);
}

// The images, 43 KB per k point at D = 10 and two sets of them in G_loc's pass, are what k_schur does without: they stay
// within 64 GB in a call, and where they cannot be had at all the pass is k_schur's.
bool dg_lat_tc_reserve(dmftgpu_ctx *ctx, int n, int D, int nk, bool block) {
    const size_t np = np_of((D + 1) / 2 * 2), img = (size_t)nk * NSB * KSTEPS * np * 16 * 2, col = (size_t)nk * np * 4;
    const bool two = block && D > 6;  // with the images of U (launch_block)
    const size_t need = img * (two ? 2 : 1);
    if (need > ctx->image_left) return false;
    const struct {
        const char *name;
        size_t bytes;
    } part[] = {{"tc.B", img}, {"tc.col", col}, {"tc.U", img}, {"tc.ucol", col}};
    const int parts = two ? 4 : 2;
    for (int i = 0; i < parts; i++)
        if (!dg_buf(ctx, part[i].name, part[i].bytes)) {
            cudaGetLastError();
            ctx->err.clear();
            for (int j = 0; j < i; j++) dg_release(ctx, part[j].name);
            return false;
        }
    if (!ctx->buf_ns.empty()) ctx->image_left -= need;
    return true;
}

int dg_lat_tc_trace(dmftgpu_ctx *ctx, const LatTcArgs &a, bool *ready, double *tr, double *dtr) {
    if (!(dtr ? dg_lat_tc_deriv_supported(a.n, a.D) : dg_lat_tc_supported(a.n, a.D)))
        return dg_fail(ctx, DMFTGPU_BADARG, "lat_tc: unsupported sizes");
    if (a.D == 4) return launch_trace<4>(ctx, a, ready, tr, dtr);
    if (a.D <= 6) return launch_trace<6>(ctx, a, ready, tr, dtr);
    if (a.D <= 8) return launch_trace<8>(ctx, a, ready, tr, dtr);
    return launch_trace<10>(ctx, a, ready, tr, dtr);
}
int dg_lat_tc_block(dmftgpu_ctx *ctx, const LatTcArgs &a, double2 *blk, double2 *blk0) {
    if (!dg_lat_tc_block_supported(a.n, a.D)) return dg_fail(ctx, DMFTGPU_BADARG, "lat_tc: unsupported sizes");
    if (a.D <= 6) return launch_block<6>(ctx, a, blk, blk0);
    if (a.D <= 8) return launch_block<8>(ctx, a, blk, blk0);
    return launch_block<10>(ctx, a, blk, blk0);
}
