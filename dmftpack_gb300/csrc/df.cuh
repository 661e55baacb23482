// df.cuh -- double-float ("split precision") complex arithmetic on the FP32 pipe.
//
// A real number is an unevaluated sum hi + lo of two floats (|lo| <= ulp(hi)/2), giving a 48-bit mantissa;
// products use the FMA error-free transformation (p = a*b, e = fma(a, b, -p)), sums the two-sum
// transformation (Knuth), so every operation is accurate to ~2^-47 relative.  On GB300 the FP32 pipe issues
// ~70x the FP64 rate, so a double-float multiply-add (~18 FP32 instructions) is still several times cheaper
// than an FP64 one.  Values enter from FP64 memory exactly (hi = rn(x), lo = rn(x - hi)) and leave as
// hi + lo in FP64.
//
// Ops policies used by the templated lattice kernels:
//   OpsD: complex FP64 (double2)       OpsF: complex double-float (cdf)       OpsP: the same on packed pairs (pdf)
//
// OpsP works on the real and imaginary parts at once with the packed FP32 instructions (add / sub / mul / fma .f32x2):
// the same roundings in the same order as OpsF, hence the same bits.  A packed instruction holds the FP32 pipe as long
// as the two scalar ones it replaces (measured: 125 of 128 lane operations per SM and clock, where 8-16 warps of
// scalar FMAs reach 85-105) but takes one issue slot, which leaves slots for pivot selects, shuffles and loads.
// Broadcast operands and negations cost nothing (they fold into the instruction, measured); putting two unrelated
// registers side by side costs two moves, so a pdf is kept as (re.h, im.h, re.l, im.l) in registers and in memory.
#pragma once
#include <cmath>
#include <cstring>

#include "common.cuh"

#define DG_HD __host__ __device__ __forceinline__

// IEEE single-precision operations rounded to nearest: the device intrinsics (never contracted into FMAs), and the
// same operations on the host, so that the double-float arithmetic below can be checked on a CPU (host code that
// includes this header is built with -ffp-contract=off)
DG_HD float f_add(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
DG_HD float f_sub(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
}
DG_HD float f_mul(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
DG_HD float f_fma(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    return __fmaf_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
DG_HD int bits_of(float a) {
#ifdef __CUDA_ARCH__
    return __float_as_int(a);
#else
    int i;
    std::memcpy(&i, &a, sizeof i);
    return i;
#endif
}
DG_HD float float_of(int i) {
#ifdef __CUDA_ARCH__
    return __int_as_float(i);
#else
    float a;
    std::memcpy(&a, &i, sizeof a);
    return a;
#endif
}
// 1/a to within an ulp: on the device the approximate reciprocal and one Newton step (the correctly rounded division
// takes ~20 issue slots, this three)
DG_HD float f_rcp(float a) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return __fmaf_rn(r, __fmaf_rn(-a, r, 1.0f), r);
#else
    return 1.0f / a;
#endif
}
DG_HD float f_from_double(double x) {
#ifdef __CUDA_ARCH__
    return __double2float_rn(x);
#else
    return (float)x;
#endif
}

struct dfl {
    float h, l;
};
struct cdf {
    dfl re, im;
};

DG_HD dfl df_make(double x) {
    const float h = f_from_double(x);
    return {h, f_from_double(x - (double)h)};
}
DG_HD double df_val(dfl a) { return (double)a.h + (double)a.l; }
DG_HD dfl fast_two_sum(float a, float b) {
    const float s = f_add(a, b);
    return {s, f_sub(b, f_sub(s, a))};
}
DG_HD dfl two_sum(float a, float b) {
    const float s = f_add(a, b);
    const float bb = f_sub(s, a);
    return {s, f_add(f_sub(a, f_sub(s, bb)), f_sub(b, bb))};
}
DG_HD dfl df_add(dfl a, dfl b) {
    dfl s = two_sum(a.h, b.h);
    const float e = f_add(s.l, f_add(a.l, b.l));
    return fast_two_sum(s.h, e);
}
DG_HD dfl df_neg(dfl a) { return {-a.h, -a.l}; }
DG_HD dfl df_sub(dfl a, dfl b) { return df_add(a, df_neg(b)); }
DG_HD dfl df_mul(dfl a, dfl b) {
    const float p = f_mul(a.h, b.h);
    float e = f_fma(a.h, b.h, -p);
    e = f_fma(a.h, b.l, e);
    e = f_fma(a.l, b.h, e);
    return fast_two_sum(p, e);
}
// c + a*b with one rounding of the product's error term
DG_HD dfl df_fma(dfl a, dfl b, dfl c) {
    const float p = f_mul(a.h, b.h);
    float e = f_fma(a.h, b.h, -p);
    e = f_fma(a.h, b.l, e);
    e = f_fma(a.l, b.h, e);
    dfl s = two_sum(c.h, p);
    const float t = f_add(s.l, f_add(c.l, e));
    return fast_two_sum(s.h, t);
}
// the product a*b as hi p plus the FP32 sum e of its error terms (p + e = a*b to ~2^-48 relative)
DG_HD float df_prod(dfl a, dfl b, float &e) {
    const float p = f_mul(a.h, b.h);
    e = f_fma(a.h, b.h, -p);
    e = f_fma(a.h, b.l, e);
    e = f_fma(a.l, b.h, e);
    return p;
}
// a*b + c*d with one renormalisation (the real or imaginary part of a complex product): the two hi products
// are added exactly (two-sum), the error terms in FP32, so the result is as accurate as two chained
// df_fma and takes 19 FP32 operations instead of 22
DG_HD dfl df_dot2(dfl a, dfl b, dfl c, dfl d) {
    float e1, e2;
    const float p1 = df_prod(a, b, e1), p2 = df_prod(c, d, e2);
    const dfl s = two_sum(p1, p2);
    return fast_two_sum(s.h, f_add(s.l, f_add(e1, e2)));
}
// acc + a*b + c*d with one renormalisation (27 FP32 operations instead of 30 for two chained df_fma)
DG_HD dfl df_fma2(dfl a, dfl b, dfl c, dfl d, dfl acc) {
    float e1, e2;
    const float p1 = df_prod(a, b, e1), p2 = df_prod(c, d, e2);
    const dfl s1 = two_sum(acc.h, p1);
    const dfl s2 = two_sum(s1.h, p2);
    const float t = f_add(f_add(s1.l, s2.l), f_add(acc.l, f_add(e1, e2)));
    return fast_two_sum(s2.h, t);
}
// Lazy accumulation for a running sum of products: acc + a*b with the hi parts added exactly (two-sum) and the
// low parts summed unnormalised in FP32 (12 FP32 operations instead of 15).  The low part of a lazy sum of n
// terms grows to ~n ulp of the hi part and its own rounding with it, so lazy sums are for short runs (the poles of
// one k point, n <= ~64) and pass through df_renorm before any other double-float operation reads them.
DG_HD dfl df_fma_lazy(dfl a, dfl b, dfl acc) {
    float e;
    const float p = df_prod(a, b, e);
    const dfl s = two_sum(acc.h, p);
    return {s.h, f_add(f_add(acc.l, e), s.l)};
}
DG_HD dfl df_renorm(dfl a) { return fast_two_sum(a.h, a.l); }
// 1/a = r / (1 - e) with the FP32 reciprocal r and the residual e = 1 - a r, which an FMA gives exactly up to its own
// rounding: r + r (e + e^2), the neglected e^3 below 2^-66 (without e^2 every reciprocal would come out low by up to
// 2^-46, and the sums over k would keep that bias)
DG_HD dfl df_rcp(dfl a) {
    const float r = f_rcp(a.h);
    const float e = f_fma(-a.l, r, f_fma(-a.h, r, 1.0f));
    return fast_two_sum(r, f_mul(r, f_fma(e, e, e)));
}

DG_HD cdf cdf_make(double2 z) { return {df_make(z.x), df_make(z.y)}; }
DG_HD double2 cdf_val(cdf z) { return make_double2(df_val(z.re), df_val(z.im)); }

struct OpsD {
    typedef double2 C;
    typedef double M;  // pivot magnitude type
    static DG_HD C zero() { return cmk(0, 0); }
    static DG_HD C one() { return cmk(1, 0); }
    static DG_HD C from(double2 z) { return z; }
    static DG_HD double2 to(C z) { return z; }
    static DG_HD C add(C a, C b) { return cadd(a, b); }
    static DG_HD C sub(C a, C b) { return csub(a, b); }
    static DG_HD C neg(C a) { return cneg(a); }
    static DG_HD C mul(C a, C b) { return cmul(a, b); }
    static DG_HD C mulc(C a, C b) { return cmulc(a, b); }  // a conj(b)
    static DG_HD C conj(C a) { return cconj(a); }
    static DG_HD C fma(C a, C b, C acc) { return cfma(a, b, acc); }
    static DG_HD C fms(C a, C b, C acc) { return cfms(a, b, acc); }
    static DG_HD C rcp(C a) { return crcp(a); }
    static DG_HD double re(C a) { return a.x; }
    static DG_HD double im(C a) { return a.y; }
    static DG_HD double mag2(C a) { return cabs2(a); }
    static __device__ __forceinline__ C shfl(C v, int src, int w) { return shfl2(v, src, w); }
    // real parts (R) for the Hermitian split of the pole sums
    typedef double R;
    static DG_HD R rzero() { return 0.0; }
    static DG_HD R rfrom(double x) { return x; }
    static DG_HD R rfma(R a, R b, R acc) { return ::fma(a, b, acc); }
    static DG_HD R rmul(R a, R b) { return a * b; }
    static DG_HD R radd(R a, R b) { return a + b; }
    static DG_HD R rsub(R a, R b) { return a - b; }
    static DG_HD R rneg(R a) { return -a; }
    static DG_HD R rrcp(R a) { return 1.0 / a; }
    static DG_HD C mk(R re, R im) { return cmk(re, im); }
    static DG_HD R cre(C a) { return a.x; }
    static DG_HD R cim(C a) { return a.y; }
    // two running sums of a few products with a common second factor, acc + (w.re, w.im) p (double-float: lazy sums,
    // unnormalised low parts, read through pnorm)
    static DG_HD C pacc(C w, R p, C acc) { return cmk(::fma(w.x, p, acc.x), ::fma(w.y, p, acc.y)); }
    static DG_HD C pnorm(C a) { return a; }
    static DG_HD C pscale(C a, R r) { return cmk(a.x * r, a.y * r); }
    static DG_HD R rdotc(C a, C b) { return ::fma(a.x, b.x, a.y * b.y); }  // Re(a conj b)
    static DG_HD void balance(C &, C &) {}
    // a d - b c from rounded products: equal products cancel to an exact zero, the sign of a singular matrix
    static DG_HD C det2(C a, C b, C c, C d) { return csub(cmul(a, d), cmul(b, c)); }
    static DG_HD C times_i(C a) { return cmk(-a.y, a.x); }
};

struct OpsF {
    typedef cdf C;
    typedef float M;
    static DG_HD C zero() { return {{0.f, 0.f}, {0.f, 0.f}}; }
    static DG_HD C one() { return {{1.f, 0.f}, {0.f, 0.f}}; }
    static DG_HD C from(double2 z) { return cdf_make(z); }
    static DG_HD double2 to(C z) { return cdf_val(z); }
    static DG_HD C add(C a, C b) { return {df_add(a.re, b.re), df_add(a.im, b.im)}; }
    static DG_HD C sub(C a, C b) { return {df_sub(a.re, b.re), df_sub(a.im, b.im)}; }
    static DG_HD C neg(C a) { return {df_neg(a.re), df_neg(a.im)}; }
    static DG_HD C mul(C a, C b) {
        return {df_dot2(a.re, b.re, df_neg(a.im), b.im), df_dot2(a.re, b.im, a.im, b.re)};
    }
    static DG_HD C conj(C a) { return {a.re, df_neg(a.im)}; }
    static DG_HD C mulc(C a, C b) {  // a conj(b)
        return {df_dot2(a.re, b.re, a.im, b.im), df_dot2(a.im, b.re, df_neg(a.re), b.im)};
    }
    static DG_HD C fma(C a, C b, C acc) {
        return {df_fma2(a.re, b.re, df_neg(a.im), b.im, acc.re), df_fma2(a.re, b.im, a.im, b.re, acc.im)};
    }
    static DG_HD C fms(C a, C b, C acc) {
        return {df_fma2(df_neg(a.re), b.re, a.im, b.im, acc.re),
                df_fma2(df_neg(a.re), b.im, df_neg(a.im), b.re, acc.im)};
    }
    static DG_HD C rcp(C a) {  // conj(a)/|a|^2
        const dfl n = df_dot2(a.re, a.re, a.im, a.im);
        const dfl r = df_rcp(n);
        return {df_mul(a.re, r), df_neg(df_mul(a.im, r))};
    }
    static DG_HD double re(C a) { return df_val(a.re); }
    static DG_HD double im(C a) { return df_val(a.im); }
    static DG_HD float mag2(C a) {  // pivot choice only: FP32 magnitude suffices
        return f_fma(a.re.h, a.re.h, f_mul(a.im.h, a.im.h));
    }
    typedef dfl R;
    static DG_HD R rzero() { return {0.f, 0.f}; }
    static DG_HD R rfrom(double x) { return df_make(x); }
    static DG_HD R rfma(R a, R b, R acc) { return df_fma(a, b, acc); }
    static DG_HD R rmul(R a, R b) { return df_mul(a, b); }
    static DG_HD R radd(R a, R b) { return df_add(a, b); }
    static DG_HD R rsub(R a, R b) { return df_sub(a, b); }
    static DG_HD R rneg(R a) { return df_neg(a); }
    static DG_HD R rrcp(R a) { return df_rcp(a); }
    static DG_HD C mk(R re, R im) { return {re, im}; }
    static DG_HD R cre(C a) { return a.re; }
    static DG_HD R cim(C a) { return a.im; }
    static __device__ __forceinline__ C shfl(C v, int src, int w) {
        C o;
        o.re.h = __shfl_sync(0xffffffffu, v.re.h, src, w);
        o.re.l = __shfl_sync(0xffffffffu, v.re.l, src, w);
        o.im.h = __shfl_sync(0xffffffffu, v.im.h, src, w);
        o.im.l = __shfl_sync(0xffffffffu, v.im.l, src, w);
        return o;
    }
};

// ---- packed pairs; on the host the same operations one after the other (OpsP::shfl: device only) ----
DG_HD float2 p2(float x, float y) { return make_float2(x, y); }
DG_HD float2 p2(float x) { return make_float2(x, x); }
#ifdef __CUDA_ARCH__
#define DG_P2_OP(NAME, INSN, SCALAR)                                                                       \
    DG_HD float2 NAME(float2 a, float2 b) {                                                                \
        float2 d;                                                                                          \
        asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t" INSN              \
            " d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"                                                       \
            : "=f"(d.x), "=f"(d.y)                                                                         \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                     \
        return d;                                                                                          \
    }
#else
#define DG_P2_OP(NAME, INSN, SCALAR) \
    DG_HD float2 NAME(float2 a, float2 b) { return p2(SCALAR(a.x, b.x), SCALAR(a.y, b.y)); }
#endif
DG_P2_OP(p2_add, "add.rn.f32x2", f_add)
DG_P2_OP(p2_sub, "sub.rn.f32x2", f_sub)
DG_P2_OP(p2_mul, "mul.rn.f32x2", f_mul)
#undef DG_P2_OP
DG_HD float2 p2_fma(float2 a, float2 b, float2 c) {
#ifdef __CUDA_ARCH__
    float2 d;
    asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
#else
    return p2(f_fma(a.x, b.x, c.x), f_fma(a.y, b.y, c.y));
#endif
}
DG_HD float2 p2_neg(float2 a) { return p2(-a.x, -a.y); }

// two double-float numbers side by side: the parts of a complex number, or two real sums
struct __align__(16) pdf {
    float2 h, l;
};
DG_HD pdf pdf_fast_two_sum(float2 a, float2 b) {
    const float2 s = p2_add(a, b);
    return {s, p2_sub(b, p2_sub(s, a))};
}
DG_HD pdf pdf_two_sum(float2 a, float2 b) {
    const float2 s = p2_add(a, b), bb = p2_sub(s, a);
    return {s, p2_add(p2_sub(a, p2_sub(s, bb)), p2_sub(b, bb))};
}
DG_HD pdf pdf_neg(pdf a) { return {p2_neg(a.h), p2_neg(a.l)}; }
DG_HD pdf pdf_add(pdf a, pdf b) {
    const pdf s = pdf_two_sum(a.h, b.h);
    return pdf_fast_two_sum(s.h, p2_add(s.l, p2_add(a.l, b.l)));
}
// df_prod on both halves
DG_HD float2 pdf_prod(pdf a, pdf b, float2 &e) {
    const float2 p = p2_mul(a.h, b.h);
    e = p2_fma(a.h, b.h, p2_neg(p));
    e = p2_fma(a.h, b.l, e);
    e = p2_fma(a.l, b.h, e);
    return p;
}
// df_mul, df_dot2 (a1 b1 + a2 b2), df_fma2 (acc + a1 b1 + a2 b2) and df_fma_lazy on both halves
DG_HD pdf pdf_mul(pdf a, pdf b) {
    float2 e;
    const float2 p = pdf_prod(a, b, e);
    return pdf_fast_two_sum(p, e);
}
DG_HD pdf pdf_dot2(pdf a1, pdf b1, pdf a2, pdf b2) {
    float2 e1, e2;
    const float2 x1 = pdf_prod(a1, b1, e1), x2 = pdf_prod(a2, b2, e2);
    const pdf s = pdf_two_sum(x1, x2);
    return pdf_fast_two_sum(s.h, p2_add(s.l, p2_add(e1, e2)));
}
DG_HD pdf pdf_fma2(pdf a1, pdf b1, pdf a2, pdf b2, pdf acc) {
    float2 e1, e2;
    const float2 x1 = pdf_prod(a1, b1, e1), x2 = pdf_prod(a2, b2, e2);
    const pdf s1 = pdf_two_sum(acc.h, x1);
    const pdf s2 = pdf_two_sum(s1.h, x2);
    return pdf_fast_two_sum(s2.h, p2_add(p2_add(s1.l, s2.l), p2_add(acc.l, p2_add(e1, e2))));
}
DG_HD pdf pdf_fma_lazy(pdf a, pdf b, pdf acc) {
    float2 e;
    const float2 x = pdf_prod(a, b, e);
    const pdf s = pdf_two_sum(acc.h, x);
    return {s.h, p2_add(p2_add(acc.l, e), s.l)};
}
DG_HD pdf pdf_both(dfl a) { return {p2(a.h), p2(a.l)}; }
// real part twice, imaginary part twice, and i z = (-im, re)
DG_HD pdf pdf_re(pdf z) { return {p2(z.h.x), p2(z.l.x)}; }
DG_HD pdf pdf_im(pdf z) { return {p2(z.h.y), p2(z.l.y)}; }
DG_HD pdf pdf_i(pdf z) { return {p2(-z.h.y, z.h.x), p2(-z.l.y, z.l.x)}; }

struct OpsP {
    typedef pdf C;
    typedef float M;
    static DG_HD C zero() { return {p2(0.f), p2(0.f)}; }
    static DG_HD C one() { return {p2(1.f, 0.f), p2(0.f)}; }
    static DG_HD C from(double2 z) { return mk(df_make(z.x), df_make(z.y)); }
    static DG_HD double2 to(C z) { return make_double2(df_val(cre(z)), df_val(cim(z))); }
    static DG_HD C add(C a, C b) { return pdf_add(a, b); }
    static DG_HD C sub(C a, C b) { return pdf_add(a, pdf_neg(b)); }
    static DG_HD C neg(C a) { return pdf_neg(a); }
    static DG_HD C conj(C a) { return {p2(a.h.x, -a.h.y), p2(a.l.x, -a.l.y)}; }
    static DG_HD C mul(C a, C b) { return pdf_dot2(pdf_re(a), b, pdf_im(a), pdf_i(b)); }
    static DG_HD C mulc(C a, C b) {  // a conj(b) = b.re a + b.im (-i a)
        return pdf_dot2(a, pdf_re(b), pdf_neg(pdf_i(a)), pdf_im(b));
    }
    static DG_HD C fma(C a, C b, C acc) { return pdf_fma2(pdf_re(a), b, pdf_im(a), pdf_i(b), acc); }
    static DG_HD C fms(C a, C b, C acc) {
        return pdf_fma2(pdf_re(a), pdf_neg(b), pdf_im(a), pdf_neg(pdf_i(b)), acc);
    }
    static DG_HD C rcp(C a) {  // conj(a)/|a|^2
        return pdf_mul(conj(a), pdf_both(df_rcp(rdotc(a, a))));
    }
    static DG_HD double re(C a) { return df_val(cre(a)); }
    static DG_HD double im(C a) { return df_val(cim(a)); }
    static DG_HD float mag2(C a) { return f_fma(a.h.x, a.h.x, f_mul(a.h.y, a.h.y)); }
    typedef dfl R;
    static DG_HD R rfrom(double x) { return df_make(x); }
    static DG_HD R rfma(R a, R b, R acc) { return df_fma(a, b, acc); }
    static DG_HD R rmul(R a, R b) { return df_mul(a, b); }
    static DG_HD R radd(R a, R b) { return df_add(a, b); }
    static DG_HD R rsub(R a, R b) { return df_sub(a, b); }
    static DG_HD R rneg(R a) { return df_neg(a); }
    static DG_HD R rrcp(R a) { return df_rcp(a); }
    static DG_HD C mk(R re, R im) { return {p2(re.h, im.h), p2(re.l, im.l)}; }
    static DG_HD R cre(C a) { return {a.h.x, a.l.x}; }
    static DG_HD R cim(C a) { return {a.h.y, a.l.y}; }
    // two lazy real sums with a common second factor: acc + (wx, wy) p
    static DG_HD C pacc(C w, R p, C acc) { return pdf_fma_lazy(w, pdf_both(p), acc); }
    static DG_HD C pnorm(C a) { return pdf_fast_two_sum(a.h, a.l); }
    static DG_HD C pscale(C a, R r) { return pdf_mul(a, pdf_both(r)); }
    static DG_HD C times_i(C a) { return pdf_i(a); }
    static DG_HD C det2(C a, C b, C c, C d) { return fms(b, c, mul(a, d)); }
    // num and den by the power of two that takes |den| to about 1, so that |den|^2 stays in the FP32 range
    static DG_HD void balance(C &num, C &den) {
        const float mx = fmaxf(fabsf(den.h.x), fabsf(den.h.y));
        const float2 sc = p2(float_of((254 << 23) - (bits_of(mx) & 0x7f800000)));
        num = {p2_mul(num.h, sc), p2_mul(num.l, sc)};
        den = {p2_mul(den.h, sc), p2_mul(den.l, sc)};
    }
    static DG_HD R rdotc(C a, C b) {  // Re(a conj b)
        float2 e;
        const float2 p = pdf_prod(a, b, e);
        const dfl s = two_sum(p.x, p.y);
        return fast_two_sum(s.h, f_add(s.l, f_add(e.x, e.y)));
    }
    static __device__ __forceinline__ C shfl(C v, int src, int w) {
        C o;
        o.h.x = __shfl_sync(0xffffffffu, v.h.x, src, w);
        o.h.y = __shfl_sync(0xffffffffu, v.h.y, src, w);
        o.l.x = __shfl_sync(0xffffffffu, v.l.x, src, w);
        o.l.y = __shfl_sync(0xffffffffu, v.l.y, src, w);
        return o;
    }
};

// warp_gj_inverse (linalg.cuh) for any Ops policy
template <class Ops, int N, int W>
__device__ __forceinline__ bool warp_gj_inverse_t(typename Ops::C (&a)[N], const int c) {
    typedef typename Ops::C C;
    typedef typename Ops::M M;
    static_assert(N <= W && W <= 32 && (W & (W - 1)) == 0, "bad lane group");
    bool singular = false;
    int perm[N];
#pragma unroll
    for (int j = 0; j < N; j++) {
        M best = M(-1);
        int p = j;
#pragma unroll
        for (int i = j; i < N; i++) {
            const M v = Ops::mag2(a[i]);
            if (v > best) {
                best = v;
                p = i;
            }
        }
        p = __shfl_sync(0xffffffffu, p, j, W);
        best = __shfl_sync(0xffffffffu, best, j, W);
        singular |= !(best > M(0));
        perm[j] = p;
#pragma unroll
        for (int i = j + 1; i < N; i++)
            if (i == p) {
                const C t = a[j];
                a[j] = a[i];
                a[i] = t;
            }
        const C piv = Ops::shfl(a[j], j, W);
        const C ipiv = Ops::rcp(piv);
        const C t = Ops::mul(a[j], ipiv);
        const bool is_piv_col = (c == j);
        // the pivot column's entries become -f ipiv = fms(f, ipiv, 0): one fms per entry on every lane
        const C tu = is_piv_col ? ipiv : t;
#pragma unroll
        for (int i = 0; i < N; i++) {
            if (i == j) continue;
            const C f = Ops::shfl(a[i], j, W);
            a[i] = Ops::fms(f, tu, is_piv_col ? Ops::zero() : a[i]);
        }
        a[j] = is_piv_col ? ipiv : t;
    }
#pragma unroll
    for (int j = N - 1; j >= 0; j--) {
        const int p = perm[j];
        const int src = (c == j) ? p : ((c == p) ? j : c);
#pragma unroll
        for (int i = 0; i < N; i++) a[i] = Ops::shfl(a[i], src, W);
    }
    return singular;
}

// warp_gj_inverse_t with the elimination steps in a rolled loop: the same arithmetic and pivot choices, but
// the rows of each lane's column are rotated by one after every step, so the current pivot row is always
// register a[0] and the loop body is the same for every step (no dynamic register indexing).  The code is N
// times shorter than the unrolled form, which matters for large N, where the kernels are bound by instruction
// fetch.  Row r of step j sits in register (r - j) mod N; after N steps every row is back in place.  The interchange
// of a step (8 selects per row) and its undoing at the end (N^2 exchanges) are skipped when no group of the warp pivots
// off the diagonal, which is the rule: above the first hundred or so Matsubara frequencies iw dominates the matrix.
template <class Ops, int N, int W>
__device__ __forceinline__ bool warp_gj_inverse_rolled(typename Ops::C (&a)[N], const int c) {
    typedef typename Ops::C C;
    typedef typename Ops::M M;
    static_assert(N <= W && W <= 32 && (W & (W - 1)) == 0, "bad lane group");
    bool singular = false, moved = false;
    int perm[N];
#pragma unroll 1
    for (int j = 0; j < N; j++) {
        // pivot search over rows j..N-1 (registers 0..N-1-j) of column j (lane j)
        M best = M(-1);
        int pp = 0;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const M v = Ops::mag2(a[i]);
            if (i <= N - 1 - j && v > best) {
                best = v;
                pp = i;
            }
        }
        pp = __shfl_sync(0xffffffffu, pp, j, W);
        best = __shfl_sync(0xffffffffu, best, j, W);
        singular |= !(best > M(0));
        perm[j] = pp + j;  // the row index of the pivot
        if (__any_sync(0xffffffffu, pp != 0)) {
            moved = true;
#pragma unroll
            for (int i = 1; i < N; i++)
                if (i == pp) {
                    const C t = a[0];
                    a[0] = a[i];
                    a[i] = t;
                }
        }
        const C piv = Ops::shfl(a[0], j, W);
        const C ipiv = Ops::rcp(piv);
        const C t = Ops::mul(a[0], ipiv);
        const bool is_piv_col = (c == j);
        const C tu = is_piv_col ? ipiv : t;  // the pivot column's entries become fms(f, ipiv, 0) = -f ipiv
#pragma unroll
        for (int i = 1; i < N; i++) {
            const C f = Ops::shfl(a[i], j, W);
            a[i] = Ops::fms(f, tu, is_piv_col ? Ops::zero() : a[i]);
        }
        a[0] = is_piv_col ? ipiv : t;
        // rotate: the finished pivot row moves to the end
        const C r0 = a[0];
#pragma unroll
        for (int i = 0; i < N - 1; i++) a[i] = a[i + 1];
        a[N - 1] = r0;
    }
    if (!moved) return singular;
#pragma unroll 1
    for (int j = N - 1; j >= 0; j--) {
        const int p = perm[j];
        const int src = (c == j) ? p : ((c == p) ? j : c);
#pragma unroll
        for (int i = 0; i < N; i++) a[i] = Ops::shfl(a[i], src, W);
    }
    return singular;
}

// warp_gj_inverse_rolled for lane groups of any width N that need not divide 32: the group is lanes
// base .. base+N-1 of the warp (lane c of the group holds column c), so 32/N groups share a warp with no idle
// padding lanes inside a group.  Every shuffle names an absolute source lane (width 32) and runs with the
// full mask under warp-uniform control flow; lanes outside any group take part with base past the last
// group and compute values that are never used.
template <class Ops, int N>
__device__ __forceinline__ bool group_gj_inverse(typename Ops::C (&a)[N], const int c, const int base) {
    typedef typename Ops::C C;
    typedef typename Ops::M M;
    bool singular = false, moved = false;
    int perm[N];
#pragma unroll 1
    for (int j = 0; j < N; j++) {
        M best = M(-1);
        int pp = 0;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const M v = Ops::mag2(a[i]);
            if (i <= N - 1 - j && v > best) {
                best = v;
                pp = i;
            }
        }
        pp = __shfl_sync(0xffffffffu, pp, base + j, 32);
        best = __shfl_sync(0xffffffffu, best, base + j, 32);
        singular |= !(best > M(0));
        perm[j] = pp + j;
        if (__any_sync(0xffffffffu, pp != 0 && base <= 32 - N)) {
            moved = true;
#pragma unroll
            for (int i = 1; i < N; i++)
                if (i == pp) {
                    const C t = a[0];
                    a[0] = a[i];
                    a[i] = t;
                }
        }
        const C piv = Ops::shfl(a[0], base + j, 32);
        const C ipiv = Ops::rcp(piv);
        const C t = Ops::mul(a[0], ipiv);
        const bool is_piv_col = (c == j);
        const C tu = is_piv_col ? ipiv : t;  // the pivot column's entries become fms(f, ipiv, 0) = -f ipiv
#pragma unroll
        for (int i = 1; i < N; i++) {
            const C f = Ops::shfl(a[i], base + j, 32);
            a[i] = Ops::fms(f, tu, is_piv_col ? Ops::zero() : a[i]);
        }
        a[0] = is_piv_col ? ipiv : t;
        const C r0 = a[0];
#pragma unroll
        for (int i = 0; i < N - 1; i++) a[i] = a[i + 1];
        a[N - 1] = r0;
    }
    if (!moved) return singular;
#pragma unroll 1
    for (int j = N - 1; j >= 0; j--) {
        const int p = perm[j];
        const int src = base + ((c == j) ? p : ((c == p) ? j : c));
#pragma unroll
        for (int i = 0; i < N; i++) a[i] = Ops::shfl(a[i], src, 32);
    }
    return singular;
}
