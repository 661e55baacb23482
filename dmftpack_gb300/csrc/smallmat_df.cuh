// smallmat_df.cuh -- the reciprocal square root in double-float, for the rotations of the double-float eigensolver (eig.cuh), and
// the square root and division its host tests are written against.
#pragma once
#include "df.cuh"

// sqrt(a), a >= 0: the FP32 root refined by one Newton step in double-float
DG_HD dfl df_sqrt(dfl a) {
    if (!(a.h > 0.f)) return {0.f, 0.f};
    const float s = sqrtf(a.h);
    const dfl e = df_sub(a, df_mul({s, 0.f}, {s, 0.f}));  // a - s^2
    return fast_two_sum(s, e.h / (2.f * s));
}
// a / b: the FP32 quotient corrected by the double-float remainder
DG_HD dfl df_div(dfl a, dfl b) {
    const float q1 = a.h / b.h;
    const dfl r = df_sub(a, df_mul(b, {q1, 0.f}));
    const float q2 = r.h / b.h;
    return fast_two_sum(q1, q2);
}

// a^-1/2, a > 0: the approximate root refined in FP32, then one double-float step on its residual e = 1 - a y^2,
// y (1 + e/2 + 3/8 e^2)
DG_HD dfl df_rsqrt(dfl a) {
#ifdef __CUDA_ARCH__
    float y = rsqrtf(a.h);
#else
    float y = 1.f / sqrtf(a.h);
#endif
    y = fmaf(0.5f * y, fmaf(-a.h * y, y, 1.f), y);
    const dfl y2 = df_mul({y, 0.f}, {y, 0.f});
    const dfl e = df_sub({1.f, 0.f}, df_mul(a, y2));
    return fast_two_sum(y, y * e.h * fmaf(0.375f, e.h, 0.5f) + 0.5f * y * e.l);
}
