// Float-float arithmetic: a value as an unevaluated sum hi + lo of two float32
// (about 48 significant bits), from error-free transforms (Knuth two-sum,
// Dekker 1971, with the fused multiply-add for products).  FP64 runs at a
// sixty-fourth of the FP32 rate on GB300 (a warp-wide FP64 instruction holds an
// SM for 16 cycles), so the kernels that need more than 24 bits use this.
#pragma once
#include "fpm_common.cuh"

struct ff {
    float h, l;
};
FPM_DEV ff ff_of(float h, float l = 0.f) { return ff{h, l}; }
// |a| >= |b| or a = 0
FPM_DEV ff ff_quick(float a, float b) {
    const float s = __fadd_rn(a, b);
    return ff{s, __fsub_rn(b, __fsub_rn(s, a))};
}
FPM_DEV ff ff_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return ff{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
FPM_DEV ff ff_two_prod(float a, float b) {
    const float p = __fmul_rn(a, b);
    return ff{p, __fmaf_rn(a, b, -p)};
}
FPM_DEV ff ff_add(ff a, ff b) {
    ff s = ff_two_sum(a.h, b.h);
    const ff t = ff_two_sum(a.l, b.l);
    s = ff_quick(s.h, __fadd_rn(s.l, t.h));
    return ff_quick(s.h, __fadd_rn(s.l, t.l));
}
FPM_DEV ff ff_add_f(ff a, float b) {
    const ff s = ff_two_sum(a.h, b);
    return ff_quick(s.h, __fadd_rn(s.l, a.l));
}
FPM_DEV ff ff_mul(ff a, ff b) {
    const ff p = ff_two_prod(a.h, b.h);
    return ff_quick(p.h, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, p.l)));
}
FPM_DEV ff ff_mul_f(ff a, float b) {
    const ff p = ff_two_prod(a.h, b);
    return ff_quick(p.h, __fmaf_rn(a.l, b, p.l));
}
FPM_DEV ff ff_neg(ff a) { return ff{-a.h, -a.l}; }
// 1 / a: one Newton step on the float32 quotient
FPM_DEV ff ff_recip(ff a) {
    const float r = __fdiv_rn(1.f, a.h);
    const float e = __fmaf_rn(-a.l, r, __fmaf_rn(-a.h, r, 1.f));
    return ff_quick(r, __fmul_rn(r, e));
}
// square root of a >= 0
FPM_DEV ff ff_sqrt(ff a) {
    const float s = __fsqrt_rn(a.h);
    if (s == 0.f) return ff{0.f, 0.f};
    const float e = __fadd_rn(__fmaf_rn(-s, s, a.h), a.l);
    return ff_quick(s, __fdiv_rn(e, __fadd_rn(s, s)));
}
FPM_DEV double ff_double(ff a) { return (double)a.h + (double)a.l; }

// host: a double as hi + lo
inline ff ff_split(double x) {
    const float h = (float)x;
    return ff{h, (float)(x - (double)h)};
}
