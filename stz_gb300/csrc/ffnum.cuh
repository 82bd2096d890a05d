// Float pairs hi + lo (~48 significant bits) and their error-free sums and
// products; plain C++, so that the arithmetic can be checked on the host.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define FF_FN __device__ __forceinline__
#else
#define FF_FN inline
#endif

namespace stzg {

struct ff {
    float hi, lo;
};

// a * b rounded, never contracted into a later addition (an error-free sum of
// the product needs the rounded value).
FF_FN float ff_prod(float a, float b) {
#ifdef __CUDACC__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}

FF_FN ff ff_fast2sum(float a, float b) {
    const float s = a + b;
    return ff{s, b - (s - a)};
}
FF_FN ff ff_add(ff a, ff b) {
    const float s = a.hi + b.hi, bb = s - a.hi;
    float e = (a.hi - (s - bb)) + (b.hi - bb);
    e += a.lo + b.lo;
    return ff_fast2sum(s, e);
}
FF_FN ff ff_neg(ff a) { return ff{-a.hi, -a.lo}; }
FF_FN ff ff_sub(ff a, ff b) { return ff_add(a, ff_neg(b)); }
FF_FN ff ff_mul(ff a, ff b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    return ff_fast2sum(p, e);
}
FF_FN ff ff_add_f(ff a, float b) {
    const float s = a.hi + b, bb = s - a.hi;
    float e = (a.hi - (s - bb)) + (b - bb);
    e += a.lo;
    return ff_fast2sum(s, e);
}


// Error-free sum and difference: hi + lo = a + b (a - b) exactly.
FF_FN ff ff_two_sum(float a, float b) {
    const float s = a + b, bb = s - a;
    return ff{s, (a - (s - bb)) + (b - bb)};
}
FF_FN ff ff_two_diff(float a, float b) {
    const float s = a - b, bb = s - a;
    return ff{s, (a - (s - bb)) - (b + bb)};
}
// (a - b) + (d - c) of pairs.
FF_FN ff ff_diffs(ff a, ff b, ff d, ff c) { return ff_add(ff_sub(a, b), ff_sub(d, c)); }
// k a: the product's high word in p, the rest returned.
FF_FN float ff_term(ff k, ff a, float &p) {
    p = ff_prod(k.hi, a.hi);
    return fmaf(k.lo, a.hi, fmaf(k.hi, a.lo, fmaf(k.hi, a.hi, -p)));
}
// b - (k1 a1 + k2 a2 + k3 a3 + d c) as one float; d c below the rounding of the others.
FF_FN float ff_residual(ff b, ff k1, ff a1, ff k2, ff a2, ff k3, ff a3, ff d, ff c) {
    float p1, p2, p3;
    const float e = (ff_term(k1, a1, p1) + ff_term(k2, a2, p2)) + fmaf(d.hi, c.hi, ff_term(k3, a3, p3));
    const ff s = ff_two_sum(p1, p2), t = ff_two_sum(s.hi, p3), r = ff_two_diff(b.hi, t.hi);
    return r.hi + ((r.lo + b.lo) - ((s.lo + t.lo) + e));
}

}  // namespace stzg
