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

}  // namespace stzg
