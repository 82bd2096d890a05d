// 64-bit fixed point: a tile's doubles as integers of one scale, 2^(1081 - E)
// for the biased exponent E of its largest magnitude.  Sums and differences
// of them are exact, on the integer pipe (64 operations per clock and SM,
// FP64 has two).
#pragma once

namespace stzg {

// d 2^(1081 - E) cut to an integer; E: the biased exponent of the largest
// magnitude of d's set, so the result is below 2^59.
__device__ __forceinline__ long long to_fixed(double d, int E) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
    const int e = (hi >> 20) & 0x7ff;
    const unsigned long long m =
        ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;  // below 2^63
    const long long v = (long long)(m >> min(4 + E - e, 63));  // zero and subnormal: shifted out
    return (int)hi < 0 ? -v : v;
}

// 2^K as a double (0 below the normal range, infinity above).
__device__ __forceinline__ double power_of_two(int K) {
    const int e = min(max(K + 1023, 0), 0x7ff);
    return __hiloint2double(e << 20, 0);
}

}  // namespace stzg
