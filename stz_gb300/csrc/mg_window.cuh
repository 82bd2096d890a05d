// Phases of a V-cycle on a window of a level that sits in shared memory,
// templated on the number type: float, or ff (a float pair, ~48 significant
// bits).  A window holds the nodes of a range of rows, either whole periodic
// rows (WRAP) or a range of columns with a halo, each row stored parity-major
// (even columns, then odd ones) so that the points of one colour, and their
// neighbours, are consecutive.  Every phase is a loop over points by thread
// index without synchronisation; the caller separates phases by barriers.
//
// The smoother is the one of mg.cu: two colours on the matrix-free top level
// (colour c updates x where (i + j) & 1 == c and y elsewhere), on coarse
// levels the even rows (even columns, odd columns, the last column of an odd
// line) and then the odd rows; float results are the bits of the streaming
// kernels' operations in their order.
#pragma once

#include <cuda_runtime.h>

#include "transfer1d.cuh"

#ifdef __CUDACC__
#define MGW_FN __device__ __forceinline__
#define MGW_BOTH __host__ __device__ inline
#else
#define MGW_FN inline
#define MGW_BOTH inline
#endif

#include "ffnum.cuh"

namespace stzg {
struct pair_range;
namespace mgw {

// ---- numbers -----------------------------------------------------------------

template <typename S> struct num;
template <> struct num<float> {
    typedef float2 node;            // x, y
    static constexpr int quads = 1; // float4 words of a 2x2 block
};
template <> struct num<ff> {
    typedef float4 node;            // x.hi, y.hi, x.lo, y.lo
    static constexpr int quads = 2; // the high parts, then the low parts
};

template <typename S> struct val2 {
    S x, y;
};

MGW_FN val2<float> get(const float2 &p) { return val2<float>{p.x, p.y}; }
MGW_FN val2<ff> get(const float4 &p) { return val2<ff>{ff{p.x, p.z}, ff{p.y, p.w}}; }
MGW_FN float2 put(const val2<float> &v) { return make_float2(v.x, v.y); }
MGW_FN float4 put(const val2<ff> &v) { return make_float4(v.x.hi, v.y.hi, v.x.lo, v.y.lo); }

// Nodes in shared memory: the x components, then the y ones, so that a sweep
// over one component (the top level's) reads consecutive words.
template <typename S> struct plane {
    S *p;    // x; y at p + ps
    int ps;
    MGW_FN plane operator+(int k) const { return plane{p + k, ps}; }
    MGW_FN S x(int k) const { return p[k]; }
    MGW_FN S y(int k) const { return p[k + ps]; }
    MGW_FN void set_x(int k, S v) const { p[k] = v; }
    MGW_FN void set_y(int k, S v) const { p[k + ps] = v; }
    MGW_FN val2<S> get(int k) const { return val2<S>{p[k], p[k + ps]}; }
    MGW_FN void set(int k, const val2<S> &v) const {
        p[k] = v.x;
        p[k + ps] = v.y;
    }
};

MGW_FN float add(float a, float b) { return a + b; }
MGW_FN ff add(ff a, ff b) { return ff_add(a, b); }
MGW_FN float sub(float a, float b) { return a - b; }
MGW_FN ff sub(ff a, ff b) { return ff_sub(a, b); }
MGW_FN float mul(float a, float b) { return a * b; }
MGW_FN ff mul(ff a, ff b) { return ff_mul(a, b); }
// by a power of two
MGW_FN float scale(float a, float w) { return a * w; }
MGW_FN ff scale(ff a, float w) { return ff{a.hi * w, a.lo * w}; }

// A running sum of products.  ff: the high parts by TwoSum, every rounding
// error and low part gathered in lo (relative 2^-48 of the terms' magnitude),
// renormalised once at the end.
struct facc {
    float v = 0.f;
    MGW_FN void mad(float a, float b) { v = fmaf(a, b, v); }
    MGW_FN float done() const { return v; }
};
struct ffacc {
    float hi = 0.f, lo = 0.f;
    MGW_FN void mad(ff a, ff b) {
        const float p = ff_prod(a.hi, b.hi);
        float e = fmaf(a.hi, b.hi, -p);
        e = fmaf(a.hi, b.lo, e);
        e = fmaf(a.lo, b.hi, e);
        const float s = hi + p, bb = s - hi;
        lo += ((hi - (s - bb)) + (p - bb)) + e;
        hi = s;
    }
    MGW_FN ff done() const { return ff_fast2sum(hi, lo); }
};
template <typename S> struct acc_of;
template <> struct acc_of<float> { typedef facc type; };
template <> struct acc_of<ff> { typedef ffacc type; };

// a + b - c - d of the corner terms, and a + b, as operands of a product (not
// renormalised for ff: the product folds the low part in).
MGW_FN float sum2(float a, float b) { return a + b; }
MGW_FN ff sum2(ff a, ff b) {
    const float s = a.hi + b.hi, bb = s - a.hi;
    return ff{s, ((a.hi - (s - bb)) + (b.hi - bb)) + (a.lo + b.lo)};
}
MGW_FN float cross4(float a, float b, float c, float d) { return a + b - c - d; }
MGW_FN ff cross4(ff a, ff b, ff c, ff d) { return sum2(sum2(a, ff_neg(c)), sum2(b, ff_neg(d))); }

// Constants of the top-level operator (top_op in mg.cuh) in the number type.
template <typename S> struct top_consts {
    S Kmx, Kmy, mx, my, qK, cxx, cyy, icxx, icyy, bcxx, bcyy, ibcxx, ibcyy;
};

MGW_FN float three(float k1, float s1, float k2, float s2, float k3, float s3) { return k1 * s1 + k2 * s2 + k3 * s3; }
MGW_FN ff three(ff k1, ff s1, ff k2, ff s2, ff k3, ff s3) {
    ffacc a;
    a.mad(k1, s1);
    a.mad(k2, s2);
    a.mad(k3, s3);
    return a.done();
}

// ---- windows -----------------------------------------------------------------

// YP: y is periodic too; rows are unwrapped (a band's halo rows continue below
// 0 and beyond n), lines in y are even.
template <typename S, bool WRAP, bool YP = false> struct window {
    plane<S> z, b, r;
    int W, He;          // columns; even ones
    int jb, rb;         // rows of local row 0 of z and b; of r
    int m, n;           // the level
    int x0;             // global column of window column 0 (even; 0 when WRAP)
    const float4 *st;   // stencils: 10 blocks each
    const int *cls;     // class per row (homog) or per point
    int homog;
    MGW_FN int lo(int j) const { return YP || j > 0 ? j : 0; }          // first row of a range from j on
    MGW_FN int hi(int j) const { return YP || j < n - 1 ? j : n - 1; }  // last row of a range up to j
    MGW_FN bool has_below(int j) const { return YP || j > 0; }
    MGW_FN bool has_above(int j) const { return YP || j < n - 1; }
    MGW_FN int wrapped(int j) const { return !YP ? j : (j < 0 ? j + n : (j >= n ? j - n : j)); }
    // halves_of(2J + q - 1, n, yp, J), q = 0, 1, 2
    MGW_FN int halves(int q, int J) const {
        if (YP) return q == 1 ? 2 : 1;
        const int fy = 2 * J + q - 1;
        if (fy < 0 || fy >= n) return 0;
        if (q == 1) return 2;
        if ((n & 1) || fy != n - 1) return 1;
        return q == 0 ? 2 : 0;
    }
    // the coarse rows (unwrapped) that feed row j and their halves
    MGW_FN int feeds(int j, int *c, int *h) const {
        if (!YP) return p1d_halves(j, n, 0, c, h);
        c[0] = j >> 1;
        c[1] = c[0] + 1;
        h[0] = j & 1 ? 1 : 2;
        h[1] = 1;
        return 1 + (j & 1);
    }
    MGW_FN int col(int w) const { return (w & 1) * He + (w >> 1); }
    MGW_FN int at(int j, int w) const { return (j - jb) * W + col(w); }
    MGW_FN int rat(int j, int w) const { return (j - rb) * W + col(w); }
    MGW_FN int left(int w) const { return WRAP && w == 0 ? W - 1 : w - 1; }
    MGW_FN int right(int w) const { return WRAP && w == W - 1 ? 0 : w + 1; }
    MGW_FN int gcol(int w) const {
        if (WRAP) return w;
        const int g = x0 + w;
        return g < 0 ? g + m : (g >= m ? g % m : g);
    }
    MGW_FN const float4 *sten(int j, int w) const {
        const int c = homog ? cls[wrapped(j)] : cls[(size_t)wrapped(j) * m + gcol(w)];
        return st + (size_t)c * (10 * num<S>::quads);
    }
};

// idx -> (idx / per, idx % per) for idx < 2^20: the half keeps the float
// quotient away from whole numbers.
struct divider {
    float inv;
    int per;
    MGW_FN explicit divider(int p) : inv(1.f / (float)(p > 0 ? p : 1)), per(p) {}
    MGW_FN int quot(int k) const { return (int)(((float)k + 0.5f) * inv); }
};

// acc += A z of block e.
MGW_FN void madd(facc &ax, facc &ay, const float4 *s, int e, const val2<float> &z) {
    const float4 A = s[e];
    ax.mad(A.x, z.x);
    ax.mad(A.y, z.y);
    ay.mad(A.z, z.x);
    ay.mad(A.w, z.y);
}
MGW_FN void madd(ffacc &ax, ffacc &ay, const float4 *s, int e, const val2<ff> &z) {
    const float4 H = s[2 * e], L = s[2 * e + 1];
    ax.mad(ff{H.x, L.x}, z.x);
    ax.mad(ff{H.y, L.y}, z.y);
    ay.mad(ff{H.z, L.z}, z.x);
    ay.mad(ff{H.w, L.w}, z.y);
}
// A v of block e (the inverse of the centre block)
MGW_FN val2<float> apply(const float4 *s, int e, const val2<float> &v) {
    const float4 A = s[e];
    return val2<float>{A.x * v.x + A.y * v.y, A.z * v.x + A.w * v.y};
}
MGW_FN val2<ff> apply(const float4 *s, int e, const val2<ff> &v) {
    ffacc ax, ay;
    madd(ax, ay, s, e, v);
    return val2<ff>{ax.done(), ay.done()};
}

// Off-diagonal products of a coarse level (tgmg_level::mul_a,
// tgmg.in.cc:536-547).  rows: whether the rows below and above take part;
// mid: whether the neighbours in the row do (a sweep that starts from zero
// skips what is still zero: adding exact zeros changes nothing).
template <typename S, bool WRAP, bool YP>
MGW_FN void offdiag(const window<S, WRAP, YP> &V, const float4 *s, int j, int w, bool rows, bool mid,
                    typename acc_of<S>::type &ax, typename acc_of<S>::type &ay) {
    const int wl = V.left(w), wr = V.right(w);
    if (rows && V.has_below(j)) {
        madd(ax, ay, s, 0, V.z.get(V.at(j - 1, wl)));
        madd(ax, ay, s, 1, V.z.get(V.at(j - 1, w)));
        madd(ax, ay, s, 2, V.z.get(V.at(j - 1, wr)));
    }
    if (mid) {
        madd(ax, ay, s, 3, V.z.get(V.at(j, wl)));
        madd(ax, ay, s, 5, V.z.get(V.at(j, wr)));
    }
    if (rows && V.has_above(j)) {
        madd(ax, ay, s, 6, V.z.get(V.at(j + 1, wl)));
        madd(ax, ay, s, 7, V.z.get(V.at(j + 1, w)));
        madd(ax, ay, s, 8, V.z.get(V.at(j + 1, wr)));
    }
}

MGW_FN int imin(int a, int b) { return a < b ? a : b; }

// Colours of a sweep: rows of parity cy, columns of parity cx (cx == 2: the
// last column of an odd line), rows jlo..jhi and window columns wlo..whi (all
// when WRAP).
template <typename S, bool WRAP, bool YP>
MGW_FN void lev_color(const window<S, WRAP, YP> &V, int jlo, int jhi, int wlo, int whi, int cx, int cy, bool from_zero,
                      int tid, int nth) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    const int j0 = jlo + ((jlo ^ cy) & 1);
    if (j0 > jhi) return;
    int w0, nw;
    if (cx == 2) {
        w0 = V.W - 1;
        nw = 1;
    } else if (WRAP) {
        w0 = cx;
        nw = V.W >> 1;  // even columns without the last one of an odd line
    } else {
        w0 = wlo + ((wlo ^ cx) & 1);
        nw = whi >= w0 ? ((whi - w0) >> 1) + 1 : 0;
    }
    const int total = (((jhi - j0) >> 1) + 1) * nw;
    const divider dv(nw);
    for (int k = tid; k < total; k += nth) {
        const int q = dv.quot(k), j = j0 + 2 * q, w = w0 + 2 * (k - q * nw);
        const float4 *s = V.sten(j, w);
        typename acc_of<S>::type ax, ay;
        offdiag(V, s, j, w, !(from_zero && cy == 0), !(from_zero && cx == 0), ax, ay);
        const int c = V.at(j, w);
        const val2<S> bb = V.b.get(c);
        V.z.set(c, apply(s, 9, val2<S>{sub(bb.x, ax.done()), sub(bb.y, ay.done())}));
    }
}

// z = 0 on the last column of an odd line (the third colour, read before its
// first update in a sweep from zero).
template <typename S, bool WRAP, bool YP>
MGW_FN void lev_clear_last(const window<S, WRAP, YP> &V, int jlo, int jhi, int tid, int nth) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    for (int j = jlo + tid; j <= jhi; j += nth) {
        val2<S> o{};
        V.z.set(V.at(j, V.W - 1), o);
    }
}

// r = b - A z after a sweep.  On an even line the odd columns of odd rows took
// the last colour: their residual is zero up to rounding and set to zero.
template <typename S, bool WRAP, bool YP>
MGW_FN void lev_residual(const window<S, WRAP, YP> &V, int jlo, int jhi, int wlo, int whi, int tid, int nth) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    if (jlo > jhi) return;
    if (WRAP) {
        wlo = 0;
        whi = V.W - 1;
    }
    const int nw = whi - wlo + 1, total = (jhi - jlo + 1) * nw;
    const bool odd_line = V.m & 1;
    const divider dv(nw);
    for (int k = tid; k < total; k += nth) {
        const int q = dv.quot(k), j = jlo + q, w = wlo + (k - q * nw);
        val2<S> o{};
        if (odd_line || !(j & w & 1)) {
            const float4 *s = V.sten(j, w);
            typename acc_of<S>::type ax, ay;
            offdiag(V, s, j, w, true, true, ax, ay);
            const int c = V.at(j, w);
            madd(ax, ay, s, 4, V.z.get(c));
            const val2<S> bb = V.b.get(c);
            o = val2<S>{sub(bb.x, ax.done()), sub(bb.y, ay.done())};
        }
        V.r.set(V.rat(j, w), o);
    }
}

// Off-diagonal sums of the top level (qs_multi::mul_a, qs_multi.hh:41-50).
template <typename S, bool WRAP, bool YP>
MGW_FN S top_off_x(const top_consts<S> &o, const window<S, WRAP, YP> &V, int j, int w) {
    const int wl = V.left(w), wr = V.right(w);
    return three(o.Kmx, sum2(V.z.x(V.at(j, wl)), V.z.x(V.at(j, wr))), o.my,
                 sum2(V.z.x(V.at(j - 1, w)), V.z.x(V.at(j + 1, w))), o.qK,
                 cross4(V.z.y(V.at(j - 1, wl)), V.z.y(V.at(j + 1, wr)), V.z.y(V.at(j - 1, wr)),
                        V.z.y(V.at(j + 1, wl))));
}
template <typename S, bool WRAP, bool YP>
MGW_FN S top_off_y(const top_consts<S> &o, const window<S, WRAP, YP> &V, int j, int w) {
    const int wl = V.left(w), wr = V.right(w);
    return three(o.mx, sum2(V.z.y(V.at(j, wl)), V.z.y(V.at(j, wr))), o.Kmy,
                 sum2(V.z.y(V.at(j - 1, w)), V.z.y(V.at(j + 1, w))), o.qK,
                 cross4(V.z.x(V.at(j - 1, wl)), V.z.x(V.at(j + 1, wr)), V.z.x(V.at(j - 1, wr)),
                        V.z.x(V.at(j + 1, wl))));
}

// One colour of the top level: a thread takes a pair of columns, the x
// equation at one and the y equation at the other, so that lanes do not
// diverge on the component.  from_zero: z is zero, so only b counts.
template <typename S, bool WRAP, bool YP>
MGW_FN void top_color(const top_consts<S> &o, const window<S, WRAP, YP> &V, int jlo, int jhi, int wlo, int whi, int color,
                      bool from_zero, int tid, int nth) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    if (jlo > jhi) return;
    if (WRAP) {
        wlo = 0;
        whi = V.W - 1;
    }
    const int p0 = wlo >> 1, np = (whi >> 1) - p0 + 1, total = (jhi - jlo + 1) * np;
    const divider dv(np);
    for (int k = tid; k < total; k += nth) {
        const int q = dv.quot(k), j = jlo + q, wa = 2 * (p0 + (k - q * np));
        const bool even_is_x = (j & 1) == color;
        const int wx = even_is_x ? wa : wa + 1, wy = even_is_x ? wa + 1 : wa;
        const bool wall = j == 0 || j == V.n - 1;
        if (wx >= wlo && wx <= whi) {
            const int c = V.at(j, wx);
            const S bb = V.b.x(c);
            if (wall) V.z.set_x(c, mul(o.ibcxx, bb));
            else if (from_zero) V.z.set_x(c, mul(o.icxx, bb));
            else V.z.set_x(c, mul(o.icxx, sub(bb, top_off_x(o, V, j, wx))));
        }
        if (wy >= wlo && wy <= whi) {
            const int c = V.at(j, wy);
            const S bb = V.b.y(c);
            if (wall) V.z.set_y(c, mul(o.ibcyy, bb));
            else if (from_zero) V.z.set_y(c, mul(o.icyy, bb));
            else V.z.set_y(c, mul(o.icyy, sub(bb, top_off_y(o, V, j, wy))));
        }
    }
}

// Residual of the colour-0 equations after a sweep (the colour-1 ones, whose
// unknowns were updated last, and the wall rows are zero up to rounding).
template <typename S, bool WRAP, bool YP>
MGW_FN void top_residual(const top_consts<S> &o, const window<S, WRAP, YP> &V, int jlo, int jhi, int wlo, int whi, int tid,
                         int nth) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    if (jlo > jhi) return;
    if (WRAP) {
        wlo = 0;
        whi = V.W - 1;
    }
    const int p0 = wlo >> 1, np = (whi >> 1) - p0 + 1, total = (jhi - jlo + 1) * np;
    const divider dv(np);
    for (int k = tid; k < total; k += nth) {
        const int q = dv.quot(k), j = jlo + q, wa = 2 * (p0 + (k - q * np));
        const int wx = (j & 1) ? wa + 1 : wa, wy = (j & 1) ? wa : wa + 1;
        const bool wall = j == 0 || j == V.n - 1;
        if (wx >= wlo && wx <= whi) {
            const int c = V.at(j, wx);
            val2<S> r{};
            if (!wall) r.x = sub(sub(V.b.x(c), top_off_x(o, V, j, wx)), mul(o.cxx, V.z.x(c)));
            V.r.set(V.rat(j, wx), r);
        }
        if (wy >= wlo && wy <= whi) {
            const int c = V.at(j, wy);
            val2<S> r{};
            if (!wall) r.y = sub(sub(V.b.y(c), top_off_y(o, V, j, wy)), mul(o.cyy, V.z.y(c)));
            V.r.set(V.rat(j, wy), r);
        }
    }
}

// Full weighting of r at the coarse points of rows Jlo..Jhi, columns
// Ilo..Ihi (global): out(J, I, value).
template <typename S, bool WRAP, bool YP, typename Out>
MGW_FN void restrict_rows(const window<S, WRAP, YP> &V, int Jlo, int Jhi, int Ilo, int Ihi, int cm, Out out, int tid,
                          int nth) {
    const int nI = Ihi - Ilo + 1, total = (Jhi - Jlo + 1) * nI;
    if (Jhi < Jlo || nI <= 0) return;
    const bool odd_line = V.m & 1;
    const divider dv(nI);
    for (int k = tid; k < total; k += nth) {
        const int qk = dv.quot(k), J = Jlo + qk, I = Ilo + (k - qk * nI), w = 2 * I - V.x0;
        // an odd periodic line: its last (even) point injects, so the two
        // coarse points at the seam have no neighbour across it
        const bool hl = !(odd_line && I == 0), hr = !(odd_line && I == cm - 1);
        val2<S> a{};
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const int hy = V.halves(q, J);
            if (!hy) continue;
            const int fy = 2 * J + q - 1;
            const float w1 = (float)hy * 0.25f, w2 = (float)(2 * hy) * 0.25f;
            if (hl) {
                const val2<S> v = V.r.get(V.rat(fy, V.left(w)));
                a.x = add(a.x, scale(v.x, w1));
                a.y = add(a.y, scale(v.y, w1));
            }
            const val2<S> c = V.r.get(V.rat(fy, w));
            a.x = add(a.x, scale(c.x, w2));
            a.y = add(a.y, scale(c.y, w2));
            if (hr) {
                const val2<S> v = V.r.get(V.rat(fy, V.right(w)));
                a.x = add(a.x, scale(v.x, w1));
                a.y = add(a.y, scale(v.y, w1));
            }
        }
        out(J, I, a);
    }
}

// z += P zc on rows jlo..jhi, window columns wlo..whi: zc(J, I) is the child's
// value at row J and the coarse column I of window column 2 (I - x0/2) (WRAP:
// 0 <= I < cm; else unwrapped).
template <typename S, bool WRAP, bool YP, typename Child>
MGW_FN void prolong_rows(const window<S, WRAP, YP> &V, int jlo, int jhi, int wlo, int whi, int cm, Child zc, int tid,
                         int nth) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    if (jlo > jhi) return;
    if (WRAP) {
        wlo = 0;
        whi = V.W - 1;
    }
    const int nw = whi - wlo + 1, total = (jhi - jlo + 1) * nw;
    const divider dv(nw);
    for (int k = tid; k < total; k += nth) {
        const int qk = dv.quot(k), j = jlo + qk, w = wlo + (k - qk * nw);
        int cy[2], hy[2];
        const int ny = V.feeds(j, cy, hy);
        const int I = (V.x0 + w) >> 1;  // floor: x0 is even
        val2<S> a{};
        if (w & 1) {
            const int I1 = WRAP && I + 1 == cm ? 0 : I + 1;
            for (int q = 0; q < ny; q++) {
                const float wy = (float)hy[q] * 0.25f;
                const val2<S> v0 = zc(cy[q], I), v1 = zc(cy[q], I1);
                a.x = add(a.x, scale(add(v0.x, v1.x), wy));
                a.y = add(a.y, scale(add(v0.y, v1.y), wy));
            }
        } else {
            for (int q = 0; q < ny; q++) {
                const float wy = (float)hy[q] * 0.25f;
                const val2<S> v0 = zc(cy[q], I);
                a.x = add(a.x, scale(v0.x, 2.f * wy));
                a.y = add(a.y, scale(v0.y, 2.f * wy));
            }
        }
        const int c = V.at(j, w);
        const val2<S> f = V.z.get(c);
        V.z.set(c, val2<S>{add(f.x, a.x), add(f.y, a.y)});
    }
}

// ---- even levels in 2 x 2 blocks --------------------------------------------------
//
// The same phases for a band of an even line with one stencil class per row
// and its tables in shared memory: a thread keeps one block of 2 x 2 nodes
// (rows 2q, 2q + 1 of the band, columns 2k, 2k + 1) through every phase, so
// that indices are formed once per level; small levels are bound by the
// latency of a phase, of which index arithmetic was the larger part.

// A thread's blocks: q, k of the first one, and the step to the next.
struct block_walk {
    int q, k, dq, dk, P;
    MGW_FN block_walk(int tid, int nth, int p) : P(p) {
        const divider dv(p);
        q = dv.quot(tid);
        k = tid - q * p;
        dq = dv.quot(nth);
        dk = nth - dq * p;
    }
    MGW_FN void next() {
        k += dk;
        q += dq;
        if (k >= P) {
            k -= P;
            q++;
        }
    }
};

// The nodes around a point: its column and its neighbours' columns as offsets
// in a parity-major row.
struct columns3 {
    int l, c, r;
    MGW_FN columns3(int k, int P, int cx)
        : l(cx ? k : P + (k ? k - 1 : P - 1)), c(cx ? P + k : k), r(cx ? (k + 1 == P ? 0 : k + 1) : P + k) {}
};

template <typename S>
MGW_FN void offdiag3(const float4 *s, const plane<S> &row, int W, const columns3 &c, bool dn, bool mid,
                     bool up, typename acc_of<S>::type &ax, typename acc_of<S>::type &ay) {
    if (dn) {
        madd(ax, ay, s, 0, row.get(c.l - W));
        madd(ax, ay, s, 1, row.get(c.c - W));
        madd(ax, ay, s, 2, row.get(c.r - W));
    }
    if (mid) {
        madd(ax, ay, s, 3, row.get(c.l));
        madd(ax, ay, s, 5, row.get(c.r));
    }
    if (up) {
        madd(ax, ay, s, 6, row.get(c.l + W));
        madd(ax, ay, s, 7, row.get(c.c + W));
        madd(ax, ay, s, 8, row.get(c.r + W));
    }
}

// Colour (cx, cy) on the rows jlo..jhi of the band (qn block rows).
template <typename S, bool YP>
MGW_FN void block_color(const window<S, true, YP> &V, block_walk w, int qn, int jlo, int jhi, int cx, int cy,
                        bool from_zero) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    for (; w.q < qn; w.next()) {
        const int lr = 2 * w.q + cy, j = V.jb + lr;
        if (j < jlo || j > jhi) continue;
        const float4 *s = V.st + V.cls[V.wrapped(j)] * (10 * num<S>::quads);
        const columns3 c(w.k, w.P, cx);
        const plane<S> row = V.z + lr * V.W;
        const bool rows = !(from_zero && cy == 0);
        const val2<S> bb = V.b.get(lr * V.W + c.c);
        typename acc_of<S>::type ax, ay;
        offdiag3<S>(s, row, V.W, c, rows && V.has_below(j), !(from_zero && cx == 0), rows && V.has_above(j), ax, ay);
        row.set(c.c, apply(s, 9, val2<S>{sub(bb.x, ax.done()), sub(bb.y, ay.done())}));
    }
}

// Residual of the rows jlo..jhi (the odd columns of odd rows: zero): the three
// points of a block on different threads.
template <typename S, bool YP>
MGW_FN void block_residual(const window<S, true, YP> &V, int P, int qn, int jlo, int jhi, int tid, int nth) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    const int blocks = P * qn;
    const divider dv(P);
    for (int t = tid; t < 3 * blocks; t += nth) {
        const int e = t >= 2 * blocks ? 2 : (t >= blocks ? 1 : 0), i = t - e * blocks, q = dv.quot(i), k = i - q * P;
        const int cx = e & 1, cy = e >> 1, lr = 2 * q + cy, j = V.jb + lr;
        if (j < jlo || j > jhi) continue;
        const columns3 c(k, P, cx);
        const float4 *s = V.st + V.cls[V.wrapped(j)] * (10 * num<S>::quads);
        const plane<S> row = V.z + lr * V.W;
        const val2<S> bb = V.b.get(lr * V.W + c.c);
        typename acc_of<S>::type ax, ay;
        offdiag3<S>(s, row, V.W, c, V.has_below(j), true, V.has_above(j), ax, ay);
        madd(ax, ay, s, 4, row.get(c.c));
        const plane<S> r = V.r + (j - V.rb) * V.W;
        r.set(c.c, val2<S>{sub(bb.x, ax.done()), sub(bb.y, ay.done())});
        if (cy) r.set(P + k, val2<S>{});
    }
}

// Restriction to the coarse rows Jlo..Jhi: coarse point (J, k) under block
// (J - jb/2, k).
template <typename S, bool YP, typename Out>
MGW_FN void block_restrict(const window<S, true, YP> &V, block_walk w, int qn, int Jlo, int Jhi, Out out) {
    for (; w.q < qn; w.next()) {
        const int J = (V.jb >> 1) + w.q;
        if (J < Jlo || J > Jhi) continue;
        const columns3 c(w.k, w.P, 0);
        val2<S> a{};
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const int hy = V.halves(q, J);
            if (!hy) continue;
            const plane<S> row = V.r + (2 * J + q - 1 - V.rb) * V.W;
            const float w1 = (float)hy * 0.25f, w2 = (float)(2 * hy) * 0.25f;
            const val2<S> l = row.get(c.l), m = row.get(c.c), r = row.get(c.r);
            a.x = add(a.x, scale(l.x, w1));
            a.y = add(a.y, scale(l.y, w1));
            a.x = add(a.x, scale(m.x, w2));
            a.y = add(a.y, scale(m.y, w2));
            a.x = add(a.x, scale(r.x, w1));
            a.y = add(a.y, scale(r.y, w1));
        }
        out(J, w.k, a);
    }
}

// Prolongation on the rows jlo..jhi: crow(J) is the child's row J, col(k) and
// next(k) the places in it of the columns under block k and right of it.
template <typename S, bool YP, typename Row, typename Col, typename Next>
MGW_FN void block_prolong(const window<S, true, YP> &V, block_walk w, int qn, int jlo, int jhi, Row crow, Col col,
                          Next next) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    for (; w.q < qn; w.next()) {
        const int je = V.jb + 2 * w.q, J = je >> 1;
        if (je > jhi || je + 1 < jlo) continue;
        const int c0 = col(w.k), c1 = next(w.k);
        const bool even = je >= jlo, odd = je + 1 <= jhi;
        // an even line injects its last point into the last coarse one
        const bool inject = !YP && !(V.n & 1) && je + 1 == V.n - 1;
        val2<S> a0{}, a1{}, b0{}, b1{};
        if (even || !inject) {
            const plane<S> r = crow(J);
            a0 = r.get(c0);
            a1 = r.get(c1);
        }
        if (odd) {
            const plane<S> r = crow(J + 1);
            b0 = r.get(c0);
            b1 = r.get(c1);
        }
        const plane<S> z = V.z + 2 * w.q * V.W;
        if (even) {
            const val2<S> f = z.get(w.k), g = z.get(w.P + w.k);
            z.set(w.k, val2<S>{add(f.x, a0.x), add(f.y, a0.y)});
            z.set(w.P + w.k,
                  val2<S>{add(g.x, scale(add(a0.x, a1.x), 0.5f)), add(g.y, scale(add(a0.y, a1.y), 0.5f))});
        }
        if (odd) {
            const plane<S> y = z + V.W;
            const val2<S> f = y.get(w.k), g = y.get(w.P + w.k);
            val2<S> u, v;
            if (inject) {
                u = b0;
                v = val2<S>{scale(add(b0.x, b1.x), 0.5f), scale(add(b0.y, b1.y), 0.5f)};
            } else {
                u = val2<S>{add(scale(a0.x, 0.5f), scale(b0.x, 0.5f)), add(scale(a0.y, 0.5f), scale(b0.y, 0.5f))};
                v = val2<S>{add(scale(add(a0.x, a1.x), 0.25f), scale(add(b0.x, b1.x), 0.25f)),
                            add(scale(add(a0.y, a1.y), 0.25f), scale(add(b0.y, b1.y), 0.25f))};
            }
            y.set(w.k, val2<S>{add(f.x, u.x), add(f.y, u.y)});
            y.set(w.P + w.k, val2<S>{add(g.x, v.x), add(g.y, v.y)});
        }
    }
}

// Off-diagonal sums of the top level around a point (comp 0: the x equation).
template <typename S>
MGW_FN S top_off3(const top_consts<S> &o, const plane<S> &row, int W, const columns3 &c, int comp) {
    if (comp == 0)
        return three(o.Kmx, sum2(row.x(c.l), row.x(c.r)), o.my,
                     sum2(row.x(c.c - W), row.x(c.c + W)), o.qK,
                     cross4(row.y(c.l - W), row.y(c.r + W), row.y(c.r - W), row.y(c.l + W)));
    return three(o.mx, sum2(row.y(c.l), row.y(c.r)), o.Kmy,
                 sum2(row.y(c.c - W), row.y(c.c + W)), o.qK,
                 cross4(row.x(c.l - W), row.x(c.r + W), row.x(c.r - W), row.x(c.l + W)));
}

// One colour of the top level on the rows jlo..jhi: of the block's four nodes
// the x equation at the two with (i + j) & 1 == color, the y one at the others.
template <typename S, bool YP>
MGW_FN void block_top_color(const top_consts<S> &o, const window<S, true, YP> &V, block_walk w, int qn, int jlo, int jhi,
                            int color, bool from_zero) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    for (; w.q < qn; w.next()) {
#pragma unroll
        for (int cy = 0; cy < 2; cy++) {
            const int lr = 2 * w.q + cy, j = V.jb + lr;
            if (j < jlo || j > jhi) continue;
            const bool wall = j == 0 || j == V.n - 1;
            const int cxx = (cy ^ color) & 1;  // the column whose x equation is due
            const plane<S> row = V.z + lr * V.W, b = V.b + lr * V.W;
            const columns3 cx(w.k, w.P, cxx), cyc(w.k, w.P, cxx ^ 1);
            const S bx = b.x(cx.c), by = b.y(cyc.c);
            if (wall) {
                row.set_x(cx.c, mul(o.ibcxx, bx));
                row.set_y(cyc.c, mul(o.ibcyy, by));
            } else if (from_zero) {
                row.set_x(cx.c, mul(o.icxx, bx));
                row.set_y(cyc.c, mul(o.icyy, by));
            } else {
                const S ex = top_off3(o, row, V.W, cx, 0), ey = top_off3(o, row, V.W, cyc, 1);
                row.set_x(cx.c, mul(o.icxx, sub(bx, ex)));
                row.set_y(cyc.c, mul(o.icyy, sub(by, ey)));
            }
        }
    }
}

template <typename S, bool YP>
MGW_FN void block_top_residual(const top_consts<S> &o, const window<S, true, YP> &V, block_walk w, int qn, int jlo,
                               int jhi) {
    jlo = V.lo(jlo);
    jhi = V.hi(jhi);
    for (; w.q < qn; w.next()) {
#pragma unroll
        for (int cy = 0; cy < 2; cy++) {
            const int lr = 2 * w.q + cy, j = V.jb + lr;
            if (j < jlo || j > jhi) continue;
            const bool wall = j == 0 || j == V.n - 1;
            const plane<S> row = V.z + lr * V.W, b = V.b + lr * V.W;
            const columns3 cx(w.k, w.P, cy), cyc(w.k, w.P, cy ^ 1);
            val2<S> rx{}, ry{};
            if (!wall) {
                rx.x = sub(sub(b.x(cx.c), top_off3(o, row, V.W, cx, 0)), mul(o.cxx, row.x(cx.c)));
                ry.y = sub(sub(b.y(cyc.c), top_off3(o, row, V.W, cyc, 1)), mul(o.cyy, row.y(cyc.c)));
            }
            const plane<S> r = V.r + (j - V.rb) * V.W;
            r.set(cx.c, rx);
            r.set(cyc.c, ry);
        }
    }
}

// ---- distributed small levels ---------------------------------------------------
//
// The levels t .. d-1 of a V-cycle in the shared memory of a cluster of blocks
// (or one block), each cut into row bands, one per block, so that block c owns
// the coarse rows that restrict from its own fine rows; a band carries the
// halo rows that make its sweep, residual and restriction exact without an
// exchange inside a level, so a level costs one cluster barrier on the way
// down (the child's right-hand side, with its halo) and one on the way up (the
// child's solution).  From level d on the rest of the V-cycle (it starts from
// zero, so it is one linear map of d's right-hand side, coarsest solve
// included) is a matrix of float pairs laid out with the operators, its rows
// shared out over the blocks: ten levels' worth of dependent phases become
// one product.

constexpr int kMaxLevels = 17;
constexpr int kTopBelow = 4, kTopAbove = 4;  // halo rows of the top level: below y0, from y1 up
constexpr int kLevBelow = 2, kLevAbove = 4;  // of a coarse level (three are read; block rows are pairs)

template <typename S> struct small_level {
    typedef typename num<S>::node node;
    int m, n, homog, nst, ncls;
    const int *cls;     // global
    const float4 *st;   // global
    int ps;             // nodes of the band's arrays (their planes' stride)
    unsigned zo, bo;    // shared offsets of the band's z and b (level d: all of them, b as nodes)
    unsigned ho;        // the three rows of the solution beyond the band (levels above t)
    unsigned so, co;    // stencils and row classes (kNone: read from global memory)
    node *zg;           // global z, b (level t)
    const node *bg;
};

constexpr unsigned kNone = 0xffffffffu;

template <typename S> struct small_plan {
    int t, d, blocks, shift;  // blocks = 1 << shift
    int rs;                  // plane stride of the residual rows
    int top;                 // level t is the matrix-free top level
    int zero_start;          // its z starts from zero
    unsigned ro;             // residual rows of the level in hand
    unsigned bytes;
    const float4 *dense;     // row-major, per column node (x.hi, x.lo, y.hi, y.lo)
    double2 *sum;            // not null: the top level's result, times a power of
                             // two, is added to this iterate
    const pair_range *range;
    int unit;                // the tables are those of A 2^-unit
    top_consts<S> op;
    small_level<S> lv[kMaxLevels];
};

// First row of block c on level l: level d's cut scaled up, the line's end
// for c == blocks.  A bounded line of even n has a coarse row beyond its last
// one, so the scaled cut of the last block can lie beyond the line's end (8 rows
// of level d cut into 8 over 50 rows: 7 << 3); its band is empty then, and what it
// owns of the coarser levels it computes from its halo rows.
template <typename S> MGW_BOTH int band_row(const small_plan<S> &P, int l, int c) {
    const int n = P.lv[l].n, row = ((c * P.lv[P.d].n) >> P.shift) << (P.d - l);
    return c >= P.blocks || row > n ? n : row;
}
template <typename S> MGW_BOTH int band_below(const small_plan<S> &P, int l) {
    return P.top && l == P.t ? kTopBelow : kLevBelow;
}
template <typename S> MGW_BOTH int band_above(const small_plan<S> &P, int l) {
    return P.top && l == P.t ? kTopAbove : kLevAbove;
}

// FAST: every level t .. d-1 is an even line with one class per row and its
// tables in shared memory (known at compile time).
template <bool FAST, bool YP, typename S>
MGW_FN window<S, true, YP> band_window(const small_plan<S> &P, int l, int c, unsigned char *base) {
    const small_level<S> &L = P.lv[l];
    window<S, true, YP> V;
    V.z = plane<S>{reinterpret_cast<S *>(base + L.zo), L.ps};
    V.b = plane<S>{reinterpret_cast<S *>(base + L.bo), L.ps};
    V.r = plane<S>{reinterpret_cast<S *>(base + P.ro), P.rs};
    V.W = V.m = L.m;
    V.He = (L.m + 1) >> 1;
    V.n = L.n;
    const int y0 = band_row(P, l, c);
    V.jb = y0 - band_below(P, l);
    V.rb = y0 - 1;
    V.x0 = 0;
    V.homog = L.homog;
    if (FAST) {
        V.st = reinterpret_cast<const float4 *>(base + L.so);
        V.cls = reinterpret_cast<const int *>(base + L.co);
    } else {
        V.st = L.so != kNone ? reinterpret_cast<const float4 *>(base + L.so) : L.st;
        V.cls = L.co != kNone ? reinterpret_cast<const int *>(base + L.co) : L.cls;
    }
    return V;
}

MGW_FN ff as_pair(float a) { return ff{a, 0.f}; }
MGW_FN ff as_pair(ff a) { return a; }
MGW_FN float from_pair(ff a, float) { return a.hi + a.lo; }
MGW_FN ff from_pair(ff a, ff) { return a; }

#ifdef __CUDACC__
// The sum of a pair over a warp, on every lane.
MGW_FN ff warp_pair_sum(ff a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ff b;
        b.hi = __shfl_xor_sync(0xffffffffu, a.hi, o);
        b.lo = __shfl_xor_sync(0xffffffffu, a.lo, o);
        a = ff_add(a, b);
    }
    return a;
}
#endif

// This lane's shares of up to R rows of the dense levels' product, `stride`
// rows apart (nr of them exist): all rows' loads are in flight together.
template <int LANES, int R, typename S>
MGW_FN void dense_share(const float4 *row, size_t stride, int nr, const typename num<S>::node *b, int nd, int lane,
                        ff (&out)[R]) {
    ffacc a[R];
#pragma unroll 3
    for (int k = lane; k < nd; k += LANES) {
        const val2<S> v = get(b[k]);
#pragma unroll
        for (int q = 0; q < R; q++) {
            const float4 *p = row + (q < nr ? q * stride : 0) + k;
#ifdef __CUDACC__
            const float4 M = __ldg(p);
#else
            const float4 M = *p;
#endif
            a[q].mad(ff{M.x, M.y}, as_pair(v.x));
            a[q].mad(ff{M.z, M.w}, as_pair(v.y));
        }
    }
#pragma unroll
    for (int q = 0; q < R; q++) out[q] = a[q].done();
}
constexpr int kDenseRows = 3;  // 34 rows per block of sixteen warps at 17 x 16 nodes

// The V-cycle on the levels of the plan.  E: the block's environment -
// rank(), local() and base(rank) (a block's shared memory, this or another
// one's), par(f) (f(thread, threads) on every thread, then a block barrier),
// csync() (a barrier of all blocks), kLanes and lane_sum(v) (threads of a
// product row and the sum over them), ld(p) (a global load), store(P, k, v)
// (the result of level t at its node k), wait_input(P) (before the first read
// of what an earlier kernel wrote).  kMeasured: the largest magnitude of level
// t's b is taken before b is loaded, each thread with measure(p), each block
// with measured() and, on one thread per block of the cluster, share(thread, nb).
template <bool FAST, bool YP, typename S, typename E> MGW_FN void small_vcycle(const small_plan<S> &P, E &env) {
    typedef typename num<S>::node node;
    const int me = env.rank(), nb = P.blocks;
    unsigned char *base = env.local();
    const small_level<S> &D = P.lv[P.d];
    const node *bd = reinterpret_cast<const node *>(base + D.bo);
    const plane<S> zd{reinterpret_cast<S *>(base + D.zo), D.ps};
    // level t's own and halo rows of b (and z)
    auto load = [&](int tid, int nth) {
        const small_level<S> &L = P.lv[P.t];
        const window<S, true, YP> V = band_window<FAST, YP>(P, P.t, me, base);
        const int y1 = band_row(P, P.t, me + 1);
        const int lo = V.lo(V.jb), hi = V.hi(y1 + band_above(P, P.t) - 1) + 1;
        const int total = (hi - lo) * L.m;
        const divider dv(L.m);
        for (int k = tid; k < total; k += nth) {
            const int q = dv.quot(k), j = lo + q, w = k - q * L.m;
            V.b.set(V.at(j, w), get(env.ld(L.bg + (size_t)V.wrapped(j) * L.m + w)));
            if (P.top && !P.zero_start) V.z.set(V.at(j, w), get(env.ld(L.zg + (size_t)V.wrapped(j) * L.m + w)));
        }
    };
    // the tables
    env.par([&](int tid, int nth) {
        for (int l = P.t; l < P.d; l++) {
            const small_level<S> &L = P.lv[l];
            if (L.so != kNone) {
                float4 *d = reinterpret_cast<float4 *>(base + L.so);
                for (int k = tid; k < L.nst * 10 * num<S>::quads; k += nth) d[k] = L.st[k];
            }
            if (L.co != kNone) {
                int *d = reinterpret_cast<int *>(base + L.co);
                for (int k = tid; k < L.ncls; k += nth) d[k] = L.cls[k];
            }
        }
        env.wait_input(P);
        if (!E::kMeasured) load(tid, nth);
    });
    if (nb > 1) env.csync();  // every block runs: its shared memory may be written
    if (E::kMeasured) {
        env.par([&](int tid, int nth) {
            const int m = P.lv[P.t].m, y0 = band_row(P, P.t, me), y1 = band_row(P, P.t, me + 1);
            const node *b = P.lv[P.t].bg + (size_t)y0 * m;
            for (int k = tid; k < (y1 - y0) * m; k += nth) env.measure(b + k);
            env.measured();
        });
        env.par([&](int tid, int nth) { env.share(tid, nb); });
        if (nb > 1) env.csync();
        env.par(load);
    }
    // down
    for (int l = P.t; l < P.d; l++) {
        const window<S, true, YP> V = band_window<FAST, YP>(P, l, me, base);
        const int y0 = band_row(P, l, me), y1 = band_row(P, l, me + 1), cm = P.lv[l + 1].m;
        const int qn = (y1 - V.jb + band_above(P, l) + 1) >> 1;
        const bool top = P.top && l == P.t;
        if (FAST) {
            const block_walk w(env.thread(), env.threads(), V.W >> 1);
            if (top) {
                env.par([&](int tid, int nth) {
                    block_top_color(P.op, V, env.walk(w, tid, nth), qn, y0 - 3, y1 + 2, 0, P.zero_start != 0);
                });
                env.par([&](int tid, int nth) {
                    block_top_color(P.op, V, env.walk(w, tid, nth), qn, y0 - 2, y1 + 1, 1, false);
                });
                env.par([&](int tid, int nth) {
                    block_top_residual(P.op, V, env.walk(w, tid, nth), qn, y0 - 1, y1 - 1);
                });
            } else {
#pragma unroll 1
                for (int c = 0; c < 4; c++)
                    env.par([&](int tid, int nth) {
                        block_color(V, env.walk(w, tid, nth), qn, y0 - 2 + (c >> 1), y1 + 2 - (c >> 1), c & 1, c >> 1,
                                    true);
                    });
                env.par([&](int tid, int nth) { block_residual(V, V.W >> 1, qn, y0 - 1, y1 - 1, tid, nth); });
            }
        } else if (top) {
            env.par([&](int tid, int nth) {
                top_color(P.op, V, y0 - 3, y1 + 2, 0, 0, 0, P.zero_start != 0, tid, nth);
            });
            env.par([&](int tid, int nth) { top_color(P.op, V, y0 - 2, y1 + 1, 0, 0, 1, false, tid, nth); });
            env.par([&](int tid, int nth) { top_residual(P.op, V, y0 - 1, y1 - 1, 0, 0, tid, nth); });
        } else {
            const int ncx = (V.m & 1) ? 3 : 2;
#pragma unroll 1
            for (int cy = 0; cy < 2; cy++)
#pragma unroll 1
                for (int cx = 0; cx < ncx; cx++)
                    env.par([&](int tid, int nth) {
                        if (ncx == 3 && cy == 0 && cx == 0) lev_clear_last(V, y0 - 2, y1 + 2, tid, nth);
                        lev_color(V, y0 - 2 + cy, y1 + 2 - cy, 0, 0, cx, cy, true, tid, nth);
                    });
            env.par([&](int tid, int nth) { lev_residual(V, y0 - 1, y1 - 1, 0, 0, tid, nth); });
        }
        // restriction: the child's own rows, and to every block whose band
        // (with its halo) holds the row; level d goes to all of them
        const int J0 = band_row(P, l + 1, me), J1 = band_row(P, l + 1, me + 1);
        env.par([&](int tid, int nth) {
            if (l + 1 < P.d) {
                const window<S, true, YP> CV = band_window<FAST, YP>(P, l + 1, me, base);
                const int He = CV.He;
                S *to[4];  // b of the neighbours at distance -2, -1, 1, 2, shifted to absolute rows
                int lo[4], hi[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    int c = me + (q < 2 ? q - 2 : q - 1), turn = 0;
                    lo[q] = 1;
                    hi[q] = 0;
                    to[q] = nullptr;
                    if (YP) {  // the bands go round
                        while (c < 0) c += nb, turn -= P.lv[l + 1].n;
                        while (c >= nb) c -= nb, turn += P.lv[l + 1].n;
                    }
                    if (c < 0 || c >= nb) continue;
                    lo[q] = band_row(P, l + 1, c) - kLevBelow + turn;
                    hi[q] = band_row(P, l + 1, c + 1) + kLevAbove - 2 + turn;  // the last row a sweep reads
                    if (lo[q] >= J1 || hi[q] < J0) hi[q] = lo[q] - 1;
                    else to[q] = reinterpret_cast<S *>((c == me ? base : env.base(c)) + P.lv[l + 1].bo);
                }
                auto out = [&](int J, int I, const val2<S> &v) {
                    const int c = (I & 1) * He + (I >> 1);
                    CV.b.set((J - CV.jb) * cm + c, v);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (J >= lo[q] && J <= hi[q]) plane<S>{to[q], CV.b.ps}.set((J - lo[q]) * cm + c, v);
                };
                if (FAST) block_restrict(V, block_walk(tid, nth, V.W >> 1), qn, J0, J1 - 1, out);
                else restrict_rows(V, J0, J1 - 1, 0, cm - 1, cm, out, tid, nth);
            } else {
                auto out = [&](int J, int I, const val2<S> &v) {
                    const node o = put(v);
                    for (int c = 0; c < nb; c++)
                        reinterpret_cast<node *>((c == me ? base : env.base(c)) + D.bo)[J * cm + I] = o;
                };
                if (FAST) block_restrict(V, block_walk(tid, nth, V.W >> 1), qn, J0, J1 - 1, out);
                else restrict_rows(V, J0, J1 - 1, 0, cm - 1, cm, out, tid, nth);
            }
        });
        if (nb > 1) env.csync();
    }
    // level d: z = M b, a group of threads per row, the result to every block
    env.par([&](int tid, int nth) {
        const int nd = D.m * D.n, r0 = 2 * (int)((long)nd * me / nb), r1 = 2 * (int)((long)nd * (me + 1) / nb);
        const int lane = tid % E::kLanes, groups = nth / E::kLanes;
        for (int r = r0 + tid / E::kLanes; r < r1; r += kDenseRows * groups) {
            const int nr = imin(kDenseRows, (r1 - r + groups - 1) / groups);
            ff v[kDenseRows];
            dense_share<E::kLanes, kDenseRows, S>(P.dense + (size_t)r * nd, (size_t)groups * nd, nr, bd, nd, lane, v);
#pragma unroll
            for (int q = 0; q < kDenseRows; q++) v[q] = env.lane_sum(v[q]);
#pragma unroll
            for (int q = 0; q < kDenseRows; q++) {
                const int rr = r + q * groups;
                if (q >= nr) break;
                const S o = from_pair(v[q], S());
                for (int c = lane; c < nb; c += E::kLanes) {
                    const plane<S> z{reinterpret_cast<S *>((c == me ? base : env.base(c)) + D.zo), D.ps};
                    if (rr & 1) z.set_y(rr >> 1, o);
                    else z.set_x(rr >> 1, o);
                }
            }
        }
    });
    if (nb > 1) env.csync();
    // up
    for (int l = P.d - 1; l >= P.t; l--) {
        const window<S, true, YP> V = band_window<FAST, YP>(P, l, me, base);
        const int y0 = band_row(P, l, me), y1 = band_row(P, l, me + 1), cm = P.lv[l + 1].m;
        const int qn = (y1 - V.jb + band_above(P, l) + 1) >> 1;
        const bool top = P.top && l == P.t, last = l + 1 == P.d;
        const window<S, true, YP> CV = band_window<FAST, YP>(P, l + 1, me, base);
        const int J0 = band_row(P, l + 1, me), J1 = band_row(P, l + 1, me + 1), cHe = CV.He;
        const plane<S> halo{reinterpret_cast<S *>(base + (last ? 0u : P.lv[l + 1].ho)), 3 * cm};
        auto crow = [&](int J) -> plane<S> {
            if (last) return zd + CV.wrapped(J) * cm;
            if (J < J0) return halo;
            if (J >= J1) return halo + (1 + J - J1) * cm;
            return CV.z + (J - CV.jb) * cm;
        };
        auto ccol = [&](int I) { return last ? I : (I & 1) * cHe + (I >> 1); };
        if (FAST) {
            const block_walk w(env.thread(), env.threads(), V.W >> 1);
            env.par([&](int tid, int nth) {
                block_prolong(V, env.walk(w, tid, nth), qn, y0 - (top ? 2 : 1), y1 + 1, crow, ccol,
                              [&](int k) { return ccol(k + 1 == cm ? 0 : k + 1); });
            });
            if (top) {
                env.par([&](int tid, int nth) {
                    block_top_color(P.op, V, env.walk(w, tid, nth), qn, y0 - 1, y1, 0, false);
                });
                env.par([&](int tid, int nth) {
                    block_top_color(P.op, V, env.walk(w, tid, nth), qn, y0, y1 - 1, 1, false);
                });
            } else {
#pragma unroll 1
                for (int c = 0; c < 4; c++)
                    env.par([&](int tid, int nth) {
                        block_color(V, env.walk(w, tid, nth), qn, y0, y1 - (c >> 1), c & 1, c >> 1, false);
                    });
            }
        } else {
            env.par([&](int tid, int nth) {
                prolong_rows(V, y0 - (top ? 2 : 1), y1 + 1, 0, 0, cm,
                             [&](int J, int I) { return crow(J).get(ccol(I)); }, tid, nth);
            });
            if (top) {
                env.par([&](int tid, int nth) { top_color(P.op, V, y0 - 1, y1, 0, 0, 0, false, tid, nth); });
                env.par([&](int tid, int nth) { top_color(P.op, V, y0, y1 - 1, 0, 0, 1, false, tid, nth); });
            } else {
                const int ncx = (V.m & 1) ? 3 : 2;
#pragma unroll 1
                for (int cy = 0; cy < 2; cy++)
#pragma unroll 1
                    for (int cx = 0; cx < ncx; cx++)
                        env.par([&](int tid, int nth) {
                            lev_color(V, y0, y1 - cy, 0, 0, cx, cy, false, tid, nth);
                        });
            }
        }
        if (l == P.t) {
            env.par([&](int tid, int nth) {
                const int total = (y1 - y0) * V.m;
                const divider dv(V.m);
                for (int k = tid; k < total; k += nth) {
                    const int q = dv.quot(k), w = k - q * V.m;
                    env.store(P, (size_t)(y0 + q) * V.m + w, put(V.z.get(V.at(y0 + q, w))));
                }
            });
        } else if (nb > 1 || YP) {
            // rows next to the band's edges, for the neighbours' prolongation
            env.par([&](int tid, int nth) {
                const int m = V.m;
                const int below = YP && me == 0 ? nb - 1 : me - 1, above = YP && me + 1 == nb ? 0 : me + 1;
                S *lo = below >= 0 ? reinterpret_cast<S *>((below == me ? base : env.base(below)) + P.lv[l].ho) : nullptr;
                S *hi = above < nb ? reinterpret_cast<S *>((above == me ? base : env.base(above)) + P.lv[l].ho) : nullptr;
                for (int k = tid; k < 2 * m; k += nth) {  // both components
                    const int c = k < m ? k : k - m, from = k < m ? 0 : V.z.ps, to = k < m ? 0 : 3 * m;
                    const S *z = V.z.p + from + c;
                    if (lo) {
                        lo[to + m + c] = z[(y0 - V.jb) * m];
                        lo[to + 2 * m + c] = z[(y0 + 1 - V.jb) * m];
                    }
                    if (hi) hi[to + c] = z[(y1 - 1 - V.jb) * m];
                }
            });
            if (nb > 1) env.csync();
        }
    }
}

}  // namespace mgw
}  // namespace stzg
