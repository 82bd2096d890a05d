// Time-step kernels: fused ENO advection + STZ plasticity, chi diffusion,
// projection source, stress correction and boundaries.
#include "ff.cuh"
#include "fixed.cuh"
#include "step.cuh"
#include "stz_law.cuh"

#include <algorithm>
#include <cmath>

namespace stzg {

// x = hi + lo as floats on the host (hi the nearest float, lo the nearest
// float of the remainder): the float-float form of a launch constant.
void split_host(double x, float *hi, float *lo) {
    *hi = (float)x;
    *lo = (float)(x - (double)*hi);
}

step_consts make_step_consts(const stz_params &p) {
    step_consts c;
    c.m = p.m;
    c.n = p.n;
    c.ax = p.ax;
    c.ay = p.ay;
    c.by = p.by;
    c.lx = p.bx - p.ax;
    c.dx = c.lx / p.m;
    c.dy = (p.by - p.ay) / p.n;
    c.xsp = 1. / c.dx;
    c.ysp = 1. / c.dy;
    c.mu = p.mu;
    c.K = p.K;
    c.stz_model = p.stz_model;
    c.t_model = p.t_model;
    c.t_scale = p.t_scale;
    c.adapt_fac = p.adapt_fac;
    c.chi_inf = p.chi_inf;
    c.s_y = p.s_y;
    c.theta = p.theta;
    c.Delta = p.Delta;
    c.Omegaeps0 = p.Omegaeps0;
    c.tau0 = p.tau0;
    c.c0 = p.c0;
    c.kappa = p.kappa;
    c.rho = p.rho;
    c.chi_diff = p.chi_diff;
    c.chi_len = p.chi_len;
    c.track_plastic = 0;
    c.substep_cap = 1 << 22;
    c.yield_cut2 = p.s_y * p.s_y * (1 - 1e-12);
    c.yield_cut2f = (float)(c.yield_cut2 * (1 - 1e-6));
    c.clock = nullptr;
    c.xbc = 0;
    c.sp_increments = 0;
    c.fixed_point = 0;
    return c;
}

namespace {

struct velo {
    const double2 *vel;
    int m, n;
    double bv;
    __device__ __forceinline__ double u(int i, int j) const {
        return j == 0 ? -bv : (j == n ? bv : vel[(size_t)j * m + i].x);
    }
    __device__ __forceinline__ double v(int i, int j) const {
        return (j == 0 || j == n) ? 0.0 : vel[(size_t)j * m + i].y;
    }
};

#define IDX(i, j) ((size_t)((j) + 1) * m + (i))

// Fused advection + STZ step over a tile of ATX x ATY cells (i,j) and their
// lower-left nodes.
//
// ENO2 through shared differences: on a line f, the first differences
// D(c+1/2) = f(c+1) - f(c) and second differences S(c) = D(c+1/2) - D(c-1/2)
// are computed once per tile (with a halo) into shared memory, and each
// point's ENO2 value is one FMA on them:
//   upwind from the left:  eno2 = 2 D(i-1/2) + (|S(i)| > |S(i-1)| ? S(i-1) : S(i))
//   upwind from the right: eno2 = -2 D(i+1/2) + (|S(i)| > |S(i+1)| ? S(i+1) : S(i))
// These are the values of eno2(p0..p3) in step.cuh operation for operation
// (p0 - p1, p1 - p2 and p2 - p3 are the D's up to exact negations, and
// (-a) - (-b) rounds as b - a), so the result is the same double.  A point
// costs three FP64 operations per direction plus its share of the tile's
// halo instead of six.  The reference map X is unwrapped across the periodic
// seam by the column's offset (+-lx) before differencing, as the per-point
// form adds it to each shifted value.
constexpr int ATX = 32, ATY = 8;
constexpr int ADXW = ATX + 3;  // D(c+1/2), tile columns c = -2..ATX
constexpr int ASXW = ATX + 2;  // S(c), c = -1..ATX
constexpr int ADYH = ATY + 3;  // D(r+1/2), tile rows r = -2..ATY
constexpr int ASYH = ATY + 2;  // S(r), r = -1..ATY
constexpr int ACOLS = ATX + 4; // tile columns -2..ATX+1

__device__ __forceinline__ double eno_left(const double *d, const double *s, int k) {
    // d[k] = D(i-1/2), s[k] = S(i), s[k-1] = S(i-1)
    const double s0 = s[k], s1 = s[k - 1];
    return fma(2.0, d[k], mag_gt(s0, s1) ? s1 : s0);
}
__device__ __forceinline__ double eno_right(const double *d, const double *s, int k) {
    // d[k+1] = D(i+1/2), s[k] = S(i), s[k+1] = S(i+1)
    const double s0 = s[k], s1 = s[k + 1];
    return fma(-2.0, d[k + 1], mag_gt(s0, s1) ? s1 : s0);
}

template <int NF> struct eno_tile {
    double dx[NF][ATY][ADXW];
    double dy[NF][ADYH][ATX];
    double sx[NF][ATY][ASXW];
    double sy[NF][ASYH][ATX];
    double xo[ACOLS];  // X offset of the unwrapped column
    int col[ACOLS];    // storage column of tile column c-2
};
typedef eno_tile<F_COUNT> adv_tile;

// Storage column and X offset of every tile column (unwrapped column
// i0 + t - 2 for t = 0..ACOLS-1); threads 0..ACOLS-1 write them.
template <int NF> __device__ __forceinline__ void tile_columns(eno_tile<NF> &T, int i0, int m, double lx) {
    const int tid = threadIdx.y * ATX + threadIdx.x;
    if (tid < ACOLS) {
        const int u = i0 + tid - 2;  // unwrapped column
        int w = u % m;
        if (w < 0) w += m;
        T.col[tid] = w;
        T.xo[tid] = u < 0 ? -lx : (u >= m ? lx : 0.0);
    }
}

// Fills the tile's first and second differences of NF fields over cell rows
// j0..j0+ATY-1 (x) and rows j0-2..j0+ATY+1 (y), after tile_columns and a
// barrier.  get(f, row, t) reads field f at row -1..n and tile column t;
// rows below low(f) (-1 for the stored fields, 0 for the node velocity) and
// above n hold no value, and the differences that would need them are never
// used.  Field xf (the reference map X) is unwrapped across the periodic
// seam.  Ends with __syncthreads.
template <int NF, typename Get, typename Low>
__device__ __forceinline__ void tile_differences(eno_tile<NF> &T, int i0, int j0, int m, int n, int xf, Get get,
                                                 Low low) {
    const int tid = threadIdx.y * ATX + threadIdx.x;
    for (int k = tid; k < NF * ATY * ADXW; k += ATX * ATY) {
        const int f = k / (ATY * ADXW), rem = k - f * (ATY * ADXW), r = rem / ADXW, cc = rem - r * ADXW;
        const int jj = j0 + r;
        double d = 0;
        if (jj < n) {
            double hi = get(f, jj, cc + 1), lo = get(f, jj, cc);
            if (f == xf) {
                if (T.xo[cc + 1] != 0) hi += T.xo[cc + 1];
                if (T.xo[cc] != 0) lo += T.xo[cc];
            }
            d = hi - lo;
        }
        T.dx[f][r][cc] = d;
    }
    for (int k = tid; k < NF * ADYH * ATX; k += ATX * ATY) {
        const int f = k / (ADYH * ATX), rem = k - f * (ADYH * ATX), r = rem / ATX, cc = rem - r * ATX;
        const int jj = j0 + r - 2, ii = i0 + cc;
        double d = 0;
        if (jj >= low(f) && jj + 1 <= n && ii < m) d = get(f, jj + 1, cc + 2) - get(f, jj, cc + 2);
        T.dy[f][r][cc] = d;
    }
    __syncthreads();
    for (int k = tid; k < NF * ATY * ASXW; k += ATX * ATY) {
        const int f = k / (ATY * ASXW), rem = k - f * (ATY * ASXW), r = rem / ASXW, cc = rem - r * ASXW;
        T.sx[f][r][cc] = T.dx[f][r][cc + 1] - T.dx[f][r][cc];
    }
    for (int k = tid; k < NF * ASYH * ATX; k += ATX * ATY) {
        const int f = k / (ASYH * ATX), rem = k - f * (ASYH * ATX), r = rem / ATX, cc = rem - r * ATX;
        T.sy[f][r][cc] = T.dy[f][r + 1][cc] - T.dy[f][r][cc];
    }
    __syncthreads();
}

// ENO2 values of a point at tile column tx / row ty from the tile (the
// factor hs is applied by the caller).
template <int NF>
__device__ __forceinline__ double tile_eno_x(const eno_tile<NF> &T, int f, int ty, int tx, bool from_left) {
    const double *d = T.dx[f][ty], *s = T.sx[f][ty];
    const int k = tx + 1;
    return from_left ? eno_left(d, s, k) : eno_right(d, s, k);
}
// y direction with the one-sided wall rows: `inner` is false on the last row
// before the wall on the upwind side.
template <int NF>
__device__ __forceinline__ double tile_eno_y(const eno_tile<NF> &T, int f, int ty, int tx, bool from_below,
                                             bool inner) {
    const int ky = ty + 1;
    const double s0 = T.sy[f][ky][tx];
    if (from_below) {
        const double d = T.dy[f][ky][tx];
        if (!inner) return 2 * d;
        const double s1 = T.sy[f][ky - 1][tx];
        return fma(2.0, d, mag_gt(s0, s1) ? s1 : s0);
    }
    const double d = T.dy[f][ky + 1][tx];
    if (!inner) return -2 * d;
    const double s1 = T.sy[f][ky + 1][tx];
    return fma(-2.0, d, mag_gt(s0, s1) ? s1 : s0);
}

// ---- TMA staging of the field tiles -----------------------------------------
// Rows of the staged tile: cell rows j0-2..j0+ATY+1 (storage rows j0-1..).
constexpr int AROWS = ATY + 4;
constexpr unsigned kTileBytes = F_COUNT * AROWS * ACOLS * sizeof(double);
// Iterations of the bounded wait on the tile copies (each try_wait itself
// suspends for a while); past it the block flags F.flags[FL_TMA].
constexpr int kTmaWaitIters = 1 << 20;

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// 2D tiled TMA load of box (x, y) of `map` into dst, completing on bar.
// x (the column) must be even for FP64 (16-byte rule); it and y may lie
// outside the tensor, whose missing elements arrive as zeros.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_addr(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// Bounded wait for a phase of bar; false when it ran out.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity = 0) {
    for (int it = 0; it < kTmaWaitIters; it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// Per-launch constants of the step that depend on dt (computed on the host
// with the same operations the per-thread code used).
struct advect_consts {
    double hx, hy;  // dt/(2 dx), dt/(2 dy)
    double xf, yf;  // 1/(2 dt dx), 1/(2 dt dy) of projection_step
};

struct adv_smem {
    double tile[F_COUNT][AROWS][ACOLS];  // staged fields, first: 128-byte aligned
    adv_tile T;
    uint64_t bar;
};

// The per-cell combinations of the advected stress (fields_dev::pre).
__device__ __forceinline__ void write_pre(const fields_dev &F, size_t ci, double xf, double yf, double pn, double qn,
                                          double sn, double tn) {
    const double pq = pn + qn, Aa = pq - sn, Bb = pq + sn;
    F.pre[0][ci] = xf * Aa + yf * tn;
    F.pre[1][ci] = xf * Aa - yf * tn;
    F.pre[2][ci] = xf * tn - yf * Bb;
    F.pre[3][ci] = xf * tn + yf * Bb;
}

// One tile (bx, by) in FP64; `use`: how often the block has done this before
// (the barrier's phase).  False when a tile copy did not arrive.
__device__ __forceinline__ bool advect_tile(const step_consts &c, const advect_consts &a, const field_boxes &maps,
                                            const fields_dev &F, int cur, double dt, double bv, int emit_source, int bx,
                                            int by, unsigned use) {
    extern __shared__ __align__(128) unsigned char adv_raw[];
    adv_smem &Sm = *reinterpret_cast<adv_smem *>(adv_raw + ((128 - (smem_addr(adv_raw) & 127)) & 127));
    adv_tile &T = Sm.T;
    const int m = c.m, n = c.n;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * ATX + tx;
    const int i0 = bx * ATX, j0 = by * ATY;
    const int i = i0 + tx, j = j0 + ty;
    const double *__restrict__ const *A = F.f[cur];
    double *const *B = F.f[cur ^ 1];
    // One thread copies the seven field tiles (columns i0-2.., storage rows
    // j0-1..) by TMA while the block sets up the column tables.
    if (tid == 0 && use == 0) mbar_init(&Sm.bar, 1);
    tile_columns(T, i0, m, c.lx);
    // the last tile's stores to the copies' destination, before the next copies
    if (use) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(&Sm.bar, kTileBytes);
        for (int f = 0; f < F_COUNT; f++) tma_load_2d(&Sm.tile[f][0][0], &maps.f[cur][f], i0 - 2, j0 - 1, &Sm.bar);
    }
    if (__syncthreads_or(!mbar_wait_bounded(&Sm.bar, use & 1))) {
        // a copy did not arrive in time: flag it, wait once more for the
        // copies in flight, and leave this tile of the next state unwritten
        if (tid == 0) atomicExch(&F.flags[FL_TMA], 1);
        mbar_wait_bounded(&Sm.bar, use & 1);
        return false;
    }
    // Columns across the periodic seam arrive as zeros: blocks at either end
    // fetch them from their wrapped columns.
    if (i0 == 0 || i0 + ACOLS - 2 > m) {
        for (int k = tid; k < F_COUNT * AROWS * ACOLS; k += ATX * ATY) {
            const int f = k / (AROWS * ACOLS), rem = k - f * (AROWS * ACOLS), r = rem / ACOLS, t = rem - r * ACOLS;
            const int u = i0 + t - 2, sr = j0 - 1 + r;
            if ((u < 0 || u >= m) && sr >= 0 && sr <= n + 1) Sm.tile[f][r][t] = A[f][(size_t)sr * m + T.col[t]];
        }
        __syncthreads();
    }
    tile_differences<F_COUNT>(
        T, i0, j0, m, n, F_X, [&](int f, int row, int t) { return Sm.tile[f][row - j0 + 2][t]; },
        [](int) { return -1; });
    if (i >= m || j >= n) return true;
    const double hx = a.hx, hy = a.hy;
    const size_t ci = (size_t)(j + 1) * m + i;
    const int ir = T.col[tx + 3];
    if (c.clock) bv = c.clock[CLK_BV_STATE];
    velo V{F.vel, m, n, bv};
    // Upwind ENO values without the factor hs = +-dt/(2 dx); it is folded
    // into the velocity: -u * (hs * eno) = -(u * hs) * eno.
    // reference map at node (i,j), rows 1..n-1 (shear_sim.cc:310-327)
    if (j > 0) {
        const double Xc = Sm.tile[F_X][ty + 2][tx + 2], Yc = Sm.tile[F_Y][ty + 2][tx + 2];
        double ex_X, ex_Y, ey_X, ey_Y;
        const double un = V.u(i, j), vn = V.v(i, j);
        const double uh = un * (un > 0 ? hx : -hx), vh = vn * (vn > 0 ? hy : -hy);
        ex_X = tile_eno_x(T, F_X, ty, tx, un > 0);
        ex_Y = tile_eno_x(T, F_Y, ty, tx, un > 0);
        const bool inner = vn > 0 ? j > 1 : j < n - 1;
        ey_X = tile_eno_y(T, F_X, ty, tx, vn > 0, inner);
        ey_Y = tile_eno_y(T, F_Y, ty, tx, vn > 0, inner);
        B[F_X][ci] = Xc + fma(-vh, ey_X, -uh * ex_X);
        B[F_Y][ci] = Yc + fma(-vh, ey_Y, -uh * ex_Y);
    }
    // staggered velocity and spin (shear_sim.cc:330-333)
    const double u00 = V.u(i, j), u10 = V.u(ir, j), u01 = V.u(i, j + 1), u11 = V.u(ir, j + 1);
    const double v00 = V.v(i, j), v10 = V.v(ir, j), v01 = V.v(i, j + 1), v11 = V.v(ir, j + 1);
    const double uc = 0.25 * (u00 + u10 + u01 + u11), vc = 0.25 * (v00 + v10 + v01 + v11);
    const double two_omega = hx * (-v00 + v10 - v01 + v11) - hy * (-u00 - u10 + u01 + u11);
    const double uh = uc * (uc > 0 ? hx : -hx), vh = vc * (vc > 0 ? hy : -hy);
    // ENO derivatives of p, q, s, tau, chi (shear_sim.cc:336-338)
    double f1[5], f2[5];
    const bool inner = vc > 0 ? j > 0 : j < n - 1;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        f1[k] = tile_eno_x(T, k, ty, tx, uc > 0);
        f2[k] = tile_eno_y(T, k, ty, tx, vc > 0, inner);
    }
    const double p = Sm.tile[F_P][ty + 2][tx + 2], q = Sm.tile[F_Q][ty + 2][tx + 2];
    const double s = Sm.tile[F_S][ty + 2][tx + 2], t = Sm.tile[F_TAU][ty + 2][tx + 2];
    double cchi = Sm.tile[F_CHI][ty + 2][tx + 2] + fma(-vh, f2[4], -uh * f1[4]), ddev, dtmp;
    const double devsq = 3 * q * q + s * s + t * t;
    // Cells far enough below the cut-offs return exactly ddev = 0 and leave
    // chi unchanged in the reference loop (sbar < 1e-12, or an athermal law
    // below yield); they skip the FP64 square root and the loop.  The margin
    // keeps the test exact under the rounding of sqrt.
    // devsq >= 0, so the cut-offs compare as integers on the bit patterns
    const bool athermal = c.stz_model >= 2;
    const long long dbits = __double_as_longlong(devsq);
    if (dbits < __double_as_longlong(0.999e-24) || (athermal && dbits < __double_as_longlong(c.yield_cut2))) {
        ddev = 0;
        dtmp = 0;
    } else {
        int iters;
        const stz_law_params<double> lp = law_params(c);
        dtmp = adaptive_plastic(lp, sqrt(devsq), cchi, ddev, dt, iters);
        if (iters >= c.substep_cap) atomicExch(&F.flags[0], 1);
        if (iters > 1) atomicMax(&F.flags[1], iters);
    }
    B[F_CHI][ci] = cchi;
    F.ddev[ci] = ddev;
    if (c.track_plastic && ddev != 0) F.eps_pl[(size_t)j * m + i] += ddev / (2 * c.mu);
    const double pn = p + fma(-vh, f2[0], -uh * f1[0]);
    // dtmp is exactly 0 outside plastic flow; the terms - dtmp * (q, s, t)
    // then add exact zeros and are skipped
    double qn, sn, tn;
    if (dtmp != 0) {
        qn = q + (fma(-vh, f2[1], -uh * f1[1]) - dtmp * q);
        sn = s + (fma(-vh, f2[2], -uh * f1[2]) + two_omega * t - dtmp * s);
        tn = t + (fma(-vh, f2[3], -uh * f1[3]) - two_omega * s - dtmp * t);
    } else {
        qn = q + fma(-vh, f2[1], -uh * f1[1]);
        sn = s + (fma(-vh, f2[2], -uh * f1[2]) + two_omega * t);
        tn = t + (fma(-vh, f2[3], -uh * f1[3]) - two_omega * s);
    }
    B[F_P][ci] = pn;
    B[F_Q][ci] = qn;
    B[F_S][ci] = sn;
    B[F_TAU][ci] = tn;
    if (emit_source) {
        write_pre(F, ci, a.xf, a.yf, pn, qn, sn, tn);
    }
    return true;
}

__global__ void __launch_bounds__(ATX * ATY) k_advect(step_consts c, advect_consts a, const __grid_constant__ field_boxes maps,
                                                      fields_dev F, int cur, double dt, double bv, int emit_source) {
    if (c.clock) cur = (int)c.clock[CLK_CUR];
    advect_tile(c, a, maps, F, cur, dt, bv, emit_source, blockIdx.x, blockIdx.y, 0);
}

// ---- float pairs of the projection kernels (mixed-precision handles) ------------

__device__ __forceinline__ ff split_ff(double d) {
    ff r;
    ff_split_d(d, r.hi, r.lo);
    return r;
}
// a + inc for the FP64 state value a with one FP64 addition (the pair formed
// as a double on the integer pipe)
__device__ __forceinline__ double add_ff(double a, ff inc) { return a + ff_to_d(inc.hi, inc.lo); }

// ---- fixed-point advection ----------------------------------------------------
//
// The same step with the ENO arithmetic in 64-bit integers: GB300 retires two
// FP64 operations per clock and SM and 64 integer ones, and the ENO part of
// the step is differences of neighbouring values, which integers form exactly.
// Every staged field of the tile is scaled by one power of two so that its
// largest magnitude lies in [2^58, 2^59) (a value within 2^-6 of the largest
// keeps all of its 53 bits, a smaller one is cut at 2^-59 of the largest, 64
// times finer than the FP64 spacing there); first and second differences, the
// comparison of their magnitudes and the ENO value (at most 2^62) are then
// exact, so near ties need no margin.  The products with the velocity times
// dt/(2 dx), scaled likewise, are the high words of 64 x 64 bit products (cut
// within four units of 2^-57 of the largest increment), and each field takes its
// increment in one FP64 addition.
// Those cuts are relative to the tile's largest values.  An update stays within
// 32 roundings of the values it is computed from, the error bound of the FP64
// form, where one value of its stencil reaches 2^50 units of the increment
// (fx_weak; with a velocity dt/(2 dx) of 0.1, 2^-7 of the tile's largest); a
// cell where none does, which takes fields over many orders of magnitude within
// a tile, lists its 32 x 8 half.  Mixed handles, whose solves and source leave
// 2^-44, ask for 2^47 units.
// The listed halves take k_advect's arithmetic in k_advect_rest, as do tiles with
// an infinity or a NaN in a field or the velocity, and the cells that the yield
// test (on the leading 24 bits, with a margin) cannot certify as elastic.
// A block takes 32 x 16 cells, two rows of eight threads after one another: the
// staged halo is 1.4 times the cells (1.7 at 32 x 8, where converting it was a
// fifth of the kernel).  At 2048^2: 290 us on FP64 handles (1390 with k_advect),
// 254 us on mixed ones (456 with float pairs); FP64 pipe 62 % busy (21 FP64
// instructions a cell, the integers' conversions among them).
constexpr int FXY = 2 * ATY, FROWS = FXY + 4;
constexpr unsigned kFxBytes = F_COUNT * FROWS * ACOLS * sizeof(double);
// Of a field's increments in a tile: minus their unit, and the quick test's
// threshold with its double (zero for a field that cannot fail it).
struct alignas(16) fx_scale {
    double unit;
    int thr;
    unsigned span;
    __device__ __forceinline__ void set(int K, int t) {
        unit = -power_of_two(K);
        thr = t;
        span = 2u * (unsigned)t;
    }
    __device__ __forceinline__ bool below(long long v) const { return (unsigned)((int)(v >> 32) + thr) < span; }
};
struct fx_smem {
    union {
        double d[F_COUNT][FROWS][ACOLS];  // TMA destination (128-byte aligned)
        long long v[F_COUNT][FROWS][ACOLS];
    } t;
    long long nu[FXY + 1][ATX + 1], nv[FXY + 1][ATX + 1];  // node velocities, walls substituted
    unsigned top[F_COUNT + 1];  // largest high word's magnitude per field; then of the velocity
    unsigned redo;              // halves to list
    fx_scale scale[F_COUNT];
    int xs[ACOLS], col[ACOLS];  // period shift and storage column of tile column c-2
    uint64_t bar;
};

// hx, hy = hmx 2^he, hmy 2^he with the larger of hmx, hmy in [2^61, 2^62).
struct advect_fx_consts {
    long long hmx, hmy;
    int he;
    int floor = 0;  // explicit step: what its viscous and diffusive sums ask of fx_threshold
    double xf, yf;  // 1/(2 dt dx), 1/(2 dt dy) of projection_step
};

// ENO2 value at c, upwind towards c[-d] (d: +-1 column or +-1 row): twice the
// upwind difference plus the smaller of the two second differences;
// `inner` false: twice the difference alone (next to a wall).
__device__ __forceinline__ long long eno_fx(const long long *c, int d, bool inner) {
    const long long c0 = c[0], c1 = c[-d], D2 = c0 - c1;
    const long long S0 = c[d] - c0 - D2, S1 = D2 - c1 + c[-2 * d];
    // |S0| > |S1| exactly where S0 - S1 and S0 + S1 have one sign (both not zero;
    // equal differences may take either)
    const long long a = S0 - S1, b = S0 + S1;
    const bool gt = (a ^ b) >= 0 && b != 0;
    long long s = gt ? S1 : S0;
    if (!inner) s = 0;
    return D2 + D2 + s;
}

// |velocity| dt/(2 dx) from four times the velocity, below 2^60, in two words
// whose lower one is halved (its last bit is dropped), so that the products
// below are signed 32 x 32 bit ones.
struct fx_factor {
    int hi, lo;
    __device__ __forceinline__ fx_factor(long long u4, long long hm) {
        const unsigned long long w =
            __umul64hi((unsigned long long)(u4 < 0 ? -u4 : u4), (unsigned long long)hm) << 1;
        hi = (int)(w >> 32);
        lo = (int)((unsigned)w >> 1);
    }
};
// (u a + v b) / 2^64 within three units: |a|, |b| <= 2^62.
__device__ __forceinline__ long long fx_products(const fx_factor &u, long long a, const fx_factor &v, long long b) {
    const int a1 = (int)(a >> 32), b1 = (int)(b >> 32), a0 = (int)((unsigned)a >> 1), b0 = (int)((unsigned)b >> 1);
    const long long mid = (long long)u.lo * a1 + (long long)u.hi * a0 + (long long)v.lo * b1 + (long long)v.hi * b0;
    return (long long)u.hi * a1 + (long long)v.hi * b1 + (mid >> 31);
}

// Whether no integer of the cross of two columns and two rows around c reaches
// 2^32 thr.
__device__ __forceinline__ bool below(long long v, int thr) {
    return (unsigned)((int)(v >> 32) + thr) < 2u * (unsigned)thr;
}
__device__ __forceinline__ bool stencil_below(const long long *c, int thr) {
    bool b = below(c[0], thr);
    for (int k = 1; k <= 2; k++)
        b = b && below(c[k], thr) && below(c[-k], thr) && below(c[k * ACOLS], thr) && below(c[-k * ACOLS], thr);
    return b;
}
// 2^(K - 32) for the test above, K = 33 at least; 2^30, which nothing reaches, for
// an increment that large.
__device__ __forceinline__ int fx_threshold(int K) { return 1 << min(max(K - 32, 1), 30); }

// Whether a cell (and node) that failed the quick test may be off by more than
// its own values' rounding: a field, unless it or the velocity is zero in the
// whole tile, or the velocity at the cell's corners, whose differences are the
// spin, is everywhere small.
__device__ __noinline__ bool fx_weak(const fx_smem &Sm, int row, int tx, bool node, int thr) {
    if (Sm.top[F_COUNT] == 0) return false;
    const int at = (row + 2) * ACOLS + tx + 2;
    for (int f = 0; f < F_COUNT; f++)
        if (Sm.top[f] != 0 && (node || (f != F_X && f != F_Y)) && stencil_below(&Sm.t.v[f][0][0] + at, thr)) return true;
    constexpr int slow = 1 << (50 - 32);
    bool b = true;
    for (int k = 0; k < 4; k++)
        b = b && below(Sm.nu[row + (k >> 1)][tx + (k & 1)], slow) && below(Sm.nv[row + (k >> 1)][tx + (k & 1)], slow);
    return b;
}

// Yield test on the leading 24 bits: 3q^2 + s^2 + tau^2 within 5e-7; a cell
// clearly below the cut-offs of k_advect (1e-24, or an athermal law below
// yield) is elastic there too, any other one takes the FP64 test and law.
__device__ __forceinline__ bool surely_elastic(const step_consts &c, double q, double s, double t) {
    const float qf = ff_hi(q), sf = ff_hi(s), tf = ff_hi(t);
    const float dv = 3.f * qf * qf + sf * sf + tf * tf;
    return dv < 0.999e-24f * (1.f - 1e-6f) || (c.stz_model >= 2 && dv < c.yield_cut2f);
}

// One tile.  PRE: also the combinations for k_source (FP64 handles).
template <bool PRE>
__global__ void __launch_bounds__(ATX * ATY, 4)
    k_advect_fx(step_consts c, advect_fx_consts h, const __grid_constant__ field_boxes maps, fields_dev F, int cur,
                double bv) {
    extern __shared__ __align__(128) unsigned char fx_raw[];
    fx_smem &Sm = *reinterpret_cast<fx_smem *>(fx_raw + ((128 - (smem_addr(fx_raw) & 127)) & 127));
    const int m = c.m, n = c.n;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * ATX + tx;
    const int i0 = blockIdx.x * ATX, j0 = blockIdx.y * FXY;
    const int i = i0 + tx;
    if (c.clock) cur = (int)c.clock[CLK_CUR];
    const double *__restrict__ const *A = F.f[cur];
    double *const *B = F.f[cur ^ 1];
    if (tid == 0) mbar_init(&Sm.bar, 1);
    if (tid < ACOLS) {
        const int u = i0 + tid - 2;
        int w = u % m;
        if (w < 0) w += m;
        Sm.col[tid] = w;
        Sm.xs[tid] = u < 0 ? -1 : (u >= m ? 1 : 0);
    }
    if (tid < F_COUNT + 1) Sm.top[tid] = 0;
    if (tid == 0) Sm.redo = 0;
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(&Sm.bar, kFxBytes);
        for (int f = 0; f < F_COUNT; f++) tma_load_2d(&Sm.t.d[f][0][0], &maps.f[cur][f], i0 - 2, j0 - 1, &Sm.bar);
    }
    // node velocities while the tile arrives (at most three per thread)
    if (c.clock) bv = c.clock[CLK_BV_STATE];
    constexpr int kNodes = (FXY + 1) * (ATX + 1), kPer = (kNodes + ATX * ATY - 1) / (ATX * ATY);
    double2 vel[kPer];
    unsigned vtop = 0;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        const int p = tid + q * ATX * ATY, r = p / (ATX + 1), cc = p - r * (ATX + 1), nj = j0 + r;
        vel[q] = make_double2(0.0, 0.0);
        if (p < kNodes && nj <= n) {
            if (nj == 0 || nj == n) vel[q].x = nj == 0 ? -bv : bv;
            else vel[q] = F.vel[(size_t)nj * m + Sm.col[cc + 2]];
        }
        vtop = max(vtop, max((unsigned)__double2hiint(vel[q].x) & 0x7fffffffu,
                             (unsigned)__double2hiint(vel[q].y) & 0x7fffffffu));
    }
    if (__syncthreads_or(!mbar_wait_bounded(&Sm.bar))) {
        if (tid == 0) atomicExch(&F.flags[FL_TMA], 1);
        mbar_wait_bounded(&Sm.bar);
        return;
    }
    // columns across the periodic seam arrive as zeros: edge blocks fetch them
    if (i0 == 0 || i0 + ACOLS - 2 > m) {
        for (int k = tid; k < F_COUNT * FROWS * ACOLS; k += ATX * ATY) {
            const int f = k / (FROWS * ACOLS), rem = k - f * (FROWS * ACOLS), r = rem / ACOLS, t = rem - r * ACOLS;
            const int u = i0 + t - 2, sr = j0 - 1 + r;
            if ((u < 0 || u >= m) && sr >= 0 && sr <= n + 1) Sm.t.d[f][r][t] = A[f][(size_t)sr * m + Sm.col[t]];
        }
        __syncthreads();
    }
    // the largest magnitude of every field and of the velocity
    {
        unsigned top[F_COUNT];
#pragma unroll
        for (int f = 0; f < F_COUNT; f++) top[f] = 0;
        for (int p = tid; p < FROWS * ACOLS; p += ATX * ATY) {
#pragma unroll
            for (int f = 0; f < F_COUNT; f++)
                top[f] = max(top[f], (unsigned)__double2hiint((&Sm.t.d[f][0][0])[p]) & 0x7fffffffu);
        }
#pragma unroll
        for (int f = 0; f < F_COUNT; f++) {
            const unsigned w = __reduce_max_sync(0xffffffffu, top[f]);
            if (tx == 0) atomicMax(&Sm.top[f], w);
        }
        vtop = __reduce_max_sync(0xffffffffu, vtop);
        if (tx == 0) atomicMax(&Sm.top[F_COUNT], vtop);
    }
    __syncthreads();
    int E[F_COUNT], Eu = max((int)(Sm.top[F_COUNT] >> 20), 128);
    bool finite = Eu < 0x7ff;
#pragma unroll
    for (int f = 0; f < F_COUNT; f++) {
        E[f] = max((int)(Sm.top[f] >> 20), 128);
        finite = finite && E[f] < 0x7ff;
    }
    const int Ku = Eu + h.he - 2037;  // an increment is its integer times -2^(E + Ku)
#pragma unroll
    for (int f = 0; f < F_COUNT; f++) finite = finite && E[f] + Ku < 1000;
    if (!finite) {  // the same for the whole block
        // two of k_advect's tiles
        if (tid < 2 && j0 + tid * ATY < n)
            F.tlist[atomicAdd(F.pcount + 1, 1u)] = (2 * blockIdx.y + tid) * gridDim.x + blockIdx.x;
        return;
    }
    // the map's values are unwrapped across the seam: room for the period
    E[F_X] = max(E[F_X], (int)((unsigned)__double2hiint(c.lx) >> 20)) + 1;
    const long long lx = to_fixed(c.lx, E[F_X]);
    const int thr = fx_threshold((PRE ? 50 : 47) + Ku + 1081);
    if (tid == 0) {
#pragma unroll
        for (int f = 0; f < F_COUNT; f++) Sm.scale[f].set(E[f] + Ku, Sm.top[f] && Sm.top[F_COUNT] ? thr : 0);
    }
    for (int p = tid; p < FROWS * ACOLS; p += ATX * ATY) {
#pragma unroll
        for (int f = 0; f < F_COUNT; f++) {
            long long v = to_fixed((&Sm.t.d[f][0][0])[p], E[f]);
            if (f == F_X) {
                const int sh = Sm.xs[p % ACOLS];
                if (sh) v += sh > 0 ? lx : -lx;
            }
            (&Sm.t.v[f][0][0])[p] = v;
        }
    }
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        const int p = tid + q * ATX * ATY;
        if (p < kNodes) {
            (&Sm.nu[0][0])[p] = to_fixed(vel[q].x, Eu);
            (&Sm.nv[0][0])[p] = to_fixed(vel[q].y, Eu);
        }
    }
    __syncthreads();
    unsigned flows = 0, unsure = 0;  // of this thread's two cells, those not surely elastic; those to look at again
#pragma unroll 1
    for (int row = ty; row < FXY && i < m && j0 + row < n; row += ATY) {
        const int j = j0 + row;
        const size_t ci = (size_t)(j + 1) * m + i;
        bool weak = false;
        auto upwind = [&](int f, const fx_factor &uh, int dx, const fx_factor &vh, int dy, bool inner) {
            const long long *q = &Sm.t.v[f][row + 2][tx + 2];
            weak = weak || Sm.scale[f].below(q[0]);
            return fx_products(uh, eno_fx(q, dx, true), vh, eno_fx(q, dy, inner));
        };
        const long long u00 = Sm.nu[row][tx], v00 = Sm.nv[row][tx];
        // reference map at node (i,j), rows 1..n-1 (shear_sim.cc:310-327)
        if (j > 0) {
            const fx_factor uh(4 * u00, h.hmx), vh(4 * v00, h.hmy);
            const int dx = u00 > 0 ? 1 : -1, dy = v00 > 0 ? ACOLS : -ACOLS;
            const bool inner = v00 > 0 ? j > 1 : j < n - 1;
#pragma unroll
            for (int f = F_X; f <= F_Y; f++)
                B[f][ci] = fma((double)upwind(f, uh, dx, vh, dy, inner), Sm.scale[f].unit, A[f][ci]);
        }
        // staggered velocity and spin (shear_sim.cc:330-333)
        const long long u10 = Sm.nu[row][tx + 1], u01 = Sm.nu[row + 1][tx], u11 = Sm.nu[row + 1][tx + 1];
        const long long v10 = Sm.nv[row][tx + 1], v01 = Sm.nv[row + 1][tx], v11 = Sm.nv[row + 1][tx + 1];
        const long long u4 = (u00 + u10) + (u01 + u11), v4 = (v00 + v10) + (v01 + v11);
        weak = weak || (below(u4, 1 << (52 - 32)) && below(v4, 1 << (52 - 32)));
        const double two_omega = (double)(__mul64hi((v10 - v00) + (v11 - v01), h.hmx) -
                                          __mul64hi((u01 - u00) + (u11 - u10), h.hmy)) *
                                 power_of_two(64 + Eu - 1081 + h.he);
        const fx_factor uh(u4, h.hmx), vh(v4, h.hmy);
        const int dx = u4 > 0 ? 1 : -1, dy = v4 > 0 ? ACOLS : -ACOLS;
        const bool inner = v4 > 0 ? j > 0 : j < n - 1;
        double a[5], v[5];
#pragma unroll
        for (int f = 0; f < 5; f++) a[f] = A[f][ci];
#pragma unroll
        for (int f = 0; f < 5; f++) {
            const double inc = (double)upwind(f, uh, dx, vh, dy, inner), sc = Sm.scale[f].unit;
            if (f == F_S) v[f] = a[f] + fma(inc, sc, two_omega * a[F_TAU]);
            else if (f == F_TAU) v[f] = a[f] + fma(inc, sc, -two_omega * a[F_S]);
            else v[f] = fma(inc, sc, a[f]);
            B[f][ci] = v[f];
        }
        if (!surely_elastic(c, a[F_Q], a[F_S], a[F_TAU])) flows |= row < ATY ? 1u : 2u;
        F.ddev[ci] = 0;
        if (PRE) write_pre(F, ci, h.xf, h.yf, v[F_P], v[F_Q], v[F_S], v[F_TAU]);
        if (weak) unsure |= row < ATY ? 1u : 2u;
    }
#pragma unroll 1
    for (int k = 0; k < 2; k++)
        if ((unsure >> k & 1) && fx_weak(Sm, ty + k * ATY, tx, j0 + ty + k * ATY > 0, thr)) atomicOr(&Sm.redo, 1u << k);
    __syncthreads();
    const unsigned redo = Sm.redo;
    if (tid < 2 && (redo >> tid & 1)) F.tlist[atomicAdd(F.pcount + 1, 1u)] = (2 * blockIdx.y + tid) * gridDim.x + blockIdx.x;
    flows &= ~redo;
    for (int k = 0; k < 2; k++)
        if (flows >> k & 1)
            F.plist[atomicAdd(F.pcount, 1u)] = (unsigned)((size_t)(j0 + ty + k * ATY + 1) * m + i);
}

// What k_advect_fx left: the listed cells' plastic part (k_advect's FP64 yield
// test and, above the cut-offs, the FP64 plastic law,
// adaptive_plastic_term, shear_sim.cc:513-548, on the advected chi, then
// q, s, tau -= dtmp times their old values, ddev and the plastic strain: the
// same operations in the same order, so the cell ends where the one-pass form
// would take it) and the listed tiles, with k_advect's arithmetic.
__global__ void __launch_bounds__(ATX * ATY)
    k_advect_rest(step_consts c, advect_consts a, const __grid_constant__ field_boxes maps, fields_dev F, int cur,
                  double dt, double bv, int emit_source, int tiles_x) {
    if (c.clock) cur = (int)c.clock[CLK_CUR];
    const unsigned cnt = F.pcount[0], tiles = F.pcount[1];
    const double *__restrict__ const *A = F.f[cur];
    double *const *B = F.f[cur ^ 1];
    const bool athermal = c.stz_model >= 2;
    const int tid = threadIdx.y * ATX + threadIdx.x;
    const stz_law_params<double> lp = law_params(c);
    const double strain = 1 / (2 * c.mu);
    for (unsigned k = blockIdx.x * (ATX * ATY) + tid; k < cnt; k += gridDim.x * (ATX * ATY)) {
        const size_t ci = F.plist[k];
        const double q = A[F_Q][ci], s = A[F_S][ci], t = A[F_TAU][ci];
        const double devsq = 3 * q * q + s * s + t * t;
        const long long dbits = __double_as_longlong(devsq);
        if (dbits < __double_as_longlong(0.999e-24) || (athermal && dbits < __double_as_longlong(c.yield_cut2)))
            continue;
        int iters;
        double chi = B[F_CHI][ci], ddev = 0;
        const double dtmp = adaptive_plastic(lp, sqrt(devsq), chi, ddev, dt, iters);
        if (iters >= c.substep_cap) atomicExch(&F.flags[FL_SUBSTEP_CAP], 1);
        if (iters > 1) atomicMax(&F.flags[FL_SUBSTEP_MAX], iters);
        B[F_CHI][ci] = chi;
        F.ddev[ci] = ddev;
        if (c.track_plastic && ddev != 0) {
            const int m = c.m, j = (int)(ci / (size_t)m) - 1, i = (int)(ci - (size_t)(j + 1) * m);
            F.eps_pl[(size_t)j * m + i] += ddev * strain;
        }
        if (dtmp != 0) {
            const double qn = B[F_Q][ci] - dtmp * q, sn = B[F_S][ci] - dtmp * s, tn = B[F_TAU][ci] - dtmp * t;
            B[F_Q][ci] = qn;
            B[F_S][ci] = sn;
            B[F_TAU][ci] = tn;
            if (emit_source) write_pre(F, ci, a.xf, a.yf, B[F_P][ci], qn, sn, tn);
        }
    }
    for (unsigned k = blockIdx.x, it = 0; k < tiles; k += gridDim.x, it++) {
        const unsigned tile = F.tlist[k];
        if (!advect_tile(c, a, maps, F, cur, dt, bv, emit_source, tile % tiles_x, tile / tiles_x, it)) return;
        __syncthreads();  // the next tile reuses the shared memory
    }
}

// Explicit step (shear_sim::step_forward, shear_sim.cc:185-276) per cell
// (i,j) and its lower-left node: the node velocity and reference map are
// advected with ENO2 and the velocity takes the net force of the old stress
// (net_force with prefactors -hx,-hy, shear_sim.cc:447-453) and a 5-point
// viscous term, divided by mu as the reference's mu_inv; the cell fields are
// advected and take the elastic rate of the old velocity gradient and the
// plastic term.  The constant chi diffusion enters cchi before the plastic
// term (and again in k_chi_diffusion, as the reference adds it twice); ddev
// is stored times the old |s| (shear_sim.cc:265).  New node velocities go to
// F.src (rows 1..n-1), the other fields to buffer cur^1.
struct direct_consts {
    double hxxv, hyyv, hcv, hxxcd, hyycd, hccd;
    double hx, hy, mu_inv;
};

// Tile fields of the explicit step: the seven stored fields, then the node
// velocity components u and v (rows 0..n, walls substituted).
enum { DF_U = F_COUNT, DF_V, DF_COUNT };
typedef eno_tile<DF_COUNT> direct_tile;

// One tile (bx, by) in FP64.
__device__ __forceinline__ void direct_tile_step(const step_consts &c, const direct_consts &d, const fields_dev &F,
                                                 int cur, double dt, double bv, int bx, int by) {
    extern __shared__ __align__(16) unsigned char dir_smem[];
    direct_tile &TT = *reinterpret_cast<direct_tile *>(dir_smem);
    const int m = c.m, n = c.n;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int i0 = bx * ATX, j0 = by * ATY;
    const int i = i0 + tx, j = j0 + ty;
    const double *__restrict__ const *A = F.f[cur];
    double *const *B = F.f[cur ^ 1];
    velo V{F.vel, m, n, bv};
    tile_columns(TT, i0, m, c.lx);
    __syncthreads();
    tile_differences<DF_COUNT>(
        TT, i0, j0, m, n, F_X,
        [&](int f, int row, int t) {
            const int col = TT.col[t];
            return f == DF_U ? V.u(col, row) : (f == DF_V ? V.v(col, row) : A[f][(size_t)(row + 1) * m + col]);
        },
        [](int f) { return f >= DF_U ? 0 : -1; });
    if (i >= m || j >= n) return;
    const double hx = d.hx, hy = d.hy, mu_inv = d.mu_inv;
    const int il = TT.col[tx + 1], ir = TT.col[tx + 3];
    const size_t ci = IDX(i, j);
    const double *P = A[F_P], *Q = A[F_Q], *S = A[F_S], *T = A[F_TAU];
    if (j > 0) {
        const double *X = A[F_X], *Y = A[F_Y];
        const double un = V.u(i, j), vn = V.v(i, j);
        const double hsx = un > 0 ? hx : -hx, hsy = vn > 0 ? hy : -hy;
        double ux = tile_eno_x(TT, DF_U, ty, tx, un > 0), vx = tile_eno_x(TT, DF_V, ty, tx, un > 0);
        double Xx = tile_eno_x(TT, F_X, ty, tx, un > 0), Yx = tile_eno_x(TT, F_Y, ty, tx, un > 0);
        const bool inner = vn > 0 ? j > 1 : j < n - 1;
        double uy = tile_eno_y(TT, DF_U, ty, tx, vn > 0, inner), vy = tile_eno_y(TT, DF_V, ty, tx, vn > 0, inner);
        double Xy = tile_eno_y(TT, F_X, ty, tx, vn > 0, inner), Yy = tile_eno_y(TT, F_Y, ty, tx, vn > 0, inner);
        ux *= hsx; vx *= hsx; Xx *= hsx; Yx *= hsx;
        uy *= hsy; vy *= hsy; Xy *= hsy; Yy *= hsy;
        // net force from the cells (i-1,j-1), (i,j-1), (i-1,j), (i,j)
        const size_t c0 = IDX(il, j - 1), c1 = IDX(i, j - 1), c2 = IDX(il, j), c3 = ci;
        const double xf = -hx, yf = -hy;
        const double fx = (-P[c0] + P[c1] - P[c2] + P[c3] - Q[c0] + Q[c1] - Q[c2] + Q[c3] + S[c0] - S[c1] + S[c2] -
                           S[c3]) * xf + (T[c0] + T[c1] - T[c2] - T[c3]) * yf;
        const double fy = (T[c0] - T[c1] + T[c2] - T[c3]) * xf +
                          (-P[c0] - P[c1] + P[c2] + P[c3] - Q[c0] - Q[c1] + Q[c2] + Q[c3] - S[c0] - S[c1] + S[c2] +
                           S[c3]) * yf;
        const double uvisc = d.hxxv * (V.u(ir, j) + V.u(il, j)) + d.hyyv * (V.u(i, j + 1) + V.u(i, j - 1)) - d.hcv * un;
        const double vvisc = d.hxxv * (V.v(ir, j) + V.v(il, j)) + d.hyyv * (V.v(i, j + 1) + V.v(i, j - 1)) - d.hcv * vn;
        F.src[(size_t)j * m + i] = make_double2(un + (-un * ux - vn * uy + mu_inv * (fx + uvisc)),
                                                vn + (-un * vx - vn * vy + mu_inv * (fy + vvisc)));
        B[F_X][ci] = X[ci] + (-un * Xx - vn * Xy);
        B[F_Y][ci] = Y[ci] + (-un * Yx - vn * Yy);
    }
    // deformation rate, staggered velocity and spin
    const double u00 = V.u(i, j), u10 = V.u(ir, j), u01 = V.u(i, j + 1), u11 = V.u(ir, j + 1);
    const double v00 = V.v(i, j), v10 = V.v(ir, j), v01 = V.v(i, j + 1), v11 = V.v(ir, j + 1);
    const double uc = 0.25 * (u00 + u10 + u01 + u11), vc = 0.25 * (v00 + v10 + v01 + v11);
    const double ux = hx * (-u00 + u10 - u01 + u11), uy = hy * (-u00 - u10 + u01 + u11);
    const double vx = hx * (-v00 + v10 - v01 + v11), vy = hy * (-v00 - v10 + v01 + v11);
    const double two_omega = vx - uy;
    const double uh = uc * (uc > 0 ? hx : -hx), vh = vc * (vc > 0 ? hy : -hy);
    double f1[5], f2[5];
    const bool inner = vc > 0 ? j > 0 : j < n - 1;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        f1[k] = tile_eno_x(TT, k, ty, tx, uc > 0);
        f2[k] = tile_eno_y(TT, k, ty, tx, vc > 0, inner);
    }
    const double *CH = A[F_CHI];
    const double p = P[ci], q = Q[ci], s = S[ci], t = T[ci];
    double cchi = CH[ci] + fma(-vh, f2[4], -uh * f1[4]) + d.hxxcd * (CH[IDX(ir, j)] + CH[IDX(il, j)]) +
                  d.hyycd * (CH[IDX(i, j + 1)] + CH[IDX(i, j - 1)]) - d.hccd * CH[ci];
    const double devsq = 3 * q * q + s * s + t * t;
    double ddev = 0, dtmp = 0, sbar = 0;
    const bool athermal = c.stz_model >= 2;
    if (!(devsq < 0.999e-24 || (athermal && devsq < c.yield_cut2))) {
        int iters;
        const stz_law_params<double> lp = law_params(c);
        sbar = sqrt(devsq);
        dtmp = adaptive_plastic(lp, sbar, cchi, ddev, dt, iters);
        if (iters >= c.substep_cap) atomicExch(&F.flags[0], 1);
        if (iters > 1) atomicMax(&F.flags[1], iters);
    }
    B[F_CHI][ci] = cchi;
    F.ddev[ci] = ddev * sbar;
    if (c.track_plastic && ddev != 0) F.eps_pl[(size_t)j * m + i] += ddev / (2 * c.mu);
    const double third = 1 / 3.0;
    B[F_P][ci] = p + (fma(-vh, f2[0], -uh * f1[0]) - c.K * (ux + vy));
    B[F_Q][ci] = q + (fma(-vh, f2[1], -uh * f1[1]) - c.mu * third * (ux + vy) - dtmp * q);
    B[F_S][ci] = s + (fma(-vh, f2[2], -uh * f1[2]) + two_omega * t + c.mu * (ux - vy) - dtmp * s);
    B[F_TAU][ci] = t + (fma(-vh, f2[3], -uh * f1[3]) - two_omega * s + c.mu * (vx + uy) - dtmp * t);
}

__global__ void __launch_bounds__(ATX * ATY) k_direct(step_consts c, direct_consts d, fields_dev F, int cur,
                                                      double dt, double bv) {
    direct_tile_step(c, d, F, cur, dt, bv, blockIdx.x, blockIdx.y);
}

// The explicit step with the arithmetic of k_advect_fx: the nine advected
// fields (the node velocity among them) in 64-bit fixed point, and with them
// the exact sums of the net force (the four stresses share one scale), the
// velocity gradient and the viscous term.  k_direct is bound by its ~160 FP64
// operations per cell (0.70 ms a step at 1024 x 768 with flow everywhere; 0.11
// this kernel, 0.14 the plastic law in k_direct_rest).  Tiles with a value that is not finite and cells near
// yield are listed for k_direct_rest, and, as in k_advect_fx, the 32 x 8 halves with
// a cell whose own values lie too far below the tile's largest (fxd_weak).
struct fxd_smem {
    union {
        double d[DF_COUNT][FROWS][ACOLS];  // TMA destination of the first seven (128-byte aligned)
        long long v[DF_COUNT][FROWS][ACOLS];
    } t;
    unsigned top[DF_COUNT];  // largest high word's magnitude per field
    int xs[ACOLS], col[ACOLS];
    // -hx, -hy times the scale of the stresses' sums; hx, hy, hxxv, hyyv times that of the velocities
    double xfs, yfs, hx[2], hy[2], vx[2], vy[2];
    fx_scale scale[DF_COUNT];
    int rates, force;        // quick thresholds of the velocity at the corners and of the stresses
    double chi;              // the unit of chi's integers
    unsigned redo;           // halves to list
    int by[DF_COUNT];        // shift to the stresses', or the velocities', common scale
    uint64_t bar;
};

// An integer at the scale of exponent E, cut to a coarser one.
__device__ __forceinline__ long long fx_cut(long long v, int by) { return v >> min(by, 63); }

// Whether a cell that failed the quick test, or its lower-left node (node), may be
// off by more than its own values' rounding (as fx_weak): a field that is
// everywhere small on its stencil, the velocity at the corners (the rates), or
// the four cells' stresses (the force on the node), unless zero in the whole tile.
// The force's and the rates' sums are cut at no more than sixteen units of 2^-59
// of the tile's largest value, and their bounds take in 16 and 8 such terms.
__device__ __noinline__ bool fxd_weak(const fxd_smem &Sm, int row, int tx, bool node, int thr, bool diffuses) {
    const int at = (row + 2) * ACOLS + tx + 2;
    constexpr int slow = 1 << (50 - 32);
    const bool moves = Sm.top[DF_U] || Sm.top[DF_V];
    for (int f = 0; f < DF_COUNT; f++) {
        if (Sm.top[f] == 0 || !(moves || (f == F_CHI && diffuses))) continue;
        if ((node || f <= F_CHI) && stencil_below(&Sm.t.v[f][0][0] + at, thr)) return true;
    }
    bool still = moves, slack = node;
    bool stressed = false;
    for (int f = 0; f < DF_COUNT; f++) {
        const bool vel = f >= DF_U;
        if (!vel && f != F_P && f != F_Q && f != F_S && f != F_TAU) continue;
        stressed = stressed || (!vel && Sm.top[f]);
        for (int k = 0; k < 4; k++) {
            const int o = vel ? (k & 1) + (k >> 1) * ACOLS : -(k & 1) - (k >> 1) * ACOLS;
            const bool b = below(fx_cut((&Sm.t.v[f][0][0])[at + o], Sm.by[f]), slow);
            if (vel) still = still && b;
            else slack = slack && b;
        }
    }
    return still || (slack && stressed);
}

__global__ void __launch_bounds__(ATX * ATY, 4)
    k_direct_fx(step_consts c, direct_consts d, advect_fx_consts h, const __grid_constant__ field_boxes maps,
                fields_dev F, int cur, double bv) {
    extern __shared__ __align__(128) unsigned char fxd_raw[];
    fxd_smem &Sm = *reinterpret_cast<fxd_smem *>(fxd_raw + ((128 - (smem_addr(fxd_raw) & 127)) & 127));
    const int m = c.m, n = c.n;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * ATX + tx;
    const int i0 = blockIdx.x * ATX, j0 = blockIdx.y * FXY;
    const int i = i0 + tx;
    const double *__restrict__ const *A = F.f[cur];
    double *const *B = F.f[cur ^ 1];
    if (tid == 0) mbar_init(&Sm.bar, 1);
    if (tid < ACOLS) {
        const int u = i0 + tid - 2;
        int w = u % m;
        if (w < 0) w += m;
        Sm.col[tid] = w;
        Sm.xs[tid] = u < 0 ? -1 : (u >= m ? 1 : 0);
    }
    if (tid < DF_COUNT) Sm.top[tid] = 0;
    if (tid == 0) Sm.redo = 0;
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(&Sm.bar, kFxBytes);
        for (int f = 0; f < F_COUNT; f++) tma_load_2d(&Sm.t.d[f][0][0], &maps.f[cur][f], i0 - 2, j0 - 1, &Sm.bar);
    }
    // node velocities of the tile's rows while it arrives
    constexpr int kTile = FROWS * ACOLS, kPer = (kTile + ATX * ATY - 1) / (ATX * ATY);
    unsigned utop = 0, vtop = 0;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        const int p = tid + q * ATX * ATY, r = p / ACOLS, t = p - r * ACOLS, nj = j0 - 2 + r;
        double2 v = make_double2(0.0, 0.0);
        if (p >= kTile) break;
        if (nj >= 0 && nj <= n) {
            if (nj == 0 || nj == n) v.x = nj == 0 ? -bv : bv;
            else v = F.vel[(size_t)nj * m + Sm.col[t]];
        }
        (&Sm.t.d[DF_U][0][0])[p] = v.x;
        (&Sm.t.d[DF_V][0][0])[p] = v.y;
        utop = max(utop, (unsigned)__double2hiint(v.x) & 0x7fffffffu);
        vtop = max(vtop, (unsigned)__double2hiint(v.y) & 0x7fffffffu);
    }
    if (__syncthreads_or(!mbar_wait_bounded(&Sm.bar))) {
        if (tid == 0) atomicExch(&F.flags[FL_TMA], 1);
        mbar_wait_bounded(&Sm.bar);
        return;
    }
    if (i0 == 0 || i0 + ACOLS - 2 > m) {
        for (int k = tid; k < F_COUNT * kTile; k += ATX * ATY) {
            const int f = k / kTile, rem = k - f * kTile, r = rem / ACOLS, t = rem - r * ACOLS;
            const int u = i0 + t - 2, sr = j0 - 1 + r;
            if ((u < 0 || u >= m) && sr >= 0 && sr <= n + 1) Sm.t.d[f][r][t] = A[f][(size_t)sr * m + Sm.col[t]];
        }
        __syncthreads();
    }
    {
        unsigned top[F_COUNT];
#pragma unroll
        for (int f = 0; f < F_COUNT; f++) top[f] = 0;
        for (int p = tid; p < kTile; p += ATX * ATY) {
#pragma unroll
            for (int f = 0; f < F_COUNT; f++)
                top[f] = max(top[f], (unsigned)__double2hiint((&Sm.t.d[f][0][0])[p]) & 0x7fffffffu);
        }
#pragma unroll
        for (int f = 0; f < F_COUNT; f++) {
            const unsigned w = __reduce_max_sync(0xffffffffu, top[f]);
            if (tx == 0) atomicMax(&Sm.top[f], w);
        }
        utop = __reduce_max_sync(0xffffffffu, utop);
        vtop = __reduce_max_sync(0xffffffffu, vtop);
        if (tx == 0) {
            atomicMax(&Sm.top[DF_U], utop);
            atomicMax(&Sm.top[DF_V], vtop);
        }
    }
    __syncthreads();
    int E[DF_COUNT];
    bool finite = true;
#pragma unroll
    for (int f = 0; f < DF_COUNT; f++) {
        E[f] = max((int)(Sm.top[f] >> 20), 128);
        finite = finite && E[f] < 0x7ff;
    }
    const int Ku = max(E[DF_U], E[DF_V]) + h.he - 2037;
#pragma unroll
    for (int f = 0; f < DF_COUNT; f++) finite = finite && E[f] + Ku < 1000;
    if (!finite) {  // the same for the whole block: two of k_direct's tiles
        if (tid < 2 && j0 + tid * ATY < n)
            F.tlist[atomicAdd(F.pcount + 1, 1u)] = (2 * blockIdx.y + tid) * gridDim.x + blockIdx.x;
        return;
    }
    E[F_X] = max(E[F_X], (int)((unsigned)__double2hiint(c.lx) >> 20)) + 1;
    const long long lx = to_fixed(c.lx, E[F_X]);
    // the stresses at one scale, and both velocities at one (cut to it)
    const int Es = max(max(E[F_P], E[F_Q]), max(E[F_S], E[F_TAU])), Eu = max(E[DF_U], E[DF_V]);
    auto cut = [](long long v, int by) { return fx_cut(v, by); };
    const int thr = fx_threshold(max(50 + Ku + 1081, h.floor));
    const bool moves = Sm.top[DF_U] || Sm.top[DF_V];
    if (tid == 0) {
#pragma unroll
        for (int f = 0; f < DF_COUNT; f++) {
            Sm.scale[f].set(E[f] + Ku, Sm.top[f] && (moves || (f == F_CHI && d.hccd != 0)) ? thr : 0);
            Sm.by[f] = (f >= DF_U ? Eu : Es) - E[f];
        }
        Sm.chi = power_of_two(E[F_CHI] - 1081);
        Sm.rates = moves ? 1 << (52 - 32) : 0;
        Sm.force = Sm.top[F_P] || Sm.top[F_Q] || Sm.top[F_S] || Sm.top[F_TAU] ? 1 << (52 - 32) : 0;
        const double ss = power_of_two(Es - 1081);
        Sm.xfs = -d.hx * ss;
        Sm.yfs = -d.hy * ss;
    }
    if (tid < 2) {
        const double su = power_of_two((tid ? E[DF_V] : E[DF_U]) - 1081);
        Sm.hx[tid] = d.hx * su;
        Sm.hy[tid] = d.hy * su;
        Sm.vx[tid] = d.hxxv * su;
        Sm.vy[tid] = d.hyyv * su;
    }
    for (int p = tid; p < kTile; p += ATX * ATY) {
#pragma unroll
        for (int f = 0; f < DF_COUNT; f++) {
            long long v = to_fixed((&Sm.t.d[f][0][0])[p], E[f]);
            if (f == F_X) {
                const int sh = Sm.xs[p % ACOLS];
                if (sh) v += sh > 0 ? lx : -lx;
            }
            (&Sm.t.v[f][0][0])[p] = v;
        }
    }
    __syncthreads();
    unsigned flows = 0, unsure = 0;
#pragma unroll 1
    for (int row = ty; row < FXY && i < m && j0 + row < n; row += ATY) {
        const int j = j0 + row;
        bool weak = false;
        const size_t ci = (size_t)(j + 1) * m + i;
        const int at = (row + 2) * ACOLS + tx + 2;
        auto fld = [&](int f) { return &Sm.t.v[f][0][0] + at; };
        auto upwind = [&](int f, const fx_factor &uh, int dx, const fx_factor &vh, int dy, bool inner) {
            weak = weak || Sm.scale[f].below(fld(f)[0]);
            return (double)fx_products(uh, eno_fx(fld(f), dx, true), vh, eno_fx(fld(f), dy, inner)) * Sm.scale[f].unit;
        };
        const long long *U = fld(DF_U), *V = fld(DF_V);
        if (j > 0) {
            const long long u0 = U[0], v0 = V[0];
            const fx_factor uh(4 * cut(u0, Sm.by[DF_U]), h.hmx), vh(4 * cut(v0, Sm.by[DF_V]), h.hmy);
            const int dx = u0 > 0 ? 1 : -1, dy = v0 > 0 ? ACOLS : -ACOLS;
            const bool inner = v0 > 0 ? j > 1 : j < n - 1;
            // net force from the cells (i-1,j-1), (i,j-1), (i-1,j), (i,j)
            long long a[4], b[4], t[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int o = (k & 1) - 1 + ((k >> 1) - 1) * ACOLS;
                const long long pq = cut(fld(F_P)[o], Sm.by[F_P]) + cut(fld(F_Q)[o], Sm.by[F_Q]);
                const long long sv = cut(fld(F_S)[o], Sm.by[F_S]);
                a[k] = pq - sv;
                b[k] = pq + sv;
                t[k] = cut(fld(F_TAU)[o], Sm.by[F_TAU]);
            }
            const int force = Sm.force;
            weak = weak || (below(a[3], force) && below(b[3], force) && below(t[3], force));
            const double xfs = Sm.xfs, yfs = Sm.yfs;
            const double fx = fma(xfs, (double)((a[1] - a[0]) + (a[3] - a[2])),
                                  yfs * (double)((t[0] - t[2]) + (t[1] - t[3])));
            const double fy = fma(xfs, (double)((t[0] - t[1]) + (t[2] - t[3])),
                                  yfs * (double)((b[2] - b[0]) + (b[3] - b[1])));
            const double uvisc = fma(Sm.vx[0], (double)((U[1] - u0) + (U[-1] - u0)),
                                     Sm.vy[0] * (double)((U[ACOLS] - u0) + (U[-ACOLS] - u0)));
            const double vvisc = fma(Sm.vx[1], (double)((V[1] - v0) + (V[-1] - v0)),
                                     Sm.vy[1] * (double)((V[ACOLS] - v0) + (V[-ACOLS] - v0)));
            const double2 w = F.vel[(size_t)j * m + i];
            F.src[(size_t)j * m + i] =
                make_double2(w.x + fma(d.mu_inv, fx + uvisc, upwind(DF_U, uh, dx, vh, dy, inner)),
                             w.y + fma(d.mu_inv, fy + vvisc, upwind(DF_V, uh, dx, vh, dy, inner)));
#pragma unroll
            for (int f = F_X; f <= F_Y; f++) B[f][ci] = A[f][ci] + upwind(f, uh, dx, vh, dy, inner);
        }
        // deformation rate, staggered velocity and spin
        const long long u00 = U[0], u10 = U[1], u01 = U[ACOLS], u11 = U[ACOLS + 1];
        const long long v00 = V[0], v10 = V[1], v01 = V[ACOLS], v11 = V[ACOLS + 1];
        const long long u4 = (u00 + u10) + (u01 + u11), v4 = (v00 + v10) + (v01 + v11);
        const long long us = cut(u4, Sm.by[DF_U]), vs = cut(v4, Sm.by[DF_V]);
        weak = weak || (below(us, Sm.rates) && below(vs, Sm.rates));
        const double ux = Sm.hx[0] * (double)((u10 - u00) + (u11 - u01));
        const double uy = Sm.hy[0] * (double)((u01 - u00) + (u11 - u10));
        const double vx = Sm.hx[1] * (double)((v10 - v00) + (v11 - v01));
        const double vy = Sm.hy[1] * (double)((v01 - v00) + (v11 - v10));
        const double two_omega = vx - uy, div = ux + vy;
        const fx_factor uh(us, h.hmx), vh(vs, h.hmy);
        const int dx = u4 > 0 ? 1 : -1, dy = v4 > 0 ? ACOLS : -ACOLS;
        const bool inner = v4 > 0 ? j > 0 : j < n - 1;
        auto inc = [&](int f) { return upwind(f, uh, dx, vh, dy, inner); };
        const double q = A[F_Q][ci], s = A[F_S][ci], t = A[F_TAU][ci];
        B[F_P][ci] = A[F_P][ci] + (inc(F_P) - c.K * div);
        B[F_Q][ci] = q + (inc(F_Q) - c.mu * (1 / 3.0) * div);
        B[F_S][ci] = s + (fma(two_omega, t, inc(F_S)) + c.mu * (ux - vy));
        B[F_TAU][ci] = t + (fma(-two_omega, s, inc(F_TAU)) + c.mu * (vx + uy));
        double cchi = A[F_CHI][ci] + inc(F_CHI);
        if (d.hccd != 0) {
            const long long *H = fld(F_CHI);
            cchi += Sm.chi *
                    fma(d.hxxcd, (double)((H[1] - H[0]) + (H[-1] - H[0])),
                        d.hyycd * (double)((H[ACOLS] - H[0]) + (H[-ACOLS] - H[0])));
        }
        B[F_CHI][ci] = cchi;
        if (!surely_elastic(c, q, s, t)) flows |= row < ATY ? 1u : 2u;
        F.ddev[ci] = 0;
        if (weak) unsure |= row < ATY ? 1u : 2u;
    }
#pragma unroll 1
    for (int k = 0; k < 2; k++)
        if ((unsure >> k & 1) && fxd_weak(Sm, ty + k * ATY, tx, j0 + ty + k * ATY > 0, thr, d.hccd != 0))
            atomicOr(&Sm.redo, 1u << k);
    __syncthreads();
    const unsigned redo = Sm.redo;
    if (tid < 2 && (redo >> tid & 1)) F.tlist[atomicAdd(F.pcount + 1, 1u)] = (2 * blockIdx.y + tid) * gridDim.x + blockIdx.x;
    flows &= ~redo;
    for (int k = 0; k < 2; k++)
        if (flows >> k & 1)
            F.plist[atomicAdd(F.pcount, 1u)] = (unsigned)((size_t)(j0 + ty + k * ATY + 1) * m + i);
}

// What k_direct_fx left: the listed cells' plastic part and the listed tiles.
__global__ void __launch_bounds__(ATX * ATY)
    k_direct_rest(step_consts c, direct_consts d, fields_dev F, int cur, double dt, double bv, int tiles_x) {
    const unsigned cnt = F.pcount[0], tiles = F.pcount[1];
    const double *__restrict__ const *A = F.f[cur];
    double *const *B = F.f[cur ^ 1];
    const int tid = threadIdx.y * ATX + threadIdx.x;
    const stz_law_params<double> lp = law_params(c);
    const double strain = 1 / (2 * c.mu);
    for (unsigned k = blockIdx.x * (ATX * ATY) + tid; k < cnt; k += gridDim.x * (ATX * ATY)) {
        const size_t ci = F.plist[k];
        const double q = A[F_Q][ci], s = A[F_S][ci], t = A[F_TAU][ci];
        const double devsq = 3 * q * q + s * s + t * t;
        if (devsq < 0.999e-24 || (c.stz_model >= 2 && devsq < c.yield_cut2)) continue;
        int iters;
        double chi = B[F_CHI][ci], ddev = 0;
        const double sbar = sqrt(devsq), dtmp = adaptive_plastic(lp, sbar, chi, ddev, dt, iters);
        if (iters >= c.substep_cap) atomicExch(&F.flags[FL_SUBSTEP_CAP], 1);
        if (iters > 1) atomicMax(&F.flags[FL_SUBSTEP_MAX], iters);
        B[F_CHI][ci] = chi;
        F.ddev[ci] = ddev * sbar;
        if (c.track_plastic && ddev != 0) {
            const int m = c.m, j = (int)(ci / (size_t)m) - 1, i = (int)(ci - (size_t)(j + 1) * m);
            F.eps_pl[(size_t)j * m + i] += ddev * strain;
        }
        if (dtmp != 0) {
            B[F_Q][ci] -= dtmp * q;
            B[F_S][ci] -= dtmp * s;
            B[F_TAU][ci] -= dtmp * t;
        }
    }
    for (unsigned k = blockIdx.x; k < tiles; k += gridDim.x) {
        const unsigned tile = F.tlist[k];
        direct_tile_step(c, d, F, cur, dt, bv, tile % tiles_x, tile / tiles_x);
        __syncthreads();  // the next tile reuses the shared memory
    }
}

__global__ void k_precombine(step_consts c, fields_dev F, int cur, double xf, double yf) {
    const int m = c.m, n = c.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= m || j >= n) return;
    const size_t k = IDX(i, j);
    const double pn = F.f[cur][F_P][k], qn = F.f[cur][F_Q][k], sn = F.f[cur][F_S][k], tn = F.f[cur][F_TAU][k];
    const double pq = pn + qn, Aa = pq - sn, Bb = pq + sn;
    F.pre[0][k] = xf * Aa + yf * tn;
    F.pre[1][k] = xf * Aa - yf * tn;
    F.pre[2][k] = xf * tn - yf * Bb;
    F.pre[3][k] = xf * tn + yf * Bb;
}

// chi_diffusion (shear_sim.cc:364-386): B.chi holds cchi; old chi in A.
__global__ void k_chi_diffusion(step_consts c, fields_dev F, int cur, double dt) {
    const int m = c.m, n = c.n;
    if (c.clock) cur = (int)c.clock[CLK_CUR];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= m || j >= n) return;
    const double hx = 0.5 * c.xsp * dt, hy = 0.5 * c.ysp * dt;
    const double hxxcd = 2 * c.xsp * hx * c.chi_diff, hyycd = 2 * c.ysp * hy * c.chi_diff,
                 hccd = 2 * (hxxcd + hyycd);
    const double dfac = 0.25 * c.chi_len * c.chi_len * (1 / c.mu), dfacx = dfac * c.xsp * c.xsp,
                 dfacy = dfac * c.ysp * c.ysp;
    const double *ch = F.f[cur][F_CHI], *dd = F.ddev;
    const int il = i == 0 ? m - 1 : i - 1, ir = i == m - 1 ? 0 : i + 1;
    const size_t k = IDX(i, j), kl = IDX(il, j), kr = IDX(ir, j), kd = IDX(i, j - 1), ku = IDX(i, j + 1);
    const double Dd = dd[k] + dd[kd], Dl = dd[k] + dd[kl], Dr = dd[k] + dd[kr], Du = dd[k] + dd[ku];
    F.f[cur ^ 1][F_CHI][k] += hxxcd * (ch[kr] + ch[kl]) + hyycd * (ch[ku] + ch[kd]) - hccd * ch[k] +
                              dfacx * (Dr * ch[kr] - (Dr + Dl) * ch[k] + Dl * ch[kl]) +
                              dfacy * (Du * ch[ku] - (Du + Dd) * ch[k] + Dd * ch[kd]);
}

// Source of the projection (shear_sim.cc:399-409): net force of the stress
// on interior nodes from the four surrounding cells (net_force,
// shear_sim.cc:447-453) as fx = U(i,j-1) - W(i-1,j-1) + W(i,j) - U(i-1,j),
// fy = Y1(i-1,j-1) - Y2(i,j-1) + Y2(i-1,j) - Y1(i,j); Dirichlet data on the
// walls.
__global__ void k_source(step_consts c, fields_dev F, double xbc_bv) {
    const int m = c.m, n = c.n;
    if (c.clock) xbc_bv = c.xbc * c.clock[CLK_BV];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= m || j > n) return;
    double2 f;
    if (j == 0) {
        f.x = -xbc_bv;
        f.y = 0;
    } else if (j == n) {
        f.x = xbc_bv;
        f.y = 0;
    } else {
        const int il = i == 0 ? m - 1 : i - 1;
        const size_t k0 = IDX(il, j - 1), k1 = IDX(i, j - 1), k2 = IDX(il, j), k3 = IDX(i, j);
        const double *U = F.pre[0], *W = F.pre[1], *Y1 = F.pre[2], *Y2 = F.pre[3];
        f.x = (U[k1] - W[k0]) + (W[k3] - U[k2]);
        f.y = (Y1[k0] - Y2[k1]) + (Y2[k2] - Y1[k3]);
    }
    F.src[(size_t)j * m + i] = f;
}

// The projection source of the float-float path (mixed handles, whose
// advection writes no per-cell combinations): net_force (shear_sim.cc:447-453) at the interior
// nodes from the stresses of the four surrounding cells.  A block of 32 x 32
// nodes (four rows per thread) first forms, for each of the 33 x 33 cells
// around it, the pairs
// A = p + q - s, B = p + q + s and tau from the split stresses (float-float
// sums, error ~2^-47 of the values) in shared memory; each node then takes
// the cell-to-cell differences of those pairs, whose high parts cancel
// exactly where the cells agree, so the force keeps ~2^-44 of its own size
// plus ~2^-47 of the stresses, and scales them by xf, yf in pairs.  The wall
// rows as k_source.
struct source_ff_consts {
    float xfh, xfl, yfh, yfl;
};

constexpr int SFX = 32, SFY = 8;  // threads of a block
constexpr int SFR = 4;            // node (cell) rows per thread: a block covers 32 x 32

__global__ void __launch_bounds__(SFX * SFY) k_source_ff(step_consts c, fields_dev F, int cur, source_ff_consts h,
                                                         double xbc_bv) {
    constexpr int TY = SFY * SFR;  // node rows of the block
    __shared__ ff cA[TY + 1][SFX + 1], cB[TY + 1][SFX + 1], cT[TY + 1][SFX + 1];
    const int m = c.m, n = c.n;
    if (c.clock) {
        xbc_bv = c.xbc * c.clock[CLK_BV];
        cur = (int)c.clock[CLK_CUR] ^ 1;  // the state the advection wrote
    }
    const int i0 = blockIdx.x * SFX, j0 = blockIdx.y * TY;
    const int tid = threadIdx.y * SFX + threadIdx.x;
    const double *P = F.f[cur][F_P], *Q = F.f[cur][F_Q], *S = F.f[cur][F_S], *T = F.f[cur][F_TAU];
    // cells (i0 - 1 + cc, j0 - 1 + r); storage rows -1 .. n exist.  The
    // passes go in two halves, each issuing all its loads before it splits
    // anything, so that more loads are in flight per thread.
    constexpr int kCells = (TY + 1) * (SFX + 1), kPasses = (kCells + SFX * SFY - 1) / (SFX * SFY);
    constexpr int kHalf = (kPasses + 1) / 2;
#pragma unroll
    for (int h0 = 0; h0 < kPasses; h0 += kHalf) {
        double vp[kHalf], vq[kHalf], vs[kHalf], vt[kHalf];
        int rr[kHalf], cw[kHalf];
#pragma unroll
        for (int it = 0; it < kHalf; it++) {
            const int k = tid + (h0 + it) * SFX * SFY;
            const int r = k / (SFX + 1), cc = k - r * (SFX + 1);
            const int cj = j0 - 1 + r;
            int ci = i0 - 1 + cc;
            ci = ci < 0 ? ci + m : (ci >= m ? ci % m : ci);
            const bool live = h0 + it < kPasses && k < kCells && cj <= n;
            rr[it] = live ? r : -1;
            cw[it] = cc;
            const size_t q = live ? IDX(ci, cj) : 0;
            vp[it] = live ? P[q] : 0.0;
            vq[it] = live ? Q[q] : 0.0;
            vs[it] = live ? S[q] : 0.0;
            vt[it] = live ? T[q] : 0.0;
        }
#pragma unroll
        for (int it = 0; it < kHalf; it++) {
            if (rr[it] < 0) continue;
            const ff pp = split_ff(vp[it]), qq = split_ff(vq[it]), ss = split_ff(vs[it]);
            const ff pq = ff_add(pp, qq);
            cA[rr[it]][cw[it]] = ff_sub(pq, ss);
            cB[rr[it]][cw[it]] = ff_add(pq, ss);
            cT[rr[it]][cw[it]] = split_ff(vt[it]);
        }
    }
    __syncthreads();
    const int tx = threadIdx.x, i = i0 + tx;
    if (i >= m) return;
    const ff xf{h.xfh, h.xfl}, yf{h.yfh, h.yfl};
#pragma unroll
    for (int q = 0; q < SFR; q++) {
        const int ty = threadIdx.y + q * SFY, j = j0 + ty;
        if (j > n) break;
        double2 out;
        if (j == 0 || j == n) {
            out.x = j == 0 ? -xbc_bv : xbc_bv;
            out.y = 0;
        } else {
            // cells k0 = (i-1, j-1), k1 = (i, j-1), k2 = (i-1, j), k3 = (i, j)
            const ff dAx = ff_add(ff_sub(cA[ty][tx + 1], cA[ty][tx]), ff_sub(cA[ty + 1][tx + 1], cA[ty + 1][tx]));
            const ff dBy = ff_add(ff_sub(cB[ty + 1][tx], cB[ty][tx]), ff_sub(cB[ty + 1][tx + 1], cB[ty][tx + 1]));
            const ff dTy = ff_add(ff_sub(cT[ty][tx], cT[ty + 1][tx]), ff_sub(cT[ty][tx + 1], cT[ty + 1][tx + 1]));
            const ff dTx = ff_add(ff_sub(cT[ty][tx], cT[ty][tx + 1]), ff_sub(cT[ty + 1][tx], cT[ty + 1][tx + 1]));
            const ff fx = ff_add(ff_mul(xf, dAx), ff_mul(yf, dTy)), fy = ff_add(ff_mul(xf, dTx), ff_mul(yf, dBy));
            out.x = ff_to_d(fx.hi, fx.lo);
            out.y = ff_to_d(fy.hi, fy.lo);
        }
        F.src[(size_t)j * m + i] = out;
    }
}

// Stress correction from the solved velocity (shear_sim.cc:418-434).
__global__ void k_project(step_consts c, fields_dev F, int cur, double hx, double hy) {
    const int m = c.m, n = c.n;
    if (c.clock) cur = (int)c.clock[CLK_CUR] ^ 1;  // the state the advection wrote
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= m || j >= n) return;
    const int ir = i == m - 1 ? 0 : i + 1;
    const double2 a = F.vel[(size_t)j * m + i], b = F.vel[(size_t)j * m + ir], cu = F.vel[(size_t)(j + 1) * m + i],
                  d = F.vel[(size_t)(j + 1) * m + ir];
    const double ux = hx * (-a.x + b.x - cu.x + d.x), uy = hy * (-a.x - b.x + cu.x + d.x),
                 vx = hx * (-a.y + b.y - cu.y + d.y), vy = hy * (-a.y - b.y + cu.y + d.y);
    const size_t k = IDX(i, j);
    double *const *S = F.f[cur];
    const double third = 1 / 3.0;
    S[F_P][k] += -c.K * (ux + vy);
    S[F_Q][k] += -c.mu * third * (ux + vy);
    S[F_S][k] += c.mu * (ux - vy);
    S[F_TAU][k] += c.mu * (uy + vx);
}

// The stress correction of the float-float path: each node's velocity is
// split into float pairs once (a block of 32 x 32 cells, four rows per
// thread, stages its 33 x 33 nodes in shared memory), the velocity differences of k_project are taken
// from the pairs, the products with hx, hy, K, mu/3 and mu in pairs, and each
// stress component takes its correction with two FP64 additions.
struct project_ff_consts {
    float hxh, hxl, hyh, hyl, Kh, Kl, m3h, m3l, muh, mul;
};

__global__ void __launch_bounds__(SFX * SFY) k_project_ff(step_consts c, fields_dev F, int cur, project_ff_consts h) {
    constexpr int TY = SFY * SFR;  // cell rows of the block
    // velocities of the block's 33 x 33 nodes as pairs, split once each
    __shared__ ff nU[TY + 1][SFX + 1], nV[TY + 1][SFX + 1];
    const int m = c.m, n = c.n;
    if (c.clock) cur = (int)c.clock[CLK_CUR] ^ 1;  // the state the advection wrote
    const int i0 = blockIdx.x * SFX, j0 = blockIdx.y * TY;
    const int tid = threadIdx.y * SFX + threadIdx.x;
#pragma unroll
    for (int k = tid; k < (TY + 1) * (SFX + 1); k += SFX * SFY) {
        const int r = k / (SFX + 1), cc = k - r * (SFX + 1);
        const int nj = j0 + r;
        int ni = i0 + cc;
        ni = ni >= m ? ni % m : ni;
        if (nj > n) continue;
        const double2 v = F.vel[(size_t)nj * m + ni];
        nU[r][cc] = split_ff(v.x);
        nV[r][cc] = split_ff(v.y);
    }
    __syncthreads();
    const int tx = threadIdx.x, i = i0 + tx;
    if (i >= m) return;
    const ff hx{h.hxh, h.hxl}, hy{h.hyh, h.hyl};
    double *const *S = F.f[cur];
#pragma unroll
    for (int q = 0; q < SFR; q++) {
        const int ty = threadIdx.y + q * SFY, j = j0 + ty;
        if (j >= n) break;
        // nodes a = (i, j), b = (i+1, j), c = (i, j+1), d = (i+1, j+1)
        const ff ax = nU[ty][tx], bx = nU[ty][tx + 1], cx = nU[ty + 1][tx], dx = nU[ty + 1][tx + 1];
        const ff ay = nV[ty][tx], by = nV[ty][tx + 1], cy = nV[ty + 1][tx], dy = nV[ty + 1][tx + 1];
        const ff ux = ff_mul(hx, ff_add(ff_sub(bx, ax), ff_sub(dx, cx)));
        const ff uy = ff_mul(hy, ff_add(ff_sub(cx, ax), ff_sub(dx, bx)));
        const ff vx = ff_mul(hx, ff_add(ff_sub(by, ay), ff_sub(dy, cy)));
        const ff vy = ff_mul(hy, ff_add(ff_sub(cy, ay), ff_sub(dy, by)));
        const ff div = ff_add(ux, vy);
        const size_t k = IDX(i, j);
        S[F_P][k] = add_ff(S[F_P][k], ff_neg(ff_mul(ff{h.Kh, h.Kl}, div)));
        S[F_Q][k] = add_ff(S[F_Q][k], ff_neg(ff_mul(ff{h.m3h, h.m3l}, div)));
        S[F_S][k] = add_ff(S[F_S][k], ff_mul(ff{h.muh, h.mul}, ff_sub(ux, vy)));
        S[F_TAU][k] = add_ff(S[F_TAU][k], ff_mul(ff{h.muh, h.mul}, ff_add(uy, vx)));
    }
}

// set_boundaries (shear_sim.cc:552-581): ghost rows by linear extrapolation,
// wall nodes of the reference map.  Wall velocities are not stored: the
// advection kernel takes them as arguments.
__global__ void k_boundaries(step_consts c, fields_dev F, int cur, double bp) {
    const int m = c.m, n = c.n;
    if (c.clock) {
        bp = c.clock[CLK_BP];
        cur = (int)c.clock[CLK_CUR] ^ 1;
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    double *const *S = F.f[cur];
    S[F_X][IDX(i, 0)] = c.ax + i * c.dx + bp;
    S[F_Y][IDX(i, 0)] = c.ay;
    S[F_X][IDX(i, n)] = c.ax + i * c.dx - bp;
    S[F_Y][IDX(i, n)] = c.by;
    // all loads before the first store, which the compiler cannot prove
    // independent of them: one memory latency instead of ten (2.2 us a step)
    double lo[5], hi[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const double *G = S[k];
        lo[k] = 2 * G[IDX(i, 0)] - G[IDX(i, 1)];
        // n = 1: the row below the last one is the ghost row set here
        hi[k] = 2 * G[IDX(i, n - 1)] - (n > 1 ? G[IDX(i, n - 2)] : lo[k]);
    }
#pragma unroll
    for (int k = 0; k < 5; k++) {
        S[k][IDX(i, -1)] = lo[k];
        S[k][IDX(i, n)] = hi[k];
    }
}

#undef IDX

inline dim3 g2(int m, int n, dim3 b) { return dim3(ceil_div(m, b.x), ceil_div(n, b.y)); }

}  // namespace

size_t tile_count(const step_consts &c) { return (size_t)ceil_div(c.m, ATX) * ceil_div(c.n, ATY); }

cudaError_t prepare_step_kernels() {
    static unsigned long long done = 0;  // per device ordinal
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && (done >> dev & 1)) return cudaSuccess;
    e = cudaFuncSetAttribute(k_advect, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(adv_smem) + 128));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_advect_fx<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(fx_smem) + 128));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_advect_fx<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(fx_smem) + 128));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_advect_rest, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(adv_smem) + 128));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_direct_fx, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(fxd_smem) + 128));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_direct_rest, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(direct_tile));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_direct, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(direct_tile));
    if (e == cudaSuccess && dev < 64) done |= 1ull << dev;
    return e;
}

int make_field_maps(const step_consts &c, const fields_dev &F, field_maps *out) {
    typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static encode_fn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn)
            return fail(STZG_ECUDA, "cuTensorMapEncodeTiled is not available");
        encode = (encode_fn)fn;
    }
    // 16-byte rules: row stride m*8 and the box's inner extent ACOLS*8
    if ((c.m * sizeof(double)) % 16 != 0) return fail(STZG_EINVAL, "tile copies need an even m");
    const cuuint64_t dims[2] = {(cuuint64_t)c.m, (cuuint64_t)c.n + 2};
    const cuuint64_t strides[1] = {(cuuint64_t)c.m * sizeof(double)};
    const cuuint32_t estr[2] = {1, 1};
    for (int k = 0; k < 4 * F_COUNT; k++) {
        const int b = k & 1, f = k / 4;
        const bool tall = k & 2;
        const cuuint32_t box[2] = {ACOLS, (cuuint32_t)(tall ? FROWS : AROWS)};
        if (((uintptr_t)F.f[b][f]) % 16 != 0) return fail(STZG_EINVAL, "field not 16-byte aligned");
        const CUresult r =
            encode(tall ? &out->tall.f[b][f] : &out->f[b][f], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, (void *)F.f[b][f],
                   dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(STZG_ECUDA, "cuTensorMapEncodeTiled failed");
    }
    return STZG_OK;
}

static advect_fx_consts fx_consts(double hx, double hy) {
    advect_fx_consts h;
    int ex, ey;
    std::frexp(hx, &ex);
    std::frexp(hy, &ey);
    h.he = std::max(ex, ey) - 62;
    h.hmx = (long long)std::ldexp(hx, -h.he);
    h.hmy = (long long)std::ldexp(hy, -h.he);
    h.xf = h.yf = 0;
    return h;
}

void advection(const step_consts &c, const field_maps &maps, fields_dev &F, int cur, double dt, double bv,
               cudaStream_t st) {
    dim3 blk(32, 8);
    advect_consts a;
    a.hx = 0.5 * c.xsp * dt;
    a.hy = 0.5 * c.ysp * dt;
    a.xf = 0.5 / dt * c.xsp;
    a.yf = 0.5 / dt * c.ysp;
    const dim3 grid(ceil_div(c.m, ATX), ceil_div(c.n, ATY));
    if (c.fixed_point && std::isfinite(a.hx + a.hy)) {
        advect_fx_consts h = fx_consts(a.hx, a.hy);
        h.xf = a.xf;
        h.yf = a.yf;
        const int pre = !c.sp_increments;
        const dim3 fgrid(grid.x, ceil_div(c.n, FXY));
        cudaMemsetAsync(F.pcount, 0, 2 * sizeof(unsigned), st);
        if (pre)
            k_advect_fx<true><<<fgrid, dim3(ATX, ATY), sizeof(fx_smem) + 128, st>>>(c, h, maps.tall, F, cur, bv);
        else
            k_advect_fx<false><<<fgrid, dim3(ATX, ATY), sizeof(fx_smem) + 128, st>>>(c, h, maps.tall, F, cur, bv);
        note_launch();
        k_advect_rest<<<2 * 152, dim3(ATX, ATY), sizeof(adv_smem) + 128, st>>>(c, a, maps, F, cur, dt, bv, pre,
                                                                              (int)grid.x);
    } else {
        k_advect<<<grid, dim3(ATX, ATY), sizeof(adv_smem) + 128, st>>>(c, a, maps, F, cur, dt, bv, 1);
    }
    note_launch();
    if (c.chi_diff != 0 || c.chi_len != 0) {
        k_chi_diffusion<<<g2(c.m, c.n, blk), blk, 0, st>>>(c, F, cur, dt);
        note_launch();
    }
}

void direct_step(const step_consts &c, const field_maps &maps, double viscosity, fields_dev &F, int cur, double dt,
                 double bv, cudaStream_t st) {
    const double hx = 0.5 * c.xsp * dt, hy = 0.5 * c.ysp * dt;
    direct_consts d;
    d.hx = hx;
    d.hy = hy;
    d.mu_inv = 1 / c.mu;
    d.hxxv = 2 * c.xsp * hx * viscosity;
    d.hyyv = 2 * c.ysp * hy * viscosity;
    d.hcv = 2 * (d.hxxv + d.hyyv);
    d.hxxcd = 2 * c.xsp * hx * c.chi_diff;
    d.hyycd = 2 * c.ysp * hy * c.chi_diff;
    d.hccd = 2 * (d.hxxcd + d.hyycd);
    dim3 blk(ATX, ATY);
    const dim3 grid = g2(c.m, c.n, blk);
    if (c.fixed_point && std::isfinite(hx + hy)) {
        advect_fx_consts h = fx_consts(hx, hy);
        // second differences times these factors, cut at four units of 2^-59
        const double second = std::max((d.hxxv + d.hyyv) * d.mu_inv, d.hxxcd + d.hyycd);
        if (second > 0) std::frexp(second, &h.floor);
        h.floor += second > 0 ? 50 : 0;
        cudaMemsetAsync(F.pcount, 0, 2 * sizeof(unsigned), st);
        k_direct_fx<<<dim3(grid.x, ceil_div(c.n, FXY)), blk, sizeof(fxd_smem) + 128, st>>>(c, d, h, maps.tall, F, cur,
                                                                                          bv);
        note_launch();
        k_direct_rest<<<2 * 152, blk, sizeof(direct_tile), st>>>(c, d, F, cur, dt, bv, (int)grid.x);
    } else {
        k_direct<<<grid, blk, sizeof(direct_tile), st>>>(c, d, F, cur, dt, bv);
    }
    note_launch();
    if (c.chi_diff != 0 || c.chi_len != 0) {
        k_chi_diffusion<<<g2(c.m, c.n, blk), blk, 0, st>>>(c, F, cur, dt);
        note_launch();
    }
}

void projection_source(const step_consts &c, fields_dev &F, int cur, double dt, double xbc_bv, cudaStream_t st) {
    dim3 blk(32, 8);
    if (c.sp_increments) {
        source_ff_consts h;
        split_host(0.5 / dt * c.xsp, &h.xfh, &h.xfl);
        split_host(0.5 / dt * c.ysp, &h.yfh, &h.yfl);
        const dim3 sb(SFX, SFY);
        k_source_ff<<<g2(c.m, c.n + 1, dim3(SFX, SFY * SFR)), sb, 0, st>>>(c, F, cur, h, xbc_bv);
    } else {
        k_source<<<g2(c.m, c.n + 1, blk), blk, 0, st>>>(c, F, xbc_bv);
    }
    note_launch();
}

void precombine(const step_consts &c, fields_dev &F, int cur, double dt, cudaStream_t st) {
    if (c.sp_increments) return;  // k_source_ff reads the stresses themselves
    dim3 blk(32, 8);
    k_precombine<<<g2(c.m, c.n, blk), blk, 0, st>>>(c, F, cur, 0.5 / dt * c.xsp, 0.5 / dt * c.ysp);
    note_launch();
}

void projection_apply(const step_consts &c, fields_dev &F, int cur, double dt, double bv, double bp,
                      cudaStream_t st) {
    dim3 blk(32, 8);
    const double hx = 0.5 * c.xsp * dt, hy = 0.5 * c.ysp * dt;
    if (c.sp_increments) {
        project_ff_consts h;
        split_host(hx, &h.hxh, &h.hxl);
        split_host(hy, &h.hyh, &h.hyl);
        split_host(c.K, &h.Kh, &h.Kl);
        split_host(c.mu * (1 / 3.0), &h.m3h, &h.m3l);
        split_host(c.mu, &h.muh, &h.mul);
        const dim3 sb(SFX, SFY);
        k_project_ff<<<g2(c.m, c.n, dim3(SFX, SFY * SFR)), sb, 0, st>>>(c, F, cur, h);
    } else {
        k_project<<<g2(c.m, c.n, blk), blk, 0, st>>>(c, F, cur, hx, hy);
    }
    note_launch();
    k_boundaries<<<ceil_div(c.m, 128), 128, 0, st>>>(c, F, cur, bp); note_launch();
    (void)bv;
}

void set_boundaries(const step_consts &c, fields_dev &F, int cur, double bp, cudaStream_t st) {
    k_boundaries<<<ceil_div(c.m, 128), 128, 0, st>>>(c, F, cur, bp); note_launch();
}

}  // namespace stzg
