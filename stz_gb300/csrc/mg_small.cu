// V-cycles on windows in shared memory (mg_window.cuh): the small levels in
// one launch over a cluster of blocks, for float and float-pair hierarchies,
// and the wide levels of float-pair hierarchies as tiles.
//
// FP64 handles run their V-cycle in correction form: the residual r = b - A z
// of the FP64 iterate in FP64, one V-cycle from zero on A d = r in float
// pairs (~48 significant bits), z += d in FP64.  That is the reference's
// V-cycle (the cycle is linear in z and b) with the rounding of d at 2^-48
// of d itself, so the iterate keeps FP64 accuracy.  Powers of two on r
// (pair_range) and on the operator's tables (hierarchy::unit), exact both ways,
// keep the pairs inside FP32's exponents whatever the problem's magnitude; r's
// is taken once per solve, from b and z, since a maximum over r in front of
// every cycle cost 3 to 5 percent of it.  What bounds the cycle on
// GB300 is the FP64 pipe, two results per clock and SM: a pair operation
// costs 10 to 20 issue slots on the FP32 pipe where an FP64 one blocks its
// quarter of the SM for 64 clocks.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "ff.cuh"
#include "fixed.cuh"
#include "mg.cuh"
#include "mg_device.cuh"
#include "mg_plan.h"
#include "mg_env.cuh"
#include "mg_tiles.cuh"

namespace stzg {

using namespace mgw;

namespace {

// The small levels of one V-cycle.  Bound by the latency of its dependent
// phases (three to six per level and direction, 0.3 to 0.5 us each) and of the
// cluster barriers (two per level, 0.6 to 1 us with their remote stores): the
// work of a phase is a few microseconds of one SM at most.  Hence bands with
// halo rows (a level needs no exchange inside), a thread per 2 x 2 block, and
// the matrix in place of the levels below 450 nodes.  V-cycle at 64^2 / 128^2 /
// 512^2, FP32: 47 / - / 79 us with one launch per level, 17 / 23 / 54 us with
// this kernel; FP64 handles: 201 / 293 / 512 us with one FP64 launch per colour,
// 31 / 43 / 93 us in pairs.

template <typename S, bool FAST>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small(const __grid_constant__ small_plan<S> P) {
    extern __shared__ __align__(16) unsigned char small_raw[];
    pdl_start();
    block_env env{small_raw, (int)blockIdx.x};  // one cluster: its rank is the block index
    small_vcycle<FAST, false>(P, env);
}

__global__ void __launch_bounds__(kSmallThreads, 1)
    k_dense_columns(const __grid_constant__ small_plan<ff> P, float2 *out) {
    extern __shared__ __align__(16) unsigned char small_raw[];
    column_env env;
    env.mem = small_raw;
    env.r = 0;
    env.b0 = P.lv[P.t].bg;
    env.out = out;
    env.col = blockIdx.x;
    env.n = gridDim.x;
    small_vcycle<false, false>(P, env);
}

// r = b - A z of the top level, times 2^range->next, as float pairs; with a sink, the norms (as
// k_top_sqnorm).
// A z is evaluated on second differences of z, exact in 64-bit fixed point
// (fixed.cuh, one scale per tile), and integer products with the
// coefficients; only b - A z and the norms are FP64.  Coefficients are cut at 2^-60
// of the largest, which is exact within a factor of 2^7 of it; the error, in
// units of 2^-53 |cxx| max|z|, is 0.05 to 0.08 with square cells and 0.15 to 0.24
// at spacings of 1 to 8 up to 1 to 4096, the plain FP64 sum's 0.8 to 2.1.  FP64 operations per node: 31 in the plain form, which was
// bound by them (56 us at 1024^2), four here.
// A block walks tiles of 32 x 8 RPT nodes (RPT rows per thread) with the next
// tile's loads in flight: two rows per thread where that still gives each SM
// two tiles, else one (latency).  Tiles with an infinity or a NaN take the FP64 form.
constexpr int kResThreads = 256, RX = 32, RC = RX + 2, kResRows = kResThreads / RX;

// A coefficient over 2^ke, in two words, the lower one halved.
struct res_factor {
    int hi, lo;
};
struct res_consts {
    res_factor Kmx, Kmy, mx, my, qK, dxx, dyy;  // dxx = cxx + 2 (Kmx + my), dyy = cyy + 2 (mx + Kmy)
    int ke;
};
struct res_sum {
    long long H, M;
    __device__ __forceinline__ void add(const res_factor &w, long long a) {
        const int a1 = (int)(a >> 32), a0 = (int)((unsigned)a >> 1);
        H += (long long)w.hi * a1;
        M += (long long)w.lo * a1 + (long long)w.hi * a0;
    }
    // sum / 2^64; the 1 is the mean of the parts dropped
    __device__ __forceinline__ double value() const { return (double)(H + (M >> 31) + 1); }
};

template <int RPT>
__global__ void __launch_bounds__(kResThreads, 4)
    k_res_pairs(top_op<double> op, res_consts C, const double2 *__restrict__ z, const double2 *__restrict__ b, int m,
                int n, int tiles_x, int tiles, float4 *__restrict__ r, pair_range *range, norm_sink sink) {
    constexpr int RY = kResRows * RPT, RR = RY + 2;
    __shared__ long long X[RR][RC], Y[RR][RC];
    __shared__ unsigned top[2];
    __shared__ double sh[32];
    constexpr int kPer = (RR * RC + kResThreads - 1) / kResThreads;
    const int tid = threadIdx.x, tx = tid & (RX - 1), ty = tid / RX;
    double sr = 0, sb = 0;
    double2 v[kPer];
    auto load = [&](int tile) {
        const int i0 = (tile % tiles_x) * RX, j0 = (tile / tiles_x) * RY;
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int p = tid + q * kResThreads, row = p / RC, t = p - row * RC, j = j0 + row - 1;
            int i = i0 + t - 1;
            v[q] = make_double2(0.0, 0.0);
            if (p >= RR * RC || j < 0 || j >= n || i > m) continue;
            if (i < 0) i += m;
            if (i == m) i = 0;
            v[q] = z[(size_t)j * m + i];
        }
    };
    if (tid < 2) top[tid] = 0;
    pdl_wait();
    const int shift = __ldcg(&range->next);
    if ((int)blockIdx.x < tiles) load(blockIdx.x);
    __syncthreads();
    int it = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, it ^= 1) {
        const int i = (tile % tiles_x) * RX + tx, j0 = (tile / tiles_x) * RY;
        double2 g[RPT];
#pragma unroll
        for (int q = 0; q < RPT; q++) {
            const int j = j0 + ty * RPT + q;
            g[q] = i < m && j < n ? b[(size_t)j * m + i] : make_double2(0.0, 0.0);
        }
        unsigned w = 0;
#pragma unroll
        for (int q = 0; q < kPer; q++)
            w = max(w, max((unsigned)__double2hiint(v[q].x) & 0x7fffffffu, (unsigned)__double2hiint(v[q].y) & 0x7fffffffu));
        w = __reduce_max_sync(0xffffffffu, w);
        if (tx == 0) atomicMax(&top[it], w);
        __syncthreads();
        const int E = max((int)(top[it] >> 20), 128);
        const bool finite = E < 0x7ff;
        if (tid == 0) top[it ^ 1] = 0;
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int p = tid + q * kResThreads;
            if (p < RR * RC && finite) {
                (&X[0][0])[p] = to_fixed(v[q].x, E);
                (&Y[0][0])[p] = to_fixed(v[q].y, E);
            }
        }
        if (tile + (int)gridDim.x < tiles) load(tile + gridDim.x);
        __syncthreads();
        const double unit = power_of_two(64 + C.ke + E - 1081);
#pragma unroll
        for (int q = 0; q < RPT; q++) {
            const int row = ty * RPT + q, j = j0 + row;
            if (i >= m || j >= n) continue;
            const size_t k = (size_t)j * m + i;
            double2 e;
            if (j == 0 || j == n - 1 || !finite) {
                e = top_res<double>(op, z, b, m, n, i, j);
            } else {
                const long long *x = &X[row + 1][tx + 1], *y = &Y[row + 1][tx + 1];
                const long long x0 = x[0], y0 = y[0];
                res_sum ax{0, 0}, ay{0, 0};
                ax.add(C.Kmx, (x[-1] - x0) + (x[1] - x0));
                ax.add(C.my, (x[-RC] - x0) + (x[RC] - x0));
                ax.add(C.qK, (y[-RC - 1] - y[-RC + 1]) + (y[RC + 1] - y[RC - 1]));
                ax.add(C.dxx, x0);
                ay.add(C.mx, (y[-1] - y0) + (y[1] - y0));
                ay.add(C.Kmy, (y[-RC] - y0) + (y[RC] - y0));
                ay.add(C.qK, (x[-RC - 1] - x[-RC + 1]) + (x[RC + 1] - x[RC - 1]));
                ay.add(C.dyy, y0);
                e = make_double2(fma(-unit, ax.value(), g[q].x), fma(-unit, ay.value(), g[q].y));
            }
            float4 o;
            ff_split_shifted(e.x, shift, o.x, o.z);
            ff_split_shifted(e.y, shift, o.y, o.w);
            r[k] = o;
            if (sink.partials) {
                sr += e.x * e.x + e.y * e.y;
                sb += g[q].x * g[q].x + g[q].y * g[q].y;
            }
        }
        __syncthreads();  // the next tile reuses the planes
    }
    if (!sink.partials) {
        if (tid == 0 && blockIdx.x == 0) range->used = shift;
        return;
    }
    const double a = block_sum(sr, sh), c = block_sum(sb, sh);
    finish_norms(a, c, sink, sh, range, shift);
}

// The power of two that brings the largest of |b| and 4 2^unit |z|, a bound on
// A z and so (with b) on the residual up to a factor of 2, to [1, 2); 1 where a
// value is not finite.
__global__ void __launch_bounds__(kResThreads)
    k_pair_begin(const double2 *__restrict__ z, const double2 *__restrict__ b, unsigned count, int unit,
                 pair_range *range) {
    __shared__ unsigned top;
    if (threadIdx.x == 0) top = 0;
    __syncthreads();
    int e = 0;
#pragma unroll 4
    for (unsigned k = blockIdx.x * kResThreads + threadIdx.x; k < count; k += gridDim.x * kResThreads) {
        const double2 v = z[k], w = b[k];
        const int ez = max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff) >> 20;
        const int eb = max(__double2hiint(w.x) & 0x7fffffff, __double2hiint(w.y) & 0x7fffffff) >> 20;
        if (ez == 0x7ff || eb == 0x7ff) e = 1 << 16;
        else e = max(e, max(eb, ez ? ez + unit + 2 : 0));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&top, (unsigned)e);
    __syncthreads();
    if (threadIdx.x != 0) return;
    atomicMax(&range->top, top);
    __threadfence();
    if (atomicAdd(&range->arrived, 1u) != gridDim.x - 1) return;
    __threadfence();
    const int all = (int)atomicExch(&range->top, 0u);
    range->arrived = 0;
    range->next = all == 0 || all >= 1 << 16 ? 0 : min(max(1023 - all, -1000), 1000);
}

// ---- host ----------------------------------------------------------------------

ff pair_of(double d) {
    ff r;
    r.hi = (float)d;
    r.lo = (float)(d - (double)r.hi);
    return r;
}

top_consts<ff> consts_of(const top_op<double> &o, int unit) {
    auto coef = [&](double d) { return pair_of(std::ldexp(d, -unit)); };
    auto inverse = [&](double d) { return pair_of(std::ldexp(d, unit)); };
    top_consts<ff> c;
    c.Kmx = coef(o.Kmx); c.Kmy = coef(o.Kmy); c.mx = coef(o.mx); c.my = coef(o.my); c.qK = coef(o.qK);
    c.cxx = coef(o.cxx); c.cyy = coef(o.cyy); c.icxx = inverse(o.icxx); c.icyy = inverse(o.icyy);
    c.bcxx = coef(o.bcxx); c.bcyy = coef(o.bcyy); c.ibcxx = inverse(o.ibcxx); c.ibcyy = inverse(o.ibcyy);
    return c;
}
top_consts<float> consts_of(const top_op<float> &o, int) {
    return top_consts<float>{o.Kmx, o.Kmy, o.mx, o.my, o.qK, o.cxx, o.cyy, o.icxx, o.icyy, o.bcxx, o.bcyy, o.ibcxx, o.ibcyy};
}

template <typename T> const float4 *table_of(const hierarchy<T> &h, int l, float) {
    return reinterpret_cast<const float4 *>(h.lv[l].st);
}
template <typename T> const float4 *table_of(const hierarchy<T> &h, int l, ff) { return h.st_pairs[l]; }
template <typename T> struct scalar_of;
template <> struct scalar_of<float> { typedef float type; };
template <> struct scalar_of<double> { typedef ff type; };

// Largest cluster the device takes for the small-level kernels (probed once
// per device; at least 1).
int max_blocks() {
    static std::atomic<int> known[64];  // several host threads may probe at once, to the same result
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    if (!known[dev]) {
        const void *k[4] = {(const void *)k_small<float, true>, (const void *)k_small<float, false>,
                            (const void *)k_small<ff, true>, (const void *)k_small<ff, false>};
        int c = 16;
        for (const void *f : k) c = std::min(c, cluster_limit(f));
        known[dev] = std::max(c, 1);
    }
    return known[dev];
}

// Levels t..d of h as a plan (not yet laid out).
template <typename S, typename T> void plan_levels(const hierarchy<T> &h, int t, int d, small_plan<S> &P) {
    std::memset(&P, 0, sizeof(P));
    for (int l = t; l <= d; l++) {
        const level_view<T> &L = h.lv[l];
        small_level<S> &D = P.lv[l];
        D.m = L.m;
        D.n = L.n;
        D.homog = L.homog;
        D.nst = L.nst;
        D.ncls = L.ncls;
        D.cls = L.cls;
        D.st = l ? table_of(h, l, S()) : nullptr;
    }
}

template <typename T>
bool plan_small(const hierarchy<T> &h, int t, int blocks, bool zero_start, small_plan<typename scalar_of<T>::type> &P) {
    typedef typename scalar_of<T>::type S;
    typedef typename num<S>::node node;
    if (t >= h.dense_from) return false;
    plan_levels(h, t, h.dense_from, P);
    P.top = t == 0;
    P.zero_start = zero_start;
    P.dense = h.dense;
    P.op = consts_of(h.op, h.unit);
    P.unit = h.unit;
    P.range = h.range;
    P.lv[t].zg = reinterpret_cast<node *>(h.lv[t].z);
    P.lv[t].bg = reinterpret_cast<const node *>(h.lv[t].b);
    return layout_small(P, t, h.dense_from, blocks, kSmallMax);
}

// Levels of at most this many nodes go to the small-level kernel, where its
// shared memory holds them.  Its blocks are one cluster, 16 of the chip's 152
// SMs, so wider levels are faster as one launch each over the whole chip.  Whole
// V-cycles with the limit at 9,000 / 17,000 / 35,000 nodes, us:
//   float pairs, 158x157 59.7 / 59.7 / 71.8, 256x256 64.1 / 60.3 / 60.2,
//     256x400 71.5 / 71.5 / 76.6, 96x256 48.2 / 48.3 / 46.4, 96x330 54.6 / 54.6
//     / 76.3; 512^2 and 1024^2 change by 1 percent or not at all (their next
//     level does not fit);
//   FP32, 158x157 40.3 / 40.2 / 45.2, 256x256 41.8 / 35.9 / 36.0, 1024^2 74.5 /
//     71.9 / 71.8 (77.8 without a limit); narrow grids would take more (64x400
//     51.2 / 51.2 / 28.5, 96x256 31.2 / 31.2 / 27.3).
constexpr long kSmallPoints = 17000;

// First level of the small-level kernel and its cluster size; false where no
// level fits.
template <typename T>
bool choose_small(const hierarchy<T> &h, bool zero_start, small_plan<typename scalar_of<T>::type> &P) {
    const int cap = std::min(max_blocks(), std::max(1, h.small_blocks));
    if (!h.dense) return false;
    for (int t = 0; t < h.dense_from; t++) {
        if ((long)h.lv[t].m * h.lv[t].n > kSmallPoints) continue;
        for (int c = cap; c >= 1; c >>= 1)
            if (plan_small(h, t, c, zero_start, P)) return true;
    }
    return false;
}

template <typename S> void launch_small(const small_plan<S> &P, bool early, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    cluster_config(cfg, at, P.blocks, P.bytes, st, early);
    if (block_phases(P)) cudaLaunchKernelEx(&cfg, k_small<S, true>, P);
    else cudaLaunchKernelEx(&cfg, k_small<S, false>, P);
    note_launch();
}

constexpr size_t kTileMax = 200 * 1024;

// A wide level's arrays and tiles on the way down (up = false) or up.
tile_level plan_tile(const hierarchy<double> &h, int l, bool up, bool &bands, size_t &bytes) {
    const level_view<double> &A = h.lv[l], &C = h.lv[l + 1];
    tile_level L;
    std::memset(&L, 0, sizeof(L));
    L.m = A.m;
    L.n = A.n;
    L.cm = C.m;
    L.cn = C.n;
    L.homog = A.homog;
    L.nst = A.nst;
    L.cls = A.cls;
    L.st = l ? h.st_pairs[l] : nullptr;
    L.staged = l && A.homog && A.nst * 320 <= 16384;
    L.b = reinterpret_cast<const float4 *>(l ? A.b : A.r);
    L.zdown = l ? reinterpret_cast<float4 *>(A.r) : h.top_pairs;
    L.zup = reinterpret_cast<float4 *>(A.z);
    L.bc = reinterpret_cast<float4 *>(C.b);
    L.zc = reinterpret_cast<const float4 *>(C.z);
    if (!l) {
        L.sum = A.z;
        L.range = h.range;
        L.unit = h.unit;
    }
    bands = l && ((A.m & 1) || !A.homog);
    const tile_shape T = shape_tile(L.m, L.cm, L.cn, L.staged ? A.nst * 320 : 0, l ? 0 : (up ? 2 : 1), bands, kTileMax);
    L.tw = T.tw;
    L.th = T.th;
    L.threads = T.threads;
    bytes = T.bytes;
    return L;
}

template <typename... K, typename... A>
void launch_tile(void (*kern)(K...), const tile_level &L, bool bands, size_t smem, bool early, cudaStream_t st,
                 A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(bands ? 1 : ceil_div(L.cm, L.tw), ceil_div(L.cn, L.th));
    cfg.blockDim = dim3(L.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = early;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, args...);
    note_launch();
}

bool prepare_tiles() {
    static std::atomic<int> known[64];  // several host threads may probe at once, to the same result
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    if (!known[dev]) {
        const void *k[6] = {(const void *)k_pair_lev_down<true>, (const void *)k_pair_lev_down<false>,
                            (const void *)k_pair_lev_up<true>,   (const void *)k_pair_lev_up<false>,
                            (const void *)k_pair_top_down,       (const void *)k_pair_top_up};
        bool ok = true;
        for (const void *f : k)
            ok = ok && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileMax) == cudaSuccess;
        known[dev] = ok ? 1 : 2;
    }
    return known[dev] == 1;
}

}  // namespace

// The matrices of the V-cycle from each level ml, ml-1 .. d on: the coarsest
// level's is its inverse; a finer one's columns are the V-cycle's results on
// unit right-hand sides, one block each, with the next matrix at its bottom.
int build_dense(hierarchy<double> &h, const std::vector<double> &inverse, std::vector<void *> &own, size_t *cap) {
    h.dense = nullptr;
    const int ml = h.nl - 1;
    if (ml < 1 || inverse.empty()) return STZG_OK;
    h.dense_from = dense_level(ml, [&](int l) { return (long)h.lv[l].m * h.lv[l].n; });
    STZG_CUDA(cudaFuncSetAttribute(k_dense_columns, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallMax));
    size_t at[17] = {0}, all = 0;
    for (int l = ml; l >= h.dense_from; l--) {
        at[l] = all;
        all += 4 * (size_t)h.lv[l].m * h.lv[l].n * h.lv[l].m * h.lv[l].n;
    }
    if (*cap < all) {
        void *p = nullptr;
        cudaError_t e = cudaMalloc(&p, all * sizeof(float2));
        if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(dense levels)");
        own.push_back(p);
        h.dense_buf = (float2 *)p;
        *cap = all;
    }
    const float4 *next = nullptr;
    for (int l = ml; l >= h.dense_from; l--) {
        const size_t N = 2 * (size_t)h.lv[l].m * h.lv[l].n, bytes = N * N * sizeof(float2);
        float2 *const M = h.dense_buf + at[l];
        if (l == ml) {
            std::vector<float2> pairs(N * N);
            for (size_t k = 0; k < N * N; k++) {
                const ff v = pair_of(std::ldexp(inverse[k], h.unit));
                pairs[k] = make_float2(v.hi, v.lo);
            }
            STZG_CUDA(cudaMemcpy(M, pairs.data(), bytes, cudaMemcpyHostToDevice));
        } else {
            small_plan<ff> P;
            plan_levels(h, l, l + 1, P);
            P.dense = next;
            if (!layout_small(P, l, l + 1, 1, kSmallMax)) return STZG_OK;  // the older kernels serve it
            k_dense_columns<<<(unsigned)N, kSmallThreads, P.bytes>>>(P, M);
            note_launch();
            STZG_CUDA(cudaGetLastError());
        }
        next = reinterpret_cast<const float4 *>(M);
    }
    STZG_CUDA(cudaStreamSynchronize(cudaStreamLegacy));  // the handle's streams do not wait for this one
    h.dense = next;
    return STZG_OK;
}

bool pair_cycle_supported(const hierarchy<double> &h) {
    if (!h.fuse || h.tail_limit >= 0 || h.nl < 2 || !h.dense || !h.top_pairs || !prepare_tiles()) return false;
    small_plan<ff> P;
    if (!choose_small(h, true, P)) return false;
    for (int l = 0; l < P.t; l++) {
        bool bands;
        size_t bytes;
        plan_tile(h, l, true, bands, bytes);
        if (bytes > kTileMax) return false;
    }
    return true;
}

void pair_residual(const hierarchy<double> &h, const norm_sink *sink, cudaStream_t st) {
    const level_view<double> &T0 = h.lv[0];
    const top_op<double> &o = h.op;
    res_consts C;
    std::frexp(std::max(std::max(std::fabs(o.Kmx), std::fabs(o.Kmy)),
                        std::max(std::max(std::fabs(o.mx), std::fabs(o.my)), std::fabs(o.qK))), &C.ke);
    C.ke -= 61;  // the largest magnitude is in [2^60, 2^61)
    auto factor = [&](double d) {
        const long long w = (long long)std::ldexp(d, -C.ke);
        return res_factor{(int)(w >> 32), (int)((unsigned)w >> 1)};
    };
    C.Kmx = factor(o.Kmx);
    C.Kmy = factor(o.Kmy);
    C.mx = factor(o.mx);
    C.my = factor(o.my);
    C.qK = factor(o.qK);
    // with the rounding error of the sums, which the second differences make up for
    auto excess = [](double c, double p, double q) {
        const double s = p + q, t = s - p, e = (p - (s - t)) + (q - t);
        return (c + 2 * s) + 2 * e;
    };
    C.dxx = factor(excess(o.cxx, o.Kmx, o.my));
    C.dyy = factor(excess(o.cyy, o.mx, o.Kmy));
    auto run = [&](auto kernel, int rows) {
        const int tiles_x = ceil_div(T0.m, RX), tiles = tiles_x * ceil_div(T0.n, rows);
        launch_early(
            !h.crowded && (long)T0.m * T0.n <= kEarlyPoints, kernel, dim3(std::min(reduction_blocks(), tiles)), dim3(kResThreads), 0, st, o, C, (const double2 *)T0.z,
            (const double2 *)T0.b, T0.m, T0.n, tiles_x, tiles, reinterpret_cast<float4 *>(T0.r), h.range,
            sink ? *sink : norm_sink{nullptr, 0, nullptr, {}});
    };
    if (ceil_div(T0.m, RX) * ceil_div(T0.n, 2 * kResRows) < 2 * 152) run(k_res_pairs<1>, kResRows);
    else run(k_res_pairs<2>, 2 * kResRows);
    note_launch();
}

void pair_begin(const hierarchy<double> &h, cudaStream_t st) {
    if (!pair_cycle_supported(h)) return;
    const level_view<double> &T0 = h.lv[0];
    const long count = (long)T0.m * T0.n;
    k_pair_begin<<<std::min(4 * 152, ceil_div(count, kResThreads)), kResThreads, 0, st>>>(T0.z, T0.b, (unsigned)count,
                                                                                          h.unit, h.range);
    note_launch();
}

void pair_cycle(const hierarchy<double> &h, cudaStream_t st) {
    small_plan<ff> P;
    if (!choose_small(h, true, P)) return;
    const top_consts<ff> op = consts_of(h.op, h.unit);
    for (int l = 0; l < P.t; l++) {
        bool bands;
        size_t bytes;
        const tile_level L = plan_tile(h, l, false, bands, bytes);
        if (l == 0) launch_tile(k_pair_top_down, L, false, bytes, !h.crowded, st, op, L);
        else if (bands) launch_tile(k_pair_lev_down<true>, L, true, bytes, !h.crowded, st, L);
        else launch_tile(k_pair_lev_down<false>, L, false, bytes, !h.crowded, st, L);
    }
    if (P.t == 0) {
        P.lv[0].bg = reinterpret_cast<const float4 *>(h.lv[0].r);
        P.sum = h.lv[0].z;
    }
    launch_small(P, !h.crowded, st);
    for (int l = P.t - 1; l >= 0; l--) {
        bool bands;
        size_t bytes;
        const tile_level L = plan_tile(h, l, true, bands, bytes);
        if (l == 0) launch_tile(k_pair_top_up, L, false, bytes, !h.crowded, st, op, L);
        else if (bands) launch_tile(k_pair_lev_up<true>, L, true, bytes, !h.crowded, st, L);
        else launch_tile(k_pair_lev_up<false>, L, false, bytes, !h.crowded, st, L);
    }
}

int small_first(const hierarchy<float> &h) {
    small_plan<float> P;
    return choose_small(h, true, P) ? P.t : -1;
}

void small_levels(const hierarchy<float> &h, bool zero_start, cudaStream_t st) {
    small_plan<float> P;
    if (choose_small(h, zero_start, P)) launch_small(P, !h.crowded, st);
}

}  // namespace stzg
