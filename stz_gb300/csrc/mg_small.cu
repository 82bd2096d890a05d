// V-cycles on windows in shared memory (mg_window.cuh): the small levels in
// one launch over a cluster of blocks, for float and float-pair hierarchies,
// and the wide levels of float-pair hierarchies as tiles.
//
// FP64 handles run their V-cycle in correction form: the residual r = b - A z
// of the FP64 iterate in FP64, one V-cycle from zero on A d = r in float
// pairs (~48 significant bits), z += d in FP64.  That is the reference's
// V-cycle (the cycle is linear in z and b) with the rounding of d at 2^-48
// of d itself, so the iterate keeps FP64 accuracy.  What bounds the cycle on
// GB300 is the FP64 pipe, two results per clock and SM: a pair operation
// costs 10 to 20 issue slots on the FP32 pipe where an FP64 one blocks its
// quarter of the SM for 64 clocks.
#include <algorithm>
#include <cstring>

#include "ff.cuh"
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
// 512^2, FP32: 47 / - / 79 us with one launch per level, 20 / 29 / 67 us with
// this kernel; FP64 handles: 201 / 293 / 512 us with one FP64 launch per colour,
// 35 / 51 / 122 us in pairs.

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

// r = b - A z of the top level in FP64 as float pairs; with partials, the sums
// of r^2 and b^2 per block (as k_top_sqnorm).
constexpr int kResThreads = 256;
__global__ void __launch_bounds__(kResThreads) k_res_pairs(top_op<double> op, const double2 *__restrict__ z,
                                                           const double2 *__restrict__ b, int m, int n,
                                                           float4 *__restrict__ r, double *partials) {
    __shared__ double sh[32];
    const unsigned total = (unsigned)m * (unsigned)n;
    double sr = 0, sb = 0;
    for (unsigned k = blockIdx.x * kResThreads + threadIdx.x; k < total; k += gridDim.x * kResThreads) {
        const int j = (int)(k / (unsigned)m), i = (int)k - j * m;
        const double2 v = top_res<double>(op, z, b, m, n, i, j);
        float4 o;
        ff_split_d(v.x, o.x, o.z);
        ff_split_d(v.y, o.y, o.w);
        r[k] = o;
        if (partials) {
            const double2 bb = b[k];
            sr += v.x * v.x + v.y * v.y;
            sb += bb.x * bb.x + bb.y * bb.y;
        }
    }
    if (!partials) return;
    const double a = block_sum(sr, sh), c = block_sum(sb, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = a;
        partials[2 * blockIdx.x + 1] = c;
    }
}

// ---- host ----------------------------------------------------------------------

ff pair_of(double d) {
    ff r;
    r.hi = (float)d;
    r.lo = (float)(d - (double)r.hi);
    return r;
}

top_consts<ff> consts_of(const top_op<double> &o) {
    top_consts<ff> c;
    c.Kmx = pair_of(o.Kmx); c.Kmy = pair_of(o.Kmy); c.mx = pair_of(o.mx); c.my = pair_of(o.my); c.qK = pair_of(o.qK);
    c.cxx = pair_of(o.cxx); c.cyy = pair_of(o.cyy); c.icxx = pair_of(o.icxx); c.icyy = pair_of(o.icyy);
    c.bcxx = pair_of(o.bcxx); c.bcyy = pair_of(o.bcyy); c.ibcxx = pair_of(o.ibcxx); c.ibcyy = pair_of(o.ibcyy);
    return c;
}
top_consts<float> consts_of(const top_op<float> &o) {
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
    static int known[64];
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
    P.op = consts_of(h.op);
    P.lv[t].zg = reinterpret_cast<node *>(h.lv[t].z);
    P.lv[t].bg = reinterpret_cast<const node *>(h.lv[t].b);
    return layout_small(P, t, h.dense_from, blocks, kSmallMax);
}

// Levels of at most this many nodes go to the small-level kernel.  Its blocks
// are one cluster, 16 of the chip's 152 SMs, so wider levels are faster as one
// launch each over the whole chip.  Measured whole V-cycles, first level at
// 17,000 / 66,000 nodes, FP32 at 512^2: 76 / 82 us; 17,000 / 27,000, float
// pairs at 1024^2: 280 / 272 us (before the matrix of the coarsest levels).
constexpr long kSmallPoints32 = 17000, kSmallPoints64 = 27000;

// First level of the small-level kernel and its cluster size; false where no
// level fits.
template <typename T>
bool choose_small(const hierarchy<T> &h, bool zero_start, small_plan<typename scalar_of<T>::type> &P) {
    const long limit = sizeof(T) == 4 ? kSmallPoints32 : kSmallPoints64;
    const int cap = std::min(max_blocks(), std::max(1, h.small_blocks));
    if (!h.dense) return false;
    for (int t = 0; t < h.dense_from; t++) {
        if ((long)h.lv[t].m * h.lv[t].n > limit) continue;
        for (int c = cap; c >= 1; c >>= 1)
            if (plan_small(h, t, c, zero_start, P)) return true;
    }
    return false;
}

template <typename S> void launch_small(const small_plan<S> &P, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    cluster_config(cfg, at, P.blocks, P.bytes, st);
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
    if (!l) L.sum = h.lv[0].z;
    bands = l && ((A.m & 1) || !A.homog);
    const tile_shape T = shape_tile(L.m, L.cm, L.cn, L.staged ? A.nst * 320 : 0, l ? 0 : (up ? 2 : 1), bands, kTileMax);
    L.tw = T.tw;
    L.th = T.th;
    L.threads = T.threads;
    bytes = T.bytes;
    return L;
}

template <typename... K, typename... A>
void launch_tile(void (*kern)(K...), const tile_level &L, bool bands, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(bands ? 1 : ceil_div(L.cm, L.tw), ceil_div(L.cn, L.th));
    cfg.blockDim = dim3(L.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, args...);
    note_launch();
}

bool prepare_tiles() {
    static int known[64];
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
template <typename T> int build_dense(hierarchy<T> &h, const std::vector<double> &inverse, std::vector<void *> &own,
                                      size_t *caps) {
    h.dense = nullptr;
    const int ml = h.nl - 1;
    if (ml < 1 || inverse.empty()) return STZG_OK;
    h.dense_from = dense_level(ml, [&](int l) { return (long)h.lv[l].m * h.lv[l].n; });
    STZG_CUDA(cudaFuncSetAttribute(k_dense_columns, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallMax));
    const float4 *next = nullptr;
    for (int l = ml; l >= h.dense_from; l--) {
        const size_t N = 2 * (size_t)h.lv[l].m * h.lv[l].n, bytes = N * N * sizeof(float2);
        if (caps[l] < bytes) {
            void *p = nullptr;
            cudaError_t e = cudaMalloc(&p, bytes);
            if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(dense levels)");
            own.push_back(p);
            h.dense_buf[l] = (float2 *)p;
            caps[l] = bytes;
        }
        if (l == ml) {
            std::vector<float2> pairs(N * N);
            for (size_t k = 0; k < N * N; k++) {
                const ff v = pair_of(inverse[k]);
                pairs[k] = make_float2(v.hi, v.lo);
            }
            STZG_CUDA(cudaMemcpy(h.dense_buf[l], pairs.data(), bytes, cudaMemcpyHostToDevice));
        } else {
            small_plan<ff> P;
            plan_levels(h, l, l + 1, P);
            P.dense = next;
            if (!layout_small(P, l, l + 1, 1, kSmallMax)) return STZG_OK;  // the older kernels serve it
            k_dense_columns<<<(unsigned)N, kSmallThreads, P.bytes>>>(P, h.dense_buf[l]);
            STZG_CUDA(cudaGetLastError());
        }
        next = reinterpret_cast<const float4 *>(h.dense_buf[l]);
    }
    STZG_CUDA(cudaStreamSynchronize(cudaStreamLegacy));  // the handle's streams do not wait for this one
    h.dense = next;
    return STZG_OK;
}
template int build_dense<float>(hierarchy<float> &, const std::vector<double> &, std::vector<void *> &, size_t *);
template int build_dense<double>(hierarchy<double> &, const std::vector<double> &, std::vector<void *> &, size_t *);

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

void pair_residual(const hierarchy<double> &h, double *partials, int npart, cudaStream_t st) {
    const level_view<double> &T0 = h.lv[0];
    const int blocks = partials ? npart : std::min(npart, ceil_div((long)T0.m * T0.n, kResThreads));
    k_res_pairs<<<blocks, kResThreads, 0, st>>>(h.op, T0.z, T0.b, T0.m, T0.n, reinterpret_cast<float4 *>(T0.r),
                                                partials);
    note_launch();
}

void pair_cycle(const hierarchy<double> &h, cudaStream_t st) {
    small_plan<ff> P;
    if (!choose_small(h, true, P)) return;
    const top_consts<ff> op = consts_of(h.op);
    for (int l = 0; l < P.t; l++) {
        bool bands;
        size_t bytes;
        const tile_level L = plan_tile(h, l, false, bands, bytes);
        if (l == 0) launch_tile(k_pair_top_down, L, false, bytes, st, op, L);
        else if (bands) launch_tile(k_pair_lev_down<true>, L, true, bytes, st, L);
        else launch_tile(k_pair_lev_down<false>, L, false, bytes, st, L);
    }
    if (P.t == 0) {
        P.lv[0].bg = reinterpret_cast<const float4 *>(h.lv[0].r);
        P.sum = h.lv[0].z;
    }
    launch_small(P, st);
    for (int l = P.t - 1; l >= 0; l--) {
        bool bands;
        size_t bytes;
        const tile_level L = plan_tile(h, l, true, bands, bytes);
        if (l == 0) launch_tile(k_pair_top_up, L, false, bytes, st, op, L);
        else if (bands) launch_tile(k_pair_lev_up<true>, L, true, bytes, st, L);
        else launch_tile(k_pair_lev_up<false>, L, false, bytes, st, L);
    }
}

int small_first(const hierarchy<float> &h) {
    small_plan<float> P;
    return choose_small(h, true, P) ? P.t : -1;
}

void small_levels(const hierarchy<float> &h, bool zero_start, cudaStream_t st) {
    small_plan<float> P;
    if (choose_small(h, zero_start, P)) launch_small(P, st);
}

}  // namespace stzg
