// The small levels of the general 2x2-block multigrid in one launch
// (mg_small.h).
#include "mg_small.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "mg_env.cuh"

namespace stzg {

using namespace mgw;

namespace {

// b and z of the first level are FP64 vectors of the size of a node.  Pairs have
// FP32's exponents, so b is taken times the power of two that brings its
// largest value to [1, 2), and z back (the tables are those of A 2^-unit).
// That value is a maximum over the cluster: one more barrier and a second
// look at b.
struct io_env : block_env {
    static constexpr bool kMeasured = true;
    unsigned *words;  // shared: the block's largest high word, the cluster's
    unsigned mine = 0;
    __device__ __forceinline__ double2 raw(const float4 *p) const {
        return __ldcg(reinterpret_cast<const double2 *>(p));
    }
    __device__ __forceinline__ void measure(const float4 *p) {
        const double2 v = raw(p);
        mine = max(mine, max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu));
    }
    __device__ __forceinline__ void measured() {
        mine = __reduce_max_sync(0xffffffffu, mine);
        if ((threadIdx.x & 31) == 0) atomicMax(&words[0], mine);
    }
    __device__ __forceinline__ void share(int tid, int nb) {
        if (tid >= nb) return;
        unsigned long long a;
        asm("mapa.u64 %0, %1, %2;\n" : "=l"(a) : "l"((unsigned long long)(words + 1)), "r"(tid));
        atomicMax((unsigned *)a, words[0]);
    }
    __device__ __forceinline__ int shift() const {
        const int e = (int)(words[1] >> 20);
        return e == 0x7ff ? 0 : 1023 - max(e, 1);
    }
    __device__ __forceinline__ float4 ld(const float4 *p) const {
        const double2 v = raw(p);
        const int s = shift();
        float4 o;
        ff_split_shifted(v.x, s, o.x, o.z);
        ff_split_shifted(v.y, s, o.y, o.w);
        return o;
    }
    __device__ __forceinline__ void store(const small_plan<ff> &P, size_t k, const float4 &v) const {
        const double back = pair_back(shift(), P.unit);
        reinterpret_cast<double2 *>(P.lv[P.t].zg)[k] =
            make_double2(ff_to_d(v.x, v.z) * back, ff_to_d(v.y, v.w) * back);
    }
};

constexpr unsigned kBlockMax = kSmallMax - 256;  // the rest for io_env's words

// FP64 V-cycle of a 512 x 256 grid of 2x2 blocks, y periodic: 520 us with one
// FP64 launch per colour on every level and a single-block FP64 tail of 215 us;
// 161 us with this kernel from level 2 (128 x 64) on, levels 0 and 1 still one
// launch per colour.  Four steps of that grid went from 25.0 to 12.8 ms.
template <bool FAST, bool YP>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small_blocks(const __grid_constant__ small_plan<ff> P) {
    extern __shared__ __align__(16) unsigned char small_raw[];
    pdl_start();
    __shared__ unsigned words[2];
    if (threadIdx.x < 2) words[threadIdx.x] = 0;  // seen by all from the first barrier on
    io_env env;
    env.mem = small_raw;
    env.r = (int)blockIdx.x;
    env.words = words;
    small_vcycle<FAST, YP>(P, env);
}

template <bool YP>
__global__ void __launch_bounds__(kSmallThreads, 1)
    k_block_columns(const __grid_constant__ small_plan<ff> P, float2 *out) {
    extern __shared__ __align__(16) unsigned char small_raw[];
    column_env env;
    env.mem = small_raw;
    env.r = 0;
    env.b0 = P.lv[P.t].bg;
    env.out = out;
    env.col = blockIdx.x;
    env.n = gridDim.x;
    small_vcycle<false, YP>(P, env);
}

int max_blocks() {
    static std::atomic<int> known[64];  // several host threads may probe at once, to the same result
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (!known[dev]) {
        const void *k[4] = {(const void *)k_small_blocks<true, true>, (const void *)k_small_blocks<true, false>,
                            (const void *)k_small_blocks<false, true>, (const void *)k_small_blocks<false, false>};
        int c = 16;
        for (const void *f : k) c = std::min(c, cluster_limit(f, kBlockMax));
        if (cudaFuncSetAttribute(k_block_columns<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallMax) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_block_columns<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSmallMax) != cudaSuccess)
            c = 0;
        known[dev] = c + 1;
    }
    return known[dev] - 1;
}

// Levels of at most this many nodes, where the blocks' shared memory holds them (a
// short grid has rows for few blocks: 256 x 128 nodes under 512 x 256, y
// periodic, do not fit, 128 x 251 under 256 x 500 do); the alternative is eleven
// FP64 launches of about 7 us per level.  V-cycles with the limit at 9,000 /
// 17,000 / 33,000: 256x500 160 / 161 / 134 us, 128x900 155 / 154 / 130, 256x256 y
// periodic 142 / 107 / 109; more than 33,000 changed nothing.
constexpr long kBlockPoints = 33000;

}  // namespace

small_cycle::~small_cycle() {
    for (int l = 0; l < 17; l++) {
        cudaFree(tab_[l].p);
        cudaFree(cls_[l].p);
        cudaFree(dense_[l].p);
    }
}

int small_cycle::need(buffer &b, size_t bytes, bool *moved) {
    if (b.cap >= bytes) return STZG_OK;
    if (b.p) cudaFree(b.p);
    b = buffer();
    *moved = true;
    const cudaError_t e = cudaMalloc(&b.p, bytes);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(small levels)");
    b.cap = bytes;
    return STZG_OK;
}

int small_cycle::setup(const std::vector<small_desc> &desc, int yp, const std::vector<double> &bottom, cudaStream_t st,
                       bool *moved) {
    const int was = t_, ml = (int)desc.size() - 1, cap = max_blocks();
    t_ = 0;
    yp_ = yp;
    auto done = [&](const small_plan<ff> *P) {
        std::vector<unsigned char> now(sizeof(small_plan<ff>));
        if (P) std::memcpy(now.data(), P, sizeof(*P));
        if (t_ != was || now != plan_) *moved = true;
        plan_.swap(now);
        return STZG_OK;
    };
    if (ml < 2 || ml > 16 || cap < 1 || bottom.empty()) return done(nullptr);
    const int d = std::max(2, dense_level(ml, [&](int l) { return (long)desc[l].m * desc[l].n; }));
    // a periodic y line is even on every level that is swept here
    int t = d;
    while (t > 1 && (long)desc[t - 1].m * desc[t - 1].n <= kBlockPoints && !(yp && (desc[t - 1].n & 1))) t--;
    for (int l = d; l < ml; l++)
        if (yp && (desc[l].n & 1)) return done(nullptr);
    small_plan<ff> P;
    std::memset(&P, 0, sizeof(P));
    double top = 0;
    for (int l = t; l <= ml; l++)
        for (size_t k = 0; k < desc[l].table.size(); k++)
            if (k % 40 < 36) top = std::max(top, std::fabs(desc[l].table[k]));
    if (top > 0 && std::isfinite(top)) std::frexp(top, &P.unit);
    for (int l = t; l <= ml; l++) {
        const small_desc &D = desc[l];
        const int nst = (int)D.table.size() / 40;
        pairs_[l].resize(20 * (size_t)nst);
        for (int c = 0; c < nst; c++)
            for (int e = 0; e < 10; e++) {
                float h[4], o[4];
                for (int q = 0; q < 4; q++) {
                    const double v = std::ldexp(D.table[(size_t)c * 40 + 4 * e + q], e < 9 ? -P.unit : P.unit);
                    h[q] = (float)v;
                    o[q] = (float)(v - (double)h[q]);
                }
                pairs_[l][20 * c + 2 * e] = make_float4(h[0], h[1], h[2], h[3]);
                pairs_[l][20 * c + 2 * e + 1] = make_float4(o[0], o[1], o[2], o[3]);
            }
        STZG_CHECK(need(tab_[l], pairs_[l].size() * sizeof(float4), moved));
        const bool sent = D.ids_kept && cls_[l].cap;
        STZG_CHECK(need(cls_[l], D.ids->size() * sizeof(int), moved));
        STZG_CUDA(cudaMemcpyAsync(tab_[l].p, pairs_[l].data(), pairs_[l].size() * sizeof(float4),
                                  cudaMemcpyHostToDevice, st));
        if (!sent)
            STZG_CUDA(cudaMemcpyAsync(cls_[l].p, D.ids->data(), D.ids->size() * sizeof(int), cudaMemcpyHostToDevice, st));
        small_level<ff> &S = P.lv[l];
        S.m = D.m;
        S.n = D.n;
        S.homog = D.rows;
        S.nst = nst;
        S.ncls = (int)D.ids->size();
        S.cls = (const int *)cls_[l].p;
        S.st = (const float4 *)tab_[l].p;
    }
    // the matrices from the coarsest level's up to level d's
    for (int l = ml; l >= d; l--) {
        const size_t N = 2 * (size_t)desc[l].m * desc[l].n;
        STZG_CHECK(need(dense_[l], N * N * sizeof(float2), moved));
        if (l == ml) {
            bottom_.resize(N * N);
            for (size_t k = 0; k < N * N; k++) {
                const double v = std::ldexp(bottom[k], P.unit);
                const float h = (float)v;
                bottom_[k] = make_float2(h, (float)(v - (double)h));
            }
            STZG_CUDA(cudaMemcpyAsync(dense_[l].p, bottom_.data(), N * N * sizeof(float2), cudaMemcpyHostToDevice, st));
            continue;
        }
        small_plan<ff> Q = P;
        Q.dense = (const float4 *)dense_[l + 1].p;
        if (!layout_small(Q, l, l + 1, 1, kSmallMax)) return done(nullptr);
        if (yp) k_block_columns<true><<<(unsigned)N, kSmallThreads, Q.bytes, st>>>(Q, (float2 *)dense_[l].p);
        else k_block_columns<false><<<(unsigned)N, kSmallThreads, Q.bytes, st>>>(Q, (float2 *)dense_[l].p);
        note_launch();
        STZG_CUDA(cudaGetLastError());
    }
    P.dense = (const float4 *)dense_[d].p;
    P.zero_start = 1;
    for (; t < d; t++)
        for (int c = cap; c >= 1; c >>= 1)
            if (layout_small(P, t, d, c, kBlockMax)) {
                t_ = t;
                return done(&P);
            }
    return done(nullptr);
}

void small_cycle::launch(const double2 *b, double2 *z, cudaStream_t st) const {
    small_plan<ff> P;
    std::memcpy(&P, plan_.data(), sizeof(P));
    P.lv[P.t].bg = reinterpret_cast<const float4 *>(b);
    P.lv[P.t].zg = reinterpret_cast<float4 *>(z);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    cluster_config(cfg, at, P.blocks, P.bytes, st);
    const bool fast = block_phases(P);
    if (yp_) fast ? cudaLaunchKernelEx(&cfg, k_small_blocks<true, true>, P) : cudaLaunchKernelEx(&cfg, k_small_blocks<false, true>, P);
    else fast ? cudaLaunchKernelEx(&cfg, k_small_blocks<true, false>, P) : cudaLaunchKernelEx(&cfg, k_small_blocks<false, false>, P);
    note_launch();
}

}  // namespace stzg
