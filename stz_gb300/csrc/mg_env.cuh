// The GPU environment of small_vcycle (mg_window.cuh).
#pragma once

#include "ff.cuh"
#include "fixed.cuh"
#include "mg.cuh"
#include "mg_plan.h"

namespace stzg {
namespace mgw {

__device__ __forceinline__ void pdl_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_input() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// z += back d in FP64, the pair formed as a double on the integer pipe.
__device__ __forceinline__ double2 add_pairs(const double2 &z, const float4 &d, double back) {
    return make_double2(fma(ff_to_d(d.x, d.z), back, z.x), fma(ff_to_d(d.y, d.w), back, z.y));
}
// The power of two that takes a solution of the system in pairs back: the
// residual was multiplied by 2^used, the operator by 2^-unit.
__device__ __forceinline__ double pair_back(int used, int unit) {
    return power_of_two(min(max(-used - unit, -1022), 1023));
}

// The environment of small_vcycle on the GPU.
struct block_env {
    static constexpr int kLanes = 32;
    static constexpr bool kMeasured = false;
    unsigned char *mem;
    int r;
    int used = 0;  // pair_range::used
    __device__ __forceinline__ int rank() const { return r; }
    __device__ __forceinline__ unsigned char *local() const { return mem; }
    __device__ __forceinline__ unsigned char *base(int k) const {
        unsigned long long a;
        asm("mapa.u64 %0, %1, %2;\n" : "=l"(a) : "l"((unsigned long long)mem), "r"(k));
        return (unsigned char *)a;
    }
    template <typename N> __device__ __forceinline__ void measure(const N *) {}
    __device__ __forceinline__ void measured() {}
    __device__ __forceinline__ void share(int, int) {}
    __device__ __forceinline__ int thread() const { return (int)threadIdx.x; }
    __device__ __forceinline__ int threads() const { return (int)blockDim.x; }
    __device__ __forceinline__ const block_walk &walk(const block_walk &w, int, int) const { return w; }
    template <typename F> __device__ __forceinline__ void par(F f) {
        f((int)threadIdx.x, (int)blockDim.x);
        __syncthreads();
    }
    __device__ __forceinline__ void csync() {
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    }
    __device__ __forceinline__ ff lane_sum(ff a) const { return warp_pair_sum(a); }
    __device__ __forceinline__ float2 ld(const float2 *p) const { return __ldcg(p); }
    __device__ __forceinline__ float4 ld(const float4 *p) const { return __ldcg(p); }
    __device__ __forceinline__ void wait_input(const small_plan<float> &) { pdl_input(); }
    __device__ __forceinline__ void wait_input(const small_plan<ff> &P) {
        pdl_input();
        if (P.sum) used = __ldcg(&P.range->used);
    }
    __device__ __forceinline__ void store(const small_plan<float> &P, size_t k, const float2 &v) const {
        P.lv[P.t].zg[k] = v;
    }
    __device__ __forceinline__ void store(const small_plan<ff> &P, size_t k, const float4 &v) const {
        if (P.sum) P.sum[k] = add_pairs(P.sum[k], v, pair_back(used, P.unit));
        else P.lv[P.t].zg[k] = v;
    }
};

constexpr int kSmallThreads = 512;
constexpr unsigned kSmallMax = 227 * 1024;

// Column c of the matrix of the V-cycle from level t on: block c runs it on
// the right-hand side that is one at unknown c.
struct column_env : block_env {
    const float4 *b0;
    float2 *out;
    int col, n;
    __device__ __forceinline__ int rank() const { return 0; }
    __device__ __forceinline__ float4 ld(const float4 *p) const {
        const int k = 2 * (int)(p - b0);
        return make_float4(k == col ? 1.f : 0.f, k + 1 == col ? 1.f : 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ void wait_input(const small_plan<ff> &) {}
    __device__ __forceinline__ void store(const small_plan<ff> &, size_t k, const float4 &v) const {
        out[(2 * k) * n + col] = make_float2(v.x, v.z);
        out[(2 * k + 1) * n + col] = make_float2(v.y, v.w);
    }
};

// Attributes of a launch of `blocks` blocks as one cluster, with programmatic
// dependent launch; at: room for two.
inline void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, int blocks, unsigned bytes, cudaStream_t st,
                           bool early = true) {
    cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = early;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = blocks;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = blocks > 1 ? 2 : 1;
}

// Largest cluster (a power of two up to 16) the device takes for a small-level
// kernel with that much dynamic shared memory; 0 where its attributes are refused.
inline int cluster_limit(const void *kernel, unsigned bytes = kSmallMax) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    for (int c = 16; c >= 2; c >>= 1) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[2];
        cluster_config(cfg, at, c, bytes, nullptr);
        cfg.attrs = at + 1;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0) return c;
    }
    cudaGetLastError();
    return 1;
}

}  // namespace mgw
}  // namespace stzg
