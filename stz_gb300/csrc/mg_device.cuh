// Device helpers shared by the multigrid kernels and the no-allocation
// residual-norm entry point.
#pragma once

#include "mg.cuh"
#include "step.cuh"

namespace stzg {

// Residual of the top level: r = b - A z (qs_multi::mul_a + a_cc).
template <typename T, typename V>
__device__ __forceinline__ V top_res(const top_op<T> &op, const V *__restrict__ z, const V *__restrict__ b, int m, int n,
                            int i, int j) {
    const size_t ij = (size_t)j * m + i;
    V r;
    if (j == 0 || j == n - 1) {
        r.x = b[ij].x - op.bcxx * z[ij].x;
        r.y = b[ij].y - op.bcyy * z[ij].y;
        return r;
    }
    const int il = i == 0 ? m - 1 : i - 1, ir = i == m - 1 ? 0 : i + 1;
    const V *zd = z + (size_t)(j - 1) * m, *zc = z + (size_t)j * m, *zu = z + (size_t)(j + 1) * m;
    T ax = op.Kmx * (zc[il].x + zc[ir].x) + op.my * (zd[i].x + zu[i].x) +
           op.qK * (zd[il].y + zu[ir].y - zd[ir].y - zu[il].y);
    T ay = op.mx * (zc[il].y + zc[ir].y) + op.Kmy * (zd[i].y + zu[i].y) +
           op.qK * (zd[il].x + zu[ir].x - zd[ir].x - zu[il].x);
    r.x = b[ij].x - ax - op.cxx * zc[i].x;
    r.y = b[ij].y - ay - op.cyy * zc[i].y;
    return r;
}

// Deterministic block reduction of a double (warp shuffles, fixed order).
__device__ __forceinline__ double block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    double t = 0;
    if (threadIdx.x < 32) {
        t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    __syncthreads();
    return t;
}

// Programmatic dependent launch within a solve: each kernel lets the next one be scheduled as soon as it starts
// (griddepcontrol.launch_dependents) and waits for its predecessor's results
// (griddepcontrol.wait) only after the set-up that needs none, so launch
// latency and set-up overlap the previous level's work.  Kernels launched
// with the attribute all execute the wait before touching data another
// kernel writes.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Where the previous kernel still has waves to run, early blocks only take
// their slots (the 512^2 to 2048^2 passes of a solve slowed by 0.2 to 1
// percent): one-pass kernels over more points than this start after it.
constexpr long kEarlyPoints = 1 << 17;

template <typename... K, typename... A>
void launch_early(bool early, void (*kern)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, args...);
}

// The end of a residual kernel: a and c are the block's sums of r^2 and b^2
// (valid in thread 0), sh 32 doubles of shared memory; range (or null): the
// residual's power of two was `used`.  While a solve converges its residual
// leaves the pairs' exponents downwards (or, from a bad guess, upwards): the
// next one is brought back to 1 once it is 2^30 below or 2^40 above.  The sums and the
// stopping rule used to be two more launches of one block each per pass (2 to
// 3 us each inside the solve's graph).
__device__ __forceinline__ void finish_norms(double a, double c, const norm_sink &s, double *sh,
                                             pair_range *range = nullptr, int used = 0) {
    __shared__ int last;
    unsigned *arrived = reinterpret_cast<unsigned *>(s.partials + 2 * s.npart);
    if (threadIdx.x == 0) {
        s.partials[2 * blockIdx.x] = a;
        s.partials[2 * blockIdx.x + 1] = c;
        __threadfence();
        last = atomicAdd(arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    a = c = 0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
        a += __ldcg(s.partials + 2 * k);
        c += __ldcg(s.partials + 2 * k + 1);
    }
    a = block_sum(a, sh);
    c = block_sum(c, sh);
    if (threadIdx.x != 0) return;
    *arrived = 0;
    if (range) {
        range->used = used;
        const int e = (__double2hiint(a) >> 20) & 0x7ff, at = (e - 1023) >> 1;  // |r| is about 2^at
        if (e > 0 && e < 0x7ff && (at + used < -30 || at + used > 40)) range->next = min(max(-at, -1000), 1000);
    }
    s.out[0] = a;
    s.out[1] = c;
    const loop_rule &r = s.rule;
    if (!r.flags) return;
    const bool conv = c > 0 ? a <= r.tol2 * c : a == 0 || (c == 0 && r.zero_ends);
    const bool nan = isnan(a);
    int it = 0;
    if (r.cap == 0) {
        r.flags[FL_PASSES] = 0;
        r.flags[FL_LOOP_ERR] = nan ? 2 : 0;
    } else {
        it = ++r.flags[FL_PASSES];
        ++r.flags[FL_PASSES_SUM];
        if (nan) r.flags[FL_LOOP_ERR] = 2;
        else if (!conv && it >= r.cap) r.flags[FL_LOOP_ERR] = 1;
    }
    if (r.flags[FL_LOOP_ERR] && !r.flags[FL_ERR_FIRST]) r.flags[FL_ERR_FIRST] = r.flags[FL_LOOP_ERR];
    const unsigned on = !conv && !nan && (r.cap == 0 || it < r.cap) ? 1u : 0u;
    cudaGraphSetConditional(r.h, on);
    if (r.has_ran) cudaGraphSetConditional(r.h_ran, on);
}

}  // namespace stzg
