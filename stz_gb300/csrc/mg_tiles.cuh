// Tile kernels of the float-pair V-cycle's wide levels (mg_small.cu).
#pragma once

#include "ff.cuh"
#include "mg_window.cuh"

namespace stzg {
namespace mgw {

__device__ __forceinline__ void pdl_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_input() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// z += d in FP64, the pair formed as a double on the integer pipe.
__device__ __forceinline__ void add_pairs(double2 *z, const float4 &d) {
    double2 v = *z;
    v.x += ff_to_d(d.x, d.z);
    v.y += ff_to_d(d.y, d.w);
    *z = v;
}

// ---- wide levels as tiles ------------------------------------------------------
//
// A block takes the coarse rows J0.. and columns I0.. of its tile and the fine
// nodes that restrict to them, with the halo that makes sweep, residual and
// restriction (or prolongation and sweep) exact: down, three to four columns
// and two to three rows on either side, recomputed by the neighbouring tiles.
// Bound by instruction issue (a block product in pairs is about 48 operations
// per neighbour) and, on levels below 512 wide, by the chain of five to six
// phases.  FP64 V-cycle at 1024^2: 782 us with one FP64 launch per colour, 265 us.
// WRAP: tiles of whole periodic rows, for odd lines and levels whose stencils
// differ along a row.

struct tile_level {
    int m, n, cm, cn;       // the level and its child
    int tw, th;             // coarse columns and rows per tile
    int homog, nst, staged; // stencils; staged: their table goes to shared memory
    const int *cls;
    const float4 *st;
    const float4 *b;
    float4 *zdown;          // written on the way down, read on the way up
    float4 *zup;            // written on the way up (coarse level)
    float4 *bc;             // the child's right-hand side
    const float4 *zc;       // the child's solution
    double2 *sum;           // top level: the iterate that takes the correction
};

constexpr int kTileThreads = 256;

template <bool WRAP> struct tile_geom {
    int I0, I1, J0, J1, x0, x1, y0, y1, xb, ow;
    __device__ __forceinline__ tile_geom(const tile_level &L, int halo) {
        J0 = blockIdx.y * L.th;
        J1 = min(J0 + L.th, L.cn);
        y0 = 2 * J0;
        y1 = min(2 * J1, L.n);
        I0 = WRAP ? 0 : blockIdx.x * L.tw;
        I1 = WRAP ? L.cm : min(I0 + L.tw, L.cm);
        x0 = 2 * I0;
        x1 = WRAP ? L.m : 2 * I1;
        xb = WRAP ? 0 : x0 - halo;
        ow = x1 - x0;
    }
};

template <bool WRAP>
__device__ __forceinline__ window<ff, WRAP> tile_window(const tile_level &L, unsigned char *raw, int W, int rows,
                                                        int jb, int x0) {
    window<ff, WRAP> V;
    V.z = reinterpret_cast<float4 *>(raw);
    V.b = V.z + W * rows;
    V.r = V.b;  // a residual replaces the right-hand side it came from
    V.W = W;
    V.He = (W + 1) >> 1;
    V.jb = V.rb = jb;
    V.m = L.m;
    V.n = L.n;
    V.x0 = x0;
    V.st = L.staged ? reinterpret_cast<const float4 *>(V.b + W * rows) : L.st;
    V.cls = L.cls;
    V.homog = L.homog;
    return V;
}

template <bool WRAP>
__device__ __forceinline__ void tile_load(const window<ff, WRAP> &V, float4 *dst, const float4 *__restrict__ src,
                                          int jlo, int jhi, int nw) {
    jlo = max(jlo, 0);
    jhi = min(jhi, V.n - 1);
    const int total = (jhi - jlo + 1) * nw;
    const divider dv(nw);
    for (int k = threadIdx.x; k < total; k += kTileThreads) {
        const int q = dv.quot(k), j = jlo + q, w = k - q * nw;
        dst[V.at(j, w)] = __ldcg(src + (size_t)j * V.m + V.gcol(w));
    }
}

__device__ __forceinline__ void tile_table(const tile_level &L, const float4 *dst) {
    if (!L.staged) return;
    float4 *d = const_cast<float4 *>(dst);
    for (int k = threadIdx.x; k < L.nst * 20; k += kTileThreads) d[k] = __ldg(L.st + k);
}

template <bool WRAP>
__device__ __forceinline__ void tile_restrict_store(const tile_level &L, const window<ff, WRAP> &V,
                                                    const tile_geom<WRAP> &G, int off, int ow) {
    const int tid = threadIdx.x;
    restrict_rows(V, G.J0, G.J1 - 1, G.I0, G.I1 - 1, L.cm,
                  [&](int J, int I, float4 v) { L.bc[(size_t)J * L.cm + I] = v; }, tid, kTileThreads);
    const int total = (G.y1 - G.y0) * ow;
    const divider dv(ow);
    for (int k = tid; k < total; k += kTileThreads) {
        const int q = dv.quot(k), w = k - q * ow;
        L.zdown[(size_t)(G.y0 + q) * L.m + G.x0 + w] = V.z[V.at(G.y0 + q, w + off)];
    }
}

template <bool WRAP> __global__ void __launch_bounds__(kTileThreads) k_pair_lev_down(tile_level L) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    pdl_start();
    const tile_geom<WRAP> G(L, 4);
    const int W = WRAP ? L.m : 2 * L.tw + 8, rows = 2 * L.th + 3;
    const window<ff, WRAP> V = tile_window<WRAP>(L, tile_raw, W, rows, G.y0 - 2, G.xb);
    const int tid = threadIdx.x, o = WRAP ? 0 : 4, ow = G.ow;
    tile_table(L, V.st);
    pdl_input();
    tile_load(V, V.b, L.b, G.y0 - 2, G.y1, WRAP ? W : ow + 7);
    if (WRAP && (L.m & 1)) lev_clear_last(V, G.y0 - 2, G.y1, tid, kTileThreads);
    __syncthreads();
    const int ncx = WRAP && (L.m & 1) ? 3 : 2;
#pragma unroll 1
    for (int cy = 0; cy < 2; cy++)
#pragma unroll 1
        for (int cx = 0; cx < ncx; cx++) {
            const int s = 2 * cy + cx;  // the columns that are still exact shrink by one per colour
            lev_color(V, G.y0 - 2 + cy, G.y1 - cy, s, ow + 6 - s, cx, cy, true, tid, kTileThreads);
            __syncthreads();
        }
    lev_residual(V, G.y0 - 1, G.y1 - 1, 3, ow + 3, tid, kTileThreads);
    __syncthreads();
    tile_restrict_store(L, V, G, o, ow);
}

// The child's values around a tile, columns Ib .. of rows Jlo ..
struct child_tile {
    const float4 *c;
    int Jlo, Ib, cw;
    __device__ __forceinline__ float4 operator()(int J, int I) const { return c[(J - Jlo) * cw + (I - Ib)]; }
};

template <bool WRAP>
__device__ __forceinline__ child_tile tile_child(const tile_level &L, const tile_geom<WRAP> &G, float4 *dst, int Ib,
                                                 int cw) {
    const int Jlo = max(0, G.J0 - 1), Jhi = min(L.cn - 1, (G.y1 >> 1) + 1);
    const int total = (Jhi - Jlo + 1) * cw;
    const divider dv(cw);
    for (int k = threadIdx.x; k < total; k += kTileThreads) {
        const int q = dv.quot(k), c = k - q * cw;
        int I = Ib + c;
        I = I < 0 ? I + L.cm : (I >= L.cm ? I % L.cm : I);
        dst[k] = __ldcg(L.zc + (size_t)(Jlo + q) * L.cm + I);
    }
    return child_tile{dst, Jlo, Ib, cw};
}

template <bool WRAP> __global__ void __launch_bounds__(kTileThreads) k_pair_lev_up(tile_level L) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    pdl_start();
    const tile_geom<WRAP> G(L, 4);
    const int W = WRAP ? L.m : 2 * L.tw + 8, rows = 2 * L.th + 3;
    const window<ff, WRAP> V = tile_window<WRAP>(L, tile_raw, W, rows, G.y0 - 1, G.xb);
    const int tid = threadIdx.x, o = WRAP ? 0 : 4, ow = G.ow, nw = WRAP ? W : ow + 8;
    float4 *cs = V.b + W * rows + (L.staged ? L.nst * 20 : 0);
    tile_table(L, V.st);
    pdl_input();
    tile_load(V, V.z, L.zdown, G.y0 - 1, G.y1 + 1, nw);
    tile_load(V, V.b, L.b, G.y0, G.y1, nw);
    const child_tile C = tile_child(L, G, cs, WRAP ? 0 : G.I0 - 2, WRAP ? L.cm : L.tw + 5);
    __syncthreads();
    prolong_rows(V, G.y0 - 1, G.y1 + 1, 0, ow + 7, L.cm, C, tid, kTileThreads);
    __syncthreads();
    const int ncx = WRAP && (L.m & 1) ? 3 : 2;
#pragma unroll 1
    for (int cy = 0; cy < 2; cy++)
#pragma unroll 1
        for (int cx = 0; cx < ncx; cx++) {
            const int s = 2 + 2 * cy + cx;
            lev_color(V, G.y0, G.y1 - cy, s, ow + 8 - s, cx, cy, false, tid, kTileThreads);
            __syncthreads();
        }
    const int total = (G.y1 - G.y0) * ow;
    const divider dv(ow);
    for (int k = tid; k < total; k += kTileThreads) {
        const int q = dv.quot(k), w = k - q * ow;
        L.zup[(size_t)(G.y0 + q) * L.m + G.x0 + w] = V.z[V.at(G.y0 + q, w + o)];
    }
}

__global__ void __launch_bounds__(kTileThreads) k_pair_top_down(top_consts<ff> op, tile_level L) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    pdl_start();
    const tile_geom<false> G(L, 4);
    const int W = 2 * L.tw + 8, rows = 2 * L.th + 5, tid = threadIdx.x, ow = G.ow;
    const window<ff, false> V = tile_window<false>(L, tile_raw, W, rows, G.y0 - 3, G.xb);
    pdl_input();
    tile_load(V, V.b, L.b, G.y0 - 3, G.y1 + 1, ow + 6);
    __syncthreads();
    top_color(op, V, G.y0 - 3, G.y1 + 1, 1, ow + 5, 0, true, tid, kTileThreads);
    __syncthreads();
    top_color(op, V, G.y0 - 2, G.y1, 2, ow + 4, 1, false, tid, kTileThreads);
    __syncthreads();
    top_residual(op, V, G.y0 - 1, G.y1 - 1, 3, ow + 3, tid, kTileThreads);
    __syncthreads();
    tile_restrict_store(L, V, G, 4, ow);
}

__global__ void __launch_bounds__(kTileThreads) k_pair_top_up(top_consts<ff> op, tile_level L) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    pdl_start();
    const tile_geom<false> G(L, 2);
    const int W = 2 * L.tw + 4, rows = 2 * L.th + 4, tid = threadIdx.x, ow = G.ow;
    const window<ff, false> V = tile_window<false>(L, tile_raw, W, rows, G.y0 - 2, G.xb);
    float4 *cs = V.b + W * rows;
    pdl_input();
    tile_load(V, V.z, L.zdown, G.y0 - 2, G.y1 + 1, ow + 4);
    tile_load(V, V.b, L.b, G.y0 - 1, G.y1, ow + 4);
    const child_tile C = tile_child(L, G, cs, G.I0 - 1, L.tw + 3);
    __syncthreads();
    prolong_rows(V, G.y0 - 2, G.y1 + 1, 0, ow + 3, L.cm, C, tid, kTileThreads);
    __syncthreads();
    top_color(op, V, G.y0 - 1, G.y1, 1, ow + 2, 0, false, tid, kTileThreads);
    __syncthreads();
    top_color(op, V, G.y0, G.y1 - 1, 2, ow + 1, 1, false, tid, kTileThreads);
    __syncthreads();
    const int total = (G.y1 - G.y0) * ow;
    const divider dv(ow);
    for (int k = tid; k < total; k += kTileThreads) {
        const int q = dv.quot(k), w = k - q * ow;
        add_pairs(L.sum + (size_t)(G.y0 + q) * L.m + G.x0 + w, V.z[V.at(G.y0 + q, w + 2)]);
    }
}

}  // namespace mgw
}  // namespace stzg
