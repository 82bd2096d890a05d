// Tile kernels of the float-pair V-cycle's wide levels (mg_small.cu).
#pragma once

#include "ff.cuh"
#include "mg_env.cuh"

namespace stzg {
namespace mgw {

// ---- wide levels as tiles ------------------------------------------------------
//
// A block takes the coarse rows J0.. and columns I0.. of its tile and the fine
// nodes that restrict to them, with the halo that makes sweep, residual and
// restriction (or prolongation and sweep) exact: two to four columns and rows
// on either side, recomputed by the neighbouring tiles.  Windows are 64
// columns wide, so that a warp takes one row of 2 x 2 blocks; what a sweep
// reads beyond the window's edge is wrong and stays in the halo.
// Bound by instruction issue (a block product in pairs is about 48 operations
// per neighbour); with nodes as (x, y) words instead of planes the top level's
// kernels were bound by shared-memory bank conflicts (41 and 51 us at 1024^2,
// now 26 and 39 with cold caches).
// BANDS: whole periodic rows, for odd lines and levels whose stencils differ
// along a row.

struct tile_level {
    int m, n, cm, cn;       // the level and its child
    int tw, th;             // coarse columns and rows per tile
    int threads;
    int homog, nst, staged; // stencils; staged: their table goes to shared memory
    const int *cls;
    const float4 *st;
    const float4 *b;
    float4 *zdown;          // written on the way down, read on the way up
    float4 *zup;            // written on the way up (coarse level)
    float4 *bc;             // the child's right-hand side
    const float4 *zc;       // the child's solution
    // top level: the iterate that takes the correction, the residual's power of
    // two and the tables'
    double2 *sum;
    const pair_range *range;
    int unit;
};

constexpr int kTileThreads = 256;  // most threads of a tile
constexpr int kTileCols = 64;
// Halo of each kernel: columns before x0 (even), rows before y0 (even) and
// block rows besides the tile's own.
constexpr int kLevCols = 4, kLevRows = 2, kLevExtra = 2;
constexpr int kTopDownCols = 4, kTopDownRows = 4, kTopDownExtra = 3;
constexpr int kTopUpCols = 2, kTopUpRows = 2, kTopUpExtra = 2;

struct tile_geom {
    int I0, I1, J0, J1, x0, x1, y0, y1, xb, qn;
    __device__ __forceinline__ tile_geom(const tile_level &L, bool bands, int halo, int extra) {
        J0 = blockIdx.y * L.th;
        J1 = min(J0 + L.th, L.cn);
        y0 = 2 * J0;
        y1 = min(2 * J1, L.n);
        I0 = bands ? 0 : blockIdx.x * L.tw;
        I1 = bands ? L.cm : min(I0 + L.tw, L.cm);
        x0 = 2 * I0;
        x1 = bands ? L.m : 2 * I1;
        xb = bands ? 0 : x0 - halo;
        qn = J1 - J0 + extra;
    }
};

__device__ __forceinline__ window<ff, true> tile_window(const tile_level &L, unsigned char *raw, int W, int rows,
                                                        int jb) {
    window<ff, true> V;
    const int np = W * rows;
    V.z = plane<ff>{reinterpret_cast<ff *>(raw), np};
    V.b = V.z + 2 * np;
    V.r = V.b;  // a residual replaces the right-hand side it came from
    V.W = W;
    V.He = (W + 1) >> 1;
    V.jb = V.rb = jb;
    V.m = L.m;
    V.n = L.n;
    V.x0 = 0;
    V.st = L.staged ? reinterpret_cast<const float4 *>(raw + (size_t)np * 4 * sizeof(ff)) : L.st;
    V.cls = L.cls;
    V.homog = L.homog;
    return V;
}

// Rows jlo..jhi of a level into a plane of the window (its column 0 at xb).
__device__ __forceinline__ void tile_load(const tile_level &L, const window<ff, true> &V, const plane<ff> &dst,
                                          const float4 *__restrict__ src, int jlo, int jhi, int xb) {
    jlo = max(jlo, 0);
    jhi = min(jhi, V.n - 1);
    const int total = (jhi - jlo + 1) * V.W;
    const divider dv(V.W);
    for (int k = threadIdx.x; k < total; k += L.threads) {
        const int q = dv.quot(k), j = jlo + q, w = k - q * V.W;
        int g = xb + w;
        g = g < 0 ? g % L.m + L.m : g;
        g = g >= L.m ? g % L.m : g;
        dst.set(V.at(j, w), get(__ldcg(src + (size_t)j * L.m + g)));
    }
}

__device__ __forceinline__ void tile_table(const tile_level &L, const float4 *dst) {
    if (!L.staged) return;
    float4 *d = const_cast<float4 *>(dst);
    for (int k = threadIdx.x; k < L.nst * 20; k += L.threads) d[k] = __ldg(L.st + k);
}

// The own nodes of a window: f(node of the level, value).
template <typename F>
__device__ __forceinline__ void tile_own(const tile_level &L, const window<ff, true> &V, const tile_geom &G, F f) {
    const int ow = G.x1 - G.x0, total = (G.y1 - G.y0) * ow;
    const divider dv(ow);
    for (int k = threadIdx.x; k < total; k += L.threads) {
        const int q = dv.quot(k), w = k - q * ow;
        f((size_t)(G.y0 + q) * L.m + G.x0 + w, V.z.get(V.at(G.y0 + q, w + G.x0 - G.xb)));
    }
}

// The child's columns xb/2 .. and rows around a tile.
struct child_tile {
    plane<ff> c;
    int Jlo, cw;
    __device__ __forceinline__ plane<ff> row(int J) const { return c + (J - Jlo) * cw; }
};

__device__ __forceinline__ child_tile tile_child(const tile_level &L, const tile_geom &G, ff *dst, int Ib, int cw) {
    child_tile C;
    C.Jlo = max(0, G.J0 - 1);
    C.cw = cw;
    C.c = plane<ff>{dst, cw * (L.th + 3)};
    const int Jhi = min(L.cn - 1, (G.y1 >> 1) + 1), total = (Jhi - C.Jlo + 1) * cw;
    const divider dv(cw);
    for (int k = threadIdx.x; k < total; k += L.threads) {
        const int q = dv.quot(k);
        int I = Ib + k - q * cw;
        I = I < 0 ? I % L.cm + L.cm : I;
        I = I >= L.cm ? I % L.cm : I;
        C.c.set(k, get(__ldcg(L.zc + (size_t)(C.Jlo + q) * L.cm + I)));
    }
    return C;
}

template <bool BANDS> __global__ void __launch_bounds__(kTileThreads) k_pair_lev_down(tile_level L) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    pdl_start();
    const tile_geom G(L, BANDS, kLevCols, kLevExtra);
    const int W = BANDS ? L.m : kTileCols, tid = threadIdx.x, nth = L.threads;
    const window<ff, true> V = tile_window(L, tile_raw, W, 2 * (L.th + kLevExtra), G.y0 - kLevRows);
    tile_table(L, V.st);
    pdl_input();
    tile_load(L, V, V.b, L.b, G.y0 - 2, G.y1, G.xb);
    if (BANDS && (L.m & 1)) lev_clear_last(V, G.y0 - 2, G.y1, tid, nth);
    __syncthreads();
    const block_walk w(tid, nth, W >> 1);
    const int ncx = BANDS && (L.m & 1) ? 3 : 2;
#pragma unroll 1
    for (int cy = 0; cy < 2; cy++)
#pragma unroll 1
        for (int cx = 0; cx < ncx; cx++) {
            if (BANDS) lev_color(V, G.y0 - 2 + cy, G.y1 - cy, 0, 0, cx, cy, true, tid, nth);
            else block_color(V, w, G.qn, G.y0 - 2 + cy, G.y1 - cy, cx, cy, true);
            __syncthreads();
        }
    if (BANDS) lev_residual(V, G.y0 - 1, G.y1 - 1, 0, 0, tid, nth);
    else block_residual(V, W >> 1, G.qn, G.y0 - 1, G.y1 - 1, tid, nth);
    __syncthreads();
    const int Ib = G.xb >> 1;
    auto out = [&](int J, int k, const val2<ff> &v) {
        const int I = BANDS ? k : Ib + k;
        if (I >= G.I0 && I < G.I1) L.bc[(size_t)J * L.cm + I] = put(v);
    };
    if (BANDS) restrict_rows(V, G.J0, G.J1 - 1, 0, L.cm - 1, L.cm, out, tid, nth);
    else block_restrict(V, w, G.qn, G.J0, G.J1 - 1, out);
    tile_own(L, V, G, [&](size_t k, const val2<ff> &v) { L.zdown[k] = put(v); });
}

template <bool BANDS> __global__ void __launch_bounds__(kTileThreads) k_pair_lev_up(tile_level L) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    pdl_start();
    const tile_geom G(L, BANDS, kLevCols, kLevExtra);
    const int W = BANDS ? L.m : kTileCols, rows = 2 * (L.th + kLevExtra), tid = threadIdx.x, nth = L.threads;
    const window<ff, true> V = tile_window(L, tile_raw, W, rows, G.y0 - kLevRows);
    ff *cs = reinterpret_cast<ff *>(tile_raw + (size_t)W * rows * 4 * sizeof(ff) + (L.staged ? L.nst * 320 : 0));
    tile_table(L, V.st);
    pdl_input();
    tile_load(L, V, V.z, L.zdown, G.y0 - 1, G.y1 + 1, G.xb);
    tile_load(L, V, V.b, L.b, G.y0, G.y1, G.xb);
    const child_tile C = tile_child(L, G, cs, G.xb >> 1, BANDS ? L.cm : kTileCols / 2 + 1);
    __syncthreads();
    const block_walk w(tid, nth, W >> 1);
    if (BANDS)
        prolong_rows(V, G.y0 - 1, G.y1 + 1, 0, 0, L.cm, [&](int J, int I) { return C.row(J).get(I); }, tid, nth);
    else
        block_prolong(V, w, G.qn, G.y0 - 1, G.y1 + 1, [&](int J) { return C.row(J); }, [](int k) { return k; },
                      [](int k) { return k + 1; });
    __syncthreads();
    const int ncx = BANDS && (L.m & 1) ? 3 : 2;
#pragma unroll 1
    for (int cy = 0; cy < 2; cy++)
#pragma unroll 1
        for (int cx = 0; cx < ncx; cx++) {
            if (BANDS) lev_color(V, G.y0, G.y1 - cy, 0, 0, cx, cy, false, tid, nth);
            else block_color(V, w, G.qn, G.y0, G.y1 - cy, cx, cy, false);
            __syncthreads();
        }
    tile_own(L, V, G, [&](size_t k, const val2<ff> &v) { L.zup[k] = put(v); });
}

__global__ void __launch_bounds__(kTileThreads) k_pair_top_down(top_consts<ff> op, tile_level L) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    pdl_start();
    const tile_geom G(L, false, kTopDownCols, kTopDownExtra);
    const window<ff, true> V = tile_window(L, tile_raw, kTileCols, 2 * (L.th + kTopDownExtra), G.y0 - kTopDownRows);
    pdl_input();
    tile_load(L, V, V.b, L.b, G.y0 - 3, G.y1 + 1, G.xb);
    __syncthreads();
    const block_walk w(threadIdx.x, L.threads, kTileCols / 2);
    block_top_color(op, V, w, G.qn, G.y0 - 3, G.y1 + 1, 0, true);
    __syncthreads();
    block_top_color(op, V, w, G.qn, G.y0 - 2, G.y1, 1, false);
    __syncthreads();
    block_top_residual(op, V, w, G.qn, G.y0 - 1, G.y1 - 1);
    __syncthreads();
    const int Ib = G.xb >> 1;
    block_restrict(V, w, G.qn, G.J0, G.J1 - 1, [&](int J, int k, const val2<ff> &v) {
        if (Ib + k >= G.I0 && Ib + k < G.I1) L.bc[(size_t)J * L.cm + Ib + k] = put(v);
    });
    tile_own(L, V, G, [&](size_t k, const val2<ff> &v) { L.zdown[k] = put(v); });
}

__global__ void __launch_bounds__(kTileThreads) k_pair_top_up(top_consts<ff> op, tile_level L) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    pdl_start();
    const tile_geom G(L, false, kTopUpCols, kTopUpExtra);
    const int rows = 2 * (L.th + kTopUpExtra);
    const window<ff, true> V = tile_window(L, tile_raw, kTileCols, rows, G.y0 - kTopUpRows);
    ff *cs = reinterpret_cast<ff *>(tile_raw + (size_t)kTileCols * rows * 4 * sizeof(ff));
    pdl_input();
    const int used = __ldcg(&L.range->used);
    tile_load(L, V, V.z, L.zdown, G.y0 - 2, G.y1 + 1, G.xb);
    tile_load(L, V, V.b, L.b, G.y0 - 1, G.y1, G.xb);
    const child_tile C = tile_child(L, G, cs, G.xb >> 1, kTileCols / 2 + 1);
    __syncthreads();
    const block_walk w(threadIdx.x, L.threads, kTileCols / 2);
    block_prolong(V, w, G.qn, G.y0 - 2, G.y1 + 1, [&](int J) { return C.row(J); }, [](int k) { return k; },
                  [](int k) { return k + 1; });
    __syncthreads();
    block_top_color(op, V, w, G.qn, G.y0 - 1, G.y1, 0, false);
    __syncthreads();
    block_top_color(op, V, w, G.qn, G.y0, G.y1 - 1, 1, false);
    __syncthreads();
    const double back = pair_back(used, L.unit);
    // z += d: four nodes' iterates are on their way at a time
    const int ow = G.x1 - G.x0, total = (G.y1 - G.y0) * ow;
    const divider dv(ow);
    for (int k0 = threadIdx.x; k0 < total; k0 += 4 * L.threads) {
        double2 *at[4], z[4];
        float4 d[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int k = min(k0 + u * L.threads, total - 1), q = dv.quot(k), w = k - q * ow;
            at[u] = L.sum + (size_t)(G.y0 + q) * L.m + G.x0 + w;
            z[u] = *at[u];
            d[u] = put(V.z.get(V.at(G.y0 + q, w + G.x0 - G.xb)));
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (k0 + u * L.threads < total) *at[u] = add_pairs(z[u], d[u], back);
    }
}

}  // namespace mgw
}  // namespace stzg
