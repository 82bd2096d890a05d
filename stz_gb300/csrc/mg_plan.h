// Host-side layout of the small levels of a V-cycle in shared memory
// (mg_window.cuh): where every array of a block lies.
#pragma once

#include "mg_window.cuh"

namespace stzg {
namespace mgw {

// Fills the offsets of P for levels t..d (their sizes, classes and stencil
// counts already in P.lv) over `blocks` blocks (a power of two) with at most max_bytes of
// shared memory each; false where it does not fit.  Every block needs a row
// of level d, so that the bands above have the two rows their neighbours'
// halos read.
template <typename S> bool layout_small(small_plan<S> &P, int t, int d, int blocks, unsigned max_bytes) {
    typedef typename num<S>::node node;
    P.t = t;
    P.d = d;
    P.blocks = blocks;
    P.shift = 0;
    while ((1 << P.shift) < blocks) P.shift++;
    if (t >= d || (blocks > 1 && P.lv[d].n < blocks)) return false;
    unsigned off = 0;
    auto place = [&](unsigned long bytes) {
        const unsigned at = off;
        off = (unsigned)((off + bytes + 15) & ~15ul);
        return at;
    };
    const unsigned long nd = (unsigned long)P.lv[d].m * P.lv[d].n;
    if (nd * sizeof(node) * 2 > max_bytes) return false;
    P.lv[d].ps = (int)nd;
    P.lv[d].zo = place(nd * sizeof(node));
    P.lv[d].bo = place(nd * sizeof(node));
    P.lv[d].ho = P.lv[d].so = P.lv[d].co = kNone;
    unsigned long rmax = 0;
    for (int l = t; l < d; l++) {
        small_level<S> &L = P.lv[l];
        int own = 0;
        for (int c = 0; c < blocks; c++) {
            const int r = band_row(P, l, c + 1) - band_row(P, l, c);
            own = r > own ? r : own;
        }
        const int rows = (own + band_below(P, l) + band_above(P, l) + 1) & ~1;
        const unsigned long nodes = (unsigned long)L.m * rows;
        if (nodes * sizeof(node) * 2 > max_bytes) return false;
        L.ps = (int)nodes;
        L.zo = place(nodes * sizeof(node));
        L.bo = place(nodes * sizeof(node));
        L.ho = l > t ? place(3ul * L.m * sizeof(node)) : kNone;
        const unsigned long rb = (unsigned long)L.m * (own + 1);
        if (rb > rmax) rmax = rb;
        if (off > max_bytes) return false;
    }
    P.rs = (int)rmax;
    P.ro = place(rmax * sizeof(node));
    if (off > max_bytes) return false;
    // tables: small ones in shared memory (one class per row, a few stencils)
    for (int l = t; l < d; l++) {
        small_level<S> &L = P.lv[l];
        L.so = L.co = kNone;
        if (P.top && l == t) continue;
        const unsigned long sb = (unsigned long)L.nst * 10 * num<S>::quads * 16, cb = 4ul * L.ncls;
        if (!L.homog || sb > 16384 || off + sb + cb + 32 > max_bytes) continue;
        L.so = place(sb);
        L.co = place(cb);
    }
    P.bytes = off;
    return true;
}

// Whether the 2 x 2 block phases apply: even lines, one stencil class per row,
// tables in shared memory.
template <typename S> bool block_phases(const small_plan<S> &P) {
    for (int l = P.t; l < P.d; l++) {
        if (P.lv[l].m & 1) return false;
        if (!(P.top && l == P.t) && P.lv[l].so == kNone) return false;
    }
    return true;
}

// Nodes of the level from which on the V-cycle is one matrix (2 x nodes
// unknowns, 8 bytes per entry, so 6.5 MB at most).  Its product streams the
// matrix from L2 through the cluster, 2.4 MB in about 1.5 us at 17 x 16 nodes,
// where the levels it stands for took 16 us (FP32) to 25 us (pairs) in their 30
// dependent phases; at 33 x 32 nodes it would be 36 MB.
constexpr long kDenseNodes = 450;

// That level of a hierarchy whose coarsest level is ml (nodes(l): m n of level
// l); at least 1, so that the top level stays a smoothed one.
template <typename F> int dense_level(int ml, F nodes) {
    int d = ml;
    while (d > 1 && nodes(d - 1) <= kDenseNodes) d--;
    return d;
}

// Tile of a wide level: coarse columns and rows, threads, shared memory of one
// launch.  top: 0 a coarse level, 1 the top level down, 2 up; bands: whole
// rows.  A row of blocks is a warp's; 8 or 4 of them per tile, the most that
// still gives three blocks per SM (the halo of a tile of 6 or 2 coarse rows
// costs 1.33 or 2 times the rows; 16 rows, 1.14 times, took 209 us per V-cycle
// of 1024x768 against 194: the last wave was nearly empty).
struct tile_shape {
    int tw, th, threads;
    unsigned long bytes;
};
inline tile_shape shape_tile(int m, int cm, int cn, int table, int top, bool bands, unsigned long max_bytes) {
    const int extra = top == 1 ? 3 : 2;
    tile_shape T;
    T.threads = 256;
    auto bytes = [&] {
        const unsigned long W = bands ? m : 64, cw = bands ? cm : 33;
        return W * 2 * (T.th + extra) * 32 + table + cw * (T.th + 3) * 16;
    };
    if (bands) {
        T.tw = cm;
        for (T.th = 4; T.th > 2 && (bytes() > max_bytes || (cn + T.th - 1) / T.th < 152); T.th >>= 1) {}
    } else {
        T.tw = top == 1 ? 29 : (top == 2 ? 30 : 28);
        for (int rows = 8; rows >= 4; rows >>= 1) {
            T.th = rows - extra;
            T.threads = rows >= 8 ? 256 : 128;
            if ((long)((cm + T.tw - 1) / T.tw) * ((cn + T.th - 1) / T.th) >= 3 * 152) break;
        }
    }
    T.bytes = bytes();
    return T;
}

}  // namespace mgw
}  // namespace stzg
