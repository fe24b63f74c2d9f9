// Arithmetic of the kernels' schedules, for the host and the device: plain C++ with no CUDA in
// it, so that a host compiler can check it at sizes that no test can run
// (tests/test_schedule.py).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MBG_HD __host__ __device__ __forceinline__
#else
#define MBG_HD inline
#endif

typedef int64_t i64;

namespace mbg {

// A reduction of k elements in slabs of `depth`: n slabs, the last of `last` elements.  A kernel
// asks for what is left from a slab's start on, never for the start itself, which passes
// 2^31 in the last slab of a reduction near 2^31.
struct KSlabs {
    i64 n;
    int last;
};
MBG_HD KSlabs k_slabs(i64 k, int depth) {
    KSlabs s;
    s.n = (k + depth - 1) / depth;
    s.last = s.n ? int(k - (s.n - 1) * depth) : 0;
    return s;
}
MBG_HD int k_left(int nkb, int last, int kb, int depth) { return kb + 1 < nkb ? depth : last; }

// Tiles in the order in which a product's CTAs take them: groups of `group` tile rows walk the tile
// columns together (L2 reuse).
struct TileGrid {
    int tiles_m, tiles_n, group;
};
struct TileAt {
    int tm, tn;
};
MBG_HD TileAt tile_at(const TileGrid& q, int t) {
    const int per_group = q.group * q.tiles_n;
    const int g = t / per_group, in_g = t - g * per_group;
    const int first_m = g * q.group, rest = q.tiles_m - first_m;
    const int gsize = rest < q.group ? rest : q.group;
    return TileAt{first_m + in_g % gsize, in_g / gsize};
}
MBG_HD i64 tile_index(const TileGrid& q, int tm, int tn) {
    const int first_m = tm / q.group * q.group, rest = q.tiles_m - first_m;
    const int gsize = rest < q.group ? rest : q.group;
    return i64(first_m) * q.tiles_n + i64(tn) * gsize + (tm - first_m);
}

// Tiles of bm x bn, tiles_m x ceil(n / bn) of them, that a triangle mask keeps (tri: 0 all, 1 those not
// strictly above the diagonal, 2 not strictly below), counted row by row: every product asks, ahead
// of its launch.
inline i64 kept_tiles(int tri, i64 tiles_m, i64 n, int bm, int bn) {
    const i64 all = (n + bn - 1) / bn;
    if (!tri) return tiles_m * all;
    i64 kept = 0;
    for (i64 tm = 0; tm < tiles_m; ++tm) {
        const i64 row = tri == 1 ? ((tm + 1) * bm + bn - 1) / bn : all - tm * bm / bn;
        kept += row > all ? all : row < 0 ? 0 : row;
    }
    return kept;
}

// Work of one persistent split launch (split_sk_kernel): one or two products (the second:
// the gemm adjoint's other gradient).  Tiles are numbered product 0's first, then product 1's.
//   whole tiles:  the first dp_tiles tiles, worker (CTA) c taking tiles c, c + G, ...
//                 (G workers); the triangle mask may skip tiles; C is stored
//                 with beta.
//   stream-K:     the slabs of the remaining tiles, [sk_begin, total) in slab positions
//                 over all tiles, cut into G equal contiguous ranges, one per worker, so
//                 the last wave leaves no SM idle.  A range runs on across tile boundaries
//                 without draining the pipeline.  Whole tiles are stored; a tile two ranges
//                 share is zeroed first (sk_zero_kernel) and both add their partial sums
//                 (beta = 0 only).  Every range is at least one tile long, so no tile gets
//                 more than two partial sums, and their fp32 sum does not depend on the
//                 order they arrive in.
struct SkWork {
    int tiles0, tiles1;   // tiles of each product (tiles1 = 0: one product)
    int nkb0, nkb1;       // k slabs of each product's tiles
    int dp_tiles;         // leading tiles taken whole
    i64 sk_begin, total;  // stream-K slab positions (sk_begin == total: none)
};

// First slab position of worker w's range.
MBG_HD i64 sk_range_begin(const SkWork& W, i64 w, i64 workers) {
    return W.sk_begin + w * (W.total - W.sk_begin) / workers;
}

// Schedule of a persistent split launch over up to G workers (SkWork): whole tiles; when
// the tiles leave a last wave partly empty (and stream_k allows), stream-K ranges over the
// last (tiles mod g) + g tiles, with g <= G workers chosen so that every range is at least
// as long as the longest tile, and only where the busiest worker then finishes clearly
// sooner than with whole tiles.  G returns the number of workers to launch.
inline SkWork sk_plan(i64 t0, int n0, i64 t1, int n1, i64& G, bool stream_k) {
    SkWork W{};
    W.tiles0 = int(t0);
    W.tiles1 = int(t1);
    W.nkb0 = n0;
    W.nkb1 = t1 ? n1 : n0;
    const i64 T = t0 + t1;
    W.dp_tiles = int(T);
    G = G < T ? G : T;
    if (!stream_k || G <= 0 || T % G == 0) return W;
    auto slab_pos = [&](i64 u) { return u <= t0 ? u * n0 : t0 * n0 + (u - t0) * n1; };
    const i64 longest = t1 && n1 > n0 ? n1 : n0;
    // all tiles in ranges of at least `longest` slabs: as many workers as that allows
    const i64 total = slab_pos(T);
    const i64 g = G < total / longest ? G : total / longest;
    const i64 dp = T > 2 * g ? T - (T % g) - g : 0;
    const i64 begin = slab_pos(dp);
    if (g <= 0 || (total - begin) / g < longest) return W;
    // worth it when the balanced ranges end before whole tiles would: whole tiles take
    // ceil(T / G) tile times on the busiest worker, the ranges (total - begin) / g slabs
    // after dp / g whole tiles
    const double whole = double((T + G - 1) / G) * double(longest);
    const double ranged = double(dp / g) * double(longest) + double(total - begin) / double(g);
    // the persistent kernel ran a slab about 5 % slower than tc_gemm_kernel (8192^3 NT, whole
    // tiles plus a stream-K tail: 4.43 against 4.26 ms): demand a tenth
    if (1.1 * ranged >= whole) return W;
    W.dp_tiles = int(dp);
    W.sk_begin = begin;
    W.total = total;
    G = g;
    return W;
}

// Where `workers` ranges cut tile t of a one-product schedule: the slab that the second part starts with, 0
// for a tile that one worker runs.
MBG_HD int sk_cut(const SkWork& W, i64 workers, i64 t) {
    if (t < W.dp_tiles || W.total == W.sk_begin) return 0;
    const i64 first = t * W.nkb0;
    // the last range to begin at or before the tile's first slab, or the one before it
    i64 w = (first - W.sk_begin) * workers / (W.total - W.sk_begin);
    while (w < workers && sk_range_begin(W, w, workers) <= first) ++w;
    const i64 cut = w < workers ? sk_range_begin(W, w, workers) - first : W.nkb0;
    return cut < W.nkb0 ? int(cut) : 0;
}

// The column block of a product that the pipelined host path computes, from tile column `tn0` of
// `whole` on: its tiles one per worker in turn, each cut where the schedule of the call over all of
// C (W, `workers`) cuts it, so that its sums are rounded as in that call.
struct SkBlock {
    SkWork W;
    i64 workers;
    TileGrid whole, block;
    int tn0;
};
MBG_HD int sk_block_cut(const SkBlock& B, int t) {
    const TileAt at = tile_at(B.block, t);
    return sk_cut(B.W, B.workers, tile_index(B.whole, at.tm, B.tn0 + at.tn));
}

}  // namespace mbg
