// Rules on sizes that launches follow, in plain C++: the tests compile this file on the host alone.
#pragma once

#include <cstdint>

namespace emg {
namespace rules {

// Column-wise dots (emg_krylov.cu): 256 threads lie over (row group, column) of a tile of up to 128
// columns; a thread sums every ``dot_groups``-th row of its block's ``dot_rows``.
constexpr int kDotThreads = 256;
constexpr int dot_tile(int64_t Bc) {                  // columns of a tile
    const int64_t ct = (Bc + 127) / 128;
    return (int)((Bc + ct - 1) / ct);
}
constexpr int dot_groups(int64_t Bc) { return kDotThreads / dot_tile(Bc); }
// Rows of a block: two blocks per SM where there are at least 64 rows for each (fewer spend more
// on the reduction than on the products).  FP32 sums go on in FP64 after a thread's rows, so these
// are at most 32, and from 32 columns on 1024, however large n is (FP32 dots have at least as many blocks as FP64 ones).
constexpr int64_t dot_rows(int64_t n, int64_t Bc, bool fp32) {
    const int64_t two = (n + 2 * 152 - 1) / (2 * 152), rows = two > 64 ? two : 64;
    const int64_t cap = (int64_t)dot_groups(Bc) * (Bc < 32 ? 32 : 1024);
    return fp32 && rows > cap ? cap : rows;
}
constexpr int64_t dot_blocks(int64_t n, int64_t Bc, bool fp32) {
    return (n + dot_rows(n, Bc, fp32) - 1) / dot_rows(n, Bc, fp32);
}

// K chunks of a tile through two shared buffers (emg_tc.cu, emg_fp64.cu): the MMAs of chunk c arrive at the
// mbarrier of its buffer, and a wait for them names the parity of that barrier's phase.  Of
// ``committed`` chunks those from pending_from on may still run: a tile that ends, also early after a
// time-out, waits for these before its tensor memory goes.
constexpr int chunk_buffer(int c) { return c & 1; }
constexpr unsigned chunk_parity(int c) { return (unsigned)(c >> 1) & 1u; }
constexpr int pending_from(int committed) { return committed > 2 ? committed - 2 : 0; }

// K splits of a tiled slab product: two CTAs per SM, at least 256 of K and at most max_splits each.
constexpr int gemm_splits(int64_t tiles, int64_t w, int max_splits) {
    int64_t sp = (2 * 152 + tiles - 1) / (tiles > 1 ? tiles : 1);
    const int64_t most = w / 256 > 1 ? w / 256 : 1;
    if (sp > most) sp = most;
    if (sp > max_splits) sp = max_splits;
    return sp > 1 ? (int)sp : 1;
}
// CTAs of a cluster of the split-TF32 product (``col_tiles`` column tiles in all groups together): doubled while the CTAs
// fit one wave and each keeps two chunks of 32.
constexpr int split_ranks(int64_t w, int64_t col_tiles, int max_splits) {
    const int64_t tiles = (w + 127) / 128 * col_tiles;
    int ranks = 1;
    while (ranks < 8 && 2 * ranks <= max_splits && tiles * 2 * ranks <= 152 && w >= 2 * ranks * 64) ranks *= 2;
    return ranks;
}
// FP32 groups of up to 16 columns on wide slabs: 128 x 16 CUDA-core tiles (k_slab_gemm16) where they are
// faster than what the slab takes else, row blocks (rows8) or split-TF32 tiles.  Estimates in us.  The
// tiles take 0.1 per K of a split, two thirds of it more for every CTA that an SM has beyond the first,
// and 4 at the launch, which the others hide under the one before; row blocks 0.0075 per K and CTA of an
// SM; the split tiles 2.4 per 32 of K of a cluster's CTA, twice where clusters of eight do not all fit.
// Measured (tiles / else): 2000 wide, one group 31 / 47, two 50 / 44, three 70 / 88; 2500, two 73 / 99;
// 1500, four 52 / 61; 1000, two 33 / 17 (row blocks).  Over 700 to 2500 wide and one to four groups of 8 and
// 16 columns the choice is within 4 % of the faster one, launches counted.
constexpr bool narrow_tiles_win(int64_t w, int G, int maxcol, int max_splits, bool rows8) {
    const int64_t tiles = (w + 127) / 128 * G;
    const int sp = gemm_splits(tiles, w, max_splits), ranks = split_ranks(w, G, max_splits);
    const int64_t rounds = (tiles * sp + 151) / 152;
    const double kper = (double)((w + sp - 1) / sp);
    const double narrow = 0.1 * kper * (0.35 + 0.65 * rounds) + 6;
    const double rows = 0.0075 * w * ((double)((w + 7) / 8 * G) / 152) * (maxcol <= 8 ? 1.0 : 1.2) + 4;
    const double chunks = (double)(((w + ranks - 1) / ranks + 31) / 32);
    const double split = 2.4 * chunks * (ranks == 8 && tiles > 14 ? 2 : 1) + 5;
    return maxcol <= 16 && narrow < (rows8 ? rows : split);
}

}  // namespace rules
}  // namespace emg
