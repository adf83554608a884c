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

}  // namespace rules
}  // namespace emg
