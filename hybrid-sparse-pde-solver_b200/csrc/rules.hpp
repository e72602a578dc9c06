// rules.hpp -- host-side rules that choose a kernel's form, without CUDA: plain functions of
// sizes, so that they are tested by themselves.
#pragma once

#include <algorithm>

namespace hamlss {

// ------------------------------------------------------------- persistent CG (cg_persist.cuh)
constexpr int kPersistMaxRows = 3584;         // rows a block
constexpr int kPersistClusterBlocks = 16;
constexpr int kPersistMaxBlocks = 256;        // sets of partial sums (all_sums)

// Whether a launch of `blocks` blocks runs all at once, as both forms of the kernel need: a
// cluster of that size fits the device (active_clusters, from the occupancy query), or the
// grid's blocks are resident together (blocks_per_sm).  Partitioned devices and contexts that
// may use a part of one report less than the whole chip.
inline bool persist_can_run(bool cluster, int blocks, int active_clusters, int blocks_per_sm, int sm_count) {
    if (blocks < 1) return false;
    if (cluster) return blocks <= kPersistClusterBlocks && active_clusters >= 1;
    return blocks <= kPersistMaxBlocks && (long long)blocks_per_sm * sm_count >= blocks;
}

// Threads a block: one a row up to 256, unless the block reads many of its neighbours' rows each
// trip (`outside`: columns of its window that are not its own), which wait for L2 four a thread
// at a time.  The sums keep their order (the other warps' are zero).  28,000 rows of 5, 300
// trips, at 256 / 512 threads: 18,000 outside 5.1 / 3.6 ms, 24,000 6.0 / 4.1 ms (two launches a
// trip: 5.2); 33,000 rows, 6,000 outside 2.9 / 2.5 ms.
inline int persist_threads(int rows, int outside) { return rows <= 256 && outside <= 4096 ? 256 : 512; }

// --------------------------------------------------------------- FP64 products (spmv.cuh)
constexpr int kProdTile = 512;                // products a warp of k_spmv_prod holds

// Whether a matrix of long rows next to one another is left to a lane a row (k_spmv): all
// entries of the rows that one warp takes (`heaviest`: the most of any warp) go through its
// tile, and where a tile holds one row's part, one lane adds it while 31 wait.  Cycles of the
// slowest warp, measured: a tile ~1,500 for its loads and ~12 an addition; a lane a row ~225 an
// entry.  The rest of the matrix runs beside that warp and prefers k_spmv_prod by about a
// 200th of a cycle an entry.  A product of 100,000 rows of 10 with 40 neighbouring rows longer,
// k_spmv_prod / k_spmv: of 100 31 / 31 us, of 300 66 / 48, of 900 184 / 108; with 8 rows of 900
// 72 / 101.
inline bool prod_uneven(int longest, long long heaviest, long long nnz) {
    const long long tiles = (heaviest + kProdTile - 1) / kProdTile;
    const long long warp = tiles * (1500 + 12LL * std::min(longest, kProdTile));
    return warp - 225LL * longest > nnz / 200;
}

// Whether the gathers of neighbouring rows mostly fall on different lines: of the places that
// two neighbouring rows both have, fewer than half with columns at most kNearColumns apart.
// (Grids in natural or coloured order: nearly all.  Rows in random order, or random columns in
// a band of +-100: nearly none; spmv_stream.cuh's WIDE form then takes 94 us for 199, and 57
// for 59.)
constexpr int kNearColumns = 8;
constexpr int kNeighbourRows = 65536;         // rows looked at, about
inline bool gathers_scattered(int pairs, int near) { return pairs > 0 && 2LL * near < pairs; }

}  // namespace hamlss
