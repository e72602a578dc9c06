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

}  // namespace hamlss
