// Layout of a graph's in-edges for the blocked PageRank gather (gg_pr.cu).
//
// The source ids are cut into blocks of kBlkSrc and the edges, in CSC order,
// into bins of kBinEdges.  The edges of one block that fall into one bin are
// its tile, stored as chunks of 8 (the last one padded), block by block and
// within a block bin by bin:
//   src[chunk * 8 + i]  the edge's source within its block (blk_slot)
//   pos[chunk * 8 + i]  the edge's place within its bin (bin_slot; kBinEdges: padding)
// and ptr[bin_ptr[b] .. bin_ptr[b + 1]) are the chunks of bin b.  A gather
// then moves values instead of fetching them one by one: block by block the
// contributions are read from shared memory in the order of src, and bin by
// bin the values are put in their places, in shared memory again.
#pragma once
#include "gg_internal.cuh"

namespace gg {

constexpr uint32_t kBlkSrcLog = 15, kBlkSrc = 1u << kBlkSrcLog;
constexpr uint32_t kBinThreads = 768, kBinEdges = 32 * kBinThreads;  // (32 edges per thread of k_pr_bins)
constexpr uint32_t kBlkMax = 2048;  // source blocks (a bin's tiles are sorted in shared memory)

// Place of a block's source in shared memory: its low bits mixed with the
// others, for in an R-MAT graph the sources of most edges have the same low
// bits and with them the same bank.
__host__ __device__ __forceinline__ uint32_t blk_slot(uint32_t v) {
    v &= kBlkSrc - 1;
    return v ^ ((v >> 6) & 63u) ^ ((v >> 9) & 63u);
}

// Place in shared memory of the bin's edge p.  A thread sums 32 edges one
// after the other; the mix puts those that the lanes of a warp read together
// into different banks.
__host__ __device__ __forceinline__ uint32_t bin_slot(uint32_t p) { return p ^ ((p >> 5) & 31u); }

struct PrPlan {
    bool tried = false, ready = false;
    uint32_t nblk = 0, nbin = 0, nparts = 0;
    uint64_t chunks = 0;
    void *base = nullptr;  // one allocation for the arrays below
    uint16_t *src = nullptr, *pos = nullptr;
    uint32_t *ptr = nullptr;
    uint32_t *bin_ptr = nullptr;   // [nbin + 1]
    uint32_t *ends = nullptr;      // [nbin * kBinThreads] a bit per edge: the last of its row
    uint32_t *bin_end = nullptr;   // [nbin + 1] rows with in-edges that end before the bin
    // the chunks cut into parts of equal work: segments {block, first chunk,
    // end} of part p are part_seg[p] .. part_seg[p + 1]
    uint4 *segs = nullptr;
    uint32_t *part_seg = nullptr;
};

// The graph's plan, built when first asked for; null where the graph does not
// fit the layout's limits, or the layout and the values not half of the free
// memory.
gg_status pr_plan(gg_graph *g, const PrPlan **out);
// Bytes of scratch that a gather of values of `size` bytes takes.
size_t pr_plan_bytes(const PrPlan *P, size_t size);
void pr_plan_free(gg_graph *g);

}  // namespace gg
