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

// The gather by blocks pays from some 25 M edges on (20 iterations, by rows
// -> by blocks, the first call of a graph with the layout's building: ER 16 M
// 2.36 -> 2.67 ms and 2.00 -> 1.71 for the next, R-MAT 20 with 31 M edges 8.7
// -> 8.1 and 3.31 -> 2.82, ER 63 M FP16 6.4 -> 5.6 and 5.9 -> 4.2, R-MAT 22 x 8
// FP32 6.8 -> 6.5 and 6.4 -> 5.1).  The layout takes the time of some 3 (ER) to
// 20 (R-MAT 24) iterations' gain to build: it is built once a graph has run that
// many, those counted that the coming run is sure to take (no tolerance to meet:
// with one it may end after a few, however many it is allowed).
constexpr uint64_t kBlockedEdges = 3ull << 23;
constexpr uint64_t kBlockedIters = 16;

// What the gather by rows takes depends on the ids: values that many edges in
// a row share, or whose sectors they share, are found in L1.  The blocked gather
// takes the same time whatever they are.  So it pays where 1024 consecutive edges
// (the work of one warp) have their values in at least kSpreadLeast * 1024 sectors
// of 32 bytes.  Time by rows over time by blocks, FP32 with double sums / BF16,
// at that share: grid 4096^2 0.90 / 0.97 (0.10, 0.05), star 2^25 0.81 / 0.93 (0.06,
// 0.03), sources within 1000 ids 0.79 / 0.77 (0.13, 0.06), 2000 1.00 / 0.90 (0.25,
// 0.13), 4000 1.16 / 1.05 (0.43, 0.24), 8000 1.28 / 1.20 (0.63, 0.43), R-MAT 20 to
// 24 and ER 1.14 to 2.9 (0.82 to 0.94).
constexpr float kSpreadLeast = 0.24f;
// L1 also holds the values of a graph of up to 2 source blocks whatever the
// order of its edges (ER of 50,000 vertices and 50 M edges 0.79 / 0.61, 60,000
// 0.98 / 0.73, 80,000 1.14 / 1.09), and those of the hubs up to 4 (R-MAT 17
// with 41 M edges 0.92 / 0.93 at 0.62 / 0.50, R-MAT 18 1.00 / 1.08, ER of 100,000 to
// 300,000 1.15 to 2.1 at 0.9).
constexpr uint32_t kBlkInL1 = 2, kBlkHubsInL1 = 4;
constexpr float kSpreadLeastHubs = 0.75f;

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
    bool sampled = false, tried = false, ready = false;
    float spread[2] = {0, 0};  // sectors per edge of 4- and 2-byte values
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

// Whether a gather of values of `size` bytes should go by blocks: not where the
// graph does not fit the layout's limits or memory, nor (unless `always`) where
// the gather by rows is the faster one (kSpreadLeast).
gg_status pr_plan_wanted(gg_graph *g, size_t size, bool always, bool *yes);
// Bytes of scratch that such a gather takes, as far as is known before the plan
// is there, and that its building takes.
size_t pr_plan_scratch(gg_graph *g, size_t size);
// The graph's plan, built in scratch of pr_plan_scratch when first asked for;
// null where the layout does not leave half of the free memory.
gg_status pr_plan(gg_graph *g, void *scratch, const PrPlan **out);
void pr_plan_free(gg_graph *g);

}  // namespace gg
