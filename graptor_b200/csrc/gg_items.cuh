// gg_items.cuh -- work items of the resident kernels (k-core peel, BFS): a
// row, or a piece of it, as {first edge, length} in one 64-bit word.  A row of
// at most kShort edges is one short item, one of at most kHuge edges is cut
// into long items of kLong, and a longer one into huge items of kHuge, which a
// whole CTA takes.  A step then spreads over all warps whatever its rows'
// lengths, and a warp that finds the hubs of an R-MAT graph lists them in a
// few items each (with long items alone, 55,000 of them for the 2256
// neighbours of an R-MAT 24 root took 190 us; 14 us with huge ones).
#pragma once
#include "gg_internal.cuh"

namespace gg {

constexpr uint32_t kShort = 32, kLong = 256, kHuge = 4096;  // edges per item
enum { IT_SHORT = 0, IT_LONG = 1, IT_HUGE = 2, IT_KINDS = 3 };

// Room for items of rows that are each listed at most once: n short ones, long
// ones of rows above kShort edges (fewer than m / kShort rows), huge ones of
// rows above kHuge.
inline uint64_t items_cap(const gg_graph *g, int kind) {
    switch (kind) {
    case IT_SHORT: return g->n + 1ull;
    case IT_LONG: return g->m / kShort + g->m / kLong + 2;
    default: return 2 * (g->m / kHuge) + 2;
    }
}
// One allocation per graph, g->resident, holds what its resident runs keep: the
// items, kind by kind, three frontier bitmaps, and a state block for each run.
// (An allocation of its own for each cost a graph's first CC some 0.3 ms apiece.)
constexpr size_t kRunState = 1024;
enum { RUN_BFS = 0, RUN_CC = 1, RUN_KCORE = 2, RUN_KINDS = 3 };
inline size_t resident_bits_at(const gg_graph *g) {
    const uint64_t items = items_cap(g, IT_SHORT) + items_cap(g, IT_LONG) + items_cap(g, IT_HUGE);
    return (items * 8 + kRunState - 1) / kRunState * kRunState;
}
inline size_t bitmap_words4(const gg_graph *g) { return ((size_t)g->n + 127) / 128; }  // 16-byte words
inline size_t resident_state_at(const gg_graph *g, int run) {
    return (resident_bits_at(g) + 3 * bitmap_words4(g) * 16 + kRunState - 1) / kRunState * kRunState + run * kRunState;
}
inline void *resident_state(const gg_graph *g, int run) { return (char *)g->resident + resident_state_at(g, run); }
gg_status resident_memory(gg_graph *g);

struct ItemLists {
    unsigned long long *p[IT_KINDS];
};
inline ItemLists item_lists(const gg_graph *g) {
    unsigned long long *items = (unsigned long long *)g->resident;
    ItemLists l;
    for (int k = 0; k < IT_KINDS; ++k) {
        l.p[k] = items;
        items += items_cap(g, k);
    }
    return l;
}

__device__ __forceinline__ unsigned long long make_item(uint64_t beg, uint32_t len) { return (beg << 14) | len; }
__device__ __forceinline__ uint64_t item_first(unsigned long long it) { return it >> 14; }
__device__ __forceinline__ uint32_t item_len(unsigned long long it) { return (uint32_t)(it & 16383u); }

// Per-warp staging of item appends (see dev::WarpAppender): `dst` is where
// this phase's items start, `dst_n` counts them.
struct ItemAppender {
    static constexpr uint32_t CAP = 64;
    unsigned long long *buf, *dst, *dst_n;
    uint32_t n = 0;
    __device__ __forceinline__ void push(bool keep, unsigned long long item) {
        const uint32_t lane = threadIdx.x & 31u;
        const unsigned mk = __ballot_sync(0xffffffffu, keep);
        if (keep) buf[n + __popc(mk & ((1u << lane) - 1u))] = item;
        n += __popc(mk);
        if (n > CAP - 32) flush();
    }
    __device__ __forceinline__ void flush() {
        __syncwarp();
        unsigned long long base = 0;
        if (n && (threadIdx.x & 31u) == 0) base = atomicAdd(dst_n, (unsigned long long)n);
        store(__shfl_sync(0xffffffffu, base, 0));
    }
    // the staged items to dst[base ...]
    __device__ __forceinline__ void store(unsigned long long base) {
        for (uint32_t i = threadIdx.x & 31u; i < n; i += 32) dst[base + i] = buf[i];
        __syncwarp();
        n = 0;
    }
};

// A warp's three lists: short and long items are staged (up to 16 long ones a
// row), the huge ones of a row of millions of edges written by all lanes
// together (by the row's lane in turn, the 4096 items of a hub with 2^24
// neighbours took 740 us; 21 us so).
struct ItemLister {
    static constexpr int STAGED = 2;
    ItemAppender a[STAGED];
    unsigned long long *huge, *huge_n;
    __device__ __forceinline__ void init(unsigned long long (*buf)[ItemAppender::CAP]) {
#pragma unroll
        for (int k = 0; k < STAGED; ++k) a[k] = {buf[k], nullptr, nullptr};
    }
    // this phase's items start `at[k]` into list k and are counted in cnt[k]
    __device__ __forceinline__ void begin(const ItemLists &l, const unsigned long long *at, unsigned long long *cnt) {
#pragma unroll
        for (int k = 0; k < STAGED; ++k) {
            a[k].dst = l.p[k] + at[k];
            a[k].dst_n = cnt + k;
        }
        huge = l.p[IT_HUGE] + at[IT_HUGE];
        huge_n = cnt + IT_HUGE;
    }
    // the last items: the counters' round trips overlap
    __device__ __forceinline__ void flush() {
        __syncwarp();
        const uint32_t lane = threadIdx.x & 31u;
        unsigned long long base = 0;
#pragma unroll
        for (int k = 0; k < STAGED; ++k)
            if (lane == (uint32_t)k && a[k].n) base = atomicAdd(a[k].dst_n, (unsigned long long)a[k].n);
#pragma unroll
        for (int k = 0; k < STAGED; ++k) a[k].store(__shfl_sync(0xffffffffu, base, k));
    }
    // the rows [beg, beg + deg) of the lanes with rec set (all lanes)
    __device__ __forceinline__ void list(bool rec, uint64_t beg, uint64_t deg) {
        a[IT_SHORT].push(rec && deg && deg <= kShort, make_item(beg, (uint32_t)deg));
        const bool is_huge = rec && deg > kHuge;
        uint32_t left = rec && deg > kShort && !is_huge ? (uint32_t)deg : 0u;
        uint64_t at = beg;
        while (__any_sync(0xffffffffu, left != 0)) {
            const uint32_t len = min(kLong, left);
            a[IT_LONG].push(left != 0, make_item(at, len));
            at += len;
            left -= len;
        }
        if (__any_sync(0xffffffffu, is_huge)) list_huge(huge, huge_n, is_huge ? deg : 0u, beg);
    }
    // room for all lanes' items in one piece, which the lanes then fill
    static __device__ __forceinline__ void list_huge(unsigned long long *huge, unsigned long long *huge_n, uint64_t deg,
                                                  uint64_t beg) {
        constexpr unsigned FULL = 0xffffffffu;
        const uint32_t lane = threadIdx.x & 31u;
        const uint32_t items = (uint32_t)((deg + kHuge - 1) / kHuge);
        uint32_t incl = items;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31), excl = incl - items;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(huge_n, (unsigned long long)total);
        base = __shfl_sync(FULL, base, 0);
        for (uint32_t e = lane; e - lane < total; e += 32) {  // warp-uniform
            uint32_t r = 0;  // the last lane whose items start at or before e
#pragma unroll
            for (uint32_t step = 16; step; step >>= 1)
                if (__shfl_sync(FULL, excl, r + step) <= e) r += step;
            const uint64_t b = __shfl_sync(FULL, beg, r), d = __shfl_sync(FULL, deg, r);
            const uint64_t o = (uint64_t)(e - __shfl_sync(FULL, excl, r)) * kHuge;
            if (e < total) huge[base + e] = make_item(b + o, (uint32_t)min((uint64_t)kHuge, d - o));
        }
    }
};

// Pieces a long item is taken in: as many as leave every one of `nw` warps a
// piece of at least 32 edges, at most 8.
__device__ __forceinline__ uint32_t long_pieces(unsigned long long nlong, uint64_t nw) {
    uint32_t s = 1;
    while (s < kLong / 32 && nlong * s * 2 <= nw) s <<= 1;
    return s;
}
// Short items a warp takes together: as few as spread them over all warps.
__device__ __forceinline__ uint32_t short_group(unsigned long long nshort, uint64_t nw) {
    uint32_t g = 1;
    while (g < 32 && (uint64_t)g * nw < nshort) g <<= 1;
    return g;
}

}  // namespace gg
