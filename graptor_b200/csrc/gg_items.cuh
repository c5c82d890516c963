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
// The graph's item buffer g->items, kind by kind, allocated on first use.
gg_status graph_items(gg_graph *g);

struct ItemLists {
    unsigned long long *p[IT_KINDS];
};
inline ItemLists item_lists(const gg_graph *g, unsigned long long *items) {
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

// A warp's three lists.
struct ItemLister {
    ItemAppender a[IT_KINDS];
    __device__ __forceinline__ void init(unsigned long long (*buf)[ItemAppender::CAP]) {
#pragma unroll
        for (int k = 0; k < IT_KINDS; ++k) a[k] = {buf[k], nullptr, nullptr};
    }
    // this phase's items start `at[k]` into list k and are counted in cnt[k]
    __device__ __forceinline__ void begin(const ItemLists &l, const unsigned long long *at, unsigned long long *cnt) {
#pragma unroll
        for (int k = 0; k < IT_KINDS; ++k) {
            a[k].dst = l.p[k] + at[k];
            a[k].dst_n = cnt + k;
        }
    }
    // the last items: the counters' round trips overlap
    __device__ __forceinline__ void flush() {
        __syncwarp();
        const uint32_t lane = threadIdx.x & 31u;
        unsigned long long base = 0;
#pragma unroll
        for (int k = 0; k < IT_KINDS; ++k)
            if (lane == (uint32_t)k && a[k].n) base = atomicAdd(a[k].dst_n, (unsigned long long)a[k].n);
#pragma unroll
        for (int k = 0; k < IT_KINDS; ++k) a[k].store(__shfl_sync(0xffffffffu, base, k));
    }
    // the rows [beg, beg + deg) of the lanes with rec set (all lanes)
    __device__ __forceinline__ void list(bool rec, uint64_t beg, uint64_t deg) {
        a[IT_SHORT].push(rec && deg && deg <= kShort, make_item(beg, (uint32_t)deg));
        uint64_t left = rec && deg > kShort ? deg : 0;
        const bool huge = left > kHuge;
        while (__any_sync(0xffffffffu, left != 0)) {
            const uint32_t len = (uint32_t)min((uint64_t)(huge ? kHuge : kLong), left);
            a[IT_LONG].push(left && !huge, make_item(beg, len));
            a[IT_HUGE].push(left && huge, make_item(beg, len));
            beg += len;
            left -= len;
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
