// Building of the blocked PageRank gather's edge layout (gg_prplan.cuh): a
// counting pass over the in-edges, a scan of the tiles' chunks, and a pass
// that sorts each bin's edges by source block in shared memory and writes
// them as whole chunks.  Ranks within a tile are taken with atomics, so their
// order may differ between builds; the gather's results do not depend on it.
#include <cub/cub.cuh>

#include <algorithm>
#include <new>
#include <vector>

#include "gg_prplan.cuh"

namespace gg {

namespace {

constexpr int kPB = 1024;
constexpr uint32_t kPer = kBinEdges / kPB;
static_assert(kBinEdges % kPB == 0 && kBinEdges < 65536, "places within a bin take 16 bits");

// sectors[0 / 1]: 32-byte sectors that the 4- / 2-byte values of each bin's first
// kPB edges lie in, those of a bin told apart by 13 bits of a hash (1000 of them
// count as 940)
__global__ void __launch_bounds__(kPB) k_plan_spread(const uint32_t *__restrict__ in_adj, uint64_t m,
                                                     uint32_t *sectors) {
    __shared__ uint32_t seen[2][256];
    const uint64_t e = (uint64_t)blockIdx.x * kBinEdges + threadIdx.x;
    if (threadIdx.x < 512) seen[threadIdx.x >> 8][threadIdx.x & 255u] = 0;
    __syncthreads();
    if (e < m) {
        const uint32_t v = __ldg(in_adj + e);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t h = (v >> (3 + k)) * 2654435761u >> 19;
            atomicOr(&seen[k][h >> 5], 1u << (h & 31u));
        }
    }
    __syncthreads();
    if (threadIdx.x < 512) {  // (a counter's bits lie in whole warps)
        const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(seen[threadIdx.x >> 8][threadIdx.x & 255u]));
        if (dev::lane_id() == 0) atomicAdd(sectors + (threadIdx.x >> 8), c);
    }
}

// chunks of every tile, and of every bin
__global__ void __launch_bounds__(kPB) k_plan_count(const uint32_t *__restrict__ in_adj, uint64_t m, uint32_t nblk,
                                                    uint32_t nbin, uint32_t *tile, uint32_t *bin_ptr) {
    __shared__ uint32_t hist[kBlkMax];
    const uint32_t b = blockIdx.x;
    const uint64_t base = (uint64_t)b * kBinEdges;
    for (uint32_t i = threadIdx.x; i < nblk; i += kPB) hist[i] = 0;
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = 0; i < kPer; ++i) {
        const uint64_t e = base + i * kPB + threadIdx.x;
        if (e < m) atomicAdd(&hist[__ldcs(in_adj + e) >> kBlkSrcLog], 1u);
    }
    __syncthreads();
    uint32_t sum = 0;
    for (uint32_t i = threadIdx.x; i < nblk; i += kPB) {
        const uint32_t c = (hist[i] + 7) / 8;
        tile[(uint64_t)i * nbin + b] = c;
        sum += c;
    }
    sum = dev::block_sum<uint32_t, kPB>(sum);
    if (threadIdx.x == 0) bin_ptr[b] = sum;
}

// each block's first chunk, and the number of chunks
__global__ void k_plan_starts(const uint32_t *tile, uint32_t nblk, uint32_t nbin, uint32_t *at) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k <= nblk) at[k] = tile[(uint64_t)k * nbin];
}

// the bin's edges sorted by block; tile holds each tile's first chunk
__global__ void __launch_bounds__(kPB) k_plan_fill(const uint32_t *__restrict__ in_adj, uint64_t m, uint32_t nblk,
                                                   uint32_t nbin, const uint32_t *__restrict__ tile,
                                                   const uint32_t *__restrict__ bin_ptr, uint16_t *src, uint16_t *pos,
                                                   uint32_t *ptr) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t cap = (kBinEdges + 7 * nblk + 7) / 8 * 8;
    uint16_t *ssrc = (uint16_t *)smem, *spos = ssrc + cap;
    __shared__ uint32_t hist[kBlkMax], first[kBlkMax + 1], wsum[kPB / 32];
    const uint32_t b = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t base = (uint64_t)b * kBinEdges;
    for (uint32_t i = threadIdx.x; i < nblk; i += kPB) hist[i] = 0;
    __syncthreads();
    uint32_t id[kPer], rank[kPer];
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i) {
        const uint64_t e = base + i * kPB + threadIdx.x;
        id[i] = e < m ? __ldcs(in_adj + e) : 0u;
    }
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i)
        rank[i] = base + i * kPB + threadIdx.x < m ? atomicAdd(&hist[id[i] >> kBlkSrcLog], 1u) : 0u;
    __syncthreads();
    // exclusive prefix of the tiles' chunks: two tiles per thread
    static_assert(kBlkMax == 2 * kPB, "two tiles per thread");
    const uint32_t t = 2 * threadIdx.x;
    const uint32_t c0 = t < nblk ? (hist[t] + 7) / 8 : 0u, c1 = t + 1 < nblk ? (hist[t + 1] + 7) / 8 : 0u;
    uint32_t incl = c0 + c1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += x;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t w = 0; w < warp; ++w) before += wsum[w];
    first[t] = before + incl - c0 - c1;
    first[t + 1] = before + incl - c1;
    if (threadIdx.x == kPB - 1) first[kBlkMax] = before + incl;
    __syncthreads();
    const uint32_t total = first[kBlkMax];
    for (uint32_t i = threadIdx.x; i < total; i += kPB) {
        ((uint4 *)ssrc)[i] = make_uint4(0, 0, 0, 0);
        ((uint4 *)spos)[i] = make_uint4(kBinEdges * 0x10001u, kBinEdges * 0x10001u, kBinEdges * 0x10001u,
                                        kBinEdges * 0x10001u);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i)
        if (base + i * kPB + threadIdx.x < m) {
            const uint32_t slot = first[id[i] >> kBlkSrcLog] * 8 + rank[i];
            ssrc[slot] = (uint16_t)blk_slot(id[i]);
            spos[slot] = (uint16_t)bin_slot(i * kPB + threadIdx.x);
        }
    __syncthreads();
    const uint64_t list = bin_ptr[b];
    for (uint32_t k = warp; k < nblk; k += kPB / 32) {
        const uint32_t f = first[k], cnt = (hist[k] + 7) / 8;
        if (!cnt) continue;
        const uint32_t to = tile[(uint64_t)k * nbin + b];
        for (uint32_t j = lane; j < cnt; j += 32) {
            ((uint4 *)src)[(uint64_t)to + j] = ((const uint4 *)ssrc)[f + j];
            ((uint4 *)pos)[(uint64_t)to + j] = ((const uint4 *)spos)[f + j];
            ptr[list + f + j] = to + j;
        }
    }
}

__global__ void k_plan_ends(const uint32_t *__restrict__ list, const uint64_t *__restrict__ count,
                            const uint64_t *__restrict__ in_off, uint32_t *ends) {
    const uint64_t nrow = *count, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nrow; k += stride) {
        const uint64_t last = in_off[list[k] + 1ull] - 1;
        atomicOr(ends + (last >> 5), 1u << (last & 31));
    }
}

__global__ void __launch_bounds__(kBinThreads) k_plan_bin_ends(const uint32_t *__restrict__ ends, uint32_t *bin_end) {
    const uint32_t c = dev::block_sum<uint32_t, kBinThreads>(
        __popc(ends[(uint64_t)blockIdx.x * kBinThreads + threadIdx.x]));
    if (threadIdx.x == 0) bin_end[blockIdx.x] = c;
}

size_t aligned(size_t b) { return (b + 255) / 256 * 256; }

size_t scan_bytes(uint64_t items) {
    size_t b = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, b, (uint32_t *)nullptr, (uint32_t *)nullptr, (int64_t)items);
    return b;
}

void plan_release(PrPlan *P) {
    cudaFree(P->base);
    cudaFree(P->segs);
    cudaFree(P->part_seg);
    *P = PrPlan();
    P->tried = true;
}

// What the building needs beside the layout, in scratch: every tile's chunks,
// every bin's, the blocks' first chunks, and the scans' own.
struct PlanTmp {
    uint32_t *tiles, *bins, *starts;
    void *scan;
    size_t scan_b, bytes;
    PlanTmp(const PrPlan *P, void *scratch) {
        const uint64_t ntile = (uint64_t)P->nblk * P->nbin;
        const size_t tb = aligned((ntile + 1) * 4), bb = aligned(((size_t)P->nbin + 1) * 4),
                     sb = aligned(((size_t)P->nblk + 1) * 4);
        scan_b = std::max(scan_bytes(ntile + 1), scan_bytes((uint64_t)P->nbin + 1));
        bytes = tb + bb + sb + scan_b;
        char *p = (char *)scratch;
        tiles = (uint32_t *)p;
        bins = (uint32_t *)(p + tb);
        starts = (uint32_t *)(p + tb + bb);
        scan = p + tb + bb + sb;
    }
};

#define PK(expr) do { cudaError_t _e = (expr); if (_e != cudaSuccess) return _e; } while (0)

// The share of sectors that a sample of the edges lies in.
cudaError_t plan_spread(gg_graph *g, PrPlan *P) {
    cudaStream_t st = g->ctx->stream;
    uint32_t *d = nullptr, h[2] = {0, 0};
    PK(cudaMalloc(&d, sizeof(h)));
    cudaError_t e = cudaMemsetAsync(d, 0, sizeof(h), st);
    if (e == cudaSuccess) {
        k_plan_spread<<<P->nbin, kPB, 0, st>>>(g->in_adj, g->m, d);
        g->ctx->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    PK(e);
    const double sampled = (double)(g->m / kBinEdges) * kPB + (double)std::min<uint64_t>(g->m % kBinEdges, kPB);
    for (int k = 0; k < 2; ++k) P->spread[k] = (float)(h[k] / sampled);
    P->sampled = true;
    return cudaSuccess;
}

// Counts the chunks of every tile; at[k]: block k's first one, of P->chunks.
cudaError_t plan_count(gg_graph *g, PrPlan *P, PlanTmp &T, std::vector<uint32_t> &at) {
    gg_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const uint64_t ntile = (uint64_t)P->nblk * P->nbin;
    PK(cudaMemsetAsync(T.tiles + ntile, 0, 4, st));
    PK(cudaMemsetAsync(T.bins + P->nbin, 0, 4, st));
    k_plan_count<<<P->nbin, kPB, 0, st>>>(g->in_adj, g->m, P->nblk, P->nbin, T.tiles, T.bins);
    PK(cudaGetLastError());
    PK(cub::DeviceScan::ExclusiveSum(T.scan, T.scan_b, T.tiles, T.tiles, (int64_t)ntile + 1, st));
    k_plan_starts<<<P->nblk / 256 + 1, 256, 0, st>>>(T.tiles, P->nblk, P->nbin, T.starts);
    PK(cudaGetLastError());
    ctx->launches += 3;
    at.resize((size_t)P->nblk + 1);
    PK(cudaMemcpyAsync(at.data(), T.starts, at.size() * 4, cudaMemcpyDeviceToHost, st));
    PK(cudaStreamSynchronize(st));
    P->chunks = at[P->nblk];
    return cudaSuccess;
}

cudaError_t plan_build(gg_graph *g, PrPlan *P, PlanTmp &T, const std::vector<uint32_t> &at) {
    gg_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const size_t cb = aligned(P->chunks * 16), pb = aligned(P->chunks * 4), bb = aligned(((size_t)P->nbin + 1) * 4),
                 eb = aligned((size_t)P->nbin * kBinThreads * 4);
    PK(cudaMalloc(&P->base, 2 * cb + pb + 2 * bb + eb));
    char *p = (char *)P->base;
    P->src = (uint16_t *)p;
    P->pos = (uint16_t *)(p + cb);
    P->ptr = (uint32_t *)(p + 2 * cb);
    P->bin_ptr = (uint32_t *)(p + 2 * cb + pb);
    P->bin_end = (uint32_t *)(p + 2 * cb + pb + bb);
    P->ends = (uint32_t *)(p + 2 * cb + pb + 2 * bb);
    PK(cudaMemsetAsync(P->bin_end, 0, bb + eb, st));
    k_plan_ends<<<ctx->sm_count * 8, 256, 0, st>>>(g->nonisolated, g->nonisolated_n, g->in_off, P->ends);
    PK(cudaGetLastError());
    k_plan_bin_ends<<<P->nbin, kBinThreads, 0, st>>>(P->ends, P->bin_end);
    PK(cudaGetLastError());
    PK(cub::DeviceScan::ExclusiveSum(T.scan, T.scan_b, T.bins, P->bin_ptr, (int64_t)P->nbin + 1, st));
    PK(cub::DeviceScan::ExclusiveSum(T.scan, T.scan_b, P->bin_end, P->bin_end, (int64_t)P->nbin + 1, st));
    const size_t smem = (size_t)((kBinEdges + 7 * P->nblk + 7) / 8 * 8) * 4;
    PK(cudaFuncSetAttribute(k_plan_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_plan_fill<<<P->nbin, kPB, smem, st>>>(g->in_adj, g->m, P->nblk, P->nbin, T.tiles, P->bin_ptr, P->src, P->pos,
                                            P->ptr);
    PK(cudaGetLastError());
    ctx->launches += 5;
    // parts of equal work: the chunks, and for each segment the load of its
    // block's contributions (as long as some kBlkSrc / 12 chunks); eight a SM,
    // fewer where loads would then take more than an eighth of a part (as many
    // regardless -> so: 20 iterations of R-MAT 20 5.13 -> 2.82 ms, of ER 63 M
    // edges 4.45 -> 4.17)
    const uint64_t load = kBlkSrc / 12;
    uint64_t work = 0;
    for (uint32_t k = 0; k < P->nblk; ++k)
        if (at[k + 1] > at[k]) work += at[k + 1] - at[k] + load;
    const uint64_t share = std::max<uint64_t>(work / ((uint64_t)ctx->sm_count * 8) + 1, 8 * load);
    std::vector<uint4> segs;
    std::vector<uint32_t> part{0};
    uint64_t room = share;
    for (uint32_t k = 0; k < P->nblk; ++k)
        for (uint32_t c = at[k]; c < at[k + 1];) {
            if (room <= load && segs.size() > part.back()) {
                part.push_back((uint32_t)segs.size());
                room = share;
            }
            const uint64_t take = std::min<uint64_t>(at[k + 1] - c, room > load ? room - load : share);
            segs.push_back(make_uint4(k, c, (uint32_t)(c + take), 0));
            c += (uint32_t)take;
            room = room > take + load ? room - take - load : 0;
        }
    part.push_back((uint32_t)segs.size());
    P->nparts = (uint32_t)part.size() - 1;
    PK(cudaMalloc(&P->segs, segs.size() * sizeof(uint4)));
    PK(cudaMalloc(&P->part_seg, part.size() * 4));
    PK(cudaMemcpyAsync(P->segs, segs.data(), segs.size() * sizeof(uint4), cudaMemcpyHostToDevice, st));
    PK(cudaMemcpyAsync(P->part_seg, part.data(), part.size() * 4, cudaMemcpyHostToDevice, st));
    PK(cudaStreamSynchronize(st));
#undef PK
    return cudaSuccess;
}

}  // namespace

gg_status pr_plan_wanted(gg_graph *g, size_t size, bool always, bool *yes) {
    *yes = false;
    if (!g->pr_plan) {
        PrPlan *P = new (std::nothrow) PrPlan();
        if (!P) return GG_OK;
        P->nblk = (uint32_t)(((uint64_t)g->n + kBlkSrc - 1) >> kBlkSrcLog);
        P->nbin = (uint32_t)((g->m + kBinEdges - 1) / kBinEdges);
        P->tried = !g->m || P->nblk > kBlkMax || g->m >> 32;  // (chunk numbers take 32 bits)
        g->pr_plan = P;
    }
    PrPlan *P = (PrPlan *)g->pr_plan;
    if ((P->tried && !P->ready) || (!always && P->nblk <= kBlkInL1)) return GG_OK;
    if (!always && !P->sampled) {
        const cudaError_t e = plan_spread(g, P);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            return GG_OK;
        }
        if (e != cudaSuccess) return cuda_error(g->ctx, e, "PageRank edge layout");
    }
    *yes = always || P->spread[size == 4 ? 0 : 1] >= (P->nblk <= kBlkHubsInL1 ? kSpreadLeastHubs : kSpreadLeast);
    return GG_OK;
}

size_t pr_plan_scratch(gg_graph *g, size_t size) {
    const PrPlan *P = (const PrPlan *)g->pr_plan;
    const size_t parts = (size_t)P->nbin * 16;  // of rows
    if (P->ready) return P->chunks * 8 * size + parts;
    return std::max(g->m * size + parts, PlanTmp(P, nullptr).bytes);
}

static gg_status plan_make(gg_graph *g, void *scratch) {
    PrPlan *P = (PrPlan *)g->pr_plan;
    P->tried = true;
    PlanTmp T(P, scratch);
    std::vector<uint32_t> at;
    cudaError_t e = plan_count(g, P, T, at);
    size_t free_b = 0, all_b = 0;
    if (e == cudaSuccess) e = cudaMemGetInfo(&free_b, &all_b);
    // the layout, 36 bytes a chunk, leaves half of the memory beside the values
    if (e == cudaSuccess && P->chunks * 72 > free_b) e = cudaErrorMemoryAllocation;
    if (e == cudaSuccess) e = plan_build(g, P, T, at);
    P->ready = e == cudaSuccess;
    if (P->ready) return GG_OK;
    plan_release(P);
    if (e != cudaErrorMemoryAllocation) return cuda_error(g->ctx, e, "PageRank edge layout");
    cudaGetLastError();
    return GG_OK;
}

gg_status pr_plan(gg_graph *g, void *scratch, const PrPlan **out) {
    *out = nullptr;
    PrPlan *P = (PrPlan *)g->pr_plan;
    if (!P->tried) {
        try {
            GG_CHECK(plan_make(g, scratch));
        } catch (const std::bad_alloc &) {  // of the host: no layout either
            plan_release(P);
        }
    }
    if (P->ready) *out = P;
    return GG_OK;
}

void pr_plan_free(gg_graph *g) {
    if (!g->pr_plan) return;
    plan_release((PrPlan *)g->pr_plan);
    delete (PrPlan *)g->pr_plan;
    g->pr_plan = nullptr;
}

}  // namespace gg
