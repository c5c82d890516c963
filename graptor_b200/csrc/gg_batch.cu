// gg_batch.cu -- batched traversals.
//
//  * Multi-source BFS (up to 64 roots at once): one uint64 word per vertex
//    holds a bit per root for the frontier, the next frontier and the visited
//    set; an iteration is a push (OR frontier bits into out-neighbours' next
//    words, 64-bit atomicOr) or a pull (OR in-neighbours' frontier words, exit
//    early once every still-unvisited root has reached the vertex), chosen by
//    the m/20 rule on the frontier's vertex and edge counts.  The whole run is
//    one cooperative launch with the bounded grid barrier of gg_grid.cuh.
//    Levels are written per (vertex, root): level[v*64 + i].
//  * Personalized PageRank for up to 128 seeds: x_s <- alpha*e_s +
//    (1-alpha)*A^T D^-1 x_s.  The contribution matrix c[v][s] = x_s[v]/deg(v)
//    is stored in bfloat16, one row of 16, 32, 64 or 128 seeds per vertex, so
//    every gathered edge is one coalesced row (lane = 4 seeds); sums are
//    float32.  Hub rows are cut into chunks (HeavyRows) summed by separate
//    warps into float32 partials.  One launch per iteration.
//  * Disjoint union of many graphs on the device (gg_graph_union), so BFS
//    from every part's root and CC of every part run as one traversal.
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "gg_batch.h"
#include "gg_grid.cuh"
#include "gg_internal.cuh"

namespace gg {

constexpr unsigned FULLB = 0xffffffffu;
constexpr int kBB = 256;
constexpr unsigned long long kMsPushDiv = 4;  // push while |F| + outdeg(F) <= m / 4

// ---------------------------------------------------------------------------
// Multi-source BFS
// ---------------------------------------------------------------------------
struct MsState {
    grid::Barrier bar;
    int iterations;
    unsigned long long nfront, efront;        // current frontier: vertices, edges
    unsigned long long nnext, enext;          // being accumulated
    unsigned long long reached_e;             // sum over roots of the out-degrees reached
    unsigned long long t_ns[GG_MAX_ITERS + 1];
    int variant[GG_MAX_ITERS];
};

struct MsArgs {
    const uint64_t *off, *in_off;
    const uint32_t *adj, *in_adj;
    uint32_t n;
    uint64_t m;
    unsigned long long *visited, *front, *next;
    int32_t *level;  // [n][64]
    unsigned long long all;  // mask of the roots in use
    MsState *st;
    unsigned long long timeout_ns;
    int max_iters;
    int K;
    HeavyRows H;     // CSC rows longer than H.T edges, cut into H.CH-edge chunks
    int symmetric;   // the chunks also cut the CSR rows (push)
};

template <typename T> __device__ __forceinline__ T ldcgb(const T *p) { return __ldcg(p); }

__device__ __forceinline__ unsigned long long warp_or64(unsigned long long x) {
    const unsigned lo = __reduce_or_sync(FULLB, (unsigned)x);
    const unsigned hi = __reduce_or_sync(FULLB, (unsigned)(x >> 32));
    return ((unsigned long long)hi << 32) | lo;
}

// Push: out-edges of frontier vertices OR their frontier bits (minus the
// target's visited bits) into the target's next word.  Light rows: a warp
// per 32 vertices (lanes alone up to K edges, then the warp per long row);
// heavy rows of a symmetric graph: a warp per chunk.
__device__ void ms_push(const MsArgs &A, uint64_t gw, uint64_t nw, uint32_t lane) {
    const uint32_t T = A.symmetric ? A.H.T : 0xFFFFFFFFu;
    for (uint64_t w = gw; w * 32 < A.n; w += nw) {
        const uint32_t v = (uint32_t)(w * 32 + lane);
        const unsigned long long f = v < A.n ? ldcgb(A.front + v) : 0ull;
        uint64_t beg = 0, end = 0;
        if (f) {
            beg = A.off[v];
            end = A.off[v + 1];
            if (end - beg > T) end = beg;  // chunked below
        }
        const uint32_t k1 = (uint32_t)min(end - beg, (uint64_t)A.K);
        for (uint32_t k = 0; k < k1; ++k) {
            const uint32_t u = __ldg(A.adj + beg + k);
            const unsigned long long nv = f & ~ldcgb(A.visited + u);
            if (nv) atomicOr(A.next + u, nv);
        }
        unsigned pend = __ballot_sync(FULLB, f && beg + k1 < end);
        while (pend) {
            const int j = __ffs(pend) - 1;
            pend &= pend - 1;
            const uint64_t ej = __shfl_sync(FULLB, beg + k1, j), endj = __shfl_sync(FULLB, end, j);
            const unsigned long long fj = __shfl_sync(FULLB, f, j);
            for (uint64_t e = ej + lane; e < endj; e += 32) {
                const uint32_t u = __ldg(A.adj + e);
                const unsigned long long nv = fj & ~ldcgb(A.visited + u);
                if (nv) atomicOr(A.next + u, nv);
            }
        }
    }
    if (!A.symmetric) return;
    for (uint64_t c = gw; c < A.H.nchunks; c += nw) {
        const uint32_t h = A.H.crow[c];
        const uint32_t v = A.H.v[h];
        const unsigned long long f = ldcgb(A.front + v);
        if (!f) continue;
        const uint64_t e0 = A.off[v] + (c - A.H.first[h]) * A.H.CH;
        const uint64_t e1 = min(e0 + A.H.CH, A.off[v + 1]);
        for (uint64_t e = e0 + lane; e < e1; e += 32) {
            const uint32_t u = __ldg(A.adj + e);
            const unsigned long long nv = f & ~ldcgb(A.visited + u);
            if (nv) atomicOr(A.next + u, nv);
        }
    }
}

// Pull: a vertex ORs its in-neighbours' frontier words until every root it
// has not been reached from is present.  Light rows: each warp a contiguous
// range of 32-vertex words of equal light-edge work; heavy rows: a warp per
// chunk, atomicOr of the chunk's new bits.
__device__ void ms_pull(const MsArgs &A, uint64_t gw, uint64_t nw, uint32_t lane) {
    const uint32_t nwords = (A.n + 31) / 32;
    uint32_t wlo, whi;
    dev::balanced_range(A.H.light_prefix, nwords, gw, nw, wlo, whi);
    for (uint32_t w = wlo; w < whi; ++w) {
        const uint32_t v = w * 32 + lane;
        const bool valid = v < A.n;
        const unsigned long long vis = valid ? ldcgb(A.visited + v) : A.all;
        uint64_t e = 0, end = 0;
        if (valid && vis != A.all) {
            e = A.in_off[v];
            end = A.in_off[v + 1];
            if (end - e > A.H.T) end = e;  // heavy: chunked below
        }
        bool act = e < end;
        unsigned long long acc = 0;
        const uint64_t lim = min(end, e + (uint64_t)A.K);
        for (; act && e < lim; ++e) {
            acc |= ldcgb(A.front + __ldg(A.in_adj + e));
            if ((acc | vis) == A.all) act = false;
        }
        unsigned pend = __ballot_sync(FULLB, act && e < end);
        while (pend) {
            const int j = __ffs(pend) - 1;
            pend &= pend - 1;
            const uint64_t ej = __shfl_sync(FULLB, e, j), endj = __shfl_sync(FULLB, end, j);
            const unsigned long long visj = __shfl_sync(FULLB, vis, j);
            unsigned long long accj = __shfl_sync(FULLB, acc, j);
            for (uint64_t base = ej; base < endj; base += 32) {
                const uint64_t ed = base + lane;
                accj |= warp_or64(ed < endj ? ldcgb(A.front + __ldg(A.in_adj + ed)) : 0ull);
                if ((accj | visj) == A.all) break;
            }
            if ((int)lane == j) acc = accj;
        }
        const unsigned long long nx = acc & ~vis;
        if (valid && nx) A.next[v] = nx;
    }
    for (uint64_t c = gw; c < A.H.nchunks; c += nw) {
        const uint32_t h = A.H.crow[c];
        const uint32_t v = A.H.v[h];
        const unsigned long long vis = ldcgb(A.visited + v);
        if (vis == A.all) continue;
        const uint64_t e0 = A.in_off[v] + (c - A.H.first[h]) * A.H.CH;
        const uint64_t e1 = min(e0 + A.H.CH, A.in_off[v + 1]);
        unsigned long long acc = 0;
        for (uint64_t base = e0; base < e1; base += 32) {
            const uint64_t ed = base + lane;
            acc |= warp_or64(ed < e1 ? ldcgb(A.front + __ldg(A.in_adj + ed)) : 0ull);
            if ((acc | vis) == A.all) break;
        }
        const unsigned long long nx = acc & ~vis;
        if (lane == 0 && nx) atomicOr(A.next + v, nx);
    }
}

__global__ void __launch_bounds__(kBB) k_msbfs(MsArgs A) {
    MsState *st = A.st;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t nw = ((uint64_t)gridDim.x * kBB) >> 5;
    const uint64_t gw = ((uint64_t)blockIdx.x * kBB + threadIdx.x) >> 5;
    const uint64_t tid = (uint64_t)blockIdx.x * kBB + threadIdx.x, nth = (uint64_t)gridDim.x * kBB;
    if (blockIdx.x == 0 && threadIdx.x == 0) st->t_ns[0] = grid::globaltimer();
    int iter = 0;
    for (; iter < A.max_iters; ++iter) {
        const unsigned long long nf = ldcgb(&st->nfront), ef = ldcgb(&st->efront);
        if (nf == 0) break;
        // a pull scans most in-edges (it stops early only once every root
        // has reached the vertex), a push only the frontier's out-edges
        const bool push = (nf + ef) <= A.m / kMsPushDiv;
        if (blockIdx.x == 0 && threadIdx.x == 0 && iter < GG_MAX_ITERS)
            st->variant[iter] = push ? GG_VAR_PUSH_DENSE : GG_VAR_PULL_DENSE;
        if (push) ms_push(A, gw, nw, lane);
        else ms_pull(A, gw, nw, lane);
        if (!grid::sync(&st->bar, A.timeout_ns)) return;
        // update: visited, levels, next frontier, counts
        unsigned long long cnt = 0, edg = 0, red = 0;
        for (uint64_t v = tid; v < A.n; v += nth) {
            const unsigned long long nx = ldcgb(A.next + v);
            A.front[v] = nx;
            if (nx) {
                A.next[v] = 0ull;
                A.visited[v] = ldcgb(A.visited + v) | nx;
                const uint64_t deg = A.off[v + 1] - A.off[v];
                cnt++;
                edg += deg;
                red += deg * (unsigned long long)__popcll(nx);
                for (unsigned long long b = nx; b; b &= b - 1) A.level[v * 64 + (__ffsll((long long)b) - 1)] = iter + 1;
            }
        }
        cnt = dev::block_sum<unsigned long long, kBB>(cnt);
        edg = dev::block_sum<unsigned long long, kBB>(edg);
        red = dev::block_sum<unsigned long long, kBB>(red);
        if (threadIdx.x == 0) {
            if (cnt) atomicAdd(&st->nnext, cnt);
            if (edg) atomicAdd(&st->enext, edg);
            if (red) atomicAdd(&st->reached_e, red);
        }
        if (!grid::sync(&st->bar, A.timeout_ns)) return;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            st->nfront = st->nnext;
            st->efront = st->enext;
            st->nnext = 0;
            st->enext = 0;
            if (iter < GG_MAX_ITERS) st->t_ns[iter + 1] = grid::globaltimer();
        }
        if (!grid::sync(&st->bar, A.timeout_ns)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) st->iterations = iter;
}

__global__ void k_ms_init(MsArgs A) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t)gridDim.x * blockDim.x;
    const int32_t inf = (int32_t)(A.n + 1);
    for (uint64_t i = tid; i < (uint64_t)A.n * 64; i += nth) A.level[i] = inf;
    for (uint64_t v = tid; v < A.n; v += nth) {
        A.visited[v] = 0;
        A.front[v] = 0;
        A.next[v] = 0;
    }
}

__global__ void k_ms_roots(MsArgs A, const uint32_t *roots, int k) {
    // one thread: roots may repeat
    if (blockIdx.x || threadIdx.x) return;
    unsigned long long nf = 0, ef = 0;
    for (int i = 0; i < k; ++i) {
        const uint32_t r = roots[i];
        if (A.front[r] == 0) {
            nf++;
            ef += A.off[r + 1] - A.off[r];
        }
        A.front[r] |= 1ull << i;
        A.visited[r] |= 1ull << i;
        A.level[(uint64_t)r * 64 + i] = 0;
        A.st->reached_e += A.off[r + 1] - A.off[r];
    }
    A.st->nfront = nf;
    A.st->efront = ef;
}

__global__ void k_ms_pack(const int32_t *level, uint32_t n, int k, int32_t *out) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = tid; i < (uint64_t)n * k; i += nth) out[i] = level[i / k * 64 + i % k];
}

// ---------------------------------------------------------------------------
// Personalized PageRank, 128 seeds, bfloat16 rows
// ---------------------------------------------------------------------------
constexpr int kPprSeeds = 128;  // 4 per lane

struct PprArgs {
    const uint64_t *in_off, *off;
    const uint32_t *in_adj;
    uint32_t n;
    const uint2 *cin;   // [n] rows of 4 L bf16 (uint2 = 4 bf16 per lane)
    uint2 *cout;        // next contributions; null in the last iteration
    uint2 *xout;        // ranks (bf16), written by the last iteration only (else null)
    const uint32_t *seeds;  // [128]
    float alpha;
    HeavyRows H;
    float4 *partial;    // [nchunks][L] float4 per lane
    uint32_t *arrived;  // [nheavy] chunks of the row that are done; wraps to 0
    uint32_t rows;      // light rows per ticket
    uint32_t tickets;   // of the chunks, 32 / L each, then of the light rows
    uint32_t *ticket;   // this iteration's; the next one's is set to 0
    uint32_t *next_ticket;
};

__device__ __forceinline__ void bf4_acc(uint2 v, float4 &a) {
    a.x += __uint_as_float(v.x << 16);
    a.y += __uint_as_float(v.x & 0xFFFF0000u);
    a.z += __uint_as_float(v.y << 16);
    a.w += __uint_as_float(v.y & 0xFFFF0000u);
}

__device__ __forceinline__ uint2 f4_to_bf4(float4 f) {
    uint2 r;
    r.x = (uint32_t)dev::bf16_rne(f.x) | ((uint32_t)dev::bf16_rne(f.y) << 16);
    r.y = (uint32_t)dev::bf16_rne(f.z) | ((uint32_t)dev::bf16_rne(f.w) << 16);
    return r;
}

// x = alpha*e_seed + (1-alpha)*acc; c = x/deg; written as bf16 rows (a
// contribution only where the vertex has an out-edge by which it is read)
template <int L>
__device__ __forceinline__ void ppr_finish(const PprArgs &A, uint32_t d, float4 acc, uint32_t lane) {
    const uint4 seed = __ldg((const uint4 *)A.seeds + lane);
    const uint64_t deg = A.off[d + 1] - A.off[d];
    const float b = 1.0f - A.alpha;
    float4 x = make_float4(b * acc.x, b * acc.y, b * acc.z, b * acc.w);
    if (seed.x == d) x.x += A.alpha;
    if (seed.y == d) x.y += A.alpha;
    if (seed.z == d) x.z += A.alpha;
    if (seed.w == d) x.w += A.alpha;
    if (A.xout) A.xout[(uint64_t)d * L + lane] = f4_to_bf4(x);
    if (A.cout && deg) {
        const float inv = 1.0f / (float)deg;
        A.cout[(uint64_t)d * L + lane] = f4_to_bf4(make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv));
    }
}

// One launch per iteration.  What bounds it: every edge reads a row of cin,
// and an SM receives about one 32-byte sector per clock from L2 (a row of 128
// seeds is eight; 9.1 TB/s over the chip where L1 holds none of them, which
// uniform ids reach).
//   * A row is as wide as its seeds need: 4 per lane over L = 4, 8, 16 or 32
//     lanes for up to 16, 32, 64 or 128 seeds.
//   * Warps draw tickets, first the chunks of the heavy rows and then small
//     sets of light rows, so that neither waits for a launch of its own; the
//     last chunk of a row to be done adds the row's partial sums.  The sums'
//     order is that of the edges within a row or chunk and of the chunks
//     within a row, whatever L.
//   * Ids are loaded for a whole batch at once and one batch ahead; 16 rows
//     are in flight (chunks of 1024 edges are a chain of that many fewer
//     round trips; 8 rows in flight and 5 CTAs per SM: R-MAT 18 5.10 ms, ER
//     4.77 ms, R-MAT 10 0.79 ms).
//   * A vertex without out-edges has no contribution to write, nor has any
//     vertex in the last iteration.
// 20 iterations, before (a warp per row, 4 rows in flight, rows of 128 seeds
// whatever their number, three launches) -> after: 128 seeds on R-MAT 18 x 16
// 8.49 -> 4.89 ms, R-MAT 10 1.07 -> 0.38, ER 2^18 x 32 4.99 -> 5.05; 50 seeds
// on R-MAT 17 4.34 -> 2.02; 5 seeds on R-MAT 18 6.72 -> 2.04; 29 and 9 seeds
// on directed ER 200001 x 12 2.09 -> 0.79 and 2.11 -> 0.54.
constexpr int kPprBlock = 256;
constexpr uint32_t kPprFlight = 16;
// most light rows per ticket
template <int L> constexpr uint32_t kPprRows = L == 32 ? 8 : 4 * (32 / L);

// Rows as wide as a warp.
__global__ void __launch_bounds__(kPprBlock, 4) k_ppr_wide(PprArgs A) {
    constexpr uint32_t FULL = 0xffffffffu, F = kPprFlight, kSkip = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint2 *cin = A.cin + lane;
    if (blockIdx.x == 0 && threadIdx.x == 0) *A.next_ticket = 0;
    uint32_t t = (blockIdx.x * kPprBlock + threadIdx.x) >> 5, next = 0;
    for (; t < A.tickets; t = __shfl_sync(FULL, next, 0)) {
        if (lane == 0) next = gridDim.x * (kPprBlock / 32) + atomicAdd(A.ticket, 1u);
        // lane r < rows holds the edges of the ticket's row d0 + r (kSkip: a
        // heavy row, done by its chunks): one chunk, or the light rows
        uint32_t d0, rows, len = kSkip;
        const uint32_t *ids;
        if (t < A.H.nchunks) {
            const uint32_t h = A.H.crow[t];
            d0 = A.H.v[h];
            rows = 1;
            const uint64_t e0 = A.in_off[d0] + (t - A.H.first[h]) * A.H.CH;
            len = (uint32_t)min((uint64_t)A.H.CH, A.in_off[d0 + 1] - e0);
            ids = A.in_adj + e0;
        } else {
            d0 = (t - (uint32_t)A.H.nchunks) * A.rows;
            rows = min(A.n - d0, A.rows);
            const uint64_t beg = __ldg(A.in_off + d0 + min(lane, rows)), end = __shfl_down_sync(FULL, beg, 1);
            if (lane < rows && end - beg <= A.H.T) len = (uint32_t)(end - beg);
            ids = A.in_adj + beg;
        }
        for (uint32_t r = 0; r < rows; ++r) {
            const uint32_t deg = __shfl_sync(FULL, len, r);
            const uint32_t *at = (const uint32_t *)__shfl_sync(FULL, (unsigned long long)ids, r) + lane;
            if (deg == kSkip) continue;
            float4 acc = make_float4(0, 0, 0, 0);
            uint32_t nid = lane < deg ? __ldg(at) : 0u;
            for (uint32_t e = 0; e < deg; e += 32) {
                const uint32_t id = nid;
                at += 32;
                nid = e + 32 + lane < deg ? __ldg(at) : 0u;
                const uint32_t cnt = min(deg - e, 32u);
                for (uint32_t j = 0; j < cnt; j += F) {
                    uint2 row[F];
                    if (j + F <= cnt) {
#pragma unroll
                        for (uint32_t u = 0; u < F; ++u)
                            row[u] = __ldg(cin + (uint64_t)__shfl_sync(FULL, id, j + u) * 32);
#pragma unroll
                        for (uint32_t u = 0; u < F; ++u) bf4_acc(row[u], acc);
                    } else {
#pragma unroll
                        for (uint32_t u = 0; u < F - 1; ++u)
                            if (j + u < cnt) row[u] = __ldg(cin + (uint64_t)__shfl_sync(FULL, id, j + u) * 32);
#pragma unroll
                        for (uint32_t u = 0; u < F - 1; ++u)
                            if (j + u < cnt) bf4_acc(row[u], acc);
                    }
                }
            }
            if (t < A.H.nchunks) {
                const uint32_t h = A.H.crow[t];
                const uint32_t c0 = (uint32_t)A.H.first[h], c1 = (uint32_t)A.H.first[h + 1];
                if (c1 - c0 > 1) {  // the last chunk of the row to be done adds them up, in their order
                    __stcg(A.partial + (uint64_t)t * 32 + lane, acc);
                    __threadfence();
                    __syncwarp();
                    uint32_t before = 0;
                    if (lane == 0) before = atomicInc(A.arrived + h, c1 - c0 - 1);
                    if (__shfl_sync(FULL, before, 0) != c1 - c0 - 1) break;
                    __threadfence();
                    acc = make_float4(0, 0, 0, 0);
                    for (uint32_t c = c0; c < c1; ++c) {
                        const float4 p = __ldcg(A.partial + (uint64_t)c * 32 + lane);
                        acc.x += p.x;
                        acc.y += p.y;
                        acc.z += p.z;
                        acc.w += p.w;
                    }
                }
            }
            ppr_finish<32>(A, d0 + r, acc, lane);
        }
    }
}

// The same for rows of L < 32 lanes: the warp's G = 32 / L groups of lanes
// work on one destination each, in step (apart, their loads would wait for one
// another: 5 seeds on R-MAT 18 3.70 ms).
template <int L>
__global__ void __launch_bounds__(kPprBlock, 3) k_ppr_narrow(PprArgs A) {
    constexpr uint32_t FULL = 0xffffffffu, G = 32 / L, F = kPprFlight;
    constexpr uint32_t IDS = L < F ? F / L : 1, BATCH = IDS * L;
    constexpr uint32_t kSkip = 0xffffffffu;
    const uint32_t wl = threadIdx.x & 31u, lane = wl & (L - 1), grp = wl / L;
    const uint2 *cin = A.cin + lane;
    if (blockIdx.x == 0 && threadIdx.x == 0) *A.next_ticket = 0;
    const uint32_t nct = ((uint32_t)A.H.nchunks + G - 1) / G;
    uint32_t t = (blockIdx.x * kPprBlock + threadIdx.x) >> 5, next = 0;
    for (; t < A.tickets; t = __shfl_sync(FULL, next, 0)) {
        if (wl == 0) next = gridDim.x * (kPprBlock / 32) + atomicAdd(A.ticket, 1u);
        // lane r holds the edges of the ticket's row r (kSkip: none, or a
        // heavy row, done by its chunks)
        const bool chunk = t < nct;
        uint32_t d = 0, rows = G, len = kSkip;
        const uint32_t *ids = A.in_adj;
        if (chunk) {
            const uint32_t c = t * G + wl;
            if (wl < G && c < A.H.nchunks) {
                const uint32_t h = A.H.crow[c];
                d = A.H.v[h];
                const uint64_t e0 = A.in_off[d] + (c - A.H.first[h]) * A.H.CH;
                len = (uint32_t)min((uint64_t)A.H.CH, A.in_off[d + 1] - e0);
                ids += e0;
            }
        } else {
            rows = A.rows;
            const uint64_t at = (uint64_t)(t - nct) * A.rows + wl;
            d = (uint32_t)at;
            if (wl < rows && at < A.n) {
                const uint64_t beg = __ldg(A.in_off + at), end = __ldg(A.in_off + at + 1);
                if (end - beg <= A.H.T) len = (uint32_t)(end - beg);
                ids += beg;
            }
        }
        for (uint32_t r = grp; r < rows; r += G) {
            uint32_t deg = __shfl_sync(FULL, len, r);
            const bool act = deg != kSkip;
            const uint32_t *at = (const uint32_t *)__shfl_sync(FULL, (unsigned long long)ids, r) + lane;
            if (!act) deg = 0;
            const uint32_t longest = __reduce_max_sync(FULL, deg);
            float4 acc = make_float4(0, 0, 0, 0);
            uint32_t nid[IDS];
#pragma unroll
            for (uint32_t i = 0; i < IDS; ++i) nid[i] = i * L + lane < deg ? __ldg(at + i * L) : 0u;
            for (uint32_t e = 0; e < longest; e += BATCH) {
                uint32_t id[IDS];
                at += BATCH;
#pragma unroll
                for (uint32_t i = 0; i < IDS; ++i) {
                    id[i] = nid[i];
                    nid[i] = e + BATCH + i * L + lane < deg ? __ldg(at + i * L) : 0u;
                }
                const uint32_t cnt = e < deg ? min(deg - e, BATCH) : 0u;
                const uint32_t steps = min(longest - e, BATCH);
#pragma unroll 1
                for (uint32_t j = 0; j < steps; j += F) {
                    uint2 row[F];
#pragma unroll
                    for (uint32_t u = 0; u < F; ++u) {
                        const uint32_t v = __shfl_sync(FULL, id[IDS == 1 ? 0 : u / L], IDS == 1 ? j + u : u % L, L);
                        if (j + u < cnt) row[u] = __ldg(cin + (uint64_t)v * L);
                    }
#pragma unroll
                    for (uint32_t u = 0; u < F; ++u)
                        if (j + u < cnt) bf4_acc(row[u], acc);
                }
            }
            bool done = act;
            if (chunk) {  // the last chunk of a row to be done adds them up, in their order
                const uint32_t c = t * G + grp;
                uint32_t h = 0, c0 = 0, c1 = 0, before = 0;
                if (act) {
                    h = A.H.crow[c];
                    c0 = (uint32_t)A.H.first[h];
                    c1 = (uint32_t)A.H.first[h + 1];
                }
                const bool several = c1 - c0 > 1;
                if (several) __stcg(A.partial + (uint64_t)c * L + lane, acc);
                __threadfence();
                __syncwarp();
                if (several && lane == 0) before = atomicInc(A.arrived + h, c1 - c0 - 1);
                before = __shfl_sync(FULL, before, 0, L);
                if (several) {
                    done = before == c1 - c0 - 1;
                    __threadfence();
                    if (done) acc = make_float4(0, 0, 0, 0);
                    for (c0 = done ? c0 : c1; c0 < c1; ++c0) {
                        const float4 p = __ldcg(A.partial + (uint64_t)c0 * L + lane);
                        acc.x += p.x;
                        acc.y += p.y;
                        acc.z += p.z;
                        acc.w += p.w;
                    }
                }
            }
            const uint32_t dr = __shfl_sync(FULL, d, r);
            if (done) ppr_finish<L>(A, dr, acc, lane);
        }
    }
}

// contributions of the seeds' own rows (x too, where no iteration writes it)
// and the counters of the first iteration
__global__ void k_ppr_init(uint2 *c, uint2 *x, const uint64_t *off, uint32_t n, int L, const uint32_t *seeds,
                           uint32_t *counters, uint64_t ncounters) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = tid; i < ncounters; i += nth) counters[i] = 0;
    const uint4 seed = __ldg((const uint4 *)seeds + tid % L);  // nth is a multiple of L
    for (uint64_t i = tid; i < (uint64_t)n * L; i += nth) {
        const uint32_t d = (uint32_t)(i / L);
        float4 xv = make_float4(seed.x == d, seed.y == d, seed.z == d, seed.w == d);
        const uint64_t deg = off[d + 1] - off[d];
        const float inv = deg ? 1.0f / (float)deg : 0.0f;
        if (x) x[i] = f4_to_bf4(xv);
        c[i] = f4_to_bf4(make_float4(xv.x * inv, xv.y * inv, xv.z * inv, xv.w * inv));
    }
}

__global__ void k_ppr_unpack(const uint2 *x, uint32_t n, int L, int k, float *out) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = tid; i < (uint64_t)n * k; i += nth) {
        const uint64_t d = i / k;
        const uint32_t s = (uint32_t)(i % k);
        const uint2 r = x[d * L + s / 4];
        const uint32_t word = (s & 2) ? r.y : r.x;
        out[i] = __uint_as_float((s & 1) ? (word & 0xFFFF0000u) : (word << 16));
    }
}

template <int L>
static void ppr_run(gg_ctx *ctx, PprArgs A, uint2 *c0, uint2 *c1, uint2 *x, uint32_t *counters, int iters) {
    void (*step)(PprArgs);
    if constexpr (L == 32) step = k_ppr_wide;
    else step = k_ppr_narrow<L>;
    constexpr uint32_t G = 32 / L;
    const uint64_t cap = (uint64_t)ctx->sm_count * resident_ctas((const void *)step, kPprBlock);
    // fewer rows per ticket where warps would go without any (always the most ->
    // so: ER 1204 x 45, 99 seeds, 14 iterations 0.355 -> 0.122 ms, R-MAT 10, 128
    // seeds, 20 iterations 0.67 -> 0.38)
    A.rows = G * (uint32_t)std::max<uint64_t>(
                     1, std::min<uint64_t>(kPprRows<L> / G, A.n / (G * cap * (kPprBlock / 32))));
    A.tickets = (uint32_t)((A.H.nchunks + G - 1) / G + ((uint64_t)A.n + A.rows - 1) / A.rows);
    const unsigned grid = (unsigned)std::min<uint64_t>(cap, ((uint64_t)A.tickets + 7) / 8);
    for (int it = 0; it < iters; ++it) {
        A.cin = (it & 1) ? c1 : c0;
        A.cout = it + 1 == iters ? nullptr : (it & 1) ? c0 : c1;
        A.xout = it + 1 == iters ? x : nullptr;  // only the ranks of the last iteration are kept
        A.ticket = counters + (it & 1);
        A.next_ticket = counters + (~it & 1);
        step<<<grid, kPprBlock, 0, ctx->stream>>>(A);
        ctx->launches++;
    }
}

// ---------------------------------------------------------------------------
// Disjoint union
// ---------------------------------------------------------------------------
__global__ void k_union_part(const uint64_t *off, const uint32_t *adj, uint32_t n, uint64_t m, uint64_t ebase,
                             uint32_t vbase, uint64_t *uoff, uint32_t *uadj) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v = tid; v < n; v += nth) uoff[vbase + v] = off[v] + ebase;
    for (uint64_t e = tid; e < m; e += nth) uadj[ebase + e] = adj[e] + vbase;
}

__global__ void k_set_u64(uint64_t *p, uint64_t v) { *p = v; }

static unsigned bgrid(gg_ctx *ctx, uint64_t work) {
    uint64_t b = (work + kBB - 1) / kBB, cap = (uint64_t)ctx->sm_count * 8;
    return (unsigned)std::max<uint64_t>(1, std::min(b, cap));
}

}  // namespace gg

using namespace gg;

extern "C" {

gg_status gg_msbfs(gg_graph *g, const uint32_t *roots, int k, int32_t *host_levels, gg_run_stats *stats) {
    if (!g || !roots || k < 1 || k > 64) return GG_ERR_ARG;
    gg_ctx *ctx = g->ctx;
    for (int i = 0; i < k; ++i)
        if (roots[i] >= g->n) return set_error(ctx, GG_ERR_ARG, "gg_msbfs: root out of range");
    cudaStream_t s = ctx->stream;
    const uint64_t n = g->n;
    // scratch: visited, front, next (8n each), levels (256n), roots, state
    const size_t words = (3 * n + 1) * 8, lev = n * 64 * 4;
    const size_t pack = host_levels && k < 64 ? n * k * 4 : 0;  // the levels as the caller wants them
    void *base;
    GG_CHECK(graph_scratch(g, words + lev + 64 * 4 + sizeof(MsState) + 512 + pack, &base));
    char *p = (char *)base;
    MsArgs A;
    std::memset(&A, 0, sizeof(A));
    A.visited = (unsigned long long *)p;
    A.front = A.visited + n;
    A.next = A.front + n;
    A.level = (int32_t *)(p + words);
    uint32_t *droots = (uint32_t *)(p + words + lev);
    MsState *st = (MsState *)(((uintptr_t)(p + words + lev + 64 * 4) + 255) & ~(uintptr_t)255);
    A.off = g->off;
    A.adj = g->adj;
    A.in_off = g->in_off;
    A.in_adj = g->in_adj;
    A.n = g->n;
    A.m = g->m;
    A.all = k == 64 ? ~0ull : ((1ull << k) - 1);
    A.st = st;
    A.timeout_ns = tuning().barrier_timeout_ns;
    A.max_iters = (int)std::min<uint64_t>(n + 2, 1u << 30);
    A.K = tuning().pull_k;
    A.H = g->heavy;
    A.symmetric = g->symmetric;
    GG_CUDA(ctx, cudaMemcpyAsync(droots, roots, k * 4, cudaMemcpyHostToDevice, s));
    GG_CUDA(ctx, cudaMemsetAsync(st, 0, sizeof(MsState), s));
    cudaEventRecord(ctx->ev0, s);
    k_ms_init<<<bgrid(ctx, n * 64), kBB, 0, s>>>(A);
    GG_LAUNCHED(ctx);
    k_ms_roots<<<1, 32, 0, s>>>(A, droots, k);
    GG_LAUNCHED(ctx);
    const int per_sm = resident_ctas((const void *)k_msbfs, kBB);
    void *args[] = {&A};
    GG_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)k_msbfs, dim3(ctx->sm_count * per_sm), dim3(kBB), args, 0, s));
    ctx->launches++;
    cudaEventRecord(ctx->ev1, s);
    MsState hs;
    GG_CUDA(ctx, cudaMemcpyAsync(&hs, st, sizeof(hs), cudaMemcpyDeviceToHost, s));
    GG_CUDA(ctx, cudaStreamSynchronize(s));
    if (hs.bar.err & DEV_ERR_TIMEOUT) return set_error(ctx, GG_ERR_TIMEOUT, "gg_msbfs: grid barrier timed out");
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        float ms = 0;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        stats->total_ms = ms;
        stats->iterations = hs.iterations;
        stats->edges_reached = hs.reached_e;
        for (int i = 0; i < std::min(hs.iterations, GG_MAX_ITERS); ++i) {
            stats->variant[i] = hs.variant[i];
            stats->iter_ms[i] = (hs.t_ns[i + 1] - hs.t_ns[i]) * 1e-6;
            stats->kernel_ms[i] = stats->iter_ms[i];
        }
    }
    if (host_levels) {
        const int32_t *out = A.level;
        if (k < 64) {
            // [n][64] -> [n][k] on the device
            int32_t *packed = (int32_t *)(st + 1);
            k_ms_pack<<<bgrid(ctx, n * k), kBB, 0, s>>>(A.level, g->n, k, packed);
            GG_LAUNCHED(ctx);
            out = packed;
        }
        GG_CHECK(host_download(ctx, host_levels, out, n * k * 4));
    }
    return GG_OK;
}

gg_status gg_ppr(gg_graph *g, const uint32_t *seeds, int k, float alpha, int iters, float *host_x,
                 gg_run_stats *stats) {
    if (!g || !seeds || k < 1 || k > kPprSeeds || !(alpha > 0 && alpha < 1) || iters < 0) return GG_ERR_ARG;
    gg_ctx *ctx = g->ctx;
    for (int i = 0; i < k; ++i)
        if (seeds[i] >= g->n) return set_error(ctx, GG_ERR_ARG, "gg_ppr: seed out of range");
    cudaStream_t s = ctx->stream;
    const uint64_t n = g->n;
    const int L = k <= 16 ? 4 : k <= 32 ? 8 : k <= 64 ? 16 : 32;  // lanes of a row, 4 seeds each
    const size_t row = (size_t)L * 8;
    const size_t part = (g->heavy.nchunks + 1) * L * sizeof(float4);
    const uint64_t ncounters = g->heavy.nheavy + 2;
    void *base;
    GG_CHECK(graph_scratch(g, 3 * n * row + part + 512 + ncounters * 4, &base));
    char *p = (char *)base;
    uint2 *c0 = (uint2 *)p, *c1 = (uint2 *)(p + n * row), *x = (uint2 *)(p + 2 * n * row);
    float4 *partial = (float4 *)(p + 3 * n * row);
    uint32_t *dseeds = (uint32_t *)(p + 3 * n * row + part), *counters = dseeds + kPprSeeds;
    std::vector<uint32_t> sd(kPprSeeds, 0xFFFFFFFFu);  // unused slots match no vertex
    std::memcpy(sd.data(), seeds, k * 4);
    GG_CUDA(ctx, cudaMemcpyAsync(dseeds, sd.data(), kPprSeeds * 4, cudaMemcpyHostToDevice, s));
    GG_CUDA(ctx, cudaStreamSynchronize(s));
    PprArgs A;
    std::memset(&A, 0, sizeof(A));
    A.in_off = g->in_off;
    A.off = g->off;
    A.in_adj = g->in_adj;
    A.n = g->n;
    A.seeds = dseeds;
    A.alpha = alpha;
    A.H = g->heavy;
    A.partial = partial;
    A.arrived = counters + 2;
    GG_CUDA(ctx, cudaEventRecord(ctx->ev0, s));
    k_ppr_init<<<bgrid(ctx, n * L), kBB, 0, s>>>(c0, iters ? nullptr : x, g->off, g->n, L, dseeds, counters,
                                                 ncounters);
    GG_LAUNCHED(ctx);
    if (L == 4) ppr_run<4>(ctx, A, c0, c1, x, counters, iters);
    else if (L == 8) ppr_run<8>(ctx, A, c0, c1, x, counters, iters);
    else if (L == 16) ppr_run<16>(ctx, A, c0, c1, x, counters, iters);
    else ppr_run<32>(ctx, A, c0, c1, x, counters, iters);
    GG_CUDA(ctx, cudaGetLastError());
    GG_CUDA(ctx, cudaEventRecord(ctx->ev1, s));
    GG_CUDA(ctx, cudaStreamSynchronize(s));
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        float ms = 0;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        stats->total_ms = ms;
        stats->iterations = iters;
        stats->scanned_edges = (uint64_t)iters * g->m;
    }
    if (host_x) {
        // (the contribution rows are free now: 16 L bytes per vertex, k <= 4 L floats)
        float *dx = (float *)c0;
        k_ppr_unpack<<<bgrid(ctx, n * k), kBB, 0, s>>>(x, g->n, L, k, dx);
        GG_LAUNCHED(ctx);
        GG_CHECK(host_download(ctx, host_x, dx, n * k * 4));
    }
    return GG_OK;
}

static gg_status graph_union_once(gg_ctx *ctx, gg_graph *const *parts, int k, gg_graph **out, uint32_t *vertex_base) {
    if (!ctx || !parts || k < 1 || !out) return GG_ERR_ARG;
    uint64_t n = 0, m = 0;
    int sym = 1;
    bool sorted = true;  // a part's rows keep their order, shifted by its vertex base
    for (int i = 0; i < k; ++i) {
        if (!parts[i] || parts[i]->ctx != ctx) return set_error(ctx, GG_ERR_ARG, "gg_graph_union: bad part");
        sorted &= parts[i]->rows_sorted;
        if (vertex_base) vertex_base[i] = (uint32_t)n;
        n += parts[i]->n;
        m += parts[i]->m;
        sym &= parts[i]->symmetric;
    }
    if (vertex_base) vertex_base[k] = (uint32_t)n;
    if (n >= 0xFFFFFFFFull) return set_error(ctx, GG_ERR_ARG, "gg_graph_union: more than 2^32-1 vertices");
    uint64_t *uoff = nullptr;
    uint32_t *uadj = nullptr;
    cudaStream_t s = ctx->stream;
    GG_CUDA(ctx, cudaMalloc(&uoff, (n + 1) * 8));
    cudaError_t e = cudaMalloc(&uadj, (m ? m : 1) * 4);
    if (e != cudaSuccess) { cudaFree(uoff); return cuda_error(ctx, e, "gg_graph_union"); }
    uint64_t eb = 0, vb = 0;
    for (int i = 0; i < k; ++i) {
        gg_graph *q = parts[i];
        k_union_part<<<bgrid(ctx, std::max<uint64_t>(q->n, q->m)), kBB, 0, s>>>(q->off, q->adj, q->n, q->m, eb,
                                                                                  (uint32_t)vb, uoff, uadj);
        ctx->launches++;
        eb += q->m;
        vb += q->n;
    }
    k_set_u64<<<1, 1, 0, s>>>(uoff + n, m);
    ctx->launches++;
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { cudaFree(uoff); cudaFree(uadj); return cuda_error(ctx, e, "gg_graph_union"); }
    return graph_adopt_device_csr(ctx, (uint32_t)n, m, uoff, uadj, sym, sorted, out);
}

gg_status gg_graph_union(gg_ctx *ctx, gg_graph *const *parts, int k, gg_graph **out, uint32_t *vertex_base) {
    if (!ctx) return GG_ERR_ARG;
    return with_room(ctx, [&] { return graph_union_once(ctx, parts, k, out, vertex_base); });
}

}  // extern "C"
