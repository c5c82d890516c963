// gg_pr.cu -- PageRank power iteration (PRv / PR_vary) and the ADD_GATHER
// edgemap.
//
// Reference loop (bench/PRv.C:115-290, bench/PR_vary.C:247-447), per
// iteration:
//   y[d]  = sum_{s->d} contrib[s]                  dense pull, PRv.C:202-212
//   s     = sum y                                   (double)   PRv.C:227-231
//   y    += (1-s)/n                                 dangling + teleport mass
//   s     = sum y ; y *= 1/s                        renormalise
//   delta = sum |x-y| (double); x = y; y = 0; contrib = d*x/outdeg
// until iter == maxiter or delta <= tol.
//
// B200 design: two kernels per iteration (three where there are heavy rows,
// four where the gather goes by blocks of sources),
// all enqueued up front; a device-resident state block carries the sums and a
// "done" flag that makes later iterations return immediately once the
// residual test passes, so the host never synchronises inside the loop.
//   k_pr_gather : the light rows' contributions staged in shared memory 32
//                 rows at a time, heavy rows chunk by chunk; contributions
//                 decoded from the storage format (FP32, BF16, FP16, FP8-E4M3
//                 with scale, customfp<6,10>, BF16-by-truncation);
//                 accumulation in float or double; the block sums of y
//                 (double) are folded in with one atomic per CTA.
//   k_pr_values, k_pr_bins, k_pr_spans : the same sums for large graphs, the
//                 values moved by blocks of sources and bins of edges.
//   k_pr_update : y += w, y *= 1/s, delta, x = y, contrib = d*x/deg encoded,
//                 one pass.  The second sum of the reference (sum of the
//                 rounded y+w) is taken as s + n*w in double: equal in exact
//                 arithmetic, different by at most n/2 float ulps of 1/n.
//   pr_finish   : (last CTA of the update, staged runs: a kernel) residual
//                 test, iteration count, FP8 scale for the next encode (from
//                 this iteration's max with 2x headroom); FP16 is scaled the
//                 same way, since contributions of order 1/n fall below its
//                 normal range.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <cmath>
#include <cstring>

#include <cstdio>
#include <cstdlib>

#include <algorithm>
#include "gg_prplan.cuh"

namespace gg {

// ---------------------------------------------------------------------------
// Storage formats
// ---------------------------------------------------------------------------
template <int DT> struct Store;
// Rank / accumulator type of the vertex passes: double for the FP64 variant
// (PR_vary's FP64 run_prec instantiation), float otherwise.
template <int DT> using XT = typename std::conditional<DT == GG_F64, double, float>::type;
template <> struct Store<GG_F64> {
    using T = double;
    __device__ static double dec(T v) { return v; }
    __device__ static T enc(double f) { return f; }
};
template <> struct Store<GG_F32> {
    using T = float;
    __device__ static float dec(T v) { return v; }
    __device__ static T enc(float f) { return f; }
};
// bfloat16 / float16 stored as raw 16-bit words: plain integer loads and
// stores (the class types' assignment made the bfloat16 update kernel several
// times slower than the float16 one).
template <> struct Store<GG_BF16> {
    using T = uint16_t;
    __device__ static float dec(T v) { return __uint_as_float((uint32_t)v << 16); }
    __device__ static T enc(float f) { return dev::bf16_rne(f); }
};
template <> struct Store<GG_F16> {
    using T = uint16_t;
    __device__ static float dec(T v) { return __half2float(__ushort_as_half(v)); }
    __device__ static T enc(float f) { return __half_as_ushort(__float2half_rn(f)); }
};
template <> struct Store<GG_FP8E4M3> {
    using T = __nv_fp8_storage_t;
    __device__ static float dec(T v) {
        __half_raw h = __nv_cvt_fp8_to_halfraw(v, __NV_E4M3);
        return __half2float(__half(h));
    }
    __device__ static T enc(float f) { return __nv_cvt_float_to_fp8(f, __NV_SATFINITE, __NV_E4M3); }
};
// Graptor customfp<6,10> (include/graptor/customfp.h:97-166): low 6 exponent
// bits + top 10 mantissa bits, truncated; decoding restores exponent bit 6.
template <> struct Store<GG_CFP_6_10> {
    using T = uint16_t;
    __device__ static float dec(T v) { return __uint_as_float(((uint32_t)v | (1u << 16)) << 13); }
    __device__ static T enc(float f) { return (T)((__float_as_uint(f) >> 13) & 0xFFFFu); }
};
// Graptor scustomfp<true,8,7>: bfloat16 by truncation.
template <> struct Store<GG_BF16_TRUNC> {
    using T = uint16_t;
    __device__ static float dec(T v) { return __uint_as_float((uint32_t)v << 16); }
    __device__ static T enc(float f) { return (T)(__float_as_uint(f) >> 16); }
};

struct PrState {
    double s1;        // sum of y after the gather
    double delta;     // L1 residual of this iteration
    float cmax;       // max contribution written by the update (for FP8 scaling)
    float scale;      // encode multiplier of the stored contributions
    float scale_inv;  // decode multiplier
    int done;
    int iters;
    int maxiter;
    double tol;
    double deltas[GG_MAX_ITERS];
    // staged runs (PR_vary's run_prec_X then run_prec_Y): the active stage,
    // each stage's dtype and residual bound, and a re-encode request raised
    // when the stage changes
    int stage, nstages, reencode;
    unsigned int updated;  // CTAs of the update kernel that have finished
    int stage_dt[4];
    double stage_tol[4];
    // BF16 stochastic rounding; tail averaging from iteration avg_from on
    int sr;
    int avg_from, avg_n;
};

// MurmurHash3's fmix32 finaliser: 16 random bits per (vertex, iteration)
__device__ __forceinline__ uint32_t sr_bits(uint32_t v, uint32_t it) {
    uint32_t h = v * 0x9E3779B1u + it * 0x85EBCA77u + 0x165667B1u;
    h ^= h >> 16;
    h *= 0x85EBCA6Bu;
    h ^= h >> 13;
    h *= 0xC2B2AE35u;
    h ^= h >> 16;
    return h & 0xFFFFu;
}
// bfloat16 of a non-negative float rounded up with probability (f - down) /
// (up - down): the low 16 bits of the pattern plus 16 random bits carry into
// bit 16 exactly that often (inf stays inf)
__device__ __forceinline__ uint16_t bf16_stochastic(float f, uint32_t v, uint32_t it) {
    const uint32_t u = __float_as_uint(f);
    if ((u & 0x7F800000u) == 0x7F800000u) return (uint16_t)(u >> 16);
    return (uint16_t)((u + sr_bits(v, it)) >> 16);
}

// true when a kernel of stage `stage` (-1: unstaged) has nothing to do
__device__ __forceinline__ bool pr_idle(const PrState *st, int stage) {
    return st && (st->done || (stage >= 0 && st->stage != stage));
}

constexpr unsigned FULL = 0xffffffffu;

// num / deg, infinite for deg 0 (a vertex without out-edges: nothing gathers
// its contribution).  Dividing by the degree 0 itself leaves the division's
// fast path, and one such lane sends its whole warp through the slow one: in
// an R-MAT graph, where half of the vertices are isolated, nearly every warp
// (k_pr_update at R-MAT 24, FP32: 908 us of a 3.05 ms iteration).  The degree
// is converted from 32 bits where it fits in them.
__device__ __forceinline__ float per_degree(float num, uint64_t deg) {
    if (deg >> 32) return num / (float)deg;
    const float q = num / (float)max((uint32_t)deg, 1u);
    return deg ? q : __int_as_float(0x7F800000);
}
__device__ __forceinline__ double per_degree(double num, uint64_t deg) {
    const double q = num / (double)(deg ? deg : 1ull);
    return deg ? q : __longlong_as_double(0x7FF0000000000000ll);
}

// Scaled formats: FP8-E4M3 (max 448) and FP16 (max 65504, min normal 2^-14)
// store contrib * scale with scale a power of two chosen so that the
// largest contribution lands at half the format's range (2x headroom).
__device__ __host__ inline bool scaled_format(int dt) { return dt == GG_FP8E4M3 || dt == GG_F16; }
__device__ __host__ inline float scale_for(int dt, float cmax) {
    if (!scaled_format(dt) || !(cmax > 0.0f)) return 1.0f;
    const float half_range = dt == GG_FP8E4M3 ? 224.0f : 32768.0f;
    int e;
    frexpf(half_range / cmax, &e);
    return ldexpf(1.0f, e - 1);
}

// a row's sum as a float rank
template <int DT, typename Acc> __device__ __forceinline__ float pr_value(Acc acc, float sinv) {
    if (DT == GG_FP8E4M3 || DT == GG_F16) acc *= (Acc)sinv;
    return (float)acc;
}

// y[d] (or its double twin) from a row's sum; returns the stored value for
// the sum of all y.
template <int DT, bool ADD_OLD, typename Acc>
__device__ __forceinline__ double pr_store_row(float *y_f32, double *y_f64, uint32_t d, Acc acc, float sinv) {
    if (DT == GG_FP8E4M3 || DT == GG_F16) acc *= (Acc)sinv;
    if (y_f64) {
        const double v = ADD_OLD ? y_f64[d] + (double)acc : (double)acc;
        y_f64[d] = v;
        return v;
    }
    const float v = ADD_OLD ? (float)((double)y_f32[d] + (double)acc) : (float)acc;
    y_f32[d] = v;
    return (double)v;
}

// Sum of the decoded contributions of in_adj[e0, e1) over the warp's lanes
// (a lane's share; the caller reduces), 8 coalesced loads per lane in flight.
template <int DT, typename Acc>
__device__ __forceinline__ Acc pr_chunk_sum(const uint32_t *__restrict__ in_adj,
                                            const typename Store<DT>::T *__restrict__ contrib, uint64_t e0,
                                            uint64_t e1, uint32_t lane) {
    using S = Store<DT>;
    Acc part = 0;
    uint64_t base = e0;
    for (; base + 256 <= e1; base += 256) {
        uint32_t s8[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) s8[u] = __ldcs(in_adj + base + 32 * u + lane);
        XT<DT> c8[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) c8[u] = S::dec(contrib[s8[u]]);
#pragma unroll
        for (int u = 0; u < 8; ++u) part += (Acc)c8[u];
    }
    if (base < e1) {
        uint32_t s8[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint64_t e = base + 32 * u + lane;
            s8[u] = e < e1 ? __ldcs(in_adj + e) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (base + 32 * u + lane < e1) part += (Acc)S::dec(contrib[s8[u]]);
    }
    return part;
}

// y[d] = sum of the contributions of d's in-neighbours (and, with st, the
// sum of all y).  What bounds it: every gathered value that misses L1 moves
// one 32-byte sector from L2, and an SM receives about one such sector per
// clock (283 G gathers/s over the chip with uniform ids, 4- or 2-byte values;
// up to 340 G/s with R-MAT ids, whose hubs hit L1), so the sums must stay off
// the load/store unit as far as they can and enough loads be in flight.
//   * Warps draw tickets: first the chunks of the heavy rows (rows above T
//     edges, cut into H.CH-edge chunks), then ranges of 32-vertex words of
//     equal light-edge work, so that no SM waits for a warp with long chunks
//     (a fixed share per warp left warps idle for 8 % of the time).
//   * The light rows of a word are one list of edges, staged in shared memory
//     kStage at a time; ids are loaded one batch ahead of their values.  Then
//     32, 16, ... or 1 lanes sum each row's part from there, depending on how
//     many rows the stage holds, parts much longer than the others by the
//     whole warp.  (A warp per row kept one id and one value per lane in
//     flight and paid a five-step reduction per row.)
//   * The edges of the heavy rows in a word are gaps in its list, which is
//     then loaded in runs between them.
// 2 KiB of stage per warp and 5 CTAs per SM: more of either takes L1 from the
// gathered lines in flight (FP32, ER: 4 KiB 2.9 ms).  Measured per iteration,
// the rest of it included, before -> after: R-MAT 24, FP32 with double sums
// 2.23 -> 1.99 ms, BF16 1.98 -> 1.85; directed ER 2^24 x 32 4.27 -> 2.38 and
// 2.78 -> 2.13; grid 2048^2 FP32 0.30 -> 0.09; R-MAT 14 0.044 -> 0.034.
constexpr uint64_t kChunkGroup = 2;  // heavy-row chunks per ticket
template <int DT> constexpr uint32_t kStage =
    2048 / sizeof(typename Store<DT>::T) < 1024 ? 2048 / sizeof(typename Store<DT>::T) : 1024;

template <int DT, bool ACC64, bool ADD_OLD, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 5)
k_pr_gather(const uint64_t *__restrict__ in_off, const uint32_t *__restrict__ in_adj,
            const typename Store<DT>::T *__restrict__ contrib, uint32_t n, float *y_f32,
            double *y_f64, PrState *st, float scale_inv_arg, HeavyRows H,
            typename std::conditional<ACC64, double, float>::type *partial, unsigned int *ticket, int stage) {
    using S = Store<DT>;
    using Acc = typename std::conditional<ACC64, double, float>::type;
    constexpr int U = 4;
    constexpr uint32_t CAP = kStage<DT>;
    __shared__ typename S::T sbuf[BLOCK / 32][CAP];
    if (pr_idle(st, stage)) return;
    const float sinv = st ? st->scale_inv : scale_inv_arg;
    const uint32_t lane = threadIdx.x & 31u;
    typename S::T *buf = sbuf[threadIdx.x >> 5];
    const uint32_t nw = (gridDim.x * BLOCK) >> 5, gw = (blockIdx.x * BLOCK + threadIdx.x) >> 5;
    const uint64_t oend = in_off[n];
    double ysum = 0;
    // offsets of the word's row, loaded one word ahead
    auto bounds = [&](uint32_t w, uint64_t &b, uint64_t &e) {
        const uint32_t d = (w << 5) + lane;
        b = e = oend;
        if (d < n) {
            b = in_off[d];
            e = in_off[d + 1];
        }
    };
    // tickets: kChunkGroup chunks each, then the light ranges
    const uint64_t ngroups = (H.nchunks + kChunkGroup - 1) / kChunkGroup;
    uint64_t t = gw, next = 0;
    for (; t < ngroups + H.ncut; t = __shfl_sync(FULL, next, 0)) {
        if (lane == 0) next = (uint64_t)nw + atomicAdd(ticket, 1u);
        if (t < ngroups) {
            const uint64_t chi = min((t + 1) * kChunkGroup, H.nchunks);
            for (uint64_t c = t * kChunkGroup; c < chi; ++c) {
                const uint32_t lo = H.crow[c];  // heavy row owning chunk c
                const uint32_t v = H.v[lo];
                const uint64_t re = in_off[v + 1];
                const uint64_t e0 = in_off[v] + (c - H.first[lo]) * H.CH;
                const Acc part = dev::warp_sum(pr_chunk_sum<DT, Acc>(in_adj, contrib, e0, min(e0 + H.CH, re), lane));
                if (lane == 0) partial[c] = part;
            }
            continue;
        }
        uint32_t w = H.light_cut[t - ngroups];
        const uint32_t whi = H.light_cut[t - ngroups + 1];
        uint64_t beg = 0, end = 0, nbeg = 0, nend = 0;
        if (w < whi) bounds(w, nbeg, nend);
        for (; w < whi; ++w) {
            const uint32_t d = (w << 5) + lane;
            const bool valid = d < n;
            beg = nbeg;
            end = nend;
            if (w + 1 < whi) bounds(w + 1, nbeg, nend);
            const bool heavy = end - beg > (uint64_t)H.T;
            unsigned gaps = __ballot_sync(FULL, heavy);
            // the word's light edges as one list: this row's are [excl, excl + deg)
            // (32 bits: H.T is at most kHeavyDegMax)
            const uint32_t deg = heavy ? 0u : (uint32_t)(end - beg);
            uint32_t stop = deg;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, stop, o);
                if (lane >= (uint32_t)o) stop += t;
            }
            const uint32_t total = __shfl_sync(FULL, stop, 31);
            const uint32_t excl = stop - deg;
            const uint32_t *first = in_adj + __shfl_sync(FULL, beg, 0);  // of the list's current run
            Acc acc = 0;
            for (uint32_t base = 0; base < total; base += CAP) {
                const uint32_t upto = min(base + CAP, total);
                for (uint32_t at = base; at < upto;) {  // runs without a gap
                    uint32_t run = upto;
                    while (gaps) {
                        const int j = __ffs(gaps) - 1;
                        const uint32_t where = __shfl_sync(FULL, excl, j);
                        if (where > at) {
                            run = min(run, where);
                            break;
                        }
                        first += __shfl_sync(FULL, end - beg, j);
                        gaps &= gaps - 1;
                    }
                    uint32_t id[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const uint32_t p = at + 32 * u + lane;
                        id[u] = p < run ? __ldcs(first + p) : 0u;
                    }
                    while (at < run) {
                        uint32_t nx[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const uint32_t p = at + 32 * (U + u) + lane;
                            nx[u] = p < run ? __ldcs(first + p) : 0u;
                        }
                        typename S::T val[U];
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            if (at + 32 * u + lane < run) val[u] = contrib[id[u]];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const uint32_t p = at + 32 * u + lane;
                            if (p < run) buf[p - base] = val[u];
                            id[u] = nx[u];
                        }
                        at += 32 * U;
                    }
                    at = run;
                }
                __syncwarp();
                // this row's part of the stage, [s, e) of buf
                const uint32_t s = excl > base ? min(excl - base, CAP) : 0u;
                const uint32_t e = stop > base ? min(stop - base, CAP) : 0u;
                // the rows of this stage, [r0, r1], by 32, 16, ... 1 lanes each
                const unsigned rows = __ballot_sync(FULL, e > s);
                const uint32_t r0 = __ffs(rows) - 1, r1 = 31 - __clz(rows);
                const uint32_t lg = r1 > r0 ? __clz(r1 - r0) - 27 : 5;  // log2 of the lanes per row
                const uint32_t q = r0 + (lane >> lg);
                const uint32_t sq = __shfl_sync(FULL, s, q & 31u), eq = __shfl_sync(FULL, e, q & 31u);
                const uint32_t most = max(16u << lg, 64u);  // a longer part is summed by the whole warp
                Acc part = 0;
                if (q <= r1 && eq - sq <= most)
                    for (uint32_t i = sq + (lane & ((1u << lg) - 1u)); i < eq; i += 1u << lg) part += (Acc)S::dec(buf[i]);
                for (uint32_t o = (1u << lg) >> 1; o; o >>= 1) part += __shfl_xor_sync(FULL, part, o);
                part = __shfl_sync(FULL, part, ((lane - r0) << lg) & 31u);
                const bool wide = e > s + most;
                if (e > s && !wide) acc += part;
                unsigned pend = __ballot_sync(FULL, wide);
                while (pend) {
                    const int j = __ffs(pend) - 1;
                    pend &= pend - 1;
                    const uint32_t sj = __shfl_sync(FULL, s, j), ej = __shfl_sync(FULL, e, j);
                    part = 0;
                    for (uint32_t i = sj + lane; i < ej; i += 32) part += (Acc)S::dec(buf[i]);
                    part = dev::warp_sum(part);
                    if ((int)lane == j) acc += part;
                }
                __syncwarp();
            }
            if (valid && !heavy) ysum += pr_store_row<DT, ADD_OLD>(y_f32, y_f64, d, acc, sinv);
        }
    }
    if (st) {
        ysum = dev::block_sum<double, BLOCK>(ysum);
        if (threadIdx.x == 0) atomicAdd(&st->s1, ysum);
    }
}

// Heavy row totals from their chunks' partial sums, in a fixed order: a lane
// per row, rows of more than 8 chunks by the whole warp (the largest hub of
// R-MAT 24 has 1400 chunks, a chain of as many additions for one thread).
template <int DT, bool ACC64, bool ADD_OLD, int BLOCK>
__global__ void __launch_bounds__(BLOCK)
k_pr_heavy_finalize(HeavyRows H, const typename std::conditional<ACC64, double, float>::type *partial,
                    float *y_f32, double *y_f64, PrState *st, float scale_inv_arg, int stage) {
    using Acc = typename std::conditional<ACC64, double, float>::type;
    if (pr_idle(st, stage)) return;
    const float sinv = st ? st->scale_inv : scale_inv_arg;
    const uint32_t lane = threadIdx.x & 31u;
    double ysum = 0;
    for (uint32_t h0 = blockIdx.x * BLOCK; h0 < H.nheavy; h0 += gridDim.x * BLOCK) {
        const uint32_t h = h0 + threadIdx.x;
        const bool have = h < H.nheavy;
        const uint64_t c0 = have ? H.first[h] : 0ull, c1 = have ? H.first[h + 1] : 0ull;
        const bool wide = c1 - c0 > 8;
        Acc acc = 0;
        if (!wide)
            for (uint64_t c = c0; c < c1; ++c) acc += partial[c];
        unsigned pend = __ballot_sync(FULL, wide);
        while (pend) {
            const int j = __ffs(pend) - 1;
            pend &= pend - 1;
            const uint64_t b = __shfl_sync(FULL, c0, j), e = __shfl_sync(FULL, c1, j);
            Acc part = 0;
            for (uint64_t c = b + lane; c < e; c += 32) part += partial[c];
            part = dev::warp_sum(part);
            if ((int)lane == j) acc = part;
        }
        if (have) ysum += pr_store_row<DT, ADD_OLD>(y_f32, y_f64, H.v[h], acc, sinv);
    }
    if (st) {
        ysum = dev::block_sum<double, BLOCK>(ysum);
        if (threadIdx.x == 0) atomicAdd(&st->s1, ysum);
    }
}

// End of an iteration (one thread): record the residual, test it, next
// stage, scales.  The sums come from other CTAs' atomics: read through L2.
__device__ __forceinline__ void pr_finish(PrState *st, int dt) {
    st->reencode = 0;
    const int it = st->iters;
    const double delta = __ldcg(&st->delta);
    if (st->avg_from >= 0 && it >= st->avg_from) st->avg_n++;
    if (it < GG_MAX_ITERS) st->deltas[it] = delta;
    st->iters = it + 1;
    if (st->nstages > 1) dt = st->stage_dt[st->stage];
    if (st->stage + 1 < st->nstages && !(delta > st->stage_tol[st->stage])) {
        // next stage: its re-encode kernels rewrite the contributions from x
        st->stage++;
        st->reencode = 1;
        if (st->iters >= st->maxiter) st->done = 1;
    } else {
        if (st->iters >= st->maxiter || !(delta > st->tol)) st->done = 1;
        st->scale_inv = 1.0f / st->scale;               // decode of what the update just wrote
        st->scale = scale_for(dt, __ldcg(&st->cmax));  // next encode
    }
    st->s1 = 0;
    st->delta = 0;
    st->cmax = 0.0f;
    st->updated = 0;
}

// Staged runs: the iteration ends after every stage's update kernel.
__global__ void k_pr_finish(PrState *st, int dt) {
    if (st->done) st->reencode = 0;
    else pr_finish(st, dt);
}

// With `last`, the last CTA to finish ends the iteration (one launch fewer).
// One thread also zeroes the next gather's ticket counter.
template <int DT, int BLOCK>
__global__ void __launch_bounds__(BLOCK)
k_pr_update(const XT<DT> *__restrict__ y, XT<DT> *__restrict__ x, typename Store<DT>::T *contrib,
            const uint64_t *__restrict__ off, uint32_t n, float damp, double damp64, int renorm_f32, PrState *st,
            int stage, unsigned int *ticket, bool last, float *acc = nullptr) {
    using S = Store<DT>;
    if (pr_idle(st, stage)) return;
    const int it = st->iters;
    const bool sr = DT == GG_BF16 && st->sr;
    const bool accum = acc && it >= st->avg_from;
    const double s1 = st->s1;
    const double w = (1.0 - s1) / (double)n;
    const double s2 = s1 + (double)n * w;
    const float wf32 = 1.0f / (float)s2;
    const double wf64 = 1.0 / s2;
    const float enc_scale = st->scale;
    double dl = 0;
    float cm = 0.0f;
    const uint32_t stride = gridDim.x * BLOCK;
    if constexpr (DT == GG_F64) {
        // all double: y += w, renormalise by 1/s, contrib = d * x / deg
        for (uint32_t v = blockIdx.x * BLOCK + threadIdx.x; v < n; v += stride) {
            const double yv = (y[v] + w) * wf64;
            dl += fabs(x[v] - yv);
            x[v] = yv;
            const uint64_t deg = off[v + 1] - off[v];
            contrib[v] = per_degree(damp64 * yv, deg);
        }
        (void)wf32;
        (void)enc_scale;
    } else
    for (uint32_t v = blockIdx.x * BLOCK + threadIdx.x; v < n; v += stride) {
        float yv = (float)((double)y[v] + w);
        yv = renorm_f32 ? yv * wf32 : (float)((double)yv * wf64);
        const float xv = x[v];
        dl += (double)fabsf(xv - yv);
        x[v] = yv;
        const uint64_t deg = off[v + 1] - off[v];
        const float c = per_degree(damp * yv, deg);
        if constexpr (DT == GG_BF16) {
            contrib[v] = sr ? bf16_stochastic(c, v, (uint32_t)it) : S::enc(c);
            if (accum) acc[v] += yv;
        } else {
            contrib[v] = S::enc(scaled_format(DT) ? c * enc_scale : c);
        }
        if (deg && c > cm) cm = c;
    }
    dl = dev::block_sum<double, BLOCK>(dl);
    // max of non-negative floats: integer order of the bit patterns
    __shared__ float sh[BLOCK / 32];
    for (int o = 16; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(FULL, cm, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = cm;
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = 0.0f;
        for (int i = 0; i < BLOCK / 32; ++i) b = fmaxf(b, sh[i]);
        atomicAdd(&st->delta, dl);
        atomicMax((int *)&st->cmax, __float_as_int(b));
        if (blockIdx.x == 0) *ticket = 0;
        if (last) {
            __threadfence();  // this CTA's sums before its arrival
            if (atomicAdd(&st->updated, 1u) == gridDim.x - 1) {
                __threadfence();
                pr_finish(st, DT);
            }
        }
    }
}

// Tail averaging: the ranks become the mean of the accumulated iterations.
__global__ void k_pr_average(float *x, const float *acc, uint32_t n, const PrState *st) {
    const int k = st->avg_n;
    if (k <= 0) return;
    const float inv = 1.0f / (float)k;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) x[v] = acc[v] * inv;
}

// Scale of the contributions about to be encoded, from the max found by the
// pass-0 kernel (one thread, between the two passes: every CTA of pass 1
// then reads the same value).  stage >= 0: only when that stage re-encodes.
__global__ void k_pr_setscale(PrState *st, int dt, int stage) {
    if (stage >= 0 && (st->done || !st->reencode || st->stage != stage)) return;
    const float sc = scale_for(dt, st->cmax);
    st->scale = sc;
    st->scale_inv = 1.0f / sc;
    st->cmax = 0.0f;
}

// A new stage's contributions from the current ranks: pass 0 finds the
// max, pass 1 encodes with st->scale.
template <int DT, int BLOCK>
__global__ void k_pr_reencode(const float *x, typename Store<DT>::T *contrib, const uint64_t *off, uint32_t n,
                              float damp, PrState *st, int stage, int pass) {
    using S = Store<DT>;
    if (st->done || !st->reencode || st->stage != stage) return;
    float cm = 0.0f;
    const float scale = st->scale;
    const uint32_t stride = gridDim.x * BLOCK;
    for (uint32_t v = blockIdx.x * BLOCK + threadIdx.x; v < n; v += stride) {
        const uint64_t deg = off[v + 1] - off[v];
        const float c = per_degree(damp * x[v], deg);
        if (pass == 0) {
            if (deg && c > cm) cm = c;
        } else {
            contrib[v] = S::enc(scaled_format(DT) ? c * scale : c);
        }
    }
    if (pass == 0) {
        for (int o = 16; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(FULL, cm, o));
        if ((threadIdx.x & 31) == 0) atomicMax((int *)&st->cmax, __float_as_int(cm));
    }
}

// Initial x = 1/n, contrib = d*x/deg (PRv.C:155-182); first pass finds the max.
template <int DT, int BLOCK>
__global__ void k_pr_init(XT<DT> *x, typename Store<DT>::T *contrib, const uint64_t *off, uint32_t n,
                          float damp, double damp64, PrState *st, int pass) {
    using S = Store<DT>;
    const float x0 = 1.0f / (float)n;
    float cm = 0.0f;
    const uint32_t stride = gridDim.x * BLOCK;
    if constexpr (DT == GG_F64) {
        if (pass == 1)
            for (uint32_t v = blockIdx.x * BLOCK + threadIdx.x; v < n; v += stride) {
                const double xd = 1.0 / (double)n;
                x[v] = xd;
                contrib[v] = per_degree(damp64 * xd, off[v + 1] - off[v]);
            }
        if (pass == 1 && blockIdx.x == 0 && threadIdx.x == 0) {
            st->scale = 1.0f;
            st->scale_inv = 1.0f;
            st->cmax = 0.0f;
        }
        return;
    }
    const float scale = pass == 1 ? st->scale : 1.0f;  // set by k_pr_setscale between the passes
    for (uint32_t v = blockIdx.x * BLOCK + threadIdx.x; v < n; v += stride) {
        const uint64_t deg = off[v + 1] - off[v];
        const float c = per_degree(damp * x0, deg);
        if (pass == 0) {
            if (deg && c > cm) cm = c;
        } else {
            x[v] = x0;
            contrib[v] = S::enc(scaled_format(DT) ? c * scale : c);
        }
    }
    if (pass == 0) {
        for (int o = 16; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(FULL, cm, o));
        if ((threadIdx.x & 31) == 0) atomicMax((int *)&st->cmax, __float_as_int(cm));
    }
}

constexpr int kBlock = 256;

static unsigned pr_grid(gg_ctx *ctx, uint64_t work) {
    uint64_t b = (work + kBlock - 1) / kBlock;
    uint64_t cap = (uint64_t)ctx->sm_count * tuning().pr_blocks_per_sm;
    if (b > cap) b = cap;
    return (unsigned)(b ? b : 1);
}

// the gather's ticket counter: the entry after the chunks' partial sums, 0
// when a gather starts (zeroed before a run, then by each update)
static unsigned int *pr_ticket(gg_graph *g, void *partial) {
    return (unsigned int *)((char *)partial + g->heavy.nchunks * 8);
}

// gather of one iteration / one API call: all rows, then heavy totals
template <int DT, bool ACC64, bool ADD_OLD>
static gg_status gather_launch(gg_graph *g, const typename Store<DT>::T *contrib, float *yf,
                               double *yd, PrState *st, float sinv, void *partial, int stage = -1) {
    gg_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    using Acc = typename std::conditional<ACC64, double, float>::type;
    const HeavyRows &H = g->heavy;
    const uint64_t warps = std::max<uint64_t>(((uint64_t)g->n + 31) / 32, H.nchunks);
    uint64_t blocks = (warps * 32 + 255) / 256;
    // tickets balance the load, so one CTA for every place on the SMs
    const uint64_t cap = (uint64_t)ctx->sm_count *
                         std::min(resident_ctas((const void *)k_pr_gather<DT, ACC64, ADD_OLD, 256>, 256),
                                  tuning().pr_blocks_per_sm);
    if (blocks > cap) blocks = cap;
    k_pr_gather<DT, ACC64, ADD_OLD, 256><<<(unsigned)(blocks ? blocks : 1), 256, 0, s>>>(
        g->in_off, g->in_adj, contrib, g->n, yf, yd, st, sinv, H, (Acc *)partial, pr_ticket(g, partial), stage);
    GG_LAUNCHED(ctx);
    if (H.nchunks) {
        const uint64_t fb = std::min<uint64_t>((H.nheavy + 255) / 256, cap);
        k_pr_heavy_finalize<DT, ACC64, ADD_OLD, 256><<<(unsigned)fb, 256, 0, s>>>(H, (const Acc *)partial, yf, yd,
                                                                                 st, sinv, stage);
        GG_LAUNCHED(ctx);
    }
    return GG_OK;
}

// ---------------------------------------------------------------------------
// The gather by blocks of sources (gg_prplan.cuh)
// ---------------------------------------------------------------------------
// k_pr_gather cannot go below one sector from L2 per gathered value.  Here a
// value is read from shared memory, written and read again in whole sectors
// and placed through shared memory: 12.5 bytes of DRAM traffic an edge with
// 4-byte values, 8.5 with 16-bit ones (0.98 and 0.68 ms for 520 M edges).
// Measured per iteration, the rest of it included, by rows -> by blocks:
// R-MAT 24 FP32 with double sums 2.02 -> 1.66 ms, directed ER 2^24 x 32 BF16
// 2.13 -> 1.42, ER 4 M x 64 FP32 1.06 -> 0.74, R-MAT 22 BF16 0.46 -> 0.36.
// Of it k_pr_values 0.60 ms and k_pr_bins 0.94 ms (R-MAT 24), 1.3 and 1.8
// times their DRAM time: the pipes of L1 and shared memory, whose accesses
// fall into some 3 banks deep where the ids lie at random, are busy for 69 %
// (86 % with 16-bit values) and 63 % of it, the issue slots of the second for
// 58 %, and its loads, sums and stores take turns with two CTAs per SM to
// overlap them.  Bins of 16384 edges (3 CTAs) 2.4 ms: tiles, and with them the runs
// read from DRAM, get shorter.  The values written by the first kernel in
// bin order instead, so that the second reads them in one piece: 1.9 ms, and
// 2.0 for BF16 (runs of half sectors).
constexpr int kValBlock = 1024;
// chunks that a thread of k_pr_values has in flight, and CTAs per SM (a block
// of float contributions takes 128 KiB, one of 16-bit ones 64)
template <typename T> constexpr int kValFlight = sizeof(T) == 4 ? 4 : 1;
template <typename T> constexpr int kValCtas = sizeof(T) == 4 ? 1 : 2;

// 8 values of a chunk, moved by one access of 16 or 32 bytes (in two halves,
// the lanes of a warp would each touch half of a sector, twice)
template <typename T> struct Val8 {
    T v[8];
};
__device__ __forceinline__ void load8(const float *p, Val8<float> &x) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(x.v[0]), "=f"(x.v[1]), "=f"(x.v[2]), "=f"(x.v[3]), "=f"(x.v[4]), "=f"(x.v[5]), "=f"(x.v[6]), "=f"(x.v[7])
        : "l"(p));
}
__device__ __forceinline__ void store8(float *p, const Val8<float> &x) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(x.v[0]), "f"(x.v[1]),
                 "f"(x.v[2]), "f"(x.v[3]), "f"(x.v[4]), "f"(x.v[5]), "f"(x.v[6]), "f"(x.v[7])
                 : "memory");
}
__device__ __forceinline__ void load8(const uint16_t *p, Val8<uint16_t> &x) {
    const uint4 q = __ldg((const uint4 *)p);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        x.v[2 * k] = (uint16_t)(w[k] & 0xFFFFu);
        x.v[2 * k + 1] = (uint16_t)(w[k] >> 16);
    }
}
__device__ __forceinline__ void store8(uint16_t *p, const Val8<uint16_t> &x) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = x.v[2 * k] | (uint32_t)x.v[2 * k + 1] << 16;
    *(uint4 *)p = make_uint4(w[0], w[1], w[2], w[3]);
}

// vals[slot] = the contribution of the slot's source, read from the block's
// contributions in shared memory.
template <typename T>
__global__ void __launch_bounds__(kValBlock, kValCtas<T>)
k_pr_values(const uint16_t *__restrict__ src, const uint4 *__restrict__ segs, const uint32_t *__restrict__ part_seg,
            const T *__restrict__ contrib, uint32_t n, T *__restrict__ vals, const PrState *st) {
    extern __shared__ __align__(16) uint8_t smem[];
    T *blk = (T *)smem;
    if (pr_idle(st, -1)) return;
    const uint32_t hi = part_seg[blockIdx.x + 1];
    for (uint32_t i = part_seg[blockIdx.x]; i < hi; ++i) {
        const uint4 seg = segs[i];
        const uint32_t v0 = seg.x << kBlkSrcLog, len = min(n - v0, kBlkSrc);
        constexpr uint32_t W = 16 / sizeof(T);
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < len / W; j += kValBlock) {
            const uint4 q = __ldg((const uint4 *)(contrib + v0) + j);
            const T *x = (const T *)&q;
#pragma unroll
            for (uint32_t k = 0; k < W; ++k) blk[blk_slot(j * W + k)] = x[k];
        }
        for (uint32_t j = len / W * W + threadIdx.x; j < len; j += kValBlock) blk[blk_slot(j)] = contrib[v0 + j];
        __syncthreads();
        constexpr int U = kValFlight<T>;
        uint4 id[U];
        auto ids = [&](uint64_t c) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (c + u * kValBlock < seg.z) id[u] = __ldcs((const uint4 *)src + c + u * kValBlock);
        };
        uint64_t c = (uint64_t)seg.y + threadIdx.x;
        ids(c);
        for (; c < seg.z; c += kValBlock * U) {
            uint4 a[U];
#pragma unroll
            for (int u = 0; u < U; ++u) a[u] = id[u];
            ids(c + kValBlock * U);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (c + u * kValBlock >= seg.z) break;
                const uint32_t w[4] = {a[u].x, a[u].y, a[u].z, a[u].w};
                Val8<T> o;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    o.v[2 * k] = blk[w[k] & 0xFFFFu];
                    o.v[2 * k + 1] = blk[w[k] >> 16];
                }
                store8(vals + (c + u * kValBlock) * 8, o);
            }
        }
    }
}

// The row sums of a bin: its values put in the edges' places in shared
// memory, then 32 edges per thread, cut where rows end; what a thread's
// first row has in the threads before comes from a segmented scan.  A bin's
// part of a row that began before it goes to parts[2 b], its edges after the
// last end of a row to parts[2 b + 1].
template <int DT, bool ACC64>
__global__ void __launch_bounds__(kBinThreads, 2)
k_pr_bins(PrPlan P, const typename Store<DT>::T *__restrict__ vals, const uint32_t *__restrict__ list, uint64_t m,
          float *y_f32, PrState *st, typename std::conditional<ACC64, double, float>::type *parts) {
    using S = Store<DT>;
    using T = typename S::T;
    using Acc = typename std::conditional<ACC64, double, float>::type;
    constexpr int WARPS = kBinThreads / 32;
    extern __shared__ __align__(16) uint8_t smem[];
    float *buf = (float *)smem;  // decoded values; in their stead, later, the sums of the thread's rows
    __shared__ uint32_t s_ends[WARPS];
    __shared__ Acc s_sum[WARPS];
    __shared__ double s_y[WARPS];
    __shared__ bool s_cut[WARPS];
    const uint32_t b = blockIdx.x, t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    // (all that does not depend on another load first)
    const uint32_t hi = __ldg(P.bin_ptr + b + 1);
    uint32_t c = __ldg(P.bin_ptr + b) + t;
    const uint32_t bits = __ldg(P.ends + (uint64_t)b * kBinThreads + t);  // the thread's edges that end rows
    const uint32_t *rows = list + __ldg(P.bin_end + b);                  // the rows that end in the bin
    const bool head = b && !(__ldg(P.ends + (uint64_t)b * kBinThreads - 1) >> 31);
    if (pr_idle(st, -1)) return;
    const float sinv = st->scale_inv;
    uint32_t at = c < hi ? __ldcs(P.ptr + c) : 0u;
    uint32_t rank = __popc(bits);  // of the thread's first row end, from here on
    const uint32_t nends = rank;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(FULL, rank, o);
        if (lane >= (uint32_t)o) rank += x;
    }
    if (lane == 31) s_ends[warp] = rank;
    rank -= nends;
    while (c < hi) {
        const uint4 ps = __ldcs((const uint4 *)P.pos + at);
        Val8<T> v;
        load8(vals + (uint64_t)at * 8, v);
        c += kBinThreads;
        if (c < hi) at = __ldcs(P.ptr + c);
        const uint32_t w[4] = {ps.x, ps.y, ps.z, ps.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            buf[w[k] & 0xFFFFu] = S::dec(v.v[2 * k]);
            buf[w[k] >> 16] = S::dec(v.v[2 * k + 1]);
        }
    }
    const uint32_t len = (uint32_t)min(m - (uint64_t)b * kBinEdges, (uint64_t)kBinEdges);
    for (uint32_t p = len + t; p < kBinEdges; p += kBinThreads) buf[bin_slot(p)] = 0.0f;  // (the last bin)
    __syncthreads();
    rank += dev::warp_sum(lane < warp ? s_ends[lane] : 0u);
    // the thread's first two rows, loaded beside the sums
    const uint32_t d0 = nends ? __ldg(rows + rank) : 0u, d1 = nends > 1 ? __ldg(rows + rank + 1) : 0u;
    const uint32_t own = bin_slot(t * 32) * 4, first = bits & (0u - bits);
    auto slot = [&](uint32_t i4) -> float & { return *(float *)(smem + (own ^ i4)); };
    Acc acc = 0, lead = 0;
    uint32_t to = 0;  // 4 times the row ends seen
#pragma unroll
    for (uint32_t i = 0; i < 32; ++i) {
        acc += (Acc)slot(i * 4);
        const bool end = bits >> i & 1u;
        if (end) slot(to) = pr_value<DT>(acc, sinv);
        lead = first >> i & 1u ? acc : lead;
        to += end ? 4u : 0u;
        acc = end ? Acc(0) : acc;
    }
    // segmented scan of the threads' ends (acc, bits != 0: cut)
    Acc v = acc;
    bool cut = bits != 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Acc x = __shfl_up_sync(FULL, v, o);
        const bool f = __shfl_up_sync(FULL, (int)cut, o);
        if (lane >= (uint32_t)o) {
            if (!cut) v += x;
            cut |= f;
        }
    }
    if (lane == 31) {
        s_sum[warp] = v;
        s_cut[warp] = cut;
    }
    __syncthreads();
    Acc carry = 0;  // of the warps before
    {
        // those from the last cut on, in their order
        const uint32_t cuts = __ballot_sync(FULL, lane < warp && s_cut[lane]);
        const uint32_t from = cuts ? 31 - __clz(cuts) : 0u;
        for (uint32_t w = from; w < warp; ++w) carry += s_sum[w];
    }
    const Acc x = __shfl_up_sync(FULL, v, 1);
    const bool f = __shfl_up_sync(FULL, (int)cut, 1);
    double ysum = 0;
    if (nends) {
        lead += lane == 0 ? carry : f ? x : carry + x;
        if (rank == 0 && head) {
            parts[2 * (uint64_t)b] = lead;
        } else {
            const float y = pr_value<DT>(lead, sinv);
            y_f32[d0] = y;
            ysum = (double)y;
        }
        uint32_t d = d1;
        for (uint32_t j = 1; j < nends; ++j) {
            const uint32_t dn = j + 1 < nends ? __ldg(rows + rank + j + 1) : 0u;
            const float y = slot(j * 4);
            y_f32[d] = y;
            ysum += (double)y;
            d = dn;
        }
    }
    if (t == kBinThreads - 1) parts[2 * (uint64_t)b + 1] = cut ? v : carry + v;
    ysum = dev::warp_sum(ysum);
    if (lane == 0) s_y[warp] = ysum;
    __syncthreads();
    if (warp == 0) {
        ysum = dev::warp_sum(lane < WARPS ? s_y[lane] : 0.0);
        if (lane == 0) atomicAdd(&st->s1, ysum);
    }
}

// Totals of the rows that end in a later bin than they begin in: a lane per
// bin in which such a row ends, rows over more than kSpanLane bins by the warp,
// 128 bins at a time from their last one back to the one they begin in (a star
// of 2^25 vertices, a row over 1365 bins, all of it by one lane: 1.03 ms an
// iteration with FP32 and 0.88 with BF16 -> 0.81 and 0.73).
constexpr uint32_t kSpanLane = 4;

template <int DT, bool ACC64>
__global__ void __launch_bounds__(256)
k_pr_spans(PrPlan P, const uint32_t *__restrict__ list, float *y_f32, PrState *st,
           const typename std::conditional<ACC64, double, float>::type *parts) {
    using Acc = typename std::conditional<ACC64, double, float>::type;
    if (pr_idle(st, -1)) return;
    const uint32_t b = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31u;
    const bool need =
        b && b < P.nbin && P.bin_end[b + 1] > P.bin_end[b] && !(P.ends[(uint64_t)b * kBinThreads - 1] >> 31);
    const auto begins = [&](uint32_t x) { return x == 0 || P.bin_end[x + 1] != P.bin_end[x]; };
    Acc acc = 0;
    bool wide = false;
    if (need) {
        uint32_t x = b - 1;
        while (b - x < kSpanLane && !begins(x)) --x;
        wide = !begins(x);
        if (!wide)
            for (; x < b; ++x) acc += parts[2 * (uint64_t)x + 1];
    }
    for (unsigned pend = __ballot_sync(FULL, wide); pend; pend &= pend - 1) {
        const int j = __ffs(pend) - 1;
        Acc part = 0;
        bool on = true;
        for (int64_t at = (int64_t)__shfl_sync(FULL, b, j) - 1; on; at -= 128) {
            Acc v[4];
            bool first[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int64_t x = at - 32 * u - lane;
                first[u] = x < 0 || begins((uint32_t)x);
                v[u] = x < 0 ? Acc(0) : parts[2 * x + 1];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const unsigned f = __ballot_sync(FULL, first[u]);
                // up to the bin that the row begins in, and none of the next 32 after it
                if (on && (!f || (int)lane < __ffs(f))) part += v[u];
                on = on && !f;
            }
        }
        part = dev::warp_sum(part);
        if ((int)lane == j) acc = part;
    }
    double ysum = 0;
    if (need) {
        acc += parts[2 * (uint64_t)b];
        ysum = pr_store_row<DT, false>(y_f32, nullptr, list[P.bin_end[b]], acc, st->scale_inv);
    }
    ysum = dev::block_sum<double, 256>(ysum);
    if (threadIdx.x == 0 && ysum != 0) atomicAdd(&st->s1, ysum);
}

template <int DT, bool ACC64>
static gg_status blocked_launch(gg_graph *g, const PrPlan &P, const typename Store<DT>::T *contrib, float *y,
                                PrState *st, void *vals, void *parts) {
    gg_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    using T = typename Store<DT>::T;
    using Acc = typename std::conditional<ACC64, double, float>::type;
    const size_t sv = (size_t)kBlkSrc * sizeof(T), sb = (size_t)(kBinEdges + 8) * 4;
    GG_CUDA(ctx, cudaFuncSetAttribute(k_pr_values<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sv));
    GG_CUDA(ctx, cudaFuncSetAttribute(k_pr_bins<DT, ACC64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sb));
    k_pr_values<T><<<P.nparts, kValBlock, sv, s>>>(P.src, P.segs, P.part_seg, contrib, g->n, (T *)vals, st);
    GG_LAUNCHED(ctx);
    k_pr_bins<DT, ACC64><<<P.nbin, kBinThreads, sb, s>>>(P, (const T *)vals, g->nonisolated, g->m, y, st, (Acc *)parts);
    GG_LAUNCHED(ctx);
    k_pr_spans<DT, ACC64><<<(P.nbin + 255) / 256, 256, 0, s>>>(P, g->nonisolated, y, st, (const Acc *)parts);
    GG_LAUNCHED(ctx);
    return GG_OK;
}

// Damping of the FP64 variant: the shortest decimal that rounds to the float
// parameter (0.85f -> 0.85), as the double-precision reference uses it.
static double damping_f64(float d) {
    char buf[32];
    for (int prec = 1; prec <= 9; ++prec) {
        std::snprintf(buf, sizeof(buf), "%.*g", prec, (double)d);
        const double v = std::strtod(buf, nullptr);
        if ((float)v == d) return v;
    }
    return (double)d;
}

template <int DT>
static gg_status pr_run(gg_graph *g, const gg_pr_params *p, XT<DT> *x, XT<DT> *y, void *contrib,
                        PrState *st, void *partial, const PrPlan *plan, void *vals, float *acc = nullptr) {
    gg_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    using T = typename Store<DT>::T;
    const uint32_t n = g->n;
    // (the blocked gather stores no row without in-edges)
    if (plan) GG_CUDA(ctx, cudaMemsetAsync(y, 0, (size_t)n * 4, s));
    void *parts = plan ? (char *)vals + plan->chunks * 8 * sizeof(T) : nullptr;
    const unsigned gv = pr_grid(ctx, n);
    const double d64 = damping_f64(p->damping);
    k_pr_init<DT, kBlock><<<gv, kBlock, 0, s>>>(x, (T *)contrib, g->off, n, p->damping, d64, st, 0);
    GG_LAUNCHED(ctx);
    k_pr_setscale<<<1, 1, 0, s>>>(st, DT, -1);
    GG_LAUNCHED(ctx);
    k_pr_init<DT, kBlock><<<gv, kBlock, 0, s>>>(x, (T *)contrib, g->off, n, p->damping, d64, st, 1);
    GG_LAUNCHED(ctx);
    float *yf = DT == GG_F64 ? nullptr : (float *)y;
    double *yd = DT == GG_F64 ? (double *)y : nullptr;
    for (int it = 0; it < p->maxiter; ++it) {
        if (plan) {
            if constexpr (DT != GG_F64 && DT != GG_FP8E4M3) {
                if (p->accum_f64)
                    GG_CHECK((blocked_launch<DT, true>(g, *plan, (const T *)contrib, yf, st, vals, parts)));
                else GG_CHECK((blocked_launch<DT, false>(g, *plan, (const T *)contrib, yf, st, vals, parts)));
            }
        } else if (p->accum_f64 || DT == GG_F64)
            GG_CHECK((gather_launch<DT, true, false>(g, (const T *)contrib, yf, yd, st, 1.0f, partial)));
        else
            GG_CHECK((gather_launch<DT, false, false>(g, (const T *)contrib, yf, yd, st, 1.0f, partial)));
        k_pr_update<DT, kBlock><<<gv, kBlock, 0, s>>>(y, x, (T *)contrib, g->off, n, p->damping, d64,
                                                      p->renorm_f32, st, -1, pr_ticket(g, partial), true, acc);
        GG_LAUNCHED(ctx);
    }
    if constexpr (DT == GG_BF16) {
        if (acc) {
            k_pr_average<<<gv, kBlock, 0, s>>>(x, acc, n, st);
            GG_LAUNCHED(ctx);
        }
    }
    return GG_OK;
}

// Staged runs (PR_vary.C:652-757, e.g. VARIANT 4620 = run_prec_46 with
// customfp<6,10> contributions until the residual is below 1e-3, then
// run_prec_20 with FP32 contributions and double sums until 1e-7): every
// iteration launches each stage's kernels and those of inactive stages return
// at once, so the switch is taken on the device without a host round trip.
enum { OP_GATHER, OP_UPDATE, OP_REENC0, OP_SETSCALE, OP_REENC1, OP_INIT0, OP_INIT1 };

template <int DT>
static gg_status stage_op(gg_graph *g, int op, int stage, bool acc64, const gg_pr_params *p, float *x, float *y,
                          void *contrib, PrState *st, void *partial) {
    using T = typename Store<DT>::T;
    gg_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    const unsigned gv = pr_grid(ctx, g->n);
    switch (op) {
    case OP_GATHER:
        if (acc64) return gather_launch<DT, true, false>(g, (const T *)contrib, y, nullptr, st, 1.0f, partial, stage);
        return gather_launch<DT, false, false>(g, (const T *)contrib, y, nullptr, st, 1.0f, partial, stage);
    case OP_UPDATE:
        k_pr_update<DT, kBlock><<<gv, kBlock, 0, s>>>(y, x, (T *)contrib, g->off, g->n, p->damping, 0.0,
                                                      p->renorm_f32, st, stage, pr_ticket(g, partial), false);
        break;
    case OP_REENC0:
    case OP_REENC1:
        k_pr_reencode<DT, kBlock><<<gv, kBlock, 0, s>>>(x, (T *)contrib, g->off, g->n, p->damping, st, stage,
                                                        op == OP_REENC1);
        break;
    case OP_SETSCALE: k_pr_setscale<<<1, 1, 0, s>>>(st, DT, stage); break;
    default:
        k_pr_init<DT, kBlock><<<gv, kBlock, 0, s>>>(x, (T *)contrib, g->off, g->n, p->damping, 0.0, st,
                                                    op == OP_INIT1);
        break;
    }
    GG_LAUNCHED(ctx);
    return GG_OK;
}

static gg_status stage_dispatch(int dt, gg_graph *g, int op, int stage, bool acc64, const gg_pr_params *p,
                                float *x, float *y, void *contrib, PrState *st, void *partial) {
    switch (dt) {
    case GG_F32: return stage_op<GG_F32>(g, op, stage, acc64, p, x, y, contrib, st, partial);
    case GG_BF16: return stage_op<GG_BF16>(g, op, stage, acc64, p, x, y, contrib, st, partial);
    case GG_F16: return stage_op<GG_F16>(g, op, stage, acc64, p, x, y, contrib, st, partial);
    case GG_FP8E4M3: return stage_op<GG_FP8E4M3>(g, op, stage, acc64, p, x, y, contrib, st, partial);
    case GG_CFP_6_10: return stage_op<GG_CFP_6_10>(g, op, stage, acc64, p, x, y, contrib, st, partial);
    default: return stage_op<GG_BF16_TRUNC>(g, op, stage, acc64, p, x, y, contrib, st, partial);
    }
}

static gg_status pr_run_staged(gg_graph *g, const gg_pr_params *p, float *x, float *y, void *contrib,
                               PrState *st, void *partial) {
    const int ns = p->nstages;
    const int *dt = p->stage_dtype;
    const int *acc = p->stage_accum_f64;
    GG_CHECK(stage_dispatch(dt[0], g, OP_INIT0, -1, false, p, x, y, contrib, st, partial));
    GG_CHECK(stage_dispatch(dt[0], g, OP_SETSCALE, -1, false, p, x, y, contrib, st, partial));
    GG_CHECK(stage_dispatch(dt[0], g, OP_INIT1, -1, false, p, x, y, contrib, st, partial));
    for (int it = 0; it < p->maxiter; ++it) {
        for (int k = 0; k < ns; ++k)
            GG_CHECK(stage_dispatch(dt[k], g, OP_GATHER, k, acc[k] != 0, p, x, y, contrib, st, partial));
        for (int k = 0; k < ns; ++k)
            GG_CHECK(stage_dispatch(dt[k], g, OP_UPDATE, k, false, p, x, y, contrib, st, partial));
        k_pr_finish<<<1, 1, 0, g->ctx->stream>>>(st, dt[0]);
        GG_LAUNCHED(g->ctx);
        for (int k = 1; k < ns; ++k) {
            GG_CHECK(stage_dispatch(dt[k], g, OP_REENC0, k, false, p, x, y, contrib, st, partial));
            GG_CHECK(stage_dispatch(dt[k], g, OP_SETSCALE, k, false, p, x, y, contrib, st, partial));
            GG_CHECK(stage_dispatch(dt[k], g, OP_REENC1, k, false, p, x, y, contrib, st, partial));
        }
    }
    return GG_OK;
}

// ADD_GATHER edgemap: y[d] += sum_{s in in(d), s active} dec(contrib[s]) * scale.
template <int DT>
static gg_status gather_api(gg_graph *g, const gg_emap_desc *d) {
    using T = typename Store<DT>::T;
    float *yf = d->a->t == GG_F32 ? (float *)d->a->d : nullptr;
    double *yd = d->a->t == GG_F64 ? (double *)d->a->d : nullptr;
    const float sc = d->src_scale != 0.0f ? d->src_scale : 1.0f;
    void *partial = nullptr;
    GG_CHECK(graph_scratch(g, (g->heavy.nchunks + 1) * 8, &partial));
    GG_CUDA(g->ctx, cudaMemsetAsync(pr_ticket(g, partial), 0, 8, g->ctx->stream));
    if (d->accum_f64)
        return gather_launch<DT, true, true>(g, (const T *)d->src->d, yf, yd, nullptr, sc, partial);
    return gather_launch<DT, false, true>(g, (const T *)d->src->d, yf, yd, nullptr, sc, partial);
}

// ADD_GATHER with a source frontier (APRv.C:477-487, api::filter(F, strong,
// src)): y[d] += sum over in-edges (s, d) with s in F of contrib[s].  The
// contributions of the vertices outside F are masked to zero in a scratch
// copy (one pass over n values), which the regular gather then sums: its
// light-row streaming and heavy-row chunks keep every warp busy whatever
// the degree mix.
template <typename T>
__global__ void k_mask_contrib(const T *__restrict__ contrib, const uint32_t *__restrict__ bits, uint32_t n,
                               T *__restrict__ out) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        out[v] = dev::bit_test(bits, v) ? contrib[v] : (T)0;
}

static gg_status gather_src_filtered(gg_graph *g, const gg_emap_desc *d, gg_frontier *in) {
    gg_ctx *ctx = g->ctx;
    const bool f64 = d->src->t == GG_F64;
    if (!(d->src->t == GG_F32 || (f64 && d->accum_f64)))
        return set_error(ctx, GG_ERR_UNSUPPORTED, "a source-filtered ADD_GATHER takes F32 or F64 contributions");
    GG_CHECK(frontier_ensure_bitmap(in));
    float *yf = d->a->t == GG_F32 ? (float *)d->a->d : nullptr;
    double *yd = d->a->t == GG_F64 ? (double *)d->a->d : nullptr;
    // scratch: the masked contributions, then the heavy rows' partial sums
    const size_t esz = f64 ? 8 : 4;
    const size_t cb = (((size_t)g->n + 1) * esz + 255) / 256 * 256;
    void *base = nullptr;
    GG_CHECK(graph_scratch(g, cb + (g->heavy.nchunks + 1) * 8, &base));
    void *partial = (char *)base + cb;
    GG_CUDA(ctx, cudaMemsetAsync(pr_ticket(g, partial), 0, 8, ctx->stream));
    const unsigned grid = pr_grid(ctx, g->n);
    if (f64) {
        k_mask_contrib<double><<<grid, 256, 0, ctx->stream>>>((const double *)d->src->d, in->bitmap, g->n,
                                                              (double *)base);
        GG_LAUNCHED(ctx);
        return gather_launch<GG_F64, true, true>(g, (const double *)base, yf, yd, nullptr, 1.0f, partial);
    }
    k_mask_contrib<float><<<grid, 256, 0, ctx->stream>>>((const float *)d->src->d, in->bitmap, g->n, (float *)base);
    GG_LAUNCHED(ctx);
    if (d->accum_f64) return gather_launch<GG_F32, true, true>(g, (const float *)base, yf, yd, nullptr, 1.0f, partial);
    return gather_launch<GG_F32, false, true>(g, (const float *)base, yf, yd, nullptr, 1.0f, partial);
}

gg_status pr_edgemap_gather(gg_graph *g, const gg_emap_desc *d, gg_frontier *in) {
    gg_ctx *ctx = g->ctx;
    if (!d->src || d->src->g != g) return set_error(ctx, GG_ERR_ARG, "ADD_GATHER needs a contribution property of g");
    if (d->a->t != GG_F32 && d->a->t != GG_F64) return set_error(ctx, GG_ERR_ARG, "ADD_GATHER accumulator must be F32 or F64");
    if (d->dst_filter != GG_FILTER_NONE) return set_error(ctx, GG_ERR_UNSUPPORTED, "ADD_GATHER takes no dst filter");
    if (d->src_scale != 0.0f && d->src->t != GG_FP8E4M3)
        return set_error(ctx, GG_ERR_UNSUPPORTED, "src_scale applies to FP8 contributions only");
    if (in && !in->all) return gather_src_filtered(g, d, in);
    switch (d->src->t) {
    case GG_F32: return gather_api<GG_F32>(g, d);
    case GG_BF16: return gather_api<GG_BF16>(g, d);
    case GG_F16: return gather_api<GG_F16>(g, d);
    case GG_FP8E4M3: return gather_api<GG_FP8E4M3>(g, d);
    case GG_CFP_6_10: return gather_api<GG_CFP_6_10>(g, d);
    case GG_BF16_TRUNC: return gather_api<GG_BF16_TRUNC>(g, d);
    case GG_F64:  // PR_vary VARIANT 11: double contributions, double sums
        if (!d->accum_f64) return set_error(ctx, GG_ERR_UNSUPPORTED, "double contributions take double sums");
        return gather_api<GG_F64>(g, d);
    default: return set_error(ctx, GG_ERR_UNSUPPORTED, "contribution dtype");
    }
}

}  // namespace gg

using namespace gg;

extern "C" gg_status gg_pagerank(gg_graph *g, const gg_pr_params *p, gg_prop *x, float *host_x,
                                 gg_run_stats *stats) {
    if (!g || !p) return GG_ERR_ARG;
    gg_ctx *ctx = g->ctx;
    if (p->maxiter < 0 || p->maxiter > GG_MAX_ITERS) return set_error(ctx, GG_ERR_ARG, "maxiter out of range");
    const bool staged = p->nstages > 1;
    const int dt = staged ? p->stage_dtype[0] : p->contrib_dtype;
    auto known = [](int t) {
        return t == GG_F32 || t == GG_BF16 || t == GG_F16 || t == GG_FP8E4M3 || t == GG_CFP_6_10 || t == GG_BF16_TRUNC;
    };
    if (p->nstages < 0 || p->nstages > 4) return set_error(ctx, GG_ERR_ARG, "nstages must be 0..4");
    if (staged)
        for (int k = 0; k < p->nstages; ++k)
            if (!known(p->stage_dtype[k])) return set_error(ctx, GG_ERR_UNSUPPORTED, "stage contribution dtype");
    if (!staged && !known(dt) && dt != GG_F64) return set_error(ctx, GG_ERR_UNSUPPORTED, "contribution dtype");
    if ((p->stochastic || p->average_last) && (staged || dt != GG_BF16))
        return set_error(ctx, GG_ERR_UNSUPPORTED, "stochastic rounding / tail averaging apply to BF16 runs only");
    if (p->average_last < 0) return set_error(ctx, GG_ERR_ARG, "average_last must be >= 0");
    const gg_dtype xt = dt == GG_F64 ? GG_F64 : GG_F32;
    if (x && (x->g != g || x->t != xt))
        return set_error(ctx, GG_ERR_ARG, "x must be an F32 property of g (F64 for the FP64 variant)");
    if (g->n == 0) return GG_OK;
    gg_prop *xp = x, *tmpx = nullptr;
    if (!xp) {
        GG_CHECK(gg_prop_create(g, xt, &tmpx));
        xp = tmpx;
    }
    // scratch: y (f32 / f64), contrib (up to 8 B), state
    const size_t esz = dt == GG_F64 ? 8 : 4;
    const size_t nb = (((size_t)g->n + 1) * esz + 255) / 256 * 256;
    const size_t sb = (sizeof(PrState) + 255) / 256 * 256;
    void *base = nullptr;
    const size_t ab = p->average_last > 0 ? (((size_t)g->n + 1) * 4 + 255) / 256 * 256 : 0;
    const size_t pb = ((g->heavy.nchunks + 1) * 8 + 255) / 256 * 256;
    const PrPlan *plan = nullptr;
    const uint64_t iters = g->pr_iters + (p->tol <= 0 ? (uint64_t)p->maxiter : 0ull);
    const size_t vsize = dt == GG_F32 ? 4 : 2, own = 2 * nb + sb + ab + pb;
    bool blocked = !staged && dt != GG_F64 && dt != GG_FP8E4M3 && tuning().pr_blocked &&
                   (tuning().pr_blocked == 2 || (g->m >= kBlockedEdges && iters >= kBlockedIters));
    // (the run's time and kernels: with the layout's, where it is built)
    const uint64_t k0 = ctx->launches;
    cudaEventRecord(ctx->ev0, ctx->stream);
    gg_status s = blocked ? pr_plan_wanted(g, vsize, tuning().pr_blocked == 2, &blocked) : GG_OK;
    if (s == GG_OK) s = graph_scratch(g, own + (blocked ? pr_plan_scratch(g, vsize) : 0), &base);
    if (s == GG_OK && blocked) {
        // (the values' space serves the building too; where it turns out too
        // small, for tiles of few edges, it grows)
        s = pr_plan(g, (char *)base + own, &plan);
        if (s == GG_OK && plan) s = graph_scratch(g, own + pr_plan_scratch(g, vsize), &base);
    }
    if (s == GG_ERR_OOM && blocked) {  // without the blocked gather, then
        plan = nullptr;
        s = graph_scratch(g, own, &base);
    }
    if (s != GG_OK) { if (tmpx) gg_prop_destroy(tmpx); return s; }
    float *y = (float *)base;
    void *contrib = (char *)base + nb;
    PrState *st = (PrState *)((char *)base + 2 * nb);
    float *acc = ab ? (float *)((char *)base + 2 * nb + sb) : nullptr;
    void *partial = (char *)base + 2 * nb + sb + ab;
    void *vals = (char *)partial + pb;
    PrState init;
    memset(&init, 0, sizeof(init));
    init.maxiter = p->maxiter;
    init.tol = p->tol;
    init.scale = 1.0f;
    init.scale_inv = 1.0f;
    init.done = p->maxiter == 0;
    init.nstages = staged ? p->nstages : 1;
    for (int k = 0; k < 4; ++k) {
        init.stage_dt[k] = staged && k < p->nstages ? p->stage_dtype[k] : dt;
        init.stage_tol[k] = staged && k + 1 < p->nstages ? p->stage_tol[k] : p->tol;
    }
    init.sr = p->stochastic ? 1 : 0;
    init.avg_from = p->average_last > 0 ? std::max(0, p->maxiter - p->average_last) : -1;
    cudaError_t e = cudaMemcpyAsync(st, &init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(pr_ticket(g, partial), 0, 8, ctx->stream);
    if (e == cudaSuccess && acc) e = cudaMemsetAsync(acc, 0, (size_t)g->n * 4, ctx->stream);
    if (e == cudaSuccess) {
        if (staged) {
            s = pr_run_staged(g, p, (float *)xp->d, y, contrib, st, partial);
        } else switch (dt) {
        case GG_F64: s = pr_run<GG_F64>(g, p, (double *)xp->d, (double *)base, contrib, st, partial, nullptr, nullptr); break;
        case GG_F32: s = pr_run<GG_F32>(g, p, (float *)xp->d, y, contrib, st, partial, plan, vals); break;
        case GG_BF16: s = pr_run<GG_BF16>(g, p, (float *)xp->d, y, contrib, st, partial, plan, vals, acc); break;
        case GG_F16: s = pr_run<GG_F16>(g, p, (float *)xp->d, y, contrib, st, partial, plan, vals); break;
        case GG_FP8E4M3: s = pr_run<GG_FP8E4M3>(g, p, (float *)xp->d, y, contrib, st, partial, nullptr, nullptr); break;
        case GG_CFP_6_10: s = pr_run<GG_CFP_6_10>(g, p, (float *)xp->d, y, contrib, st, partial, plan, vals); break;
        default: s = pr_run<GG_BF16_TRUNC>(g, p, (float *)xp->d, y, contrib, st, partial, plan, vals); break;
        }
    } else {
        s = cuda_error(ctx, e, "gg_pagerank state upload");
    }
    cudaEventRecord(ctx->ev1, ctx->stream);
    PrState fin;
    if (s == GG_OK) {
        e = cudaMemcpyAsync(&fin, st, sizeof(fin), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) s = cuda_error(ctx, e, "gg_pagerank");
    }
    if (s == GG_OK && !staged) g->pr_iters += (uint64_t)fin.iters;
    if (s == GG_OK && stats) {
        memset(stats, 0, sizeof(*stats));
        float ms = 0;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        stats->total_ms = ms;
        stats->iterations = fin.iters;
        stats->kernels = ctx->launches - k0;
        for (int i = 0; i < fin.iters && i < GG_MAX_ITERS; ++i) {
            stats->delta[i] = fin.deltas[i];
            stats->variant[i] = GG_VAR_PULL_DENSE;
            stats->scanned[i] = g->m;
            stats->nactv[i] = g->n;
            stats->nacte[i] = g->m;
        }
        stats->scanned_edges = (uint64_t)fin.iters * g->m;
    }
    if (s == GG_OK && host_x) {
        if (xt == GG_F64) {  // the float copy of the double ranks
            std::vector<double> hx(g->n);
            s = gg_prop_download(xp, hx.data());
            for (uint32_t v = 0; s == GG_OK && v < g->n; ++v) host_x[v] = (float)hx[v];
        } else {
            s = gg_prop_download(xp, host_x);
        }
    }
    if (tmpx) gg_prop_destroy(tmpx);
    return s;
}
