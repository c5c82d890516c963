// gg_bfs.cu -- BFS levels as one resident launch.
//
// A level-synchronous BFS (bench/BFSLVLv.C:110-254) alternates sparse pushes
// and dense pulls, chosen per step from the frontier's counts (api.h:130-222
// or the learned network).  Here a cooperative grid runs the whole search with
// one grid barrier per step: the counts a step leaves are read by every CTA
// after the barrier, each takes the same decision, and the next step starts.
//   push : the frontier is a list of items (gg_items.cuh: rows and pieces of
//          rows), so a step spreads over all warps whatever its rows'
//          lengths; the taker of a vertex sets its frontier bit and, unless
//          the step is so large that a pull will follow, appends its row's
//          items.
//   pull : a lane per vertex of the candidate list reads the vertex's record
//          (its first three in-neighbours and degree) and probes their
//          frontier bits; rows the record leaves open are gathered per warp
//          and walked 32 at a time, so no lane waits for another's long row.
//   A pull leaves the frontier as bits only; a push after it first builds the
//   items from them (one more barrier).
// Three frontier bitmaps are used in turn: step i reads i mod 3, writes i+1
// mod 3 and clears i+2 mod 3, the input of the step before.  Counters are
// three slots in turn as well (phase q adds to slot q mod 3 and clears q+1
// mod 3, last read before the barrier that ended phase q-2).
//
// Data written during the launch are read with plain loads through L1: the
// barrier's fences order them (and drop the SM's L1 lines), so frontier bits
// and levels are cached within a step.
//
// The graph-driven run it replaces cost about 20 us per step outside the
// step's own kernel (the conditional graph node, the chain of idle kernels,
// the decision); a step here costs 5 to 7 us in all where the frontier is
// small.  Per search, before -> after: R-MAT 12 0.139 -> 0.054 ms, R-MAT 20
// relabelled 0.27 -> 0.12, R-MAT 22 relabelled 0.39 -> 0.23, ER 3 M directed
// 0.58 -> 0.25, R-MAT 24 0.68 -> 0.47 (its large push, 195 us, is bound by the
// random level and row-bound accesses, its large pull, 127 us, by the
// latency of records and probes; 213 MB of lists, records and levels would
// take 33 us).
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstring>

#include <cuda_bf16.h>

#include "gg_grid.cuh"
#include "gg_internal.cuh"
#include "gg_items.cuh"
#include "gg_mlp.cuh"
#include "gg_persist.cuh"

namespace gg {

constexpr int kBB = 512;                 // threads per CTA
constexpr int kBW = kBB / 32;            // warps
constexpr uint32_t kRestCap = 64;        // open rows a warp gathers
constexpr int kPull = 3;                 // candidate groups a warp has in flight
constexpr uint32_t kKeepCap = 128;       // candidate appends a warp stages
// A push that finds many edges makes a frontier to pull, whose items nobody
// reads.  So a step over more than kListEdges edges lists none, and a warp
// stops listing after rows of kListWarp edges (the 33,483 vertices that six
// hubs reach on a relabelled R-MAT 22 have 45 M edges: 76 -> 34 us); a push
// that follows all the same builds the items from the bits.
constexpr unsigned long long kListEdges = 1ull << 19;
constexpr uint32_t kListWarp = 8192;

struct alignas(128) BSlot {
    unsigned long long nv, ne, scanned;   // the frontier made: vertices, out-edges; edges examined
    unsigned long long unlisted;          // warps that left rows of it unlisted
    unsigned long long items[IT_KINDS];   // items appended
    unsigned long long ncand;             // candidates left
};

struct BState {
    grid::Arrivals bar;
    BSlot slot[3];
};

struct BArgs {
    const uint64_t *off, *in_off;
    const uint32_t *adj, *in_adj;
    const uint4 *first_in;
    uint32_t n, nw4;                      // vertices; 16-byte words of a bitmap
    uint64_t m;
    int32_t *level;
    uint32_t *bits[3];
    ItemLists items;
    uint32_t *cand[2];
    const uint32_t *nonisolated;
    const unsigned long long *nonisolated_n;
    BState *bs;
    PState *st;
    PState *rec;                          // page-locked copy of *st, written at the end (or null)
    PFront fr[2];
    // the first frontier: root (nroots = 0), a list of roots, or (resumed)
    // the list in fr[resume_cur]
    uint32_t root, nroots;
    const uint32_t *roots;
    int resumed, resume_cur, iter0;
    int threshold, threshold_k;
    const __nv_bfloat16 *sel_w;           // learned choice, or null
    float gini, sel_x4, sel_x9;
    int K;                                // edges a lane walks alone
    int max_iters;
    unsigned long long give_up;           // from the fourth step on: stop at a frontier below this (0: never)
    unsigned long long timeout_ns;
    uint32_t smax, mmax;
    int small_ok, small_from;             // small frontiers leave for k_small_bfs
};

// level = n + 1, bitmaps and state cleared
__global__ void k_bfs_start(BArgs A) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t)gridDim.x * blockDim.x;
    if (!A.resumed) {
        const int32_t inf = (int32_t)A.n + 1;
        for (uint64_t v = tid; v < A.n; v += nth) A.level[v] = inf;
    }
    for (uint64_t w = tid; w < 3ull * A.nw4; w += nth) ((uint4 *)A.bits[0])[w] = make_uint4(0, 0, 0, 0);
    if (tid == 0) {
        A.bs->bar.n = 0;
        A.bs->bar.err = 0;
        for (int i = 0; i < 3; ++i) {
            BSlot *s = &A.bs->slot[i];
            s->nv = s->ne = s->scanned = s->unlisted = s->ncand = 0;
            s->items[0] = s->items[1] = s->items[2] = 0;
        }
        PState *st = A.st;
        st->err = 0;
        st->exit_small = st->small_done = 0;
        if (!A.resumed) {
            st->iterations = 0;
            st->reached_v = st->reached_e = 0;
            st->f_seen = 0;
            for (int f = 0; f < 2; ++f)
                for (int i = 0; i < FC_WORDS; ++i) A.fr[f].cnt[i] = 0;
        }
    }
}

// What warp 0 tells the CTA after a barrier.
struct BNext {
    unsigned long long nv, ne, scanned, unlisted, items[IT_KINDS], ncand;
    int push, err;
};

// Two CTAs per SM leave a thread 64 registers and no spills to speak of (with
// three, R-MAT 24 gained 2 % and ER 3 M lost 12 %, R-MAT 20 20 %).
__global__ void __launch_bounds__(kBB, 2) k_bfs_run(BArgs A) {
    constexpr unsigned FULL = 0xffffffffu;
    // staging of a push (items) and of a pull (kept candidates, open rows):
    // never in use at the same time
    __shared__ union {
        unsigned long long items[kBW][ItemLister::STAGED][ItemAppender::CAP];
        struct {
            uint32_t keep[kBW][kKeepCap], rest[kBW][kRestCap];
        } pull;
    } sm;
    __shared__ float s_selw[GG_SEL_NPARAMS];  // both hidden layers by input unit (lane = output unit)
    __shared__ unsigned long long s_tally[4];
    __shared__ BNext s_next;
    __shared__ unsigned long long s_sel[3];  // last network evaluation: nactv, nacte, unreached
    __shared__ int s_sel_iter, s_sel_push, s_sel_valid;
    PState *st = A.st;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint64_t nw = (uint64_t)gridDim.x * kBW, gw = (uint64_t)blockIdx.x * kBW + wib;
    const uint64_t tid = (uint64_t)blockIdx.x * kBB + threadIdx.x, nth = (uint64_t)gridDim.x * kBB;
    const bool first_thread = blockIdx.x == 0 && threadIdx.x == 0;
    const bool sym = A.off == A.in_off;
    if (threadIdx.x < 4) s_tally[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_sel_valid = 0;
    if (A.sel_w)
        for (int i = threadIdx.x; i < GG_SEL_NPARAMS; i += kBB) s_selw[mlp::by_input(i)] = __bfloat162float(A.sel_w[i]);
    __syncthreads();

    unsigned long long epoch = 0;
    uint32_t q = 0;
    int iter = A.iter0;
    unsigned long long head[IT_KINDS] = {0, 0, 0};  // items of the phases before the last one
    unsigned long long reached_v = A.resumed ? st->reached_v : 0ull, reached_e = A.resumed ? st->reached_e : 0ull;
    unsigned long long nv = 0, ne = 0, sc = 0;  // this thread's share of a phase's tally
    uint32_t listed = 0;  // edges of the rows this warp listed
    bool full = false;    // it left rows unlisted
    ItemLister lister;
    lister.init(sm.items[wib]);

    auto begin = [&]() -> BSlot * {
        if (first_thread) {
            BSlot *s = &A.bs->slot[(q + 1) % 3];
            s->nv = s->ne = s->scanned = s->unlisted = s->ncand = 0;
            s->items[0] = s->items[1] = s->items[2] = 0;
        }
        BSlot *out = &A.bs->slot[q % 3];
        lister.begin(A.items, head, out->items);
        return out;
    };
    // The push / pull choice for the frontier just made (one warp, the same
    // in every CTA).  The learned network replaces the threshold's choice
    // where it predicts a clear gain; an evaluation is reused while the counts
    // stay within 1/16 of its own.
    auto choose = [&](unsigned long long fv, unsigned long long fe, int it, unsigned long long rv) -> int {
        bool push;
        switch (A.threshold) {
        case GG_THRESH_ALWAYS_SPARSE: push = true; break;
        case GG_THRESH_ALWAYS_DENSE: push = false; break;
        case GG_THRESH_FRAC: push = (float)(fv + fe) <= (float)A.m / (float)(100.0 / (float)A.threshold_k); break;
        default: push = fv + fe <= A.m / 20;
        }
        if (!A.sel_w || fv == 0) return push;
        const unsigned long long unr = rv < A.n ? A.n - rv : 0ull;
        const auto close = [](unsigned long long a, unsigned long long b) {
            const unsigned long long d = a > b ? a - b : b - a, mx = a > b ? a : b;
            return d * 16 <= mx;
        };
        if (s_sel_valid && close(fv, s_sel[0]) && close(fe, s_sel[1]) && close(unr, s_sel[2]) &&
            min(it, 255) - s_sel_iter < 8)
            return s_sel_push;
        const float n = (float)A.n, m = (float)A.m, v = (float)fv, e = (float)fe;
        float x[GG_SEL_FEATURES], o[GG_SEL_VARIANTS];
        x[0] = log2f(1.0f + v) / 32;
        x[1] = log2f(1.0f + e) / 40;
        x[2] = log2f(1.0f + (float)unr) / 32;
        x[3] = log2f(1.0f + (float)min(it, 255)) / 8;
        x[4] = A.sel_x4;
        x[5] = A.gini;
        x[6] = n > 0 ? v / n : 0.0f;
        x[7] = m > 0 ? e / m : 0.0f;
        x[8] = fminf(4.0f, m > 0 ? (v + e) / m : 0.0f);
        x[9] = A.sel_x9;
        mlp::warp_forward_by_input(s_selw, x, o);
        const int tv = push ? GG_VAR_PUSH_SPARSE : GG_VAR_PULL_DENSE;
        const int best = o[GG_VAR_PUSH_SPARSE] < o[GG_VAR_PULL_DENSE] ? GG_VAR_PUSH_SPARSE : GG_VAR_PULL_DENSE;
        if (o[best] < o[tv] - mlp::kSelMargin) push = best == GG_VAR_PUSH_SPARSE;
        __syncwarp();
        if (lane == 0) {
            s_sel[0] = fv;
            s_sel[1] = fe;
            s_sel[2] = unr;
            s_sel_iter = min(it, 255);
            s_sel_push = push;
            s_sel_valid = 1;
        }
        __syncwarp();
        return push;
    };
    // Ends a phase: the CTA's tally, the barrier, the phase's counters and
    // (with `decide`) the next step's choice.  False: a barrier timed out.
    auto end_phase = [&](BSlot *out, bool decide) -> bool {
        nv = dev::warp_sum(nv);
        ne = dev::warp_sum(ne);
        sc = dev::warp_sum(sc);
        if (lane == 0) {
            if (nv) atomicAdd(&s_tally[0], nv);
            if (ne) atomicAdd(&s_tally[1], ne);
            if (sc) atomicAdd(&s_tally[2], sc);
            if (full) atomicAdd(&s_tally[3], 1ull);
        }
        nv = ne = sc = 0;
        listed = 0;
        full = false;
        __syncthreads();
        ++epoch;
        if (wib == 0) {
            // (one thread adds, arrives, waits and reads: its fences order
            // its own accesses and those it saw through the CTA's barrier)
            unsigned long long x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            int err = 0;
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const unsigned long long t = s_tally[i];
                    if (t) atomicAdd(&out->nv + i, t);
                    s_tally[i] = 0;
                }
                err = !grid::arrive_and_wait(&A.bs->bar, epoch, A.timeout_ns);
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = __ldcg(&out->nv + i);
            }
            err = __shfl_sync(FULL, err, 0);
            const unsigned long long fv = __shfl_sync(FULL, x[0], 0), fe = __shfl_sync(FULL, x[1], 0);
            const int push = decide && !err ? choose(fv, fe, iter + 1, reached_v) : 0;
            if (lane == 0) {
                s_next.nv = fv;
                s_next.ne = fe;
                s_next.scanned = x[2];
                s_next.unlisted = x[3];
                for (int k = 0; k < IT_KINDS; ++k) s_next.items[k] = x[4 + k];
                s_next.ncand = x[7];
                s_next.err = err;
                s_next.push = push;
            }
        }
        __syncthreads();
        ++q;
        return s_next.err == 0;
    };
    // a vertex joins the frontier being made, with `list` as a row of items
    // too (all lanes)
    auto record = [&](bool rec, uint32_t d, uint32_t *bits, bool list) {
        if (!__any_sync(FULL, rec)) return;
        uint64_t b = 0, dg = 0;
        if (rec) {
            b = A.off[d];
            dg = A.off[d + 1] - b;
            nv++;
            ne += dg;
            atomicOr(bits + (d >> 5), 1u << (d & 31));
        }
        if (!list) return;
        if (listed > kListWarp) {
            full = true;
            return;
        }
        listed += __reduce_add_sync(FULL, (uint32_t)min(dg, (uint64_t)kListWarp));
        lister.list(rec, b, dg);
    };

    // ---- the first frontier
    {
        BSlot *out = begin();
        uint32_t *F = A.bits[iter % 3];
        const PFront &R = A.fr[A.resume_cur];
        uint64_t c0 = 0, c1 = 0, k = A.nroots ? A.nroots : 1;
        if (A.resumed) {
            c0 = R.cnt[FC_BIN0];
            c1 = R.cnt[FC_BIN1];
            k = c0 + c1 + R.cnt[FC_BIN2];
        }
        for (uint64_t base = gw * 32; base < k; base += nw * 32) {
            const uint64_t i = base + lane;
            uint32_t v = 0;
            if (i < k) {
                if (A.resumed) v = i < c0 ? R.bins[0][i] : (i < c0 + c1 ? R.bins[1][i - c0] : R.bins[2][i - c0 - c1]);
                else {
                    v = A.nroots ? A.roots[i] : A.root;
                    A.level[v] = 0;
                }
            }
            record(i < k, v, F, true);
        }
        lister.flush();
        if (first_thread && iter <= GG_MAX_ITERS) st->t_ns[iter] = grid::globaltimer();
        --iter;  // (the choice below is for step `iter`)
        const bool ok = end_phase(out, true);
        ++iter;
        if (!ok) goto timed_out;
        if (A.resumed && first_thread)
            for (int i = 0; i < FC_WORDS; ++i) A.fr[A.resume_cur].cnt[i] = 0;
    }
    {
    bool have_items = s_next.unlisted == 0, prev_pull = false, cand_valid = false, handed = false;
    int cc = 0;                            // candidate list in use
    unsigned long long ncand = 0;
    unsigned long long cnt[IT_KINDS] = {s_next.items[0], s_next.items[1], s_next.items[2]};  // the frontier's items
    while (true) {
        const unsigned long long fv = s_next.nv, fe = s_next.ne;
        const bool push = s_next.push != 0;
        if (fv == 0 || iter >= A.max_iters || (iter >= 3 && fv < A.give_up)) break;
        uint32_t *F = A.bits[iter % 3], *O = A.bits[(iter + 1) % 3], *C = A.bits[(iter + 2) % 3];
        if (A.small_ok && push && iter >= A.small_from && fv <= kSmallEnterV && fe <= kSmallEnterE) {
            // the frontier as the binned list that k_small_bfs takes
            __syncthreads();
            const PFront &R = A.fr[0];
            // (the appenders' 32-entry buffers in the keep area)
            uint32_t *buf = sm.pull.keep[wib];
            dev::WarpAppender<32> a0{buf, 0, R.bins[0], R.cnt + FC_BIN0}, a1{buf + 32, 0, R.bins[1], R.cnt + FC_BIN1},
                a2{buf + 64, 0, R.bins[2], R.cnt + FC_BIN2};
            unsigned long long x = 0, y = 0;
            dev::bitmap_to_bins<32>(F, A.n, A.off, A.smax, A.mmax, a0, a1, a2, x, y);
            a0.flush();
            a1.flush();
            a2.flush();
            handed = true;
            break;
        }
        if (first_thread && iter < GG_MAX_ITERS) {
            st->variant[iter] = push ? GG_VAR_PUSH_SPARSE : GG_VAR_PULL_DENSE;
            st->nactv[iter] = fv;
            st->nacte[iter] = fe;
        }
        const int32_t fk = iter + 1;
        if (push && !have_items) {
            // items of the rows whose bits a pull left
            BSlot *out = begin();
            const uint32_t nwords = (A.n + 31u) >> 5, group = max(short_group(nwords, nw), 4u);
            for (uint64_t base = gw * group; base < nwords; base += nw * group) {
                const uint64_t w = base + lane;
                const uint32_t mine = lane < group && w < nwords ? F[w] : 0u;
                unsigned nz = __ballot_sync(FULL, mine != 0);
                while (nz) {  // warp-uniform: four words' row bounds in flight
                    uint64_t b[4], e[4];
                    bool on[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int j = nz ? __ffs(nz) - 1 : -1;
                        if (j >= 0) nz &= nz - 1;
                        const uint32_t word = __shfl_sync(FULL, mine, max(j, 0));
                        const uint32_t v = (uint32_t)((base + (uint32_t)max(j, 0)) * 32) + lane;
                        on[k] = j >= 0 && ((word >> lane) & 1u);
                        b[k] = on[k] ? A.off[v] : 0;
                        e[k] = on[k] ? A.off[v + 1] : 0;
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) lister.list(on[k], b[k], e[k] - b[k]);
                }
            }
            lister.flush();
            if (!end_phase(out, false)) goto timed_out;
            for (int k = 0; k < IT_KINDS; ++k) cnt[k] = s_next.items[k];
        }
        // a step over many edges most likely makes a frontier to pull, whose
        // items nobody would read: it leaves bits only
        const bool list = push && fe <= kListEdges;
        BSlot *out = begin();
        for (uint64_t w = tid; w < A.nw4; w += nth) ((uint4 *)C)[w] = make_uint4(0, 0, 0, 0);
        if (push) {
            const unsigned long long *is = A.items.p[IT_SHORT] + head[IT_SHORT], *il = A.items.p[IT_LONG] + head[IT_LONG],
                                     *ih = A.items.p[IT_HUGE] + head[IT_HUGE];
            const unsigned long long ns = cnt[IT_SHORT], nl = cnt[IT_LONG], nh = cnt[IT_HUGE];
            for (int k = 0; k < IT_KINDS; ++k) head[k] += cnt[k];
            lister.begin(A.items, head, out->items);
            auto take = [&](uint32_t d) -> bool {
                if (A.level[d] <= fk) return false;
                return atomicMin(A.level + d, fk) > fk;
            };
            // up to kLong edges from `first`, four per lane in flight
            auto piece = [&](uint64_t first, uint32_t len) {
                const uint32_t *row = A.adj + first;
                if (lane == 0) sc += len;
                for (uint32_t h = 0; h < len; h += 128) {
                    uint32_t d[4];
                    bool rec[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) d[u] = h + 32 * u + lane < len ? __ldg(row + h + 32 * u + lane) : 0u;
#pragma unroll
                    for (int u = 0; u < 4; ++u) rec[u] = h + 32 * u + lane < len && take(d[u]);
#pragma unroll
                    for (int u = 0; u < 4; ++u) record(rec[u], d[u], O, list);
                }
            };
            for (uint64_t i = blockIdx.x; i < nh; i += gridDim.x) {
                const unsigned long long it = ih[i];
                const uint32_t len = item_len(it);
                for (uint32_t o = wib * kLong; o < len; o += kBW * kLong) piece(item_first(it) + o, min(kLong, len - o));
            }
            const uint32_t parts = long_pieces(nl, nw), width = kLong / parts;
            for (uint64_t i = gw; i < nl * parts; i += nw) {
                const unsigned long long it = il[i / parts];
                const uint32_t len = item_len(it), o = (uint32_t)(i % parts) * width;
                if (o < len) piece(item_first(it) + o, min(width, len - o));
            }
            const uint32_t group = short_group(ns, nw);
            for (uint64_t base = gw * group; base < ns; base += nw * group) {
                unsigned long long it = 0;
                if (lane < group && base + lane < ns) it = is[base + lane];
                sc += item_len(it);
                dev::warp_flat_rows<4>(
                    A.adj, item_first(it), item_len(it), 0u, [&](uint32_t d, uint32_t) { return take(d); },
                    [&](bool rec, uint32_t d) { record(rec, d, O, list); });
            }
            lister.flush();
        } else {
            const uint32_t *cand = cand_valid ? A.cand[cc] : A.nonisolated;
            const unsigned long long nc = cand_valid ? ncand : *A.nonisolated_n;
            const bool fresh = cand_valid && prev_pull;  // the last pull's open candidates: all unvisited
            dev::WarpAppender<kKeepCap> keep{sm.pull.keep[wib], 0, A.cand[cand_valid ? cc ^ 1 : 0], &out->ncand};
            uint32_t *rest = sm.pull.rest[wib];
            uint32_t nrest = 0;
            auto probe = [&](uint32_t s) -> bool { return (F[s >> 5] >> (s & 31u)) & 1u; };
            // vertices found: level, frontier bit (one atomic per distinct
            // word; lists are mostly ascending), counts (all lanes)
            auto settle = [&](bool found, uint32_t d, uint64_t deg) {
                if (found) {
                    A.level[d] = fk;
                    nv++;
                    ne += sym ? deg : A.off[d + 1] - A.off[d];
                }
                unsigned todo = __ballot_sync(FULL, found);
                while (todo) {
                    const int leader = __ffs(todo) - 1;
                    const uint32_t w0 = __shfl_sync(FULL, d >> 5, leader);
                    const bool mine = found && (d >> 5) == w0;
                    const unsigned b = __reduce_or_sync(FULL, mine ? 1u << (d & 31) : 0u);
                    if ((int)lane == leader) atomicOr(O + w0, b);
                    todo &= ~__ballot_sync(FULL, mine);
                }
            };
            // up to 32 gathered rows from their fourth edge: K edges by their
            // lane, the rest of long rows by the whole warp
            auto walk = [&](uint32_t count) {
                __syncwarp();
                const bool on = lane < count;
                const uint32_t d = on ? rest[nrest - count + lane] : 0u;
                uint64_t beg = 0, end = 0;
                if (on) {
                    beg = A.in_off[d];
                    end = A.in_off[d + 1];
                }
                uint64_t e = beg + 3;
                const uint64_t lim = min(end, beg + (uint64_t)max(A.K, 3));
                bool found = false;
                while (on && !found && e < lim) {
                    const int cnt = (int)min((uint64_t)4, lim - e);
                    uint32_t s[4];
                    bool hit[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[j] = j < cnt ? __ldg(A.in_adj + e + j) : 0u;
#pragma unroll
                    for (int j = 0; j < 4; ++j) hit[j] = j < cnt && probe(s[j]);
                    int used = cnt;
#pragma unroll
                    for (int j = 3; j >= 0; --j)
                        if (hit[j]) {
                            found = true;
                            used = j + 1;
                        }
                    e += used;
                }
                if (on) sc += e - beg - 3;
                unsigned pend = __ballot_sync(FULL, on && !found && e < end);
                while (pend) {
                    const int j = __ffs(pend) - 1;
                    pend &= pend - 1;
                    const uint64_t ej = __shfl_sync(FULL, e, j), endj = __shfl_sync(FULL, end, j);
                    bool hit = false;
                    for (uint64_t base = ej; base < endj && !hit; base += 32) {
                        if (lane == 0) sc += min((uint64_t)32, endj - base);
                        hit = __any_sync(FULL, base + lane < endj && probe(__ldg(A.in_adj + base + lane)));
                    }
                    if ((int)lane == j) found = hit;
                }
                settle(found, d, end - beg);
                keep.push(on && !found, d);
                nrest -= count;
                __syncwarp();
            };
            // kPull groups of 32 candidates at a time: their ids, then their
            // records and levels, are in flight together
            for (uint64_t w0 = gw; w0 * 32 < nc; w0 += kPull * nw) {
                uint32_t dd[kPull];
                uint4 rr[kPull];
                int32_t lv[kPull];
#pragma unroll
                for (int u = 0; u < kPull; ++u) {
                    const uint64_t i = (w0 + u * nw) * 32 + lane;
                    dd[u] = i < nc ? cand[i] : 0xFFFFFFFFu;
                }
#pragma unroll
                for (int u = 0; u < kPull; ++u) {
                    rr[u] = make_uint4(0u, 0u, 0u, 0u);
                    lv[u] = INT_MAX;
                    if (dd[u] != 0xFFFFFFFFu) {
                        rr[u] = A.first_in[dd[u]];
                        if (!fresh) lv[u] = A.level[dd[u]];
                    }
                }
#pragma unroll
                for (int u = 0; u < kPull; ++u) {
                    if ((w0 + u * nw) * 32 >= nc) break;  // warp-uniform
                    const uint32_t d = dd[u];
                    const uint4 r = rr[u];
                    const bool open = lv[u] > fk && r.z != 0;  // (r.z is 0 past the list's end)
                    bool found = false;
                    if (open) {
                        found = probe(r.x);
                        uint32_t used = 1;
                        if (!found && r.z > 1) {
                            const bool h1 = probe(r.y), h2 = r.z > 2 && probe(r.w);
                            found = h1 || h2;
                            used = h1 || r.z == 2 ? 2u : 3u;
                        }
                        sc += used;
                    }
                    uint64_t deg = r.z;
                    if (r.z == 0xFFFFFFFFu) deg = A.in_off[d + 1] - A.in_off[d];
                    settle(found, d, deg);
                    const bool more = open && !found && r.z > 3;
                    keep.push(open && !found && !more, d);
                    const unsigned mk = __ballot_sync(FULL, more);
                    if (more) rest[nrest + __popc(mk & ((1u << lane) - 1u))] = d;
                    nrest += __popc(mk);
                    if (nrest > kRestCap - 32) walk(32);
                }
            }
            if (nrest > 0) walk(min(nrest, 32u));
            keep.flush();
            cc = cand_valid ? cc ^ 1 : 0;
            cand_valid = true;
        }
        reached_v += fv;
        reached_e += fe;
        if (!end_phase(out, true)) goto timed_out;
        if (first_thread) {
            if (iter < GG_MAX_ITERS) st->scanned[iter] = s_next.scanned;
            if (iter + 1 <= GG_MAX_ITERS) st->t_ns[iter + 1] = grid::globaltimer();
        }
        if (!push) ncand = s_next.ncand;
        for (int k = 0; k < IT_KINDS; ++k) cnt[k] = s_next.items[k];
        have_items = list && s_next.unlisted == 0;
        prev_pull = !push;
        ++iter;
    }
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            st->iterations = iter;
            st->reached_v = reached_v + (handed ? 0ull : s_next.nv);  // (a search cut short: its last frontier)
            st->reached_e = reached_e;
            st->cand_valid = cand_valid;
            st->cand_cur = cc;
            st->cand_n[0] = ncand;
            st->t_end = grid::globaltimer();
            st->exit_small = handed;
            st->small_done = !handed;
            st->small_iter = iter;
            st->small_cur = 0;
        }
        if (handed || !A.rec) return;
        // the records to the host (whole 16-byte words over the link)
        __syncthreads();
        const uint4 *src = (const uint4 *)st;
        for (uint32_t i = threadIdx.x; i < sizeof(PState) / 16; i += kBB) ((uint4 *)A.rec)[i] = src[i];
    }
    return;
    }
timed_out:
    if (threadIdx.x == 0) atomicOr(&st->err, DEV_ERR_TIMEOUT);
}

const void *selector_weights(gg_graph *g);

static_assert(sizeof(PState) <= kRunRecord && sizeof(BState) <= kRunState, "records and state block");

static gg_status bfs_resident_buffers(gg_graph *g) {
    gg_ctx *ctx = g->ctx;
    for (auto &f : g->tmp_front)
        if (!f) GG_CHECK(gg_frontier_create(g, &f));
    for (auto *f : g->tmp_front) {
        GG_CHECK(frontier_alloc_bins(f));
        GG_CHECK(frontier_alloc_bitmap(f));
    }
    GG_CHECK(cand_lists_alloc(g));
    if (!g->pstate) GG_CUDA(ctx, cudaMalloc(&g->pstate, sizeof(PState)));
    GG_CHECK(run_record(ctx));
    return resident_memory(g);
}

// What the resident runs of g allocated for themselves goes back: the drivers
// taken instead need room too (their frontiers and candidate lists are the same).
gg_status resident_give_up(gg_graph *g, gg_status s) {
    if (s != GG_ERR_OOM) return s;
    cudaFree(g->resident);
    g->resident = nullptr;
    return GG_OK;
}

// Buffers for a run on g.  *ok = false (and nothing kept but what other
// drivers use) where they do not fit in memory: the caller takes another one.
gg_status bfs_resident_prepare(gg_graph *g, bool *ok) {
    const gg_status s = bfs_resident_buffers(g);
    *ok = s == GG_OK;
    return resident_give_up(g, s);
}

static gg_status bfs_args(gg_graph *g, gg_prop *level, const gg_run_opts &opt, PState *st, BArgs &A) {
    const Tuning &t = tuning();
    std::memset(&A, 0, sizeof(A));
    A.off = g->off;
    A.in_off = g->in_off;
    A.adj = g->adj;
    A.in_adj = g->in_adj;
    A.first_in = g->first_in;
    A.n = g->n;
    A.nw4 = (uint32_t)bitmap_words4(g);
    A.m = g->m;
    A.level = (int32_t *)level->d;
    uint32_t *bits = (uint32_t *)((char *)g->resident + resident_bits_at(g));
    for (int i = 0; i < 3; ++i) A.bits[i] = bits + (size_t)i * A.nw4 * 4;
    A.items = item_lists(g);
    A.cand[0] = g->cand.list[0];
    A.cand[1] = g->cand.list[1];
    A.nonisolated = g->nonisolated;
    A.nonisolated_n = (const unsigned long long *)g->nonisolated_n;
    A.bs = (BState *)resident_state(g, RUN_BFS);
    A.st = st;
    for (int i = 0; i < 2; ++i) {
        gg_frontier *f = g->tmp_front[i];
        for (int b = 0; b < NBINS; ++b) A.fr[i].bins[b] = f->bins[b];
        A.fr[i].bitmap = f->bitmap;
        A.fr[i].cnt = (unsigned long long *)f->d_cnt;
        f->host_valid = f->has_list = f->has_bitmap = f->all = false;
    }
    A.threshold = opt.threshold;
    A.threshold_k = opt.threshold_k;
    if (opt.threshold == GG_THRESH_LEARNED && selector_weights(g)) {
        if (g->gini < 0) {
            float gi;
            GG_CHECK(graph_gini(g, &gi));
        }
        A.sel_w = (const __nv_bfloat16 *)selector_weights(g);
        A.gini = g->gini < 0 ? 0.0f : g->gini;
        float xs[GG_SEL_FEATURES];
        selector_features(xs, 0, 0, 0, 0, (double)g->n, (double)g->m, A.gini);
        A.sel_x4 = xs[4];
        A.sel_x9 = xs[9];
    }
    A.K = t.pull_k;
    A.max_iters = (int)std::min<uint64_t>((uint64_t)g->n + 2, (uint64_t)INT_MAX / 2);
    A.timeout_ns = t.barrier_timeout_ns;
    A.smax = t.bin_small_max;
    A.mmax = t.bin_medium_max;
    return GG_OK;
}

static gg_status bfs_launch(gg_graph *g, BArgs &A) {
    gg_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    const uint64_t start = A.resumed ? 3ull * A.nw4 : (uint64_t)g->n;
    const unsigned sg = (unsigned)std::min<uint64_t>((start + 255) / 256, (uint64_t)ctx->sm_count * 8);
    k_bfs_start<<<sg ? sg : 1, 256, 0, s>>>(A);
    GG_LAUNCHED(ctx);
    // a CTA per 8192 edges or 4096 vertices, all that fit at most: the
    // barriers of a small graph's steps are cheaper with fewer
    const uint64_t most = (uint64_t)ctx->sm_count * resident_ctas((const void *)k_bfs_run, kBB);
    const uint64_t want = std::max<uint64_t>(std::max<uint64_t>(g->m / 8192, g->n / 4096), 1);
    void *args[] = {&A};
    GG_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)k_bfs_run, dim3((unsigned)std::min(most, want)), dim3(kBB),
                                             args, 0, s));
    ctx->launches++;
    return GG_OK;
}

// Enqueues a search from `nroots` distinct roots (device list) with its state
// in `st`; nothing waits on the host and no host memory is read later (may be
// captured).  bfs_resident_prepare() has been called.
gg_status bfs_resident_enqueue(gg_graph *g, gg_prop *level, const uint32_t *d_roots, uint32_t nroots,
                               const gg_run_opts &opt, PState *st) {
    BArgs A;
    GG_CHECK(bfs_args(g, level, opt, st, A));
    A.roots = d_roots;
    A.nroots = nroots;
    return bfs_launch(g, A);
}

// Enqueues at most `steps` levels from one root, fewer where the fourth step
// or a later one starts from fewer than `give_up` vertices (those of the last
// frontier have their levels); may be captured.
gg_status bfs_resident_search(gg_graph *g, gg_prop *level, uint32_t root, int steps, unsigned long long give_up,
                              PState *st) {
    gg_run_opts opt;
    std::memset(&opt, 0, sizeof(opt));
    opt.threshold = GG_THRESH_DEFAULT;
    opt.variant = GG_VAR_AUTO;
    BArgs A;
    GG_CHECK(bfs_args(g, level, opt, st, A));
    A.root = root;
    A.max_iters = std::min(A.max_iters, steps);
    A.give_up = give_up;
    return bfs_launch(g, A);
}

// Levels from one root.
gg_status bfs_resident(gg_graph *g, gg_prop *level, uint32_t root, const gg_run_opts &opt, gg_run_stats *st,
                       int *iters_out) {
    gg_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    const Tuning &t = tuning();
    PState *ds = (PState *)g->pstate;
    BArgs A;
    GG_CHECK(bfs_args(g, level, opt, ds, A));
    A.root = root;
    A.rec = (PState *)ctx->d_run;
    A.small_ok = t.small_frontier;
    A.small_from = t.graph_handoff > 0 ? t.graph_handoff : 32;
    PState &hs = *(PState *)ctx->h_run;
    while (true) {
        hs.small_done = -1;  // written by the run's end
        GG_CHECK(bfs_launch(g, A));
        GG_CUDA(ctx, cudaStreamSynchronize(s));
        if (hs.small_done == 1) break;
        GG_CUDA(ctx, cudaMemcpy(&hs, ds, sizeof(PState), cudaMemcpyDeviceToHost));
        if (hs.err & DEV_ERR_TIMEOUT) return set_error(ctx, GG_ERR_TIMEOUT, "traversal grid barrier timed out");
        if (hs.err || !hs.exit_small) return set_error(ctx, GG_ERR_STATE, "traversal device error");
        // a small frontier of a long run: levels in one cluster
        GG_CHECK(enqueue_small_bfs(g, ds, A.fr, A.level, A.max_iters, A.threshold, A.threshold_k));
        GG_CUDA(ctx, cudaMemcpyAsync(&hs, ds, sizeof(PState), cudaMemcpyDeviceToHost, s));
        GG_CUDA(ctx, cudaStreamSynchronize(s));
        if (hs.small_done == 1) break;
        A.resumed = 1;
        A.resume_cur = hs.small_cur;
        A.iter0 = hs.small_iter;
        A.small_from = A.iter0 + 1;  // at least one step here before the next hand-over
    }
    *iters_out = hs.iterations;
    if (st) {
        st->vertices_reached = hs.reached_v;
        st->edges_reached = hs.reached_e;
        for (int i = 0; i < std::min(hs.iterations, GG_MAX_ITERS); ++i) {
            st->variant[i] = hs.variant[i];
            st->nactv[i] = hs.nactv[i];
            st->nacte[i] = hs.nacte[i];
            st->scanned[i] = hs.scanned[i];
            st->scanned_edges += hs.scanned[i];
            st->iter_ms[i] = (double)(hs.t_ns[i + 1] - hs.t_ns[i]) * 1e-6;
            st->kernel_ms[i] = st->iter_ms[i];
        }
    }
    return GG_OK;
}

}  // namespace gg
