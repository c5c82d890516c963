// gg_cc.cu -- connected components of a symmetric graph: a short search from
// the vertex of largest degree, then min-id hooking of what it did not reach,
// two resident launches without a host round trip.
//
// CCv (bench/CCv.C:221-471) lowers labels along every edge until nothing
// moves; its labels are the smallest id of each component, whatever the order.
//   search : where the degrees let it reach far, at most kSearchSteps levels
//            of the resident BFS (gg_bfs.cu).  On a graph with hubs they reach
//            the giant component, most of it by pulls that look at one or two
//            edges per vertex;
//   count  : the vertices reached and their smallest id.  Where they are half
//            of the vertices with edges, that id is their label and only the
//            others hook their edges (gg_uf.cuh);
//   hook   : else (grids, unions of graphs, sparse random graphs: the search
//            stopped or found a small component) label[v] = min(v, its first
//            neighbour) for every vertex, then every vertex hooks its edges to
//            smaller ids, long rows in chunks of a warp each;
//   finish : label[v] = its root.
// Per run, before (label propagation and, on graphs that pass CCv's
// road-network test, hooking after its first step) -> here: R-MAT 24 0.71 ->
// 0.45 ms, R-MAT 20 relabelled 0.26 -> 0.12, R-MAT 12 0.12 -> 0.065, star of 2^24
// 0.52 -> 0.24, grid 2896^2 1.17 -> 0.49, a union of 100 graphs (134 M edges, hubs)
// 8.7 -> 1.1, sparse ER (3 M vertices, average degree 2.6) 0.89 -> 0.45, 2 M vertices
// of degree 16 within 1000 ids 1.51 -> 1.33.  The search takes 0.42 of R-MAT 24's
// 0.45 ms; the sparse graphs are bound by the chains of dependent label reads of
// the hooks (0.36 ms for ER's).
#include <algorithm>
#include <climits>
#include <cstring>

#include "gg_grid.cuh"
#include "gg_internal.cuh"
#include "gg_items.cuh"
#include "gg_persist.cuh"
#include "gg_uf.cuh"

namespace gg {

constexpr int kCB = 512;                   // threads per CTA, two CTAs per SM
// The search stops early at a frontier of fewer than kSearchLeast vertices: on
// a grid or a sparse random graph it would not reach far, on a graph with hubs
// little is left by then.
// For the same reason there is none where even the largest hub's neighbours,
// each with average rows, and theirs would be fewer (with the search -> without:
// grid 85 x 84 less a third of its edges 161 -> 133 us a call, ER of 3001
// vertices and average degree 3 163 -> 139, of 300001 and 2 212 -> 189).
constexpr int kSearchSteps = 10;
constexpr unsigned long long kSearchLeast = 1024;

struct CcState {
    grid::Arrivals bar;
    uint32_t smallest;
    uint32_t nleft;  // vertices listed in `left`
    uint32_t moved[3];  // a doubling round changed a label (three in turn)
    unsigned long long hooked;  // edges that the hooks looked at
};

// What the host reads after a run: the records, written by the first CTA at
// its end, and a word of their own for the CTAs that gave up at a barrier (the
// first one may have left the last barrier in time and write its records all
// the same).
struct CcRecord {
    PState st;
    unsigned int gave_up;
};
static_assert(sizeof(CcRecord) <= kRunRecord && sizeof(CcState) <= kRunState, "records and state block");

struct CcArgs {
    const uint64_t *off;
    const uint32_t *adj;
    const uint4 *first_in;
    const uint32_t *nonisolated;
    const unsigned long long *nonisolated_n;
    HeavyRows H;
    uint32_t n;
    uint64_t m;
    int searched;          // level, cand and st's reached_v are a search's
    const int32_t *level;
    const uint32_t *cand[2];  // its candidate lists: st->cand_cur holds the vertices the last pull left open
    uint32_t *left;        // room for the vertices outside the giant component
    uint32_t *label;
    CcState *cs;
    PState *st;   // records
    CcRecord *rec;  // page-locked copy of them, or null
    unsigned long long timeout_ns;
};

__global__ void __launch_bounds__(kCB, 2) k_cc_run(CcArgs A) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int U = 4;  // vertices a thread has in flight
    uint32_t *lab = A.label;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t tid = (uint64_t)blockIdx.x * kCB + threadIdx.x, nth = (uint64_t)gridDim.x * kCB;
    const uint64_t nw = nth >> 5, gw = tid >> 5;
    const int32_t inf = (int32_t)A.n + 1;
    const bool first_thread = blockIdx.x == 0 && threadIdx.x == 0;
    unsigned long long epoch = 0;
    const unsigned long long t0 = grid::globaltimer();
    const uint64_t nn = *A.nonisolated_n, reached = A.st->reached_v;
    const bool giant = A.searched && 2 * reached >= nn;
    bool ok = true;

    // ---- label
    uint32_t top = 0xFFFFFFFFu;
    if (giant) {
        // its smallest vertex: of the first ids, or else of all
        __shared__ uint32_t s_top;
        if (threadIdx.x == 0) s_top = 0xFFFFFFFFu;
        __syncthreads();
        if (threadIdx.x < A.n && A.level[threadIdx.x] != inf) atomicMin(&s_top, threadIdx.x);
        __syncthreads();
        top = s_top;
        if (top == 0xFFFFFFFFu) {  // the same in every CTA
            uint32_t least = 0xFFFFFFFFu;
            for (uint64_t v = tid; v < A.n; v += nth)
                if (A.level[v] != inf) least = min(least, (uint32_t)v);
            least = __reduce_min_sync(FULL, least);
            if (lane == 0 && least != 0xFFFFFFFFu) atomicMin(&A.cs->smallest, least);
            ok = grid::sync(&A.cs->bar, epoch, A.timeout_ns);
            top = __ldcg(&A.cs->smallest);
        }
    }
    if (ok) {
        for (uint64_t v0 = tid; v0 < A.n; v0 += U * nth) {
            if (giant) {
                int32_t l[U];
#pragma unroll
                for (int u = 0; u < U; ++u) l[u] = v0 + u * nth < A.n ? A.level[v0 + u * nth] : inf;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (v0 + u * nth < A.n) lab[v0 + u * nth] = l[u] != inf ? top : (uint32_t)(v0 + u * nth);
            } else {
                uint4 r[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    r[u] = v0 + u * nth < A.n ? __ldcs(A.first_in + v0 + u * nth) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint64_t v = v0 + u * nth;
                    if (v < A.n) lab[v] = r[u].z ? min((uint32_t)v, r[u].x) : (uint32_t)v;
                }
            }
        }
        ok = grid::sync(&A.cs->bar, epoch, A.timeout_ns);
    }
    // without a giant component: every label becomes its tree's root, the
    // walks halved by all vertices at once (a grid's trees are columns of
    // thousands of vertices: twelve rounds)
    for (int round = 0; ok && !giant; ++round) {
        if (first_thread) A.cs->moved[(round + 1) % 3] = 0;
        bool move = false;
        for (uint64_t v0 = tid; v0 < A.n; v0 += U * nth) {
            uint32_t l[U], p[U];
#pragma unroll
            for (int u = 0; u < U; ++u) l[u] = v0 + u * nth < A.n ? __ldcg(lab + v0 + u * nth) : 0u;
#pragma unroll
            for (int u = 0; u < U; ++u) p[u] = __ldcg(lab + l[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (v0 + u * nth < A.n && p[u] != l[u]) {
                    lab[v0 + u * nth] = p[u];
                    move = true;
                }
        }
        if (__syncthreads_or(move) && threadIdx.x == 0) atomicOr(&A.cs->moved[round % 3], 1u);
        ok = grid::sync(&A.cs->bar, epoch, A.timeout_ns);
        if (__ldcg(&A.cs->moved[round % 3]) == 0) break;
    }
    const unsigned long long t1 = grid::globaltimer();
    if (ok) {
        unsigned long long looked = 0;  // edges, this thread's share
        // ---- hook.  With a giant component its vertices are done: an edge
        // that leaves the part reached is taken from its other end, and all of
        // the other vertices' edges are.  Without one, an edge is taken from
        // its larger end.
        // Four edges' labels are read together before any is hooked.
        auto edges = [&](const uint32_t *w, const uint32_t *v, const bool *on) {
            uint32_t lu[4], lv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool mine = on[u] && (giant || w[u] < v[u]);
                lu[u] = mine ? lab[w[u]] : 0u;
                lv[u] = mine ? __ldcg(lab + v[u]) : 0u;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (lu[u] != lv[u]) uf_hook(lab, lv[u], lu[u]);  // (their trees: nearly roots)
        };
        // rows above H.T edges: a lane looks whether a chunk's vertex is done,
        // the warp takes the chunks left
        for (uint64_t c0 = gw * 32; c0 < A.H.nchunks; c0 += nw * 32) {
            const uint64_t c = c0 + lane;
            uint32_t v = 0;
            uint64_t e0 = 0, e1 = 0;
            if (c < A.H.nchunks) {
                const uint32_t lo = A.H.crow[c];
                v = A.H.v[lo];
                if (!giant || A.level[v] == inf) {
                    e0 = A.off[v] + (c - A.H.first[lo]) * A.H.CH;
                    e1 = min(e0 + A.H.CH, A.off[v + 1]);
                }
            }
            looked += e1 - e0;
            for (unsigned todo = __ballot_sync(FULL, e0 < e1); todo; todo &= todo - 1) {
                const int j = __ffs(todo) - 1;
                const uint32_t vj = __shfl_sync(FULL, v, j);
                const uint64_t end = __shfl_sync(FULL, e1, j);
                for (uint64_t b = __shfl_sync(FULL, e0, j); b < end; b += 128) {
                    uint32_t w[4], from[4];
                    bool on[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        on[u] = b + 32 * u + lane < end;
                        w[u] = on[u] ? __ldg(A.adj + b + 32 * u + lane) : 0u;
                        from[u] = vj;
                    }
                    edges(w, from, on);
                }
            }
        }
        // the other rows: a warp per 32 vertices, their edges as one list.
        // Beside a giant component only vertices that the search's last pull
        // left open (all with edges, if it never pulled) are looked at, and
        // those outside it are kept for the last pass.
        const bool few = giant && A.st->cand_valid;
        const uint32_t *list = few ? A.cand[A.st->cand_cur] : A.nonisolated;
        const uint64_t nl = few ? A.st->cand_n[0] : nn;
        for (uint64_t i0 = gw * 32; i0 < nl; i0 += U * nw * 32) {
            uint32_t v[U];
            bool need[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint64_t i = i0 + u * nw * 32 + lane;
                need[u] = i < nl;
                v[u] = need[u] ? list[i] : 0u;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (giant && need[u]) need[u] = A.level[v[u]] == inf;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const unsigned who = __ballot_sync(FULL, need[u]);
                if (!who) continue;
                if (giant) {
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(&A.cs->nleft, (uint32_t)__popc(who));
                    at = __shfl_sync(FULL, at, 0) + __popc(who & ((1u << lane) - 1u));
                    if (need[u]) A.left[at] = v[u];
                }
                uint64_t beg = 0, deg = 0;
                if (need[u]) {
                    beg = A.off[v[u]];
                    deg = A.off[v[u] + 1] - beg;
                    if (deg > A.H.T) deg = 0;  // above
                }
                looked += deg;
                uint32_t incl = (uint32_t)deg;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= (uint32_t)o) incl += t;
                }
                const uint32_t total = __shfl_sync(FULL, incl, 31), excl = incl - (uint32_t)deg;
                for (uint32_t e0 = 0; e0 < total; e0 += 128) {  // warp-uniform
                    uint32_t w[4], from[4];
                    bool on[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t idx = e0 + 32 * k + lane;
                        uint32_t r = 0;  // the last lane whose row starts at or before idx
#pragma unroll
                        for (uint32_t step = 16; step; step >>= 1)
                            if (__shfl_sync(FULL, excl, r + step) <= idx) r += step;
                        const uint64_t b = __shfl_sync(FULL, beg, r);
                        const uint32_t x = __shfl_sync(FULL, excl, r);
                        from[k] = __shfl_sync(FULL, v[u], r);
                        on[k] = idx < total;
                        w[k] = on[k] ? __ldg(A.adj + b + (idx - x)) : 0u;
                    }
                    edges(w, from, on);
                }
            }
        }
        looked = dev::block_sum<unsigned long long, kCB>(looked);
        if (threadIdx.x == 0 && looked) atomicAdd(&A.cs->hooked, looked);
        ok = grid::sync(&A.cs->bar, epoch, A.timeout_ns);
    }
    if (!ok) {
        if (threadIdx.x == 0) {
            atomicOr(&A.st->err, DEV_ERR_TIMEOUT);
            if (A.rec) *(volatile unsigned int *)&A.rec->gave_up = 1u;
        }
        return;
    }
    // ---- finish: every label written once, by its own thread, with its root
    if (giant && __ldcg(lab + top) == top) {
        // (those reached have theirs, unless a search cut short left out a
        // smaller id of their component; isolated vertices keep their own)
        const uint32_t k = __ldcg(&A.cs->nleft);
        for (uint64_t i = tid; i < k; i += nth) {
            const uint32_t v = __ldcg(A.left + i);
            lab[v] = uf_root(lab, v);
        }
    } else {
        for (uint64_t v0 = tid; v0 < A.n; v0 += U * nth) {
            uint32_t l[U], p[U];
#pragma unroll
            for (int u = 0; u < U; ++u) l[u] = v0 + u * nth < A.n ? __ldcg(lab + v0 + u * nth) : 0u;
#pragma unroll
            for (int u = 0; u < U; ++u) p[u] = __ldcg(lab + l[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (v0 + u * nth < A.n && p[u] != l[u]) lab[v0 + u * nth] = uf_root(lab, p[u]);
        }
    }
    if (blockIdx.x != 0) return;
    if (threadIdx.x == 0) {
        PState *st = A.st;
        // CCv's road-network test: few zeros
        const bool road = (giant && top == 0 ? reached : 1ull) * 10 < (unsigned long long)A.n;
        // edges examined: the search's or, without a giant component, each
        // vertex's first one as well; then those of the hooks
        unsigned long long first = giant ? 0ull : nn;
        for (int i = 0; i < (A.searched ? st->iterations : 0); ++i) first += st->scanned[i];
        st->iterations = 2;
        st->reached_v = A.n;
        st->reached_e = A.m;
        st->variant[0] = GG_VAR_PULL_DENSE;
        st->variant[1] = road ? GG_VAR_HOOK : GG_VAR_PULL_DENSE;
        for (int i = 0; i < 2; ++i) {
            st->nactv[i] = A.n;
            st->nacte[i] = A.m;
        }
        st->scanned[0] = first;
        st->scanned[1] = __ldcg(&A.cs->hooked);
        st->t_ns[0] = t0;
        st->t_ns[1] = t1;
        st->t_ns[2] = st->t_end = grid::globaltimer();
        st->f_seen = 0;
    }
    if (!A.rec) return;
    __syncthreads();
    const uint4 *src = (const uint4 *)A.st;
    for (uint32_t i = threadIdx.x; i < sizeof(PState) / 16; i += kCB) ((uint4 *)&A.rec->st)[i] = src[i];
}

__global__ void k_cc_start(CcState *cs, PState *st, int searched) {
    if (!searched) {
        st->err = 0;
        st->reached_v = 0;
        st->exit_small = st->small_done = 0;
    }
    cs->bar.n = 0;
    cs->bar.err = 0;
    cs->smallest = 0xFFFFFFFFu;
    cs->nleft = 0;
    cs->moved[0] = cs->moved[1] = cs->moved[2] = 0;
    cs->hooked = 0;
}

// The search's buffers, its levels among them, and with them this run's.
static gg_status cc_resident_buffers(gg_graph *g) {
    bool search;
    GG_CHECK(bfs_resident_prepare(g, &search));
    if (!search) return GG_ERR_OOM;
    gg_prop *level;
    return run_tmp_prop(g, 1, GG_I32, &level);
}

// Whether CC of g with these options runs here, its buffers made: symmetric
// graphs with the threshold's choice of variants (which no pass here takes)
// and no per-step records wanted.  Not where the buffers do not fit in memory.
gg_status cc_resident_prepare(gg_graph *g, const gg_run_opts &opt, bool *ok) {
    const Tuning &t = tuning();
    *ok = false;
    if (!g->symmetric || g->n == 0 || !t.resident || !(t.persistent & 4) || t.cc_hook != 1 || (t.fusion & 4) ||
        g->force_iter >= 0 || opt.variant != GG_VAR_AUTO || opt.collect_stats ||
        (opt.threshold != GG_THRESH_DEFAULT && opt.threshold != GG_THRESH_FRAC))
        return GG_OK;
    const gg_status s = cc_resident_buffers(g);
    *ok = s == GG_OK;
    return resident_give_up(g, s);
}

// Enqueues the run with its records in `st` (and, with to_host, copied to the
// host); may be captured.
gg_status cc_resident_enqueue(gg_graph *g, gg_prop *label, PState *st, bool to_host) {
    gg_ctx *ctx = g->ctx;
    CcState *cs = (CcState *)resident_state(g, RUN_CC);
    CcArgs A;
    std::memset(&A, 0, sizeof(A));
    A.off = g->off;
    A.adj = g->adj;
    A.first_in = g->first_in;
    A.nonisolated = g->nonisolated;
    A.nonisolated_n = (const unsigned long long *)g->nonisolated_n;
    A.H = g->heavy;
    A.n = g->n;
    A.m = g->m;
    A.label = (uint32_t *)label->d;
    A.cs = cs;
    A.st = st;
    A.rec = to_host ? (CcRecord *)ctx->d_run : nullptr;
    A.timeout_ns = tuning().barrier_timeout_ns;
    gg_prop *level;
    GG_CHECK(run_tmp_prop(g, 1, GG_I32, &level));
    A.level = (const int32_t *)level->d;
    const double avg = (double)g->m / (double)g->n;
    A.searched = (double)g->maxdeg * avg * avg >= (double)kSearchLeast;
    if (A.searched) GG_CHECK(bfs_resident_search(g, level, g->maxdeg_v, kSearchSteps, kSearchLeast, st));
    A.cand[0] = g->cand.list[0];
    A.cand[1] = g->cand.list[1];
    A.left = g->tmp_front[0]->bins[0];
    k_cc_start<<<1, 1, 0, ctx->stream>>>(cs, st, A.searched);
    GG_LAUNCHED(ctx);
    // a CTA per 2048 vertices or 16384 edges, all that fit at most
    const uint64_t most = (uint64_t)ctx->sm_count * resident_ctas((const void *)k_cc_run, kCB);
    const uint64_t want = std::max<uint64_t>(std::max<uint64_t>(g->n / 2048, g->m / 16384), 1);
    void *args[] = {&A};
    GG_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)k_cc_run, dim3((unsigned)std::min(most, want)), dim3(kCB),
                                             args, 0, ctx->stream));
    ctx->launches++;
    return GG_OK;
}

gg_status cc_resident(gg_graph *g, gg_prop *label, gg_run_stats *stats, int *iters_out) {
    gg_ctx *ctx = g->ctx;
    if (!g->pstate) GG_CUDA(ctx, cudaMalloc(&g->pstate, sizeof(PState)));
    PState *st = (PState *)g->pstate;
    CcRecord &rec = *(CcRecord *)ctx->h_run;
    PState &hs = rec.st;
    hs.iterations = -1;  // written by the run's end
    rec.gave_up = 0;
    GG_CHECK(cc_resident_enqueue(g, label, st, true));
    GG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    // (the search's error word is in the records, which follow it on the stream)
    if (hs.iterations < 0 || rec.gave_up || (hs.err & DEV_ERR_TIMEOUT))
        return set_error(ctx, GG_ERR_TIMEOUT, "gg_cc: grid barrier timed out");
    *iters_out = hs.iterations;
    if (stats) {
        stats->vertices_reached = hs.reached_v;
        stats->edges_reached = hs.reached_e;
        for (int i = 0; i < hs.iterations; ++i) {
            stats->variant[i] = hs.variant[i];
            stats->nactv[i] = hs.nactv[i];
            stats->nacte[i] = hs.nacte[i];
            stats->scanned[i] = hs.scanned[i];
            stats->scanned_edges += hs.scanned[i];
            stats->iter_ms[i] = stats->kernel_ms[i] = (double)(hs.t_ns[i + 1] - hs.t_ns[i]) * 1e-6;
        }
    }
    return GG_OK;
}

}  // namespace gg
