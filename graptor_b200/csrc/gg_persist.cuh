// gg_persist.cuh -- what the device-driven traversals share: the frontier
// handed between them and the state block of a run.
#pragma once
#include "gg_internal.cuh"

namespace gg {

// BFS levels: a listed frontier of at most this many vertices and edges
// continues in the one-cluster kernel k_small_bfs
constexpr unsigned long long kSmallEnterV = 8192, kSmallEnterE = 65536;

struct PFront {
    uint32_t *bins[NBINS];
    uint32_t *bitmap;
    unsigned long long *cnt;  // FC_WORDS
};

struct PState {
    unsigned int bar_count;
    unsigned int bar_gen;
    unsigned int err;
    int iterations;
    int has_list[2];
    int all[2];
    unsigned long long cand_n[2];
    int cand_valid;
    int cand_cur;
    int variant[GG_MAX_ITERS];
    unsigned long long nactv[GG_MAX_ITERS];
    unsigned long long nacte[GG_MAX_ITERS];
    unsigned long long scanned[GG_MAX_ITERS];
    unsigned long long t_ns[GG_MAX_ITERS + 1];
    unsigned long long reached_v, reached_e;
    // timing collection: the forced iteration's input counts, its start and
    // end, and the end of the run (any iteration index)
    unsigned long long f_nactv, f_nacte, f_reached, f_t0, f_t1, t_end;
    int f_seen;
    unsigned long long zeros;  // CC: vertices labelled 0 after the first step
    // fused push work queue counters (reset between iterations), one
    // 128-byte line each so that claims, appends and completions do not
    // contend for one L2 line
    struct alignas(128) Line { unsigned long long v; };
    Line wq_head, wq_tail, wq_done;
    // small-frontier hand-over (BFS levels): the traversal left the frontier
    // at small_cur after small_iter iterations for k_small_bfs (exit_small),
    // which either finishes the run (small_done) or hands back the same way
    int exit_small, small_done, small_iter, small_cur;
    // learned policy: the next step's choice, taken by one warp of CTA 0
    // while the grid finishes the current step (slot = iteration & 1)
    int next_choice[2];
};

// Levels from the listed frontier st->small_cur of fr[] in one thread-block
// cluster until the run ends (st->small_done) or the frontier outgrows it
// (then it is listed in fr[st->small_cur] at iteration st->small_iter).
gg_status enqueue_small_bfs(gg_graph *g, PState *st, const PFront *fr, int32_t *level, int max_iters, int threshold,
                            int threshold_k);

}  // namespace gg
