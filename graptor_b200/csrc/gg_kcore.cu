// gg_kcore.cu -- the k-core peel as one cooperative launch.
//
// KC_bucket's peel (bench/KC_bucket.C:290-420) is a chain of about a thousand
// small steps (R-MAT 20: 651 peel steps on 204 floors).  Driven from the host
// each step cost a launch, a wait for the frontier's counts and the frontier's
// conversions: 29 us, of which the edges took a few.  Here a resident grid
// runs all of it, one grid barrier per step:
//   scan of floor L : the alive vertices whose count is L are peeled, those
//                     above stay alive, the smallest count left is kept;
//   peel step       : the rows of the vertices peeled by the phase before are
//                     counted down towards L; the take that brings a vertex
//                     to L peels it (its row is the next step's work).
// A peeled row becomes items (gg_items.cuh), so that a step's work spreads
// over all warps whatever the rows' lengths (the late floors of R-MAT peel a
// few hubs of thousands of edges).  Every vertex is peeled once, so the item
// arrays are only ever appended to.
//
// A phase's counters (items, vertices at the floor and above) live in one of
// three slots used in turn: phase q adds to slot q mod 3 and clears slot q+1
// mod 3, which every CTA read before it entered phase q-1's barrier, so a
// slow CTA never reads a counter that a fast one already moves on.
//
// R-MAT 20 (n 2^20, m 31 M): 24.4 -> 6.3 ms, 7.4 us a phase, of which 5 us are
// the barrier and the chain of dependent accesses (item, edge, count, take,
// row bounds, append) that the smallest graphs show.
#include <algorithm>
#include <cstring>

#include "gg_grid.cuh"
#include "gg_internal.cuh"
#include "gg_items.cuh"

namespace gg {

constexpr int kKcBlock = 512;

struct alignas(128) KcSlot {
    unsigned long long items[IT_KINDS];  // appended
    unsigned long long at, above;      // scan: vertices at the floor, above it
    unsigned long long min_above;      // scan: smallest count above it
};

struct KcState {
    grid::Arrivals bar;
    KcSlot slot[3];
    unsigned long long many;  // vertices of degree above one
    uint32_t floors, steps, largest;
};

static_assert(sizeof(KcState) <= kRunState, "state block");

struct KcArgs {
    const uint64_t *off;
    const uint32_t *adj;
    uint32_t n;
    uint32_t *count;
    uint32_t *alive[2];
    ItemLists items;
    KcState *st;
    unsigned long long timeout_ns;
};

__global__ void __launch_bounds__(kKcBlock, 2) k_kc_run(KcArgs A) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ unsigned long long s_items[kKcBlock / 32][ItemLister::STAGED][ItemAppender::CAP];
    __shared__ uint32_t s_alive[kKcBlock / 32][128];
    KcState *st = A.st;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * kKcBlock) >> 5;
    const uint64_t gw = ((uint64_t)blockIdx.x * kKcBlock + threadIdx.x) >> 5;
    const bool first_thread = blockIdx.x == 0 && threadIdx.x == 0;
    unsigned long long epoch = 0;
    unsigned long long head[IT_KINDS] = {0, 0, 0};  // items of the phases before the last one
    uint32_t q = 0, floors = 0, steps = 0, largest = 0;
    uint64_t L = 0, na = A.n;
    int cur = -1;  // alive list in use; -1: every vertex

    ItemLister lister;
    lister.init(s_items[wib]);
    // d loses one while it is above the floor; true for the take that brings
    // it there.  A take that finds it at the floor already (others took it
    // meanwhile) is given back; counts stay below 2^31, so one read as
    // negative has been carried below the floor for a moment.
    auto take = [&](uint32_t d) -> bool {
        if ((uint64_t)__ldcg(A.count + d) <= L) return false;
        const uint32_t old = atomicSub(A.count + d, 1u);
        if ((int32_t)old < 0 || (uint64_t)old <= L) {
            atomicAdd(A.count + d, 1u);
            return false;
        }
        return (uint64_t)old == L + 1;
    };
    auto record = [&](bool rec, uint32_t d) {
        if (!__any_sync(FULL, rec)) return;
        uint64_t b = 0, dg = 0;
        if (rec) {
            b = A.off[d];
            dg = A.off[d + 1] - b;
        }
        lister.list(rec, b, dg);
    };
    auto begin = [&](KcSlot *out) {
        if (first_thread) {
            KcSlot *next = &st->slot[(q + 1) % 3];
            next->items[0] = next->items[1] = next->items[2] = next->at = next->above = 0;
            next->min_above = ~0ull;
        }
        lister.begin(A.items, head, out->items);
    };

    for (;;) {
        // ---- scan of floor L
        KcSlot *out = &st->slot[q % 3];
        begin(out);
        {
            const uint32_t *alive = cur < 0 ? nullptr : A.alive[cur];
            dev::WarpAppender<128> keep{s_alive[wib], 0, A.alive[cur < 0 ? 0 : cur ^ 1], &out->above};
            unsigned long long at_n = 0;
            uint32_t mn = 0xFFFFFFFFu;
            for (uint64_t base = gw * 32; base < na; base += nw * 32) {
                const uint64_t i = base + lane;
                uint32_t v = 0;
                bool at = false, above = false;
                uint64_t beg = 0, deg = 0;
                if (i < na) {
                    v = alive ? __ldcg(alive + i) : (uint32_t)i;
                    const uint32_t c = __ldcg(A.count + v);
                    at = c == L;
                    above = c > L;
                    if (at) {
                        beg = A.off[v];
                        deg = A.off[v + 1] - beg;
                    }
                    if (above) mn = min(mn, c);
                }
                at_n += at;
                if (__any_sync(FULL, at)) lister.list(at, beg, deg);
                keep.push(above, v);
            }
            lister.flush();
            keep.flush();
            mn = __reduce_min_sync(FULL, mn);
            if (lane == 0 && mn != 0xFFFFFFFFu) atomicMin(&out->min_above, (unsigned long long)mn);
            at_n = dev::block_sum<unsigned long long, kKcBlock>(at_n);
            if (threadIdx.x == 0 && at_n) atomicAdd(&out->at, at_n);
        }
        if (!grid::sync(&st->bar, epoch, A.timeout_ns)) return;
        ++q;
        ++floors;
        const unsigned long long at = __ldcg(&out->at), above = __ldcg(&out->above);
        const unsigned long long smallest = __ldcg(&out->min_above);
        unsigned long long ns = __ldcg(&out->items[IT_SHORT]), nl = __ldcg(&out->items[IT_LONG]),
                           nh = __ldcg(&out->items[IT_HUGE]);
        cur = cur < 0 ? 0 : cur ^ 1;
        na = above;
        if (at == 0) {
            if (above == 0) break;
            L = smallest;  // no vertex at this floor: the next count that exists
            continue;
        }
        largest = (uint32_t)L;
        // ---- peel steps at floor L
        while (ns || nl || nh) {
            out = &st->slot[q % 3];
            const unsigned long long *is = A.items.p[IT_SHORT] + head[IT_SHORT], *il = A.items.p[IT_LONG] + head[IT_LONG],
                                     *ih = A.items.p[IT_HUGE] + head[IT_HUGE];
            head[IT_SHORT] += ns;
            head[IT_LONG] += nl;
            head[IT_HUGE] += nh;
            begin(out);
            // up to kLong edges from `first`, all in flight
            auto piece = [&](uint64_t first, uint32_t len) {
                const uint32_t *row = A.adj + first;
                constexpr int U = kLong / 32;
                uint32_t d[U];
                bool rec[U];
#pragma unroll
                for (int u = 0; u < U; ++u) d[u] = 32 * u + lane < len ? __ldg(row + 32 * u + lane) : 0u;
#pragma unroll
                for (int u = 0; u < U; ++u) rec[u] = 32 * u + lane < len && take(d[u]);
#pragma unroll
                for (int u = 0; u < U; ++u) record(rec[u], d[u]);
            };
            for (uint64_t i = blockIdx.x; i < nh; i += gridDim.x) {
                const unsigned long long it = __ldcg(ih + i);
                const uint32_t len = item_len(it);
                for (uint32_t o = wib * kLong; o < len; o += (kKcBlock / 32) * kLong)
                    piece(item_first(it) + o, min(kLong, len - o));
            }
            const uint32_t parts = long_pieces(nl, nw), width = kLong / parts;
            for (uint64_t i = gw; i < nl * parts; i += nw) {
                const unsigned long long it = __ldcg(il + i / parts);
                const uint32_t len = item_len(it), o = (uint32_t)(i % parts) * width;
                if (o < len) piece(item_first(it) + o, min(width, len - o));
            }
            const uint32_t group = short_group(ns, nw);
            for (uint64_t base = gw * group; base < ns; base += nw * group) {
                unsigned long long it = 0;
                if (lane < group && base + lane < ns) it = __ldcg(is + base + lane);
                dev::warp_flat_rows<4>(
                    A.adj, item_first(it), item_len(it), 0u, [&](uint32_t d, uint32_t) { return take(d); }, record);
            }
            lister.flush();
            if (!grid::sync(&st->bar, epoch, A.timeout_ns)) return;
            ++q;
            ++steps;
            ns = __ldcg(&out->items[IT_SHORT]);
            nl = __ldcg(&out->items[IT_LONG]);
            nh = __ldcg(&out->items[IT_HUGE]);
        }
        if (above == 0) break;
        ++L;
    }
    // KC_bucket's rule for isolated vertices (k_kc_isolated)
    if (__ldcg(&st->many) < (unsigned long long)(A.n / 2)) {
        for (uint64_t v = (uint64_t)blockIdx.x * kKcBlock + threadIdx.x; v < A.n; v += (uint64_t)gridDim.x * kKcBlock)
            if (A.off[v + 1] == A.off[v]) A.count[v] = 1u;
        largest = max(largest, 1u);
    }
    if (first_thread) {
        st->floors = floors;
        st->steps = steps;
        st->largest = largest;
    }
}

// count = degree; `many` counts the vertices of degree above one
__global__ void __launch_bounds__(256) k_kc_start(const uint64_t *__restrict__ off, uint32_t n,
                                                  uint32_t *__restrict__ count, KcState *st) {
    unsigned long long k = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t deg = off[v + 1] - off[v];
        count[v] = deg > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)deg;
        k += deg > 1;
    }
    k = dev::block_sum<unsigned long long, 256>(k);
    if (threadIdx.x == 0 && k) atomicAdd(&st->many, k);
}

gg_status resident_memory(gg_graph *g) {
    if (!g->resident) GG_CUDA(g->ctx, cudaMalloc(&g->resident, resident_state_at(g, RUN_KINDS)));
    return GG_OK;
}

// The whole peel of g into count[] (g->n entries, alive lists allocated).
// *ran = false, and nothing done, where its buffers do not fit in memory.
gg_status kcore_resident(gg_graph *g, uint32_t *count, bool *ran, uint32_t *largest, int *steps, int *floors) {
    gg_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    *ran = false;
    const gg_status fit = resident_memory(g);
    if (fit != GG_OK) return resident_give_up(g, fit);
    KcState *st = (KcState *)resident_state(g, RUN_KCORE);
    KcArgs A;
    A.off = g->off;
    A.adj = g->adj;
    A.n = g->n;
    A.count = count;
    A.alive[0] = g->kc_alive[0];
    A.alive[1] = g->kc_alive[1];
    A.items = item_lists(g);
    A.st = st;
    A.timeout_ns = tuning().barrier_timeout_ns;
    KcState init;
    std::memset(&init, 0, sizeof(init));
    init.slot[0].min_above = ~0ull;
    GG_CUDA(ctx, cudaMemcpyAsync(st, &init, sizeof(init), cudaMemcpyHostToDevice, s));
    k_kc_start<<<(unsigned)std::min<uint64_t>((g->n + 255ull) / 256, (uint64_t)ctx->sm_count * 8), 256, 0, s>>>(
        g->off, g->n, count, st);
    GG_LAUNCHED(ctx);
    // A CTA per 16384 edges, 8 at least and one per SM at most: each of the
    // thousand barriers costs more with more CTAs (R-MAT 20: 7.6 ms with 148,
    // 8.5 with 296, 8.8 with 37; R-MAT 16: 2.7 with 37 to 111, 3.3 with 222)
    const uint64_t most = (uint64_t)ctx->sm_count * std::min(1, resident_ctas((const void *)k_kc_run, kKcBlock));
    const unsigned ctas = (unsigned)std::min(most, std::max<uint64_t>(8, g->m / 16384));
    void *args[] = {&A};
    GG_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)k_kc_run, dim3(ctas), dim3(kKcBlock), args, 0, s));
    ctx->launches++;
    KcState fin;
    GG_CUDA(ctx, cudaMemcpyAsync(&fin, st, sizeof(fin), cudaMemcpyDeviceToHost, s));
    GG_CUDA(ctx, cudaStreamSynchronize(s));
    if (fin.bar.err) return set_error(ctx, GG_ERR_TIMEOUT, "gg_kcore: grid barrier timed out");
    *ran = true;
    *largest = fin.largest;
    *steps = (int)fin.steps;
    *floors = (int)fin.floors;
    return GG_OK;
}

}  // namespace gg
