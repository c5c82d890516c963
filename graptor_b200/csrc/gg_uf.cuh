// gg_uf.cuh -- connected components by min-id hooking.
//
// label[] is a forest: every label is the id of a vertex of the same
// component and never above the vertex's own id, so following labels ends at
// a vertex labelled with itself (a root).  Hooking an edge's two roots, the
// larger under the smaller (compare-and-swap on the larger root), and
// repeating until they agree merges the trees; the root of a component is
// then its minimum id, the CCv label.  Finds halve paths with plain stores
// (a label only ever moves to an ancestor, so racing stores stay valid).
#pragma once
#include "gg_internal.cuh"

namespace gg {

__device__ __forceinline__ uint32_t uf_find(uint32_t *lab, uint32_t x) {
    for (int guard = 0; guard < (1 << 26); ++guard) {  // a chain of n links at most
        const uint32_t p = __ldcg(lab + x);
        if (p == x) return x;
        const uint32_t gp = __ldcg(lab + p);
        if (gp != p) lab[x] = gp;
        x = gp;
    }
    return x;
}

__device__ __forceinline__ void uf_hook(uint32_t *lab, uint32_t u, uint32_t v) {
    uint32_t ru = uf_find(lab, u), rv = uf_find(lab, v);
    for (int guard = 0; ru != rv && guard < (1 << 26); ++guard) {
        const uint32_t lo = ru < rv ? ru : rv, hi = ru ^ rv ^ lo;
        const uint32_t old = atomicCAS(lab + hi, hi, lo);
        if (old == hi) break;
        ru = uf_find(lab, old);
        rv = uf_find(lab, lo);
    }
}

// The root of x without path halving: in the final pass every vertex's
// entry is written once, by its own thread, with its root; a halving store
// from another thread's walk could land after it and leave a non-root there.
__device__ __forceinline__ uint32_t uf_root(const uint32_t *lab, uint32_t x) {
    for (int guard = 0; guard < (1 << 26); ++guard) {  // a chain of n links at most
        const uint32_t p = __ldcg(lab + x);
        if (p == x) return x;
        x = p;
    }
    return x;
}

}  // namespace gg
