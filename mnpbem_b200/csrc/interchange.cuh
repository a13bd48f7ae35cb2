// Interchanges of an LU panel composed into a gather (FP64 and FP32 strips).
#pragma once
#include "common.cuh"

namespace mnpb {
namespace swp {

// ---------------------------------------------------------------------------
// Row interchanges.  A sequence of interchanges (c, p_c), c ascending, p_c >= c,
// is composed into a gather before any row moves: row c ends with the value
// that row p_c held just before step c, which is V(c') of the last earlier
// step c' with the same target, or the original row p_c; V(c), the value of
// row c before step c, is V of the last earlier step that targeted c, or the
// original row c.  Steps with one target are chained (next), so each step
// walks the few that share its target instead of all that precede it.
// Shared memory: head of every target row met, by its slot.
// ---------------------------------------------------------------------------
constexpr int SWN = 128;   // interchanges composed by one CTA

struct Swaps {             // in shared memory
    int p[SWN];            // target of step c, relative to the first step's row
    int par[SWN];          // last earlier step that targeted row c, or -1
    int out[SWN];          // row (relative) whose value ends in row c
    int tail[SWN];         // for the last step of a target below the steps' own rows:
                           // the row whose value ends there; else -1
};

// compose steps [0, ns), ns <= SWN <= blockDim.x, one thread a step; ends with a barrier
__device__ __forceinline__ void compose(Swaps &w, const int32_t *ipiv, int base, int ns) {
    const int c = threadIdx.x;
    if (c < ns) w.p[c] = ipiv[c] - base;
    __syncthreads();
    const int t = c < ns ? w.p[c] : -1;
    int par = -1, prev = -1;              // last earlier step with target c / target t
    bool last = t >= ns;
    for (int e = 0; e < ns; ++e) {
        const int pe = w.p[e];
        if (e < c) {
            if (pe == c && e != c) par = e;
            if (pe == t) prev = e;
        } else if (e > c && pe == t) {
            last = false;
        }
    }
    if (c < ns) w.par[c] = par;
    __syncthreads();
    if (c < ns) {
        auto before = [&](int e) {        // V(e)
            while (w.par[e] >= 0) e = w.par[e];
            return e;
        };
        w.out[c] = t == c ? before(c) : prev >= 0 ? before(prev) : t;
        w.tail[c] = last ? before(c) : -1;
    }
    __syncthreads();
}

}  // namespace swp
}  // namespace mnpb
