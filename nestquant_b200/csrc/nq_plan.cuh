// The pass list of the prefill GEMM, built on the device without a host sync.
#pragma once
#include "nq_format.cuh"
#include "nq_scan.cuh"

namespace nq {

constexpr int kPfTokens = 384;                       // most tokens per pass (accumulator columns)
struct PfPass { int expert, row0, ntok, pad; };

// A pass = one expert x up to 384 of its pairs (pairs are sorted by expert); experts at level 0 get none.  plan: [0] passes,
// [1] pairs covered, then PfPass records from int 4 on, in expert order.
//   WINDOW = false  from[e] = routed pairs of expert e, in the order of the pair list; the plan covers the whole list
//   WINDOW = true   from[e] = first pair of expert e in the sorted list (from[E] = end of the last expert's pairs); the plan covers
//                   the pairs [pair0, pair0 + npairs) with rows counted from pair0
// from: global or shared memory; s_warp: 32 ints.  One CTA of kPlanThreads, a thread per expert: sums over the CTA (passes before the expert,
// pairs before it) place every record.  One thread that walks the experts alone pays two dependent loads for each of them.
constexpr int kPlanThreads = 1024;

template <bool WINDOW>
__device__ __forceinline__ void plan_passes(const int* from, const int64_t* table, int E, int pair0, int npairs, int* plan, int max_passes,
                                            int* s_warp)
{
    PfPass* out = (PfPass*)(plan + 4);
    int n = 0, rows = 0, covered = 0;     // passes, pairs and covered pairs of the experts handled so far
    for (int e0 = 0; e0 < E; e0 += kPlanThreads)
    {
        const int e = e0 + (int)threadIdx.x;
        int first = 0, c = 0, total;
        bool live = false;
        if (e < E)
        {
            live = table[(int64_t)e * kTableWidth] > 0;
            if constexpr (WINDOW)
            {
                const int a = max(from[e], pair0), b = min(from[e + 1], pair0 + npairs);
                first = a - pair0; c = b - a;
            }
            else c = from[e];
        }
        if constexpr (!WINDOW)
        {
            first = rows + cta_exclusive_sum(c, s_warp, total);
            rows += total;
        }
        const int np = live && c > 0 ? (c + kPfTokens - 1) / kPfTokens : 0;
        const int at = n + cta_exclusive_sum(np, s_warp, total);
        const int kept = max(min(np, max_passes - at), 0);
        for (int i = 0; i < kept; ++i)
        {
            PfPass ps;
            ps.expert = e; ps.row0 = first + i * kPfTokens; ps.ntok = min(c - i * kPfTokens, kPfTokens); ps.pad = 0;
            out[at + i] = ps;
        }
        n = min(n + total, max_passes);
        cta_exclusive_sum(kept > 0 ? min(c, kept * kPfTokens) : 0, s_warp, total);
        covered += total;
    }
    if (threadIdx.x == 0) { plan[0] = n; plan[1] = covered; plan[2] = plan[3] = 0; }
}

}  // namespace nq
