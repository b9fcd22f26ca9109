// Prefill path, the permutation: the (token, pick) pairs of a window sorted by expert, as a stable counting sort in one kernel
// (up to 8,192 picks and 369 experts, whose counts fit into 48 KB of shared memory) or three, and without a host sync.
//
// Replaces the host side of the reference's prefill (sm120/moe.py:293-298: torch.argsort of the flattened expert ids,
// scatter_add for the counts, a .cpu() of the counts) and this library's earlier use of the same torch operators.
//   bins     expert id 0 .. E - 1, plus bin E for the picks that contribute nothing (id outside [0, E), expert not resident
//            on this GPU, routing weight 0): they sort behind every real pair and no kernel touches their rows.
//   slices   a warp owns up to 256 consecutive picks.  Pass 1 counts its picks per bin; pass 2 turns the counts into the
//            offset of every (slice, bin) and the size of every bin; pass 3 walks the slice again, 32 picks at a time in pick
//            order, and places each pick at start[bin] + offset[slice][bin] + its rank among the slice's earlier picks of that
//            bin (match.any gives the lanes of a step that share a bin).  Equal experts keep pick order: the result does
//            not depend on timing, nor on where the slices are cut.
// Everything here is latency (65,536 picks are 0.7 MB), so every pass loads independently: with pass 2 as one CTA whose threads
// walked the slices, and a pass list written by one thread, sort and pass list of the full layer (256 experts) took 80 us
// longer at 8,000 picks and 130 us longer at 65,536 (whole prefill call, same GPU).
// Outputs: pe[p] = expert (or E) and pt[p] = token of sorted pair p, pos[t * topk + k] = sorted index of a pick,
// start[0 .. E + 1] = first pair of each bin (start[E] = number of live pairs, start[E + 1] = all pairs), and, optionally,
// the routing-hit counts of this call (every pick with a valid id and a non-zero weight, whatever the expert's level) added
// to a device array that the caller zeroed.
#include <cuda_fp16.h>

#include "nq_common.cuh"
#include "nq_format.cuh"
#include "nq_plan.cuh"

namespace nq {

constexpr int kSortSlice = 256;      // picks per warp
constexpr int kSortWarps = 8;        // warps per CTA
constexpr int kSortMaxBins = 1025;   // experts + 1
constexpr size_t kSortSmallShared = 48 * 1024 - 256;      // the one-kernel form stays within the default shared memory of a CTA

__device__ __forceinline__ int pick_bin(const int64_t* sel, const __half* rw, const int64_t* table,
                                        int E, int i, bool* hit)
{
    const int64_t e = sel[i];
    const bool valid = e >= 0 && e < E && __half2float(rw[i]) != 0.f;
    *hit = valid;
    return valid && table[e * kTableWidth] > 0 ? (int)e : E;
}

// pass 1: hist[slice][bin] (and hits[e] += picks with a weight)
__global__ void __launch_bounds__(32 * kSortWarps) sort_count_kernel(const int64_t* sel, const __half* rw,
                                                                    const int64_t* table, int P, int E, int* hist, int* hits)
{
    launch_dependents();
    grid_dependency_wait();
    extern __shared__ int s_hist[];      // [kSortWarps][E + 1]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slice = blockIdx.x * kSortWarps + warp, nb = E + 1;
    int* h = s_hist + warp * nb;
    for (int b = lane; b < nb; b += 32) h[b] = 0;
    __syncwarp();
    const int i0 = slice * kSortSlice;
    for (int i = i0 + lane; i < i0 + kSortSlice && i < P; i += 32)
    {
        bool hit;
        const int b = pick_bin(sel, rw, table, E, i, &hit);
        atomicAdd(h + b, 1);
        if (hits && hit) atomicAdd(hits + (int)sel[i], 1);
    }
    __syncwarp();
    if (i0 < P)
        for (int b = lane; b < nb; b += 32) hist[(size_t)slice * nb + b] = h[b];
}

// pass 2: hist[slice][bin] -> picks of the bin in earlier slices; the row of slice 0, whose offsets are zero, takes the size of
// the bin instead.  A CTA takes 32 bins (a lane each), its 32 warps equal runs of slices: every load is independent.
__global__ void __launch_bounds__(1024) sort_offset_kernel(int* hist, int nslices, int E)
{
    launch_dependents();
    grid_dependency_wait();
    __shared__ int s_sum[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = E + 1, b = blockIdx.x * 32 + lane;
    const int per = (nslices + 31) / 32, s0 = warp * per, s1 = min(s0 + per, nslices);
    int sum = 0;
    if (b < nb)
#pragma unroll 8
        for (int s = s0; s < s1; ++s) sum += __ldcg(hist + (size_t)s * nb + b);
    s_sum[warp][lane] = sum;
    __syncthreads();
    int run = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 32; ++w)
    {
        const int v = s_sum[w][lane];
        run += w < warp ? v : 0;
        total += v;
    }
    if (b >= nb) return;
    for (int s = s0; s < s1; ++s)
    {
        const int c = __ldcg(hist + (size_t)s * nb + b);
        hist[(size_t)s * nb + b] = s ? run : total;
        run += c;
    }
}

// size[b] -> s_start[b] = picks of earlier bins, s_start[nb] = all picks; whole CTA.  size and s_start may be the same array.
// GLOBAL: size is an array that the kernel before this one both read and wrote (its CTAs share lines of it), so it comes from L2, not from what
// that kernel left in this SM's L1.
template <bool GLOBAL>
__device__ __forceinline__ void scan_bins(const int* size, int nb, int* s_start, int* s_warp)
{
    auto at = [&](int b) { return GLOBAL ? __ldcg(size + b) : size[b]; };
    const int per = (nb + (int)blockDim.x - 1) / (int)blockDim.x, b0 = (int)threadIdx.x * per, b1 = min(b0 + per, nb);
    int sum = 0, total;
    for (int b = b0; b < b1; ++b) sum += at(b);
    int run = cta_exclusive_sum(sum, s_warp, total);
    for (int b = b0; b < b1; ++b) { const int c = at(b); s_start[b] = run; run += c; }
    if (threadIdx.x == 0) s_start[nb] = total;
    __syncthreads();
}

// 32 picks of a warp (pick i of bin b per lane; lanes without one: b < 0 and different from every other lane's) take their
// places: nx[bin] = next free place of the bin for this warp
__device__ __forceinline__ void place_picks(int* nx, int b, int i, int topk, int lane, int* pe, int* pt, int* pos)
{
    const unsigned same = __match_any_sync(0xffffffffu, b);
    const int rank = __popc(same & ((1u << lane) - 1u));
    int p = 0;
    if (b >= 0) p = nx[b] + rank;
    __syncwarp();
    if (b >= 0 && rank == __popc(same) - 1) nx[b] = p + 1;                     // the last lane of each bin moves the bin on
    __syncwarp();
    if (b >= 0) { pe[p] = b; pt[p] = i / topk; pos[i] = p; }
}

// pass 3: place every pick.  Every CTA adds up the bin sizes itself (row 0 of hist); CTA 0 writes them out as start.
__global__ void __launch_bounds__(32 * kSortWarps) sort_place_kernel(const int64_t* sel, const __half* rw,
                                                                    const int64_t* table, int P, int E, int topk,
                                                                    const int* hist, int* start, int* pe, int* pt, int* pos)
{
    launch_dependents();
    grid_dependency_wait();
    extern __shared__ int s_next[];      // [kSortWarps][E + 1]: next free place of each bin for this slice
    __shared__ int s_start[kSortMaxBins + 1], s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slice = blockIdx.x * kSortWarps + warp, nb = E + 1;
    scan_bins<true>(hist, nb, s_start, s_warp);
    if (blockIdx.x == 0)
        for (int b = threadIdx.x; b <= nb; b += blockDim.x) start[b] = s_start[b];
    int* nx = s_next + warp * nb;
    const int i0 = slice * kSortSlice;
    if (i0 >= P) return;                 // warp-uniform
    for (int b = lane; b < nb; b += 32) nx[b] = s_start[b] + (slice ? __ldcg(hist + (size_t)slice * nb + b) : 0);
    __syncwarp();
    for (int base = i0; base < i0 + kSortSlice && base < P; base += 32)
    {
        const int i = base + lane;
        bool hit;
        place_picks(nx, i < P ? pick_bin(sel, rw, table, E, i, &hit) : -1 - lane, i, topk, lane, pe, pt, pos);
    }
}

// The three passes in one CTA of 32 warps, the counts in shared memory: up to 32 slices (8,192 picks).  A slice is a multiple of
// 32 picks, no longer than needed, and a lane keeps its picks' bins in registers between the passes.  If the whole list is one chunk, its
// pass list too.
constexpr int kSortSmallPicks = 32 * kSortSlice;
__global__ void __launch_bounds__(1024) sort_small_kernel(const int64_t* sel, const __half* rw,
                                                          const int64_t* table, int P, int E, int topk, int* start, int* hits,
                                                          int* pe, int* pt, int* pos, int* plan, int max_passes)
{
    launch_dependents();
    grid_dependency_wait();
    extern __shared__ int s_hist[];      // [32][E + 1] counts, then next free places; [E + 2] bin sizes, then starts
    __shared__ int s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = E + 1;
    const int slice = (P + 1023) / 1024 * 32, i0 = warp * slice;
    int* h = s_hist + warp * nb;
    int* s_start = s_hist + 32 * nb;
    int bin[kSortSlice / 32];
    for (int b = lane; b < nb; b += 32) h[b] = 0;
#pragma unroll
    for (int j = 0; j < kSortSlice / 32; ++j)
    {
        const int i = i0 + 32 * j + lane;
        bin[j] = -1 - lane;
        if (32 * j < slice && i < P)
        {
            bool hit;
            bin[j] = pick_bin(sel, rw, table, E, i, &hit);
            if (hits && hit) atomicAdd(hits + (int)sel[i], 1);
        }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kSortSlice / 32; ++j)
        if (bin[j] >= 0) atomicAdd(h + bin[j], 1);
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += blockDim.x)
    {
        int run = 0;
#pragma unroll 8
        for (int w = 0; w < 32; ++w) { const int c = s_hist[w * nb + b]; s_hist[w * nb + b] = run; run += c; }
        s_start[b] = run;
    }
    __syncthreads();
    scan_bins<false>(s_start, nb, s_start, s_warp);
    for (int b = threadIdx.x; b <= nb; b += blockDim.x) start[b] = s_start[b];
    for (int b = lane; b < nb; b += 32) h[b] += s_start[b];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kSortSlice / 32; ++j)
        if (32 * j < slice) place_picks(h, bin[j], i0 + 32 * j + lane, topk, lane, pe, pt, pos);
    if (plan) plan_passes<true>(s_start, table, E, 0, P, plan, max_passes, s_warp);
}

// the sort, and the pass list of the whole window if plan is given
int sort_pairs(const int64_t* sel, const void* rw, const int64_t* table, int T, int topk, int E, int32_t* pe, int32_t* pt, int32_t* pos, int32_t* start,
               int32_t* hits, int32_t* scratch, int scratch_ints, int32_t* plan, int plan_ints, void* stream)
{
    NQ_REQUIRE(T >= 0 && topk >= 1 && E >= 1 && E + 1 <= kSortMaxBins, "nq_pf_sort: T = %d, topk = %d, E = %d", T, topk, E);
    NQ_REQUIRE((long long)T * topk <= 0x7fffffffLL, "nq_pf_sort: too many pairs");
    const int P = T * topk;
    NQ_REQUIRE(start, "nq_pf_sort: null start array");
    cudaStream_t st = (cudaStream_t)stream;
    if (P == 0) return cudaMemsetAsync(start, 0, sizeof(int32_t) * (E + 2), st) == cudaSuccess ? NQ_OK : fail(NQ_ERR_CUDA, "nq_pf_sort: memset failed");
    NQ_REQUIRE(sel && rw && table && pe && pt && pos && scratch, "nq_pf_sort: null pointer");
    NQ_REQUIRE(scratch_ints >= nq_pf_sort_scratch_ints(P, E), "nq_pf_sort: scratch needs %d ints", nq_pf_sort_scratch_ints(P, E));
    const size_t small = sizeof(int) * (33 * (size_t)(E + 1) + 1);
    if (P <= kSortSmallPicks && small <= kSortSmallShared)
    {
        launch_dependent(sort_small_kernel, dim3(1), dim3(1024), small, st, sel, (const __half*)rw, table, P, E, topk, start, hits, pe, pt, pos, plan, (plan_ints - 4) / 4);
        return check_launch("nq_pf_sort");
    }
    const int slices = (P + kSortSlice - 1) / kSortSlice, ctas = (slices + kSortWarps - 1) / kSortWarps;
    const size_t smem = sizeof(int) * kSortWarps * (E + 1);
    launch_dependent(sort_count_kernel, dim3(ctas), dim3(32 * kSortWarps), smem, st, sel, (const __half*)rw, table, P, E, scratch, hits);
    if (int e = check_launch("nq_pf_sort(count)")) return e;
    launch_dependent(sort_offset_kernel, dim3((E + 1 + 31) / 32), dim3(1024), 0, st, scratch, slices, E);
    if (int e = check_launch("nq_pf_sort(offset)")) return e;
    launch_dependent(sort_place_kernel, dim3(ctas), dim3(32 * kSortWarps), smem, st, sel, (const __half*)rw, table, P, E, topk, scratch, start, pe, pt, pos);
    if (int e = check_launch("nq_pf_sort(place)")) return e;
    return plan ? nq_pf_plan_window(start, table, E, 0, P, plan, plan_ints, stream) : NQ_OK;
}

}  // namespace nq

extern "C" {

int nq_pf_sort_scratch_ints(int pairs, int E)
{
    if (pairs < 0 || E < 1) return 0;
    const long long slices = ((long long)pairs + nq::kSortSlice - 1) / nq::kSortSlice;
    const long long n = slices * (E + 1);
    return n > 0x7fffffffLL ? 0 : (int)n;
}

int nq_pf_sort(const int64_t* sel, const void* rw, const int64_t* table, int T, int topk, int E, int32_t* pe, int32_t* pt, int32_t* pos,
               int32_t* start, int32_t* hits, int32_t* scratch, int scratch_ints, void* stream)
{
    return nq::sort_pairs(sel, rw, table, T, topk, E, pe, pt, pos, start, hits, scratch, scratch_ints, nullptr, 4, stream);
}

}  // extern "C"
