// Decode path of the MoE layer (1..32 tokens): routing, input rotation, gate|up GEMV + SwiGLU, down GEMV + combine, in
// ONE persistent launch of one 640-thread CTA per SM.
//
// Replaces moe_forward() of the reference (sm120/nqmoe.cu:858-907 and the kernels it launches, :375-824).  Every routing,
// level and pointer decision is read on the device (graph-capturable).
//
//   route      every CTA groups the picks into runs (one expert + the tokens that picked it, level 4 first) in its own
//              shared memory: no CTA waits for another one's routing.
//   lists      the 16 x 128 units of the runs, in storage order, form two lists, gate|up and down, that every CTA goes through in
//              this order.  (Two lists per phase, each of half of the runs, would hide the hand-over of h, but their rows,
//              barriers and cuts cost more than that: 1 token of the full layer 132 us against 117, 4 tokens 379 against 369,
//              7 tokens over 90 experts at H = 2048, I = 640 101 against 75.)
//   shares     a list is cut by cost into one share per CTA, at piece boundaries (a piece = 16-row strip x k-slice), and a share
//              into one range per warp, at unit boundaries.  The cut points follow from the run list, so a CTA computes its
//              own: no queue, and a warp walks a contiguous range of each plane.  (A share whose token rows do not fit into
//              shared memory is worked off in several jobs.)
//   rows       the token rows a job multiplies with sit in shared memory: for gate|up x * su -> WHT128 -> fp16, computed by every
//              CTA for the runs of its share (1 to 2 rows of a 1-token call), for down copies of h; both in the k order the
//              lanes read (see "operand order").
//   units      a warp decodes a unit in registers and feeds mma.m16n8k16 with the run's tokens as N.  A piece that spans warps is
//              added up in warp order through shared memory.  The last piece of a (run, 128-column group) of gate|up to arrive
//              sums the k-slices in a fixed order and applies WHT128, sv, SwiGLU, su_d, WHT128 -> h (fp16); the last piece of
//              a (token, 128-row group) of down combines out[b] = sum_k rw * sv_o * WHT128(y).
//   waits      down jobs need h of their runs (one counter per run), a piece that spans warps needs the following warps'
//              first units.  CTAs draw their shares from counters and leave a list only when no share of it is left, so
//              whatever a warp waits for is in the hands of a running CTA, however many CTAs are resident (with all of them
//              resident each draws one share of every list).  The waits are bounded all the same (2 s, then status[0] = 1
//              and the launch drains).
//   operand order   inside a 128-wide chunk the fp16 element k = 16 T + 2 t4 + 8 hi + e sits at position 32 t4 + 4 T + 2 hi + e,
//              so lane (g, t4) finds the B fragments of all 8 k-steps of a unit in 64 contiguous bytes.
// Split-k partial sums go to separate buffers and are added in a fixed order, so results are bitwise repeatable
// (the reference accumulates with fp32 atomics and is not, sm120/check.py:21).  The cut points follow from all picks of a call, so the
// order in which a token's fp32 sums are added, and with it its last bits, depend on what the other tokens of the call picked; they do not
// depend on timing nor on how many CTAs are resident.
//
// Bound: the integer decode.  A loop that does nothing but decode and multiply units from registers runs at 382 clocks per
// unit and SM sub-partition at level 2 and 645 at level 4 (the multiplies and byte sums on the FMA-heavy pipe, half rate,
// are 320 and 576 of them, 8 legacy MMAs that overlap with nothing 64), whatever the number of warps from 8 on; HBM would
// allow 70 and 140.
#include "nq_common.cuh"
#include "nq_rotate.cuh"
#include "nq_unit.cuh"

namespace nq {

// residual window codes built into the decode-path kernel (bit c = code c; code 0 always)
#ifndef NQ_GEMV_CODES
#define NQ_GEMV_CODES 0x3FF
#endif
// One CTA of 20 warps per SM, 96 registers per thread.  Clocks per unit and sub-partition of the unit loop (level 2 / level 4 with
// residual code 0 / 7) on data in L2: 408 / 662 / 677 with 20 warps; 432 / 681 / 769 with 16 warps of 128 registers; 24 warps
// of 80 registers gain under 2 %.  Token fragments read through L1 instead of shared memory: 424 / 694 / 732, through a
// generic pointer 449 / 712 / 746; copied per unit through a cp.async ring, as an earlier version of this kernel did,
// 530 / 777 / 802.
constexpr int kWarps = 20, kThreads = 32 * kWarps;
static_assert(kThreads >= NQ_MAX_PICKS, "the run list is built by one thread per pick");
// Shared memory of the CTA: route, slots, token rows.  It stays below 164 KB, which leaves 64 KB of L1: registers that the
// decoder functions save live in local memory.  With 224 KB calls take 2 to 4 us more (1 token of the full layer 117.7 -> 119.5,
// 4 tokens 368.6 -> 375.2, 16 tokens of a small layer 65.1 -> 68.3).
constexpr int kGemvSmem = 160 * 1024;
constexpr int kRunTiles = 4;     // most column tiles (8 tokens each) of mma.m16n8k16 per run
constexpr int kTileFloats = 4 * 32;      // accumulators of a column tile
constexpr int kRowStep = 272;    // a token row in shared memory: 256 bytes per chunk, 272 from chunk to chunk (the eight chunks that
                                 // a warp stores at once fall on different banks)
constexpr unsigned long long kWaitNs = 2000000000ull;
constexpr int kEpRanks = 8, kEpTokens = NQ_MAX_TOKENS, kEpGroups = 64;   // limits of the in-kernel all-reduce

struct RunRec { int expert, level, first, count; };   // picks of the run: order[first .. first + count)

struct MoeArgs
{
    const __half* x; const int64_t* sel; const __half* rw;
    int B, topk, E, H, I, nm_gu, nm_dn, force_level, ks_gu, ks_dn, which;
    int run_cap, slot_floats;    // most tokens of a run (their rows fit into shared memory), floats of a slot
    const int64_t* table;
    int* status;       // [0] != 0: a device-side wait ran out
    float* part_gu;    // [ks_gu][S][2I]
    __half* h;         // [S][I], operand order
    float* part_d;     // [ks_dn][S][H]
    int* cnt_gu;       // [S * I/128] (run, group) arrivals, [S * I/128] (run, 512-block) arrivals, [S] finished groups per run
    int* cnt_d;        // [B][H/128] (token, group) arrivals
    int* wq;           // [0], [2] shares drawn so far of gate|up and down, [1] CTAs that left ([3] unused)
    float* zd;         // [S][I/128][4] down low-rank partials
    float* out;        // [B][H]
    int* hits;         // optional [E] pick counters (may be host-mapped)
    // expert parallelism (world > 1): the all-reduce of the partial outputs runs inside this kernel, over peer memory
    int world, rank;
    float* recv[kEpRanks];   // every rank's receive buffer [2][world][32][H] fp32, as seen from this GPU
    int* rcnt[kEpRanks];     // every rank's arrival counters [2][32 * 64], as seen from this GPU
    int* epoch;              // this rank's call counter (device): its parity picks the half of recv / rcnt
};

// What a pick refers to.  The fields of the table row are fetched together, not one decision after the other.
struct Pick { int expert, level; const __half *scales, *lr; bool masked_gu, masked_dn; };
__device__ __forceinline__ bool read_pick(const MoeArgs& a, int s, Pick& p)
{
    const int64_t e = a.sel[s];
    const __half w = a.rw[s];
    if (e < 0 || e >= a.E) return false;
    const int64_t* row = a.table + e * kTableWidth;
    const int64_t lv = row[0], fg = row[4], fd = row[8], sc = row[9], lr = row[14];
    p.expert = (int)e; p.level = a.force_level > 0 ? a.force_level : (int)lv; p.scales = (const __half*)sc; p.lr = (const __half*)lr;
    p.masked_gu = fg != 0; p.masked_dn = fd != 0;
    return (int)lv > 0 && __half2float(w) != 0.f;
}

__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Arrival on a counter: publishes what the warp stored before it.  The one that finds itself last acquires (ld_acquire on the
// counter) before it reads what the others published; everybody else keeps its L1, which an acquire drops.
__device__ __forceinline__ int add_release(int* p, int v)
{
    int prev;
    asm volatile("atom.add.release.gpu.global.s32 %0, [%1], %2;" : "=r"(prev) : "l"(p), "r"(v) : "memory");
    return prev;
}
// Every lane polls (one broadcast transaction) until *p >= target; false = gave up (status raised by this or another warp).
// The polls are relaxed: an acquiring load drops the SM's L1, where the other warps find their token rows.
__device__ __forceinline__ int ld_relaxed(const int* p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool wait_counter(const int* p, int target, int* status)
{
    unsigned long long t0 = 0;
    for (uint32_t i = 0;; ++i)
    {
        if (ld_relaxed(p) >= target) { ld_acquire(p); return true; }
        if ((i & 63u) == 63u)
        {
            if (ld_relaxed(status) != 0) return false;
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            else if (t - t0 > kWaitNs) break;
        }
        __nanosleep(32);
    }
    atomicExch(status, 1);
    return false;
}

// ---------------------------------------------------------------- shared state of a CTA
// Relative cost of a unit, by which the lists are cut: measured clocks of the unit loop, 410 at level 2 and 690 at level 4, and 80
// for a further column tile (its 8 legacy MMAs are 64 of them, the reads of its fragments the rest).  A unit of a strip in mask mode costs 75
// more than its mix of refined and unrefined units (the loop decides unit by unit): without them, CTAs with masked experts took 455 us for a
// gate|up share that took the others 400 (8 tokens of the full layer, a third of the level-4 experts masked).
constexpr float kCostUnit = 410.f, kCostRefined = 280.f, kCostTile = 80.f, kCostMasked = 75.f;
constexpr int kLists = 2, kCachedRows = 2;
constexpr int kQueue = 64;       // finishers waiting in a CTA
// The units [at, stop) of list positions that this CTA is working on, and the token rows it needs for them.
struct Job
{
    int at, stop, end;               // this job; the end of the share
    int seq;                         // number of the job (of either list), not 0 once it is cut
    int run0, row0, nrows;           // first run, its first row's number, rows
    int bound[kWarps + 1];           // the warps' ranges
    int64_t row[kCachedRows][kTableWidth];   // table rows of run0 and the runs behind it
};
struct Shape
{
    int S, ng, ngH, KSg, KSd, nruns;
    int nu_gu, nu_dn;                // units per run of the two projections (0: that half is not wanted)
};
// What a warp does with (part of) a piece: read by the decoder functions.
struct StripJob
{
    ProjPlanes P;
    size_t nrec, res_nrec;           // records of the base and of the residual plane
    size_t unit0, res0;              // plane index of the first unit, of the strip's first refined unit
    unsigned long long flags;        // mask mode: refined chunks of the strip
    int c0, n;                       // first chunk, units
    uint32_t x;                      // shared-space address of the run's first token row
    int row_bytes, count;            // bytes from row to row, tokens of the run
    // what becomes of the sums: list (0 gate|up, 1 down), run, strip, k-slice, units of the piece behind the warp's range, whether it begins in it
    int l, r, strip, ks, left, starts;
};
// The state of a CTA, at the start of its shared memory.  (Reached through route(): the functions that are not inlined get
// neither pointers nor structures, which would go through local memory.)
struct Route
{
    MoeArgs a;
    Shape sh;
    int par;
    StripJob strip[kWarps];
    int key[NQ_MAX_PICKS];                // expert of a valid pick, else -1 - pick
    RunRec runs[NQ_MAX_PICKS];
    const __half* scales[NQ_MAX_PICKS];   // scale vector of a valid pick's expert
    const __half* lr[NQ_MAX_PICKS];       // its low-rank plane, or null
    short lead[NQ_MAX_PICKS];             // run ordinal (by first pick) -> its first pick
    short first_of[NQ_MAX_PICKS];         // first pick of a run -> offset of the run in order[]
    unsigned char lvl[NQ_MAX_PICKS], order[NQ_MAX_PICKS], nvalid[NQ_MAX_TOKENS];
    int warp_sum[NQ_MAX_PICKS / 32], nruns;
    float cost[2][NQ_MAX_PICKS];          // cost of one unit of a run (gate|up, down)
    float base[2][NQ_MAX_PICKS + 1];      // cost of the units before a run
    int ks[2];                            // k-slices per strip in use
    int draws[kLists], drawn[kLists];     // this CTA's first shares of the lists, and how many shares were drawn when it last looked
    __align__(16) float zg[NQ_MAX_PICKS][4];   // low-rank inputs x V_gu^T of the picks of this CTA's gate|up shares
    int slot_seq[kWarps];                 // job whose share of a piece is in the warp's slot
    int queue[kQueue], q_head, q_tail;    // finishers to be done, [q_head, q_tail) of them not taken yet (0: entry not written yet)
    int ended[kLists];                    // warps that are through with their ranges of the jobs of a list
    int share_tasks;                      // some run has more than one token: finishers go through the queue
    Job job[kLists];
};
constexpr int kRouteBytes = (sizeof(Route) + 127) / 128 * 128;
extern __shared__ __align__(128) uint8_t nq_gemv_smem[];      // Route, [2][kWarps][slot_floats], token rows
__device__ __forceinline__ Route& route() { return *(Route*)nq_gemv_smem; }
// slots of a warp: 0 its share of a piece that an earlier warp adds up (read before the next job starts), 1 the sums of its current
// piece; fragment order [tile][i][lane]
__device__ __forceinline__ float* slot_of(const Route& R, int which, int warp) { return (float*)(nq_gemv_smem + kRouteBytes) + (which * kWarps + warp) * R.a.slot_floats; }
__device__ __forceinline__ uint32_t rows_base(const Route& R) { return smem_addr(nq_gemv_smem) + kRouteBytes + 2 * kWarps * R.a.slot_floats * 4; }
__host__ __device__ constexpr int rows_room(int slot_floats) { return kGemvSmem - kRouteBytes - 2 * kWarps * slot_floats * 4; }

// quotient of small non-negative integers (a < 2^20) without the ~130 clocks of an integer division
__device__ __forceinline__ int quot(int a, int b) { return (int)__fdividef((float)a + 0.5f, (float)b); }
__device__ __forceinline__ int quot_any(int a, int b) { return a < (1 << 20) ? quot(a, b) : a / b; }

// Group the picks into runs: a run = one expert and up to run_cap of its picks in pick order; runs are numbered by first
// pick, then ordered level 4 before level 2.
__device__ __forceinline__ void set_costs(const MoeArgs& a, Route& R, int rank, const Pick& p, int count)
{
    const int C[2] = {a.H / 128, a.I / 128}, nm[2] = {a.nm_gu, a.nm_dn};
#pragma unroll
    for (int d = 0; d < 2; ++d)
    {
        const bool masked = d ? p.masked_dn : p.masked_gu;
        const float refined = p.level < 4 ? 0.f : masked ? fminf(__fdividef((float)nm[d], (float)C[d]), 1.f) : 1.f;
        R.cost[d][rank] = kCostUnit + kCostRefined * refined + (p.level >= 4 && masked ? kCostMasked : 0.f) + kCostTile * (float)((count - 1) >> 3);
    }
}
// up to 32 picks, none of them more than run_cap times the same expert (false otherwise): one warp, a lane per pick
__device__ __forceinline__ bool build_route_warp(const MoeArgs& a, Route& R, int lane)
{
    const int S = a.B * a.topk;
    Pick p{-1, 0, nullptr, nullptr, false, false};
    const bool tv = lane < S && read_pick(a, lane, p);
    const unsigned valid = __ballot_sync(0xffffffffu, tv), below = (1u << lane) - 1u;
    const unsigned same = __match_any_sync(0xffffffffu, tv ? p.expert : -1 - lane);
    const int pos = __popc(same & below), count = __popc(same), leader = __ffs(same) - 1;
    if (__any_sync(0xffffffffu, count > a.run_cap)) return false;
    const bool lead = tv && pos == 0;
    const unsigned lead4 = __ballot_sync(0xffffffffu, lead && p.level >= 4), lead2 = __ballot_sync(0xffffffffu, lead && p.level < 4);
    const int rank = p.level >= 4 ? __popc(lead4 & below) : __popc(lead4) + __popc(lead2 & below), nruns = __popc(lead4 | lead2);
    // picks of the runs before this one: the leaders' counts, in run order, added up
    if (lead) R.first_of[rank] = (short)count;
    __syncwarp();
    const int mine_count = lane < nruns ? R.first_of[lane] : 0;
    int sum = mine_count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += u; }
    const int first = __shfl_sync(0xffffffffu, sum - mine_count, rank & 31);
    if (lead) { R.runs[rank] = RunRec{p.expert, p.level, first, count}; set_costs(a, R, rank, p, count); }
    const int base = __shfl_sync(0xffffffffu, first, leader);
    if (lane < S) { R.key[lane] = tv ? p.expert : -1 - lane; R.lvl[lane] = (unsigned char)p.level; R.scales[lane] = p.scales; R.lr[lane] = p.lr; }
    if (tv) R.order[base + pos] = (unsigned char)lane;
    if (lane < a.B)
    {
        const unsigned mine = a.topk >= 32 ? 0xffffffffu : ((1u << a.topk) - 1u) << (lane * a.topk);
        R.nvalid[lane] = (unsigned char)__popc(valid & mine);
    }
    if (lane == 0) R.nruns = nruns;
    return true;
}
// up to 256 picks: thread t = pick t; every thread of the CTA must call it
__device__ __forceinline__ void build_route_cta(const MoeArgs& a, Route& R)
{
    const int S = a.B * a.topk, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool in = t < NQ_MAX_PICKS;
    Pick p{-1, 0, nullptr, nullptr, false, false};
    const bool tv = t < S && read_pick(a, t, p);
    const int e = p.expert, lv = p.level;
    if (in) { R.key[t] = tv ? e : -1 - t; R.lvl[t] = (unsigned char)lv; R.scales[t] = p.scales; R.lr[t] = p.lr; }
    __syncthreads();
    int pos = 0, cnt = 0, first_pick = t;
    if (tv)
        for (int q = 0; q < S; ++q)
            if (R.key[q] == e) { if (cnt == 0) first_pick = q; ++cnt; pos += q < t; }
    const bool lead = tv && pos % a.run_cap == 0;
    const unsigned bal = __ballot_sync(0xffffffffu, lead);
    if (lane == 0 && in) R.warp_sum[warp] = __popc(bal);
    __syncthreads();
    int ord = __popc(bal & ((1u << lane) - 1u)), nruns = 0;
    for (int w = 0; w < NQ_MAX_PICKS / 32; ++w) { const int c = R.warp_sum[w]; ord += w < warp ? c : 0; nruns += c; }
    const int my_count = cnt - pos < a.run_cap ? cnt - pos : a.run_cap;
    if (lead) { R.lead[ord] = (short)t; R.first_of[t] = (short)my_count; }      // first_of holds the run's size until the ranks are known
    if (t == 0) R.nruns = nruns;
    __syncthreads();
    int rank = 0, first = 0;
    if (lead)
        for (int q = 0; q < nruns; ++q)
        {
            const int lp = R.lead[q], ol = R.lvl[lp];
            const bool before = ol > lv || (ol == lv && q < ord);
            rank += before; first += before ? (int)R.first_of[lp] : 0;
        }
    __syncthreads();
    if (lead) { R.runs[rank] = RunRec{e, lv, first, my_count}; R.first_of[t] = (short)first; set_costs(a, R, rank, p, my_count); }
    __syncthreads();
    if (tv)
    {
        int lp = first_pick;
        const int want = pos - pos % a.run_cap;
        if (want)                                   // an expert with more than one run: find the first pick of my run
            for (int q = 0, seen = 0; q < S; ++q)
                if (R.key[q] == e) { if (seen == want) { lp = q; break; } ++seen; }
        R.order[R.first_of[lp] + pos % a.run_cap] = (unsigned char)t;
    }
    if (t < a.B)
    {
        int n = 0;
        for (int k = 0; k < a.topk; ++k) n += R.key[t * a.topk + k] >= 0;
        R.nvalid[t] = (unsigned char)n;
    }
    __syncthreads();
}

// ---------------------------------------------------------------- GEMV
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Tokens of the run as the N operand: lane (g, t4) supplies k = 16 T + 2 t4 (+8) of token 8 nt + g, i.e. column g of the
// tile: 64 contiguous bytes per unit in shared memory, read 16 bytes per two k-steps.  A tile column without a token reads the
// run's first token instead: MMA columns are independent, so whatever is multiplied there lands in accumulators that are
// never stored.
template <int NT>
struct TokenSink
{
    float (&acc)[NT][4];
    const uint32_t (&x)[NT];     // shared-space address of this lane's 64 bytes per tile, at chunk 0
    uint32_t off;                // kRowStep * chunk
    uint4 (&b)[NT];              // fragments of k-steps T and T + 1 (T even)
    template <int T>
    __device__ __forceinline__ void operator()(std::integral_constant<int, T>, const uint32_t (&a)[4]) const
    {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
        {
            if constexpr ((T & 1) == 0) { b[nt] = lds128(x[nt] + off + T * 8); mma_16816(acc[nt], a, b[nt].x, b[nt].y); }
            else mma_16816(acc[nt], a, b[nt].z, b[nt].w);
        }
    }
};

// n units of one strip: stream, decode, multiply; the 16 x (8 NT) partial sums go to the warp's slot 1.  MODE 0: level 2, 1: level 4, 2: level 4 in
// mask mode (chunks without a flag decode as level 2).  The records of the next unit are fetched into registers while the
// current one is decoded.
// Not inlined on purpose: each of the decoder variants gets a register allocation of its own, and the caller's state is
// saved once per piece around the call instead of being squeezed into the unit loop (an inlined loop saves 10 to 35
// clocks per unit, a loop that shares its function with the piece bookkeeping loses 200 to spills).
template <int MODE, int RC, int BK, int NT>
__device__ __noinline__ void strip_gemv()
{
    const StripJob& J = route().strip[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, nxt = ring_successor(lane), n = J.n;
    RecordReader<BK> rb;
    rb.init(J.P.base, J.nrec, J.unit0, lane);
    rb.fetch();
    RecordReader<RC> rr;
    const int c0 = MODE == 2 ? J.c0 : 0;
    unsigned long long flags = 0;
    size_t res = 0;                                       // residual index of the first refined unit at or behind c0
    if constexpr (MODE == 1) res = J.res0 + J.c0;
    if constexpr (MODE == 2) { flags = J.flags; res = J.res0 + __popcll(flags & ((1ull << c0) - 1ull)); flags >>= c0; }
    if constexpr (MODE > 0)
    {
        rr.init(J.P.p4, J.res_nrec, res, lane);
        if (MODE == 1 || (flags & 1ull)) rr.fetch();
    }
    uint32_t x[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
    {
        const int j = nt * 8 + (lane >> 2);
        x[nt] = J.x + (j < J.count ? j : 0) * J.row_bytes + (lane & 3) * 64;
    }
    uint32_t off = J.c0 * kRowStep;
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[nt][i] = 0.f;
    for (int s = 0; s < n; s += 32)
    {
        // per-unit scalars of units s .. s + 31, one unit per lane: ring signs and block word (meta = word | signs << 16) and the
        // block word's multipliers
        uint32_t meta = 0, ac = 0;
        const int m = n - s < 32 ? n - s : 32;
        const uint32_t now = MODE == 2 ? (uint32_t)(flags >> s) : 0u;
        const unsigned long long after = MODE == 2 ? flags >> s >> 1 : 0ull;     // bit i: the unit behind unit s + i is refined
        if (lane < m)
        {
            if (J.P.var) meta = (uint32_t)__ldg(J.P.var + J.unit0 + s + lane) << 16;
            if (MODE == 1 || (MODE == 2 && (now >> lane & 1u)))
            {
                const size_t at = MODE == 1 ? res + s + lane : res + __popcll(flags & ((1ull << (s + lane)) - 1ull));
                const uint32_t word = __ldg(J.P.d4 + at) & 0xFFFFu;
                meta |= word;
                ac = block_multipliers(word);
            }
        }
#pragma unroll 1
        for (int i = 0; i < m; ++i)
        {
            uint32_t wb[Pattern<BK>::kWords + 2], wr[Pattern<RC>::kWords + 2];
            bool refined = MODE == 1;
            if constexpr (MODE == 2) refined = now >> i & 1u;
            rb.words(wb, lane);
            if constexpr (MODE > 0)
                if (refined) rr.words(wr, lane);
            if (s + i + 1 < n)
            {
                rb.fetch();
                if constexpr (MODE > 0)
                    if (MODE == 1 || ((uint32_t)after >> i & 1u)) rr.fetch();
            }
            continue_stream<Pattern<BK>::kBits>(wb, __shfl_sync(0xffffffffu, wb[0], nxt));
            const uint32_t um = __shfl_sync(0xffffffffu, meta, i), sign2 = sign_mask(um >> 16, lane);
            uint4 b[NT];
            const TokenSink<NT> sink{acc, x, off, b};
            if (MODE > 0 && refined)
            {
                if constexpr (MODE > 0)
                {
                    continue_stream<Pattern<RC>::kBits>(wr, __shfl_sync(0xffffffffu, wr[0], nxt));
                    decode_words<true, RC, BK>(wb, wr, consts_level4(__shfl_sync(0xffffffffu, ac, i), um, sign2), sink);
                }
            }
            else if constexpr (MODE != 1) decode_words<false, 0, BK>(wb, wr, consts_level2(sign2), sink);
            off += kRowStep;
        }
    }
    float* out = slot_of(route(), 1, threadIdx.x >> 5) + lane;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) out[(nt * 4 + i) * 32] = acc[nt][i];
}

// 4 consecutive elements k = 4 lane + i of a 128-chunk -> operand order (two 4-byte stores)
__device__ __forceinline__ void store4h_operand(__half* chunk, int lane, const float (&v)[4])
{
    const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    uint32_t* w = (uint32_t*)chunk + (lane & 1) * 32 + (lane >> 2) * 2 + ((lane & 3) >> 1);
    w[0] = *(const uint32_t*)&a;
    w[16] = *(const uint32_t*)&b;
}

// A list (d = 0 gate|up, 1 down): position p is unit p mod NU of run p / NU.
struct List { int d, C, NU, cps, NH; };        // chunks per strip, units per run, chunks per piece, units of a half (gate, up)
__device__ __forceinline__ List list_of(const MoeArgs& a, const Shape& sh, int d)
{
    List L;
    L.d = d;
    L.C = (d ? a.I : a.H) >> 7; L.NU = d ? sh.nu_dn : sh.nu_gu; L.NH = d ? L.NU : L.NU >> 1;
    const int KS = d ? sh.KSd : sh.KSg;
    L.cps = KS == 1 ? L.C : quot(L.C, KS);
    return L;
}

// ---------------------------------------------------------------- token rows
__device__ __forceinline__ void unpack4h(const uint2& w, float (&f)[4])
{
    const __half2 a = *(const __half2*)&w.x, b = *(const __half2*)&w.y;
    f[0] = __low2float(a); f[1] = __high2float(a); f[2] = __low2float(b); f[3] = __high2float(b);
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// Rows are numbered run by run: gate|up has the gate rows of a run's picks, then their up rows, down one row per pick.
__device__ __forceinline__ int row_id(const RunRec& run, int d, int up) { return d ? run.first : 2 * run.first + up * run.count; }
// The rows of a gate|up job.  A warp task = eight blocks of 128 of one row: lanes 4 v .. 4 v + 3 hold block v (wht128_x8, map H).
__device__ __forceinline__ void rotate_rows(const MoeArgs& a, const Shape& sh, const Route& R, const Job& job, uint32_t rows, int lane, int warp)
{
    const int oct = (sh.ngH + 7) >> 3, n = job.nrows * oct, q = lane & 3;
    int run = job.run0;
    for (int t = warp; t < n; t += kWarps)
    {
        const int p = quot(t, oct), blk = (t - p * oct) * 8 + (lane >> 2);
        while (job.row0 + p >= 2 * (R.runs[run].first + R.runs[run].count)) ++run;
        const RunRec rr = R.runs[run];
        const int at = job.row0 + p - 2 * rr.first, u = at >= rr.count ? 1 : 0, s = R.order[rr.first + at - u * rr.count];
        const bool live = blk < sh.ngH;
        float v[32];
        if (live)
        {
            uint32_t xw[16], sw[16];
            load16w_mapH(a.x + (size_t)quot(s, a.topk) * a.H + blk * 128, q, xw);
            load16w_mapH_align8(R.scales[s] + (u ? 2 * a.H + 3 * a.I : 0) + blk * 128, q, sw);
            mul32w(xw, sw, v);
        }
        else
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.f;
        wht128_x8(v, lane);
        if (!live) continue;
        // element 32 j + 8 q + 2 t4 + e of the block -> operand position 32 t4 + 8 j + 2 q + e
        const uint32_t dst = rows + (p * sh.ngH + blk) * kRowStep + 4 * q;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int t4 = 0; t4 < 4; ++t4)
            {
                const __half2 h = __floats2half2_rn(v[8 * j + 2 * t4], v[8 * j + 2 * t4 + 1]);
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + 64 * t4 + 16 * j), "r"(*(const uint32_t*)&h) : "memory");
            }
    }
}
// low-rank inputs x V_gu^T (unrotated input) of the picks of a gate|up job that ends in run `last`, a warp per pick
__device__ __forceinline__ void low_rank_inputs(const MoeArgs& a, Route& R, const Job& job, int last, int lane, int warp)
{
    const int p0 = R.runs[job.run0].first, p1 = R.runs[last].first + R.runs[last].count;
    for (int p = p0 + warp; p < p1; p += kWarps)
    {
        const int s = R.order[p];
        const __half* lr = R.lr[s];
        if (!lr) continue;
        const int rg = (int)a.table[(int64_t)R.key[s] * kTableWidth + 16];
        const __half* xr = a.x + (size_t)(s / a.topk) * a.H;
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int k = lane * 4; k < a.H; k += 128)
        {
            float f[4], w[4];
            load4h(xr + k, f);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < rg)
                {
                    load4h(lr + (size_t)q * a.H + k, w);
                    d[q] += f[0] * w[0] + f[1] * w[1] + f[2] * w[2] + f[3] * w[3];
                }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int o = 16; o; o >>= 1) d[q] += __shfl_xor_sync(0xffffffffu, d[q], o);
        if (lane == 0) *(float4*)R.zg[s] = make_float4(d[0], d[1], d[2], d[3]);
    }
}
// The rows of a down job: h of its runs, once they are complete.  A warp task = 512 bytes of a row.  false = the wait ran out.
__device__ __forceinline__ bool copy_rows(const MoeArgs& a, const Shape& sh, const Route& R, const Job& job, uint32_t rows, int lane, int warp)
{
    const int per = (sh.ng + 1) >> 1, n = job.nrows * per;
    int run = job.run0, seen = -1;
    for (int t = warp; t < n; t += kWarps)
    {
        const int p = quot(t, per), blk = (t - p * per) * 2 + (lane >> 4);
        while (job.row0 + p >= R.runs[run].first + R.runs[run].count) ++run;
        if ((a.which & 1) && run != seen)
        {
            if (!wait_counter(a.cnt_gu + 2 * sh.S * sh.ng + run, sh.ng * R.runs[run].count, a.status)) return false;
            seen = run;
        }
        if (blk < sh.ng)
        {
            const uint4 v = __ldcg((const uint4*)(a.h + (size_t)R.order[job.row0 + p] * a.I + blk * 128) + (lane & 15));
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(rows + (p * sh.ng + blk) * kRowStep + (lane & 15) * 16), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
        }
    }
    return true;
}

// ---------------------------------------------------------------- finishers
// (run, group) complete, token j of the run: WHT128, sv, (+ low rank), SwiGLU, su_d, WHT128 -> h.
__device__ __forceinline__ float4 sum_slices(const float* p, size_t stride, int KS)
{
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = 0; q < KS; ++q)
    {
        const float4 f = __ldcg((const float4*)(p + q * stride));
        v.x += f.x; v.y += f.y; v.z += f.z; v.w += f.w;
    }
    return v;
}
__device__ __noinline__ void finish_gate_up(int r, int grp, int j)
{
    const Route& R = route();
    const MoeArgs& a = R.a;
    const Shape& sh = R.sh;
    const int lane = threadIdx.x & 31;
    __syncwarp();        // the acquiring look at the queue or at the counter is ordered before every lane's loads below
    const RunRec run = R.runs[r];
    const int64_t* row = a.table + (int64_t)run.expert * kTableWidth;
    const int S = sh.S, N = 2 * a.I, KS = sh.KSg, ng = sh.ng;
    const size_t slice = (size_t)S * N;
    const int col = grp * 128 + lane * 4;
    const float* part = a.part_gu + col;
    const int slot = R.order[run.first + j];
    const float4 fg = sum_slices(part + (size_t)slot * N, slice, KS), fu = sum_slices(part + (size_t)slot * N + a.I, slice, KS);
    const __half* scales = R.scales[slot];
    const uint2 sv_g = *(const uint2*)(scales + a.H + col), sv_u = *(const uint2*)(scales + a.H + a.I + col),
                su_d = *(const uint2*)(scales + a.H + 2 * a.I + col);
    const __half* lr = R.lr[slot];
    const int rg = lr ? (int)row[16] : 0, rd = lr ? (int)row[17] : 0, hw = (int)row[18];
    const __half* lr4 = lr && run.level == 4 ? (const __half*)row[15] : nullptr;
    const float4 cur[2] = {fg, fu};
    float z[4] = {0.f, 0.f, 0.f, 0.f};
    if (rg)
    {
        const float4 f = *(const float4*)R.zg[slot];
        z[0] = f.x; z[1] = f.y; z[2] = f.z; z[3] = f.w;
    }
    float gu[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u)
    {
        float v[4] = {cur[u].x, cur[u].y, cur[u].z, cur[u].w}, sc[4];
        wht128(v, lane);
        unpack4h(u ? sv_u : sv_g, sc);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] *= sc[i];
        for (int q = 0; q < rg; ++q)
        {
            float u2[4], u4[4] = {0.f, 0.f, 0.f, 0.f};
            const size_t o = (size_t)(u * rg + q) * a.I + col;
            load4h(lr + (size_t)rg * a.H + o, u2);
            if (lr4) load4h(lr4 + o, u4);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] += z[q] * u2[i] + z[q] * u4[i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) gu[u][i] = v[i];
    }
    float v[4], sc[4];
    unpack4h(su_d, sc);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = silu(gu[0][i]) * gu[1][i];
    for (int q = 0; q < rd; ++q)          // this group's share of z_dn = sw V_dn^T
    {
        float w[4];
        load4h(lr + (size_t)rg * a.H + 2 * (size_t)rg * a.I + (size_t)q * a.I + col, w);
        float d = v[0] * w[0] + v[1] * w[1] + v[2] * w[2] + v[3] * w[3];
#pragma unroll
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (lane == 0) a.zd[((size_t)slot * ng + grp) * 4 + q] = d;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] *= sc[i];
    wht128(v, lane);
    if (hw <= 128) store4h_operand(a.h + (size_t)slot * a.I + grp * 128, lane, v);
    else __stcg((float4*)(a.part_gu + (size_t)slot * N + col), make_float4(v[0], v[1], v[2], v[3]));   // fp32 stage: gate columns, k-slice 0
    int done = 1;       // groups of this token whose h is now complete
    if (hw > 128)
    {
        // 512-wide rotation = H_4 (x) WHT128 / 2: the last of the hw/128 groups of a block combines their fp32 results
        const int nb = hw / 128, b0 = grp / nb * nb;
        __syncwarp();
        int last = 0;
        if (lane == 0)
        {
            int* ch = a.cnt_gu + (S + slot) * ng + b0;
            last = add_release(ch, 1) == nb - 1;
            if (last) { ld_acquire(ch); *ch = 0; }
        }
        last = __shfl_sync(0xffffffffu, last, 0);
        done = 0;
        if (last)
        {
            __syncwarp();
            const float rs = rsqrtf((float)nb);
            const float* p = a.part_gu + (size_t)slot * N + b0 * 128 + lane * 4;
            for (int ob = 0; ob < nb; ++ob)
            {
                float o[4] = {0.f, 0.f, 0.f, 0.f};
                for (int b = 0; b < nb; ++b)
                {
                    const float4 f = __ldcg((const float4*)(p + b * 128));
                    const float sg = (__popc(ob & b) & 1) ? -1.f : 1.f;
                    o[0] += sg * f.x; o[1] += sg * f.y; o[2] += sg * f.z; o[3] += sg * f.w;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) o[i] *= rs;
                store4h_operand(a.h + (size_t)slot * a.I + (b0 + ob) * 128, lane, o);
            }
            done = nb;
        }
    }
    if (done)
    {
        __syncwarp();
        if (lane == 0) add_release(a.cnt_gu + 2 * S * ng + r, done);
    }
}

// ---- all-reduce of the partial outputs inside the kernel (expert parallelism) --------------------------------------------
// Every rank computes, for each (token, 128-column group), the weighted sum over ITS experts.  It stores that slice into
// slot [parity][its rank][token] of every rank's receive buffer (plain peer stores over NVLink, its own buffer included),
// then adds 1 to the (token, group) arrival counter of every rank (release, system scope).  After its own pieces are done, a
// rank's warps take (token, group) tasks: wait until the counter shows all `world` slices (acquire; bounded), add the slices
// in rank order - every rank gets bitwise the same sums - and write out.  The parity of a per-rank call counter alternates
// two halves of the buffers: a rank can run at most one call ahead of a peer (it needs the peer's slices of call n to finish
// call n), so the slices of call n + 1 never land on slices of call n that are still being read.
__device__ __forceinline__ void ep_send(const MoeArgs& a, const Shape& sh, int par, int b, int grp, int lane, const float (&o)[4])
{
    const size_t at = (((size_t)par * a.world + a.rank) * kEpTokens + b) * a.H + grp * 128 + lane * 4;
    for (int p = 0; p < a.world; ++p) *(float4*)(a.recv[p] + at) = make_float4(o[0], o[1], o[2], o[3]);
    __syncwarp();       // the lanes' stores happen before the releasing adds below, which publish them (cumulativity)
    if (lane < a.world)
        asm volatile("red.release.sys.global.add.s32 [%0], 1;" ::"l"(a.rcnt[lane] + (par * kEpTokens + b) * kEpGroups + grp) : "memory");
}
// false = the wait ran out
__device__ __forceinline__ bool ep_sum(const MoeArgs& a, const Shape& sh, int par, int b, int grp, int lane)
{
    int* cnt = a.rcnt[a.rank] + (par * kEpTokens + b) * kEpGroups + grp;
    unsigned long long t0 = 0;
    for (uint32_t i = 0;; ++i)
    {
        int v;
        asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
        if (v >= a.world) break;
        if ((i & 31u) == 31u)
        {
            if (ld_acquire(a.status) != 0) return false;
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            else if (t - t0 > kWaitNs) { atomicExch(a.status, 1); return false; }
        }
        if (i > 8) __nanosleep(50);
    }
    __syncwarp();
    float o[4] = {0.f, 0.f, 0.f, 0.f};
    for (int p = 0; p < a.world; ++p)
    {
        const float4 v = __ldcg((const float4*)(a.recv[a.rank] + (((size_t)par * a.world + p) * kEpTokens + b) * a.H + grp * 128 + lane * 4));
        o[0] += v.x; o[1] += v.y; o[2] += v.z; o[3] += v.w;
    }
    *(float4*)(a.out + (size_t)b * a.H + grp * 128 + lane * 4) = make_float4(o[0], o[1], o[2], o[3]);
    __syncwarp();
    if (lane == 0) *cnt = 0;          // this half is next used two calls from now
    return true;
}

// output rows [grp * 128, +128) of token b are complete in every k-slice of every pick: weighted combine, four picks at a time
// (their loads and their rotations overlap).
__device__ __noinline__ void finish_down(int b, int grp)
{
    const Route& R = route();
    const MoeArgs& a = R.a;
    const Shape& sh = R.sh;
    const int lane = threadIdx.x & 31;
    __syncwarp();        // the acquiring look at the queue or at the counter is ordered before every lane's loads below
    const int N = a.H, KS = sh.KSd, col = grp * 128 + lane * 4, s0 = b * a.topk;
    const size_t slice = (size_t)sh.S * N;
    float o[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k0 = 0; k0 < a.topk; k0 += 4)
    {
        float v[4][4], w[4];
        uint2 sv[4];
        bool any_lr = false;
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const int s = s0 + k0 + i;
            const bool on = k0 + i < a.topk && R.key[s] >= 0;
            w[i] = on ? __half2float(a.rw[s]) : 0.f;
            sv[i] = on ? *(const uint2*)(R.scales[s] + a.H + 3 * a.I + col) : make_uint2(0u, 0u);
            const float4 f = on ? sum_slices(a.part_d + (size_t)s * N + col, slice, KS) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i][0] = f.x; v[i][1] = f.y; v[i][2] = f.z; v[i][3] = f.w;
            any_lr = any_lr || (on && R.lr[s] != nullptr);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) wht128(v[i], lane);
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            float sc[4];
            unpack4h(sv[i], sc);
#pragma unroll
            for (int e = 0; e < 4; ++e) v[i][e] *= sc[e];
        }
        if (any_lr)
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                const int s = s0 + k0 + i;
                if (k0 + i >= a.topk || R.key[s] < 0) continue;
                const __half* lr = R.lr[s];
                if (!lr) continue;
                const int64_t* erow = a.table + (int64_t)R.key[s] * kTableWidth;
                const int rd = (int)erow[17], rg = (int)erow[16], ng = sh.ng;
                const __half* lr4 = R.lvl[s] == 4 ? (const __half*)erow[15] : nullptr;
                const size_t ou = (size_t)rg * a.H + 2 * (size_t)rg * a.I + (size_t)rd * a.I;
                float z[4] = {0.f, 0.f, 0.f, 0.f};           // z_dn: the column groups' shares, a lane per group
                for (int gq = lane; gq < ng; gq += 32)
                {
                    const float* zp = a.zd + ((size_t)s * ng + gq) * 4;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (q < rd) z[q] += __ldcg(zp + q);
                }
                for (int q = 0; q < rd; ++q)
                {
                    float zq = q == 0 ? z[0] : q == 1 ? z[1] : q == 2 ? z[2] : z[3];
#pragma unroll
                    for (int m = 16; m; m >>= 1) zq += __shfl_xor_sync(0xffffffffu, zq, m);
                    float u2[4], u4[4] = {0.f, 0.f, 0.f, 0.f};
                    load4h(lr + ou + (size_t)q * a.H + col, u2);
                    if (lr4) load4h(lr4 + 2 * (size_t)rg * a.I + (size_t)q * a.H + col, u4);
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[i][e] += zq * u2[e] + zq * u4[e];
                }
            }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] += w[i] * v[i][e];
    }
    if (a.world > 1) ep_send(a, sh, R.par, b, grp, lane, o);
    else *(float4*)(a.out + (size_t)b * a.H + col) = make_float4(o[0], o[1], o[2], o[3]);
}

// The finishers of a CTA's pieces: one entry per token of a gate|up (run, group) or per down (token, group).  The warp whose piece
// arrives last puts them in, the warps that are through with their ranges take them out.  A finisher takes 3 to 11 us (chains of
// loads and shuffles beside 19 busy warps); done by that one warp for all tokens of the run, they held up its range, its CTA and
// whoever waits for the h: 24 tokens over 16 experts, H = 1024, I = 1280, low rank: 573 us per call against 148; 32 tokens
// over 16 experts, H = 4096: 325 against 310; 15 tokens over 54 experts, H = 896: 52 against 43.
// Calls in which no expert has two tokens gain nothing and do them in place; for one token (SHARE = false) the queue is not even
// compiled in, as its code alone costs 1 to 1.5 us.
constexpr int kTask = 1 << 30, kDownTask = 1 << 29;
__device__ __forceinline__ void finish_task(int t)
{
    if (t & kDownTask) finish_down(t >> 16 & 0xFF, t >> 8 & 0xFF);
    else finish_gate_up(t >> 16 & 0xFF, t >> 8 & 0xFF, t & 0xFF);
}
// every lane with `has` puts in its task; what does not fit is done here, and so is everything if the call does not share
template <bool SHARE>
__device__ __forceinline__ void put_tasks(Route& R, bool has, int task, int lane)
{
    const unsigned all = __ballot_sync(0xffffffffu, has);
    if (!all) return;
    __syncwarp();        // some lane's acquiring arrival is ordered before the releasing stores below
    int at = kQueue;
    if (SHARE && R.share_tasks)
    {
        if (lane == 0) at = atomicAdd(&R.q_tail, __popc(all));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(all & ((1u << lane) - 1u));
    }
    if (has && at < kQueue) asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_addr(&R.queue[at])), "r"(task) : "memory");
    unsigned left = __ballot_sync(0xffffffffu, has && at >= kQueue);
    while (left)
    {
        const int src = __ffs(left) - 1;
        left &= left - 1;
        finish_task(__shfl_sync(0xffffffffu, task, src));
    }
}
// lane 0: a task, 0 if there is none (or the next one is being written: its writer looks again when its range is through)
__device__ __forceinline__ int take_task(Route& R)
{
    int h = *(volatile int*)&R.q_head;
    for (;;)
    {
        const int tail = *(volatile int*)&R.q_tail;
        if (h >= (tail < kQueue ? tail : kQueue)) return 0;
        int t;
        asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(t) : "r"(smem_addr(&R.queue[h])) : "memory");
        if (!t) return 0;
        const int seen = atomicCAS(&R.q_head, h, h + 1);
        if (seen == h) return t;
        h = seen;
    }
}
// This warp is through with its range of list l's job: it takes finishers until no warp of the CTA can put in more (a barrier
// follows).
__device__ __noinline__ void do_tasks(int l)
{
    Route& R = route();
    const int lane = threadIdx.x & 31;
    int through = 0;
    unsigned long long t0 = 0;
    __syncwarp();
    if (lane == 0) through = (atomicAdd(&R.ended[l], 1) / kWarps + 1) * kWarps;
    for (uint32_t i = 0;; ++i)
    {
        int t = 0, more = 0;
        if (lane == 0)
        {
            more = *(volatile int*)&R.ended[l] < through;
            t = take_task(R);
        }
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t) { finish_task(t); continue; }
        if (!__shfl_sync(0xffffffffu, more, 0)) break;
        if ((i & 63u) == 63u)
        {
            // (leaving early is harmless: whoever puts in a task takes it out again if nobody else does.  A warp that gave up a
            // wait does not get here)
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            now = __shfl_sync(0xffffffffu, now, 0);
            if (t0 == 0) t0 = now;
            else if (now - t0 > kWaitNs) break;
            if (ld_relaxed(R.a.status) != 0) break;
        }
        __nanosleep(64);
    }
}
// empties the queue; one warp, between two barriers of the CTA with no finisher left
__device__ __forceinline__ void reset_queue(Route& R, int lane)
{
    for (int i = lane; i < kQueue; i += 32) R.queue[i] = 0;
    if (lane == 0) { R.q_head = 0; R.q_tail = 0; }
}

// ---------------------------------------------------------------- shares and jobs
// k-slices actually used, a divisor of the caller's: the fewest that keep the fullest CTA within 3 % of what any divisor
// gives it (every slice adds arrivals and partial sums; calls for one half of the layer use the caller's count, whose
// partial sums stay readable).  A lane per candidate; a count beyond 32 stands as it is.
__device__ __forceinline__ int choose_ksplit(int strips, int C, int ks, int ctas, int lane)
{
    if (ks == 1) return 1;
    const int d = lane + 1, q = quot(ks, d);
    int load = 0x7fffffff;
    if (ks <= 32 && q * d == ks)
    {
        const int share = quot_any(strips * d + ctas - 1, ctas) * quot(C, d);
        load = share < kWarps ? kWarps : share;
    }
    const int best = __reduce_min_sync(0xffffffffu, load);
    const unsigned good = __ballot_sync(0xffffffffu, load != 0x7fffffff && load * 32 <= best * 33);
    return good ? __ffs(good) : ks;
}
__device__ __forceinline__ Shape make_shape(const MoeArgs& a, int nruns)
{
    Shape sh;
    sh.S = a.B * a.topk; sh.ng = a.I >> 7; sh.ngH = a.H >> 7; sh.nruns = nruns;
    sh.nu_gu = (a.which & 1) ? (a.I >> 3) * sh.ngH : 0;
    sh.nu_dn = (a.which & 2) ? (a.H >> 4) * sh.ng : 0;
    sh.KSg = sh.KSd = 1;             // filled in once the lists are cut
    return sh;
}
// costs of the units before each run of phase d, by one warp
__device__ __forceinline__ void prefix_costs(const Shape& sh, Route& R, int d, float NU, int lane)
{
    float run = 0.f;
    for (int r0 = 0; r0 < sh.nruns; r0 += 32)
    {
        const int r = r0 + lane;
        const float own = r < sh.nruns ? R.cost[d][r] * NU : 0.f;
        float v = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
        if (r < sh.nruns) R.base[d][r] = run + v - own;
        run += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) R.base[d][sh.nruns] = run;
    __syncwarp();
}
// list position at which `cost` has been passed, rounded to whole steps of `step` units.  The
// arithmetic is approximate, but every CTA evaluates the same expression for the same cut.
__device__ __forceinline__ int position_at(const Route& R, const List& L, float cost, int step)
{
    const float* base = R.base[L.d];
    const int nruns = R.nruns;
    int lo = 0, hi = nruns;                      // base[lo] <= cost < base[hi + 1]
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= cost) lo = mid; else hi = mid - 1;
    }
    const int at = lo * L.NU;
    if (lo >= nruns) return at;
    const int n = __float2int_rn(__fdividef(cost - base[lo], R.cost[L.d][lo] * (float)step)) * step;
    return at + (n < 0 ? 0 : n < L.NU ? n : L.NU);
}
__device__ __forceinline__ float cost_at(const Route& R, const List& L, int p)
{
    const int r = quot_any(p, L.NU);
    return R.base[L.d][r] + (r < R.nruns ? (float)(p - r * L.NU) * R.cost[L.d][r] : 0.f);
}
// The job that starts at position `at` of the share in work, by one warp: how far its rows fit, the warps' ranges, the table rows
// of its first runs.
__device__ __forceinline__ void cut_job(const MoeArgs& a, const Shape& sh, Route& R, const List& L, Job& job, int at, int lane)
{
    int stop = job.end, run0 = 0, row0 = 0, nrows = 0;
    if (at < stop)
    {
        const int row_bytes = (L.d ? sh.ng : sh.ngH) * kRowStep, room = quot(rows_room(a.slot_floats), row_bytes);
        int h = quot_any(at, L.NH), up = L.d ? 0 : h & 1, run = L.d ? h : h >> 1;
        run0 = run; row0 = row_id(R.runs[run], L.d, up);
        for (; h * L.NH < stop; ++h)           // (run) or (run, gate / up) by (run, gate / up)
        {
            const int c = R.runs[run].count;
            if (nrows + c > room) { stop = h * L.NH; break; }
            nrows += c;
            if (L.d || up) { ++run; up = 0; } else up = 1;
        }
    }
    if (lane <= kWarps)
    {
        int g = at;
        if (at < stop)
        {
            const float ca = cost_at(R, L, at), cb = cost_at(R, L, stop);
            g = lane == 0 ? at : lane == kWarps ? stop : position_at(R, L, ca + (cb - ca) * ((float)lane / kWarps), 1);
            g = g < at ? at : g > stop ? stop : g;
        }
        job.bound[lane] = g;
    }
    if (at < stop)
        for (int i = lane; i < kCachedRows * kTableWidth; i += 32)
        {
            const int k = i / kTableWidth, run = run0 + k;
            if (run < R.nruns) job.row[k][i - k * kTableWidth] = a.table[(int64_t)R.runs[run].expert * kTableWidth + i - k * kTableWidth];
        }
    if (lane == 0)
    {
        job.at = at; job.stop = stop; job.seq += kLists;
        job.run0 = run0; job.row0 = row0; job.nrows = nrows;
    }
    __syncwarp();
}
// share k of a list (an empty one if k >= the number of CTAs), by one warp
__device__ __forceinline__ void cut_share(const MoeArgs& a, const Shape& sh, Route& R, const List& L, Job& job, int k, int lane)
{
    const float each = __fdividef(R.base[L.d][R.nruns], (float)gridDim.x);
    const bool any = k < (int)gridDim.x && L.NU > 0 && R.nruns > 0;
    const int A = any ? position_at(R, L, __fmul_rn(each, (float)k), L.cps) : 0;
    const int B = !any ? 0 : k + 1 == (int)gridDim.x ? R.nruns * L.NU : position_at(R, L, __fmul_rn(each, (float)(k + 1)), L.cps);
    if (lane == 0) job.end = B;
    __syncwarp();
    cut_job(a, sh, R, L, job, A < B ? A : B, lane);
}
// ---------------------------------------------------------------- a warp's share of a job
__device__ __forceinline__ int ld_slot_seq(const int* p)
{
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
// Part of a piece is through.  The warp in whose range the piece starts owns it: it adds the following warps' shares (if the
// piece goes on behind its range), stores the sums to part[ks][slot][row] and counts the piece; the others leave theirs in
// their slot (fragment order [tile][i][lane]).  false = a wait ran out.
template <int NT, bool SHARE>
__device__ __noinline__ bool piece_done()
{
    Route& R = route();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const StripJob& pc = R.strip[warp];
    const MoeArgs& a = R.a;
    const Shape& sh = R.sh;
    const Job& job = R.job[pc.l];
    const int g = lane >> 2, t4 = lane & 3, d = pc.l, N = d ? a.H : 2 * a.I;
    const RunRec run = R.runs[pc.r];
    float acc[NT][4];
    {
        const float* from = slot_of(R, 1, warp) + lane;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[nt][i] = from[(nt * 4 + i) * 32];
    }
    if (!pc.starts)
    {
        float* to = slot_of(R, 0, warp) + lane;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) to[(nt * 4 + i) * 32] = acc[nt][i];
        __syncwarp();
        if (lane == 0) asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_addr(&R.slot_seq[warp])), "r"(job.seq) : "memory");
        return true;
    }
    int left = pc.left;
    for (int v = warp + 1; left > 0 && v < kWarps; ++v)
    {
        const int n = job.bound[v + 1] - job.bound[v];
        if (n <= 0) continue;
        unsigned long long t0 = 0;
        for (uint32_t i = 0; ld_slot_seq(&R.slot_seq[v]) != job.seq; ++i)
            if ((i & 63u) == 63u)
            {
                if (ld_relaxed(a.status) != 0) return false;
                unsigned long long t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                if (t0 == 0) t0 = t;
                else if (t - t0 > kWaitNs) { atomicExch(a.status, 1); return false; }
            }
        __syncwarp();
        const float* from = slot_of(R, 0, v) + lane;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[nt][i] += from[(nt * 4 + i) * 32];
        left -= n;
    }
    float* part = (d ? a.part_d : a.part_gu) + (size_t)pc.ks * sh.S * N + pc.strip * 16 + g;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e)
        {
            const int j = nt * 8 + t4 * 2 + e;
            if (j < run.count)
            {
                float* to = part + (size_t)R.order[run.first + j] * N;
                __stcg(to, acc[nt][e]);
                __stcg(to + 8, acc[nt][e + 2]);
            }
        }
    // Every arrival below is a releasing atomic issued after this warp barrier: the barrier orders all lanes' partial-sum
    // stores before it, the release publishes them, the acquire of the last one to arrive sees everybody's.
    __syncwarp();
    int last = 0;
    if (!d)
    {
        const int half = a.I >> 4, grp = (pc.strip >= half ? pc.strip - half : pc.strip) >> 3;
        if (lane == 0)
        {
            int* cnt = a.cnt_gu + pc.r * sh.ng + grp;
            last = add_release(cnt, 1) == 2 * sh.KSg * 8 - 1;
            if (last) { ld_acquire(cnt); *cnt = 0; }
        }
        last = __shfl_sync(0xffffffffu, last, 0);
        put_tasks<SHARE>(R, last && lane < run.count, kTask | pc.r << 16 | grp << 8 | lane, lane);
    }
    else
    {
        // one arrival per token of the run on its (token, group) counter
        const int grp = pc.strip >> 3;
        int b = 0;
        if (lane < run.count)
        {
            b = quot(R.order[run.first + lane], a.topk);
            int* cnt = a.cnt_d + b * sh.ngH + grp;
            last = add_release(cnt, 1) == (int)R.nvalid[b] * sh.KSd * 8 - 1;
            if (last) { ld_acquire(cnt); *cnt = 0; }
        }
        put_tasks<SHARE>(R, last, kTask | kDownTask | b << 16 | grp << 8, lane);
    }
    return true;
}

// this warp's range of a job, piece by piece; false = a wait ran out
template <int NT, bool SHARE>
__device__ __forceinline__ bool run_piece(int mode, int rc, int bk)
{
#define NQ_RUN(RES, RCV, BKV) do { if (RES && mode == 2) strip_gemv<RES ? 2 : 0, RCV, BKV, NT>(); else strip_gemv<RES ? 1 : 0, RCV, BKV, NT>(); } while (0)
    NQ_WITH_CODES(mode > 0, rc, bk, NQ_GEMV_CODES, NQ_RUN);
#undef NQ_RUN
    return piece_done<NT, SHARE>();
}
template <bool SHARE>
__device__ __noinline__ bool run_job(int l)
{
    Route& R = route();
    const MoeArgs& a = R.a;
    const List L = list_of(a, R.sh, l);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Job& job = R.job[l];
    StripJob& J = R.strip[warp];
    const int d = L.d, row_bytes = ((d ? a.I : a.H) >> 7) * kRowStep, NS = (d ? a.H : 2 * a.I) >> 4;
    const uint32_t rows = rows_base(R);
    const int end = job.bound[warp + 1];
    bool ok = true;
    for (int at = job.bound[warp]; at < end;)
    {
        const int r = quot_any(at, L.NU), u = at - r * L.NU, s = quot(u, L.C), ch = u - s * L.C, up = u >= L.NH;
        const int ks = L.cps == L.C ? 0 : quot(ch, L.cps), stop = (ks + 1) * L.cps, n = stop - ch < end - at ? stop - ch : end - at;
        at += n;
        const RunRec run = R.runs[r];
        const int64_t* row = a.table + (int64_t)run.expert * kTableWidth;
        const bool cached = r - job.run0 < kCachedRows;
        const int64_t* crow = job.row[cached ? r - job.run0 : 0];
        const int rc = (int)(cached ? crow[10 + d] : row[10 + d]), bk = (int)((cached ? crow[19] : row[19]) >> (8 * d)) & 0xFF;
        const ProjPlanes P = cached ? planes_from_row(crow, d) : planes_from_row(row, d);
        const int mode = run.level < 4 ? 0 : P.flags ? 2 : 1, nm = mode == 2 ? (d ? a.nm_dn : a.nm_gu) : L.C;
        if (lane == 0)
        {
            J.P = P;
            J.nrec = (size_t)NS * L.C * 32; J.res_nrec = (size_t)NS * nm * 32;
            J.unit0 = (size_t)s * L.C + ch; J.res0 = (size_t)s * nm;
            J.flags = mode == 2 ? (unsigned long long)__ldg((const unsigned long long*)P.flags + s) : 0ull;
            J.c0 = ch; J.n = n;
            J.x = rows + (row_id(run, d, up) - job.row0) * row_bytes; J.row_bytes = row_bytes; J.count = run.count;
            J.l = l; J.r = r; J.strip = s; J.ks = ks; J.left = stop - ch - n; J.starts = ch == ks * L.cps;
        }
        __syncwarp();
        if (run.count <= 8) ok = run_piece<1, SHARE>(mode, rc, bk);
        else if (run.count <= 16) ok = run_piece<2, SHARE>(mode, rc, bk);
        else ok = run_piece<kRunTiles, SHARE>(mode, rc, bk);
        if (!ok) break;
        __syncwarp();
    }
    if (SHARE && R.share_tasks) do_tasks(l);
    return ok;
}
// the first unit of this warp's range on its way to L2, and the output scales of the strips of the job
__device__ __forceinline__ void prefetch_job(const MoeArgs& a, const Route& R, const List& L, const Job& job, int lane, int warp)
{
    const int at = job.bound[warp];
    if (at >= job.bound[warp + 1]) return;
    const int r = quot_any(at, L.NU), u = at - r * L.NU;
    const RunRec run = R.runs[r];
    const int64_t* row = r - job.run0 < kCachedRows ? job.row[r - job.run0] : a.table + (int64_t)run.expert * kTableWidth;
    const ProjPlanes P = planes_from_row(row, L.d);
    prefetch_l2((const uint8_t*)P.base + ((size_t)u * 32 + lane) * (kWideCodes >> (int)(row[19] >> (8 * L.d) & 0xFF) & 1 ? 16 : 8));
    if (run.level >= 4 && !P.flags) prefetch_l2(P.p4 + ((size_t)u * 32 + lane) * (kWideCodes >> (int)row[10 + L.d] & 1 ? 16 : 8));
    const __half* sc = (const __half*)row[9];
    const int col = quot(u, L.C) * 16;
    if (lane == 0) prefetch_l2(L.d ? sc + a.H + 3 * a.I + col : sc + a.H + col);
    if (lane == 1 && !L.d) prefetch_l2(sc + a.H + 2 * a.I + (col >= a.I ? col - a.I : col));
}

// one CTA per SM, warps independent of one another inside a job; SHARE: finishers may be shared (calls of two tokens or more)
template <bool SHARE>
__global__ void __launch_bounds__(kThreads, 1) moe_decode_kernel(const __grid_constant__ MoeArgs a)
{
    Route& R = route();
    __shared__ int s_small;
    launch_dependents();
    grid_dependency_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ctas = (int)gridDim.x, nwarps = ctas * kWarps;
    if (warp == kWarps - 1)
    {
        // this CTA's shares: one of each list that there is
        if (SHARE) reset_queue(R, lane);
        if (lane < kLists) { R.draws[lane] = (a.which >> lane & 1) ? atomicAdd(a.wq + 2 * lane, 1) : ctas; R.job[lane].seq = lane; R.ended[lane] = 0; }
        if (lane < kWarps) R.slot_seq[lane] = 0;
        for (int i = lane; i < (int)sizeof(MoeArgs) / 4; i += 32) ((int*)&R.a)[i] = ((const int*)&a)[i];
    }
    if (a.B * a.topk <= 32)
    {
        if (warp == 0)
        {
            const bool done = build_route_warp(a, R, lane);
            if (lane == 0) s_small = done;
        }
        __syncthreads();
    }
    else if (threadIdx.x == 0) s_small = 0;
    if (a.B * a.topk > 32 || !s_small) build_route_cta(a, R);
    Shape sh = make_shape(a, R.nruns);
    if (warp < kLists)
    {
        // a warp per list
        const int d = warp, ks = d ? a.ks_dn : a.ks_gu;
        const int use = a.which == 3 ? choose_ksplit(sh.nruns * (d ? a.H >> 4 : a.I >> 3), d ? sh.ng : sh.ngH, ks, ctas, lane) : ks;
        if (lane == 0) R.ks[d] = use;
        sh.KSg = sh.KSd = use;
        prefix_costs(sh, R, d, (float)(d ? sh.nu_dn : sh.nu_gu), lane);
        cut_share(a, sh, R, list_of(a, sh, d), R.job[d], R.draws[d], lane);
    }
    else if (SHARE && warp == kLists)
    {
        bool any = false;
        for (int r = lane; r < sh.nruns; r += 32) any = any || R.runs[r].count > 1;
        any = __any_sync(0xffffffffu, any);
        if (lane == 0) R.share_tasks = any;
    }
    __syncthreads();
    sh.KSg = R.ks[0]; sh.KSd = R.ks[1];
    const uint32_t rows = rows_base(R);
    if (threadIdx.x == 0) R.sh = sh;
    int drawn = 0;
    if (warp == kWarps - 1 && lane < kLists) drawn = ld_relaxed(a.wq + 2 * lane);      // (on its way while the rows are rotated)
    if (a.which & 1)
    {
        const Job& job = R.job[0];
        if (job.at < job.stop)
        {
            rotate_rows(a, sh, R, job, rows, lane, warp);
            low_rank_inputs(a, R, job, quot_any(job.stop - 1, sh.nu_gu), lane, warp);
        }
        prefetch_job(a, R, list_of(a, sh, 0), job, lane, warp);
    }
    if (blockIdx.x == 0 && a.hits && (int)threadIdx.x < sh.S)
    {
        const int64_t es = a.sel[threadIdx.x];
        if (es >= 0 && es < a.E && __half2float(a.rw[threadIdx.x]) != 0.f) atomicAdd(a.hits + es, 1);   // every pick with a weight, any level
    }
    const bool ep = a.world > 1 && a.which == 3;
    const int par = ep ? (*(volatile int*)a.epoch & 1) : 0;
    if (threadIdx.x == 0) R.par = par;
    const int gw = warp * ctas + (int)blockIdx.x;    // tasks below are dealt out CTA by CTA
    // rows of tokens none of whose picks is resident here are defined as zero (nothing else writes them); under expert
    // parallelism this rank's slice of such a token is a zero slice, sent like any other
    if (a.which & 2)
    {
        if (!ep)
        {
            for (int b = blockIdx.x; b < a.B; b += ctas)
                if (R.nvalid[b] == 0)
                    for (int i = threadIdx.x; i < a.H; i += kThreads) a.out[(size_t)b * a.H + i] = 0.f;
        }
        else
        {
            const float zero[4] = {0.f, 0.f, 0.f, 0.f};
            for (int task = gw; task < a.B * sh.ngH; task += nwarps)
                if (R.nvalid[task / sh.ngH] == 0) ep_send(a, sh, par, task / sh.ngH, task % sh.ngH, lane, zero);
        }
    }
    if (warp == kWarps - 1 && lane < kLists) R.drawn[lane] = drawn;
    __syncthreads();
    bool ok = true, ready = a.which & 1;      // the rows of the first gate|up job are
#pragma unroll 1
    for (int l = 0; l < kLists; ++l)
    {
        if (!(a.which >> l & 1) || sh.nruns == 0) continue;
        const List L = list_of(a, sh, l);
        Job& job = R.job[l];
        for (;;)
        {
            if (job.at < job.stop)
            {
                if (!ready)
                {
                    if (l) prefetch_job(a, R, L, job, lane, warp);
                    __syncthreads();            // the rows of the job before are no longer needed
                    if (SHARE && warp == kWarps - 1) reset_queue(R, lane);
                    if (!l)
                    {
                        rotate_rows(a, sh, R, job, rows, lane, warp);
                        low_rank_inputs(a, R, job, quot_any(job.stop - 1, L.NU), lane, warp);
                    }
                    else ok = copy_rows(a, sh, R, job, rows, lane, warp) && ok;
                    __syncthreads();
                }
                if (ok) ok = run_job<SHARE>(l);
            }
            ready = false;
            // the rest of the share, or a share that nobody has drawn (all of them were by the time the rows were rotated if every
            // CTA was resident then; an empty share ends the list)
            const bool rest = job.stop < job.end;
            if (!rest && R.drawn[l] >= ctas) break;
            __syncthreads();
            if (warp == 0)
            {
                if (rest) cut_job(a, sh, R, L, job, job.stop, lane);
                else
                {
                    int k = lane == 0 ? atomicAdd(a.wq + 2 * l, 1) : 0;
                    k = __shfl_sync(0xffffffffu, k, 0);
                    cut_share(a, sh, R, L, job, k, lane);
                    if (lane == 0) R.drawn[l] = k + 1;
                }
            }
            __syncthreads();
        }
    }
    // this rank's units are done: add up the slices of all ranks, one (token, group) at a time (tasks are dealt out by warp
    // index: there are more warps than tasks for every supported shape, and no counter to fight over)
    if (ep)
        for (int task = gw; task < a.B * sh.ngH; task += nwarps)
            if (!ep_sum(a, sh, par, task / sh.ngH, task % sh.ngH, lane)) break;
    // the last CTA to leave resets the counters (graph replays start from zero)
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        if (atomicAdd(a.wq + 1, 1) == ctas - 1)
        {
            a.wq[0] = 0; a.wq[1] = 0; a.wq[2] = 0;
            if (ep) *a.epoch = *(volatile int*)a.epoch + 1;
            for (int r = 0; r < sh.nruns; ++r) a.cnt_gu[2 * sh.S * sh.ng + r] = 0;
            if (ld_acquire(a.status) != 0)      // a wait ran out: leave every counter clean all the same
            {
                for (int i = 0; i < 2 * sh.S * sh.ng; ++i) a.cnt_gu[i] = 0;
                for (int i = 0; i < a.B * sh.ngH; ++i) a.cnt_d[i] = 0;
            }
            __threadfence();
        }
    }
}

constexpr int kMaxDevices = 64;

// CTAs that fit on the current device at once (the kernel is persistent); the first call on a device also opts the kernel
// into its shared memory there.  0 = failure.
static int resident_ctas()
{
    static int cached[kMaxDevices] = {0};
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    if (cached[dev]) return cached[dev];
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int fits = 1;
    for (const void* k : {(const void*)moe_decode_kernel<false>, (const void*)moe_decode_kernel<true>})
    {
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemvSmem) != cudaSuccess) return 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, kThreads, kGemvSmem);
        fits = fits && per > 0;
    }
    cached[dev] = fits ? sms : 0;
    return cached[dev];
}

// Most tokens of a run: their rows (of H or I halves) have to fit into shared memory behind the slots, whose size goes with the
// number of column tiles.  Calls of up to 8 tokens have one tile.  An expert with more tokens than that (8 at 6,144 columns, 6 at 8,192,
// 11 at 4,096, 32 up to about 900) is decoded once per run.  That costs less than it seems: a second decode of a unit keeps
// every warp busy, while fragments of 32 tokens from L2 stalled the loop (an earlier version of this kernel): 32 tokens, top-8
// of 16 experts, H = 6,144: 520 us against 1,070; all 32 tokens on one expert: 112 against 793.
static void run_limits(int B, int H, int I, int* run_cap, int* slot_floats)
{
    const int row = (H > I ? H : I) / 128 * kRowStep;
    *run_cap = 0;
    for (int tiles = 1; tiles <= (B <= 8 ? 1 : kRunTiles); tiles *= 2)
    {
        const int fit = rows_room(tiles * kTileFloats) / row, cap = fit < 8 * tiles ? fit : 8 * tiles;
        if (cap > *run_cap) { *run_cap = cap; *slot_floats = tiles * kTileFloats; }
    }
}

}  // namespace nq

extern "C" {

int nq_moe_workspace(int B, int topk, int H, int I, int ks_gu, int ks_dn, NqMoeWorkspace* w)
{
    NQ_REQUIRE(w, "nq_moe_workspace: null output");
    NQ_REQUIRE(B >= 1 && B <= NQ_MAX_TOKENS && topk >= 1 && B * topk <= NQ_MAX_PICKS, "nq_moe_workspace: B = %d, topk = %d", B, topk);
    NQ_REQUIRE(H > 0 && I > 0 && H % 128 == 0 && I % 128 == 0 && H / 128 <= 64 && I / 128 <= 64, "nq_moe_workspace: H = %d, I = %d", H, I);
    NQ_REQUIRE(ks_gu >= 1 && (H / 128) % ks_gu == 0 && ks_dn >= 1 && (I / 128) % ks_dn == 0, "nq_moe_workspace: k-splits %d / %d must divide %d / %d chunks", ks_gu, ks_dn, H / 128, I / 128);
    const size_t S = (size_t)B * topk;
    w->acc_gu_floats = (size_t)ks_gu * S * 2 * I;
    w->h_halves = S * I + S * 2 * H;                    // h [S][I]; the rest is not used (what the allocation-free entry refuses hangs on it)
    w->acc_d_floats = (size_t)ks_dn * S * H;
    w->cnt_gu_ints = 2 * S * (I / 128) + S;
    w->cnt_d_ints = (size_t)B * (H / 128);
    w->wq_ints = 4;
    w->zd_floats = S * (I / 128) * 4;
    w->cnt_h_ints = 4;                                  // [0] status
    return NQ_OK;
}

static int moe_forward(const NqMoeForward* p, const NqMoeEp* ep, void* stream)
{
    NQ_REQUIRE(p, "nq_moe_forward: null arguments");
    NQ_REQUIRE(p->G == 4, "nq_moe_forward: ring width G = %d (only 4 is built)", p->G);
    NqMoeWorkspace need;
    const int rc = nq_moe_workspace(p->B, p->topk, p->H, p->I, p->ks_gu, p->ks_dn, &need);
    if (rc) return rc;
    NQ_REQUIRE(p->x && p->sel && p->rw && p->table && p->out && p->acc_gu && p->h && p->acc_d && p->cnt_gu && p->cnt_d && p->wq && p->cnt_h && p->zd,
               "nq_moe_forward: null tensor");
    NQ_REQUIRE(p->E > 0, "nq_moe_forward: E = %d", p->E);
    NQ_REQUIRE(p->acc_gu_floats >= need.acc_gu_floats && p->h_halves >= need.h_halves && p->acc_d_floats >= need.acc_d_floats &&
               p->cnt_gu_ints >= need.cnt_gu_ints && p->cnt_d_ints >= need.cnt_d_ints && p->wq_ints >= need.wq_ints && p->cnt_h_ints >= need.cnt_h_ints &&
               p->zd_floats >= need.zd_floats,
               "nq_moe_forward: workspace too small (see nq_moe_workspace)");
    NQ_REQUIRE(p->out_floats >= (size_t)p->B * p->H, "nq_moe_forward: out too small");
    NQ_REQUIRE(nq::aligned16(p->x) && nq::aligned16(p->out) && nq::aligned16(p->acc_gu) && nq::aligned16(p->acc_d) && nq::aligned16(p->h),
               "nq_moe_forward: x, out and workspaces must be 16-byte aligned");
    NQ_REQUIRE(p->force_level == 0 || p->force_level == 2 || p->force_level == 4, "nq_moe_forward: force_level = %d", p->force_level);
    nq::MoeArgs a{};
    a.x = (const __half*)p->x; a.sel = p->sel; a.rw = (const __half*)p->rw;
    a.B = p->B; a.topk = p->topk; a.E = p->E; a.H = p->H; a.I = p->I; a.nm_gu = p->nm_gu; a.nm_dn = p->nm_dn;
    a.force_level = p->force_level; a.ks_gu = p->ks_gu; a.ks_dn = p->ks_dn; a.which = p->which & 3; a.table = p->table;
    a.status = p->cnt_h; a.h = (__half*)p->h; 
    a.part_gu = p->acc_gu; a.part_d = p->acc_d; a.zd = p->zd; a.cnt_gu = p->cnt_gu; a.cnt_d = p->cnt_d; a.wq = p->wq; a.out = p->out; a.hits = p->hits;
    a.world = 1; a.rank = 0;
    nq::run_limits(p->B, p->H, p->I, &a.run_cap, &a.slot_floats);
    if (ep && ep->world > 1)
    {
        NQ_REQUIRE(ep->world <= nq::kEpRanks && ep->rank >= 0 && ep->rank < ep->world, "nq_moe_forward_ep: rank %d of %d", ep->rank, ep->world);
        NQ_REQUIRE(ep->peer_recv && ep->peer_counters && ep->epoch, "nq_moe_forward_ep: null exchange buffers");
        NQ_REQUIRE((p->which & 3) == 3, "nq_moe_forward_ep: the in-kernel all-reduce needs the whole layer call (which = 3)");
        NQ_REQUIRE(p->H / 128 <= nq::kEpGroups && p->B <= nq::kEpTokens, "nq_moe_forward_ep: shape beyond the exchange buffers");
        a.world = ep->world; a.rank = ep->rank; a.epoch = ep->epoch;
        for (int r = 0; r < ep->world; ++r)
        {
            NQ_REQUIRE(ep->peer_recv[r] && ep->peer_counters[r] && nq::aligned16(ep->peer_recv[r]), "nq_moe_forward_ep: buffers of rank %d are null or misaligned", r);
            a.recv[r] = (float*)ep->peer_recv[r]; a.rcnt[r] = (int*)ep->peer_counters[r];
        }
    }
    const int ctas = nq::resident_ctas();
    if (ctas <= 0) return nq::fail(NQ_ERR_CUDA, "nq_moe_forward: cannot reserve %d bytes of shared memory", nq::kGemvSmem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas); cfg.blockDim = dim3(nq::kThreads); cfg.dynamicSmemBytes = nq::kGemvSmem; cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, p->B > 1 ? nq::moe_decode_kernel<true> : nq::moe_decode_kernel<false>, a);
    if (e != cudaSuccess) return nq::fail(NQ_ERR_CUDA, "nq_moe_forward: %s", cudaGetErrorString(e));
    return nq::check_launch("nq_moe_forward");
}

int nq_moe_forward(const NqMoeForward* p, void* stream) { return moe_forward(p, nullptr, stream); }

int nq_moe_forward_ep(const NqMoeForward* p, const NqMoeEp* ep, void* stream)
{
    NQ_REQUIRE(ep, "nq_moe_forward_ep: null exchange description");
    return moe_forward(p, ep, stream);
}

size_t nq_moe_ep_recv_floats(int world, int H) { return world >= 1 && H > 0 ? (size_t)2 * world * nq::kEpTokens * H : 0; }
size_t nq_moe_ep_counter_ints(void) { return (size_t)2 * nq::kEpTokens * nq::kEpGroups; }

}  // extern "C"
