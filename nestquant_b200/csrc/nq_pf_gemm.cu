// Prefill grouped GEMM with the trellis decode fused in: acc[pair][n] = sum_k act[pair][k] * W_expert(pair)[n][k].
//
// Replaces the reference's prefill sequence pf_decode -> dense fp16 weights in VRAM -> cuBLAS / Triton grouped GEMM
// (sm120/moe.py:303-324, sm120/pf_gemm.py, sm120/nqmoe.cu:1013-1080): the dense weights are never written to HBM.
//
// One work item = (pass, 128-row weight group): a pass is one expert and up to 384 of its tokens.  Per item a CTA
// walks K in blocks of 64:
//   warp 0        TMA: the tokens' activation tiles [ntok x 64] fp16 (SWIZZLE_128B boxes of 64 rows) -> shared memory; the pass
//                 record and table row of the next item -> shared memory, the first lines of its planes -> L2
//   warps 2..17   decode: a warp streams every other chunk of one strip with cp.async, decodes each unit in registers
//                 (bit-exact fp16) and stores it with tcgen05.st as two weight tiles [128 x 64] in TENSOR MEMORY
//                 (k-blocks 2 c and 2 c + 1): the m16n8k16-style fragment a lane holds is exactly what the 16x256b
//                 store shape takes, so a tile costs one store per warp and no shared memory at all
//   warp 1        one elected lane issues tcgen05.mma with the A operand in tensor memory (M 128 = weight rows, N =
//                 tokens, K 16) into a [128 x 384] fp32 accumulator, also in tensor memory; tcgen05.commit frees the
//                 stages.  Token tiles run 2 or 4 chunks of two k-blocks ahead, 3 k-blocks in passes of more than 320 tokens
//                 (160 KB), weight tiles 2, 4 or 6 units of two (64 columns each), as many as the accumulator of the pass leaves
//                 room for
//   warps 2..17   epilogue: tcgen05.ld the accumulator and store fp32 rows acc[pair][128 columns] (coalesced); it runs
//                 after the first unit of the CTA's next item has been decoded
// A lane's fragment registers of a k-step hold k = 2 t4 + {0, 1} and 8 + 2 t4 + {0, 1}; stored side by side they make
// the tile's k order inside every 16: position 4 i + {0, 1} = k 2 i + {0, 1}, position 4 i + {2, 3} = k 8 + 2 i + {0, 1}.
// The activation matrices must be in the same order (nq_pf_pre / nq_pf_mid with kperm = 1).
// Each decoded weight is used for every token of the pass, so decode cost is paid once per expert (for up to 384
// tokens).  Tensor-pipe bound by intent; the decode instruction rate is the practical limit.  With 31 tokens per expert a unit takes a
// scheduler ~1,000 clocks at level 4 and ~640 at level 2; the decode warps of this kernel alone, without MMAs, need ~810 and ~480, a bare
// loop of records through the ring, decode and tensor-memory store 658 and 388 (without the ring 598 and 355).  Warps 0 and 1 share their schedulers with four decode warps each, so what
// their loops cost is instructions, branches and operand moves, not memory or tensor time: see mbar_wait_warp and uniform.
// Every mbarrier wait is bounded: on time-out the CTA raises status[0], waits for its TMA loads and MMAs in flight, frees its tensor
// memory and returns.
#include <cuda.h>

#include "nq_common.cuh"
#include "nq_scan.cuh"
#include "nq_unit.cuh"

namespace nq {

#ifndef NQ_PF_SPLIT
#define NQ_PF_SPLIT 256      // token tiles wider than this are multiplied as two column halves
#endif
constexpr int kPfGroups = 2;                         // groups of 8 decode warps; group g takes the chunks c = g (mod 2) of its strips.  (3 groups,
                                                     // 24 decode warps at 72 registers, were slower on narrow passes and no faster on wide ones.)
constexpr int kPfDecodeWarps = 8 * kPfGroups;
constexpr int kPfACols = 32;                         // weight tile [128 lanes x 64 k] fp16 = 32 columns; a unit stage is two of them
constexpr int kPfTmemCols = 512;                     // the accumulator from column 0 on, unit stages from the top down
constexpr int kPfTokens = 384;                       // most tokens per pass (accumulator columns)
constexpr int kPfUnitStages = 6;                     // most unit stages
constexpr int kPfBoxRows = 64;                       // token rows per TMA box
constexpr int kPfBoxBytes = kPfBoxRows * 128;        // [64 rows][64 k] fp16
constexpr int kPfBBoxes = 20;                        // token-tile region: 8 x 2, 5 x 4, 4 x 5 or 3 x 6 boxes per stage
constexpr int kPfBStages = 8;                        // most token-tile stages
constexpr int kPfRingDepth = 2;
constexpr int kPfThreads = 32 * (2 + kPfDecodeWarps);
constexpr long long kPfWaitNs = 2000000000ll;             // a wait that lasts 2 s is treated as a hang, unless the caller has another limit

struct PfPass { int expert, row0, ntok, pad; };

struct PfGemmArgs
{
    const int64_t* table;
    const int* plan;          // [0] number of passes, then PfPass records from int 4 on
    float* out0; float* out1; // gate|up: acc_g, acc_u [pairs][I]; down: y [pairs][H]
    int* status;              // [0] != 0: a wait timed out (device side), the results are invalid
    int H, I, nm_gu, nm_dn, down;
    long long wait_ns;        // limit of a wait
};
// What the bounded waits of a CTA look at (shared memory).
struct PfWaits
{
    volatile int aborted;                // a wait has run out
    unsigned long long limit_ns;
};

// ---------------------------------------------------------------- mbarrier / tcgen05 / TMA primitives
__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}
// The producer and MMA warps run their loops with all 32 lanes converged (so that addresses, descriptors and
// coordinates are warp-uniform values) and one elected lane issues the asynchronous instruction.
// Waits of a whole warp, `bar` a shared-space address.  What a wait costs that finds its phase complete is the branches around the
// poll, not the poll: 200 to 240 clocks as a loop (beside 16 busy warps), 95 as a poll, a vote and a branch that falls through, 15
// the poll alone.  So the poll that nearly always succeeds stands in line and the bounded loop behind a call.
// A wait returns false if it has run out, here or in another warp of the CTA.
__device__ __forceinline__ uint32_t mbar_poll(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, PfWaits* waits)
{
    unsigned long long t0 = 0;
    for (;;)
    {
        if (__all_sync(0xffffffffu, mbar_poll(bar, parity))) return true;
        if (__any_sync(0xffffffffu, waits->aborted)) return false;
        unsigned long long t;            // (a poll that fails has waited for some time itself)
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t0 == 0) t0 = t;
        else if (__any_sync(0xffffffffu, t - t0 > waits->limit_ns)) break;
    }
    waits->aborted = 1;
    return false;
}
// Wait of a warp for what it has issued itself, whether or not the CTA has given up: no shared memory or tensor memory may be given back
// that a load or an MMA still touches.
__device__ __noinline__ void mbar_wait_own(uint32_t bar, uint32_t parity)
{
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    do
    {
        if (__all_sync(0xffffffffu, mbar_poll(bar, parity))) return;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    } while (__all_sync(0xffffffffu, t - t0 < (unsigned long long)kPfWaitNs));
}
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, PfWaits* waits)
{
    if (__builtin_expect(__all_sync(0xffffffffu, mbar_poll(bar, parity)), 1)) return true;
    return mbar_wait_slow(bar, parity, waits);
}
// Token boxes of the two k-blocks of a chunk, 64 columns apart, on one election.  first: with what the two barriers have to expect.
__device__ __forceinline__ void tma_load_chunk_elect(uint32_t dst0, uint32_t dst1, const CUtensorMap* map, int x, int y, uint32_t bar0, uint32_t bar1,
                                                     uint32_t bytes)
{
    asm volatile("{\n\t.reg .pred e;\n\t.reg .b32 x1;\n\telect.sync _|e, 0xffffffff;\n\tadd.s32 x1, %3, 64;\n\t"
                 "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%5], %7;\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%3, %4}], [%5];\n\t"
                 "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%6], %7;\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {x1, %4}], [%6];\n\t}"
                 ::"r"(dst0), "r"(dst1), "l"(map), "r"(x), "r"(y), "r"(bar0), "r"(bar1), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_more_elect(uint32_t dst0, uint32_t dst1, const CUtensorMap* map, int x, int y, uint32_t bar0, uint32_t bar1)
{
    asm volatile("{\n\t.reg .pred e;\n\t.reg .b32 x1;\n\telect.sync _|e, 0xffffffff;\n\tadd.s32 x1, %3, 64;\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%3, %4}], [%5];\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {x1, %4}], [%6];\n\t}"
                 ::"r"(dst0), "r"(dst1), "l"(map), "r"(x), "r"(y), "r"(bar0), "r"(bar1) : "memory");
}
// The boxes of one k-block, one below the other.
__device__ __forceinline__ void tma_load_kblock_elect(uint32_t dst, const CUtensorMap* map, int x, int y, int nbox, uint32_t bar)
{
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}"
                 ::"r"(bar), "r"((uint32_t)(nbox * kPfBoxBytes)) : "memory");
    for (int j = 0; j < nbox; ++j)
        asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                     "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}"
                     ::"r"(dst + j * kPfBoxBytes), "l"(map), "r"(x), "r"(y + j * kPfBoxRows), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit_elect(uint64_t* bar)
{
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(saddr(bar)) : "memory");
}
// The four K = 16 steps of one 64-wide k-block and the commits that release its two stages, issued by one elected lane of a
// converged warp (one election for all six: the warp that issues shares its scheduler with four decode warps, and what it
// spends per k-block is what paces the kernel when passes are narrow).  The weight operand is in tensor memory (8 columns per
// step), the token operand in shared memory (descriptor advances by 32 B, in 16-byte units on the low word: shared-memory
// addresses fit its 14-bit field).  first == 0: the first MMA overwrites the accumulator.
__device__ __forceinline__ void tc_mma_kblock(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t first,
                                              uint32_t free_a, uint32_t free_b)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t.reg .b32 ta, tb;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t"
        "setp.eq.b32 p, %4, %4;\n\t"
        "add.u32 ta, %1, 8;\n\tadd.u32 tb, %2, 2;\n\tmov.b64 db, {tb, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %4, p;\n\t"
        "add.u32 ta, %1, 16;\n\tadd.u32 tb, %2, 4;\n\tmov.b64 db, {tb, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %4, p;\n\t"
        "add.u32 ta, %1, 24;\n\tadd.u32 tb, %2, 6;\n\tmov.b64 db, {tb, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %4, p;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
        "}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(first), "r"(free_a), "r"(free_b) : "memory");
}
// The same for a token tile cut into two column halves with their own accumulator columns (alternating chains).
__device__ __forceinline__ void tc_mma_kblock2(uint32_t tmem_d0, uint32_t tmem_d1, uint32_t tmem_a, uint32_t b_lo0, uint32_t b_lo1,
                                               uint32_t b_hi, uint32_t idesc0, uint32_t idesc1, uint32_t first, uint32_t free_a, uint32_t free_b)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t.reg .b32 ta, tb;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %8, 0;\n\t"
        "mov.b64 db, {%3, %5};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], db, %6, p;\n\t"
        "mov.b64 db, {%4, %5};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], db, %7, p;\n\t"
        "setp.eq.b32 p, %6, %6;\n\t"
        "add.u32 ta, %2, 8;\n\tadd.u32 tb, %3, 2;\n\tmov.b64 db, {tb, %5};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %6, p;\n\t"
        "add.u32 tb, %4, 2;\n\tmov.b64 db, {tb, %5};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%1], [ta], db, %7, p;\n\t"
        "add.u32 ta, %2, 16;\n\tadd.u32 tb, %3, 4;\n\tmov.b64 db, {tb, %5};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %6, p;\n\t"
        "add.u32 tb, %4, 4;\n\tmov.b64 db, {tb, %5};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%1], [ta], db, %7, p;\n\t"
        "add.u32 ta, %2, 24;\n\tadd.u32 tb, %3, 6;\n\tmov.b64 db, {tb, %5};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %6, p;\n\t"
        "add.u32 tb, %4, 6;\n\tmov.b64 db, {tb, %5};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%1], [ta], db, %7, p;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%9];\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%10];\n\t"
        "}"
        ::"r"(tmem_d0), "r"(tmem_d1), "r"(tmem_a), "r"(b_lo0), "r"(b_lo1), "r"(b_hi), "r"(idesc0), "r"(idesc1), "r"(first), "r"(free_a), "r"(free_b)
        : "memory");
}
// 16 lanes x 4 x 256 bits of tensor memory from a warp, for columns 8 i .. 8 i + 7: lane (g, t4) supplies lane g columns
// 2 t4, 2 t4 + 1 (r[4 i], r[4 i + 1]) and lane g + 8, same columns (r[4 i + 2], r[4 i + 3]) - the layout of m16n8 fragments
__device__ __forceinline__ void tmem_st_16x256b_x4(uint32_t taddr, const uint32_t* r)
{
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// shared-memory operand descriptor: start address, leading / stride byte offsets (all >> 4), descriptor version 1,
// layout 0 = no swizzle, 2 = 128-byte swizzle
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout)
{
    const uint32_t lo = ((addr >> 4) & 0x3FFFu) | (((lbo >> 4) & 0x3FFFu) << 16);
    const uint32_t hi = ((sbo >> 4) & 0x3FFFu) | (1u << 14) | (layout << 29);
    return ((uint64_t)hi << 32) | lo;
}
// kind::f16 instruction descriptor: D fp32, A/B fp16 K-major, M 128, N tokens
__device__ __forceinline__ uint32_t instr_desc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, "
                 "%26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                   "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
                   "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
                   "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---------------------------------------------------------------- decode warps
struct PfShared
{
    uint64_t full_b[kPfBStages], empty_b[kPfBStages], full_a[kPfUnitStages], empty_a[2 * kPfUnitStages], acc_full, acc_empty;
    uint64_t head_full[2], head_empty[2], mma_done;
    // What the warps need to know of an item, put here by the producer warp one item ahead: read by every warp for itself, pass
    // record and table row are two dependent loads from L2 (~0.7 us) at the start of an item of 10 to 30 us.
    int64_t row[2][kTableWidth];
    PfPass pass[2];
    uint32_t tmem_base;
    PfWaits waits;
};
constexpr int kPfSmem = kPfBBoxes * kPfBoxBytes + kPfDecodeWarps * kPfRingDepth * kStageBytes + 1024 + (int)sizeof(PfShared);
static_assert(kPfSmem <= 232448, "shared memory of the prefill GEMM");
// Unit stages beside the accumulator of a pass.  Group g uses the stages of its parity, so it is 1, 2 or 3 units ahead of the MMAs.
// The stages of a narrow pass reach into columns that the accumulator of a wide one before it used (see decode_strip).
__device__ __forceinline__ int unit_stages(int ntok) { return ntok <= 128 ? 6 : ntok <= 256 ? 4 : 2; }
// The token-tile region (20 boxes) is cut into stages of 2, 4, 5 or 6 boxes (8, 5, 4 or 3 stages) for a pass of nbox
// boxes per k-block.  Passes with the same stage size share the stage barriers freely; when the stage size changes
// between two items of a CTA the new stages overlap old ones at other indices, so the producer first waits until every
// stage of the old layout has been released.
__device__ __forceinline__ int b_stage_boxes(int nbox) { return nbox <= 2 ? 2 : nbox <= 4 ? 4 : nbox <= 5 ? 5 : 6; }
__device__ __forceinline__ int b_stages(int nbox) { return nbox <= 2 ? 8 : nbox <= 4 ? 5 : nbox <= 5 ? 4 : 3; }
// Producer and MMA warp take the stages two at a time, the two k-blocks of a chunk at one wait, except where there are only three (passes
// of more than 320 tokens): there a pair would come free only with the last k-block but one multiplied, and its load would find nothing
// to hide behind.  16 experts x 384 tokens, H 6,144, I 2,048, us, pairs / one by one: gate|up 378 / 250 at level 2, 387 / 277 at level 4,
// down 193 / 146 and 205 / 173 (the kernel that took every pass one by one: 277, 301, 166, 187).  (A poll does not help: try_wait may wait itself, so the second one of a pair does.)  Four stages one by
// one: gate|up of 320 tokens 237 / 211 at level 2, 257 / 262 at level 4; five: 160 tokens 167 / 172 and 224 / 224.
__device__ __forceinline__ bool stages_one_by_one(int nbox) { return b_stages(nbox) == 3; }

// A unit is decoded whole (8 k-steps) by one warp: k-steps 0..3 fill the weight tile of k-block 2 c, k-steps 4..7 the
// tile of k-block 2 c + 1.  The sink keeps the fragments of four k-steps in registers and hands them over as one: wait until
// the MMAs that last read the stage are done, one 32-column store, and after the second half wait for the stores and signal "full".  The four k-steps are
// one straight run of arithmetic with nothing to wait for in it (a store and a branch after every k-step cut the unit into
// ten pieces that were scheduled one by one).
struct UnitSink
{
    uint32_t tmem_a;      // tensor-memory address of the unit stage, at the warp's 16 lanes
    PfShared* sh; uint32_t stage, parity; bool deep; int lane; bool* ok; uint32_t* frag;      // frag: 16 registers
    template <int T>
    __device__ __forceinline__ void operator()(std::integral_constant<int, T>, const uint32_t (&a)[4]) const
    {
        // a[0], a[2]: row g, k = 2 t4 + {0,1} and 8 + 2 t4 + {0,1}; a[1], a[3]: row g + 8
        constexpr int o = 4 * (T & 3), h = T >> 2;
        frag[o] = a[0]; frag[o + 1] = a[2]; frag[o + 2] = a[1]; frag[o + 3] = a[3];
        if constexpr ((T & 3) == 3)
        {
            // two units or more ahead of the MMAs (deep), both halves are nearly always free when the first is written: one vote and
            // branch for the two; one unit ahead, the second half comes back while the first is decoded
            if (h == 0 ? *ok : *ok && !deep)
            {
                const uint32_t bar = saddr(&sh->empty_a[2 * stage + h]);
                uint32_t free = mbar_poll(bar, parity ^ 1u);
                if (h == 0) free &= mbar_poll(deep ? bar + 8 : bar, parity ^ 1u);
                if (__builtin_expect(!__all_sync(0xffffffffu, free), 0))
                {
                    *ok = mbar_wait_slow(bar, parity ^ 1u, &sh->waits);
                    if (h == 0 && *ok && deep) *ok = mbar_wait_slow(bar + 8, parity ^ 1u, &sh->waits);
                }
            }
            tc_fence_after();
            // an aborted launch stores too (the columns are this CTA's until the end, the results are discarded) but signals nothing
            tmem_st_16x256b_x4(tmem_a + h * kPfACols, frag);
            if constexpr (T == 7)
            {
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (*ok && lane == 0) mbar_arrive(&sh->full_a[stage]);
            }
        }
    }
};

// Decode warps: accumulator [128 weight rows x ntok] of an item -> out (row of the item's first token, column of the weight group's
// first row).  TMEM lanes 32 q .. 32 q + 31 (the quarter this warp may read) are weight rows; the four warps of a quarter take
// 32-column chunks in turn.
__device__ __forceinline__ void write_accumulator(PfShared* sh, uint32_t tmem, float* out, int ld, int ntok, uint32_t parity)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (!mbar_wait_warp(saddr(&sh->acc_full), parity, &sh->waits)) return;
    tc_fence_after();
    const int q = warp & 3, cpart = (warp - 2) >> 2;
    for (int c0 = cpart * 32; c0 < ntok; c0 += 32 * (kPfDecodeWarps / 4))
    {
        uint32_t v[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + c0, v);
        float* o = out + (size_t)c0 * ld + q * 32 + lane;
#pragma unroll
        for (int j = 0; j < 32; ++j, o += ld)
            if (c0 + j < ntok) *o = __uint_as_float(v[j]);
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh->acc_empty);
}
// Between two units it is a call, because the registers of the decode loop are all taken there; after the last unit it is in line.  A warp
// with one unit per item has no other place for it than after that unit, and every item pays what the call costs: 128 experts x 31
// tokens, H 6,144, down projection of 256 columns, us, call / in line: 153 / 122 at level 2, 225 / 187 at level 4.  In line between units
// too, down projection of 2,048 columns, 64 experts: 255 / 246 and 404 / 415.
__device__ __noinline__ void write_accumulator_between(PfShared* sh, uint32_t tmem, float* out, int ld, int ntok, uint32_t parity)
{
    write_accumulator(sh, tmem, out, ld, ntok, parity);
}

// One decode warp, one item: its strip over the chunks c = GROUP, GROUP + 2, ... (the other group of 8 warps takes the
// other parity), i.e. k-blocks 4 i + 2 GROUP and + 1.  nstages = unit stages of this item, par_a =
// parity of the times every stage was used; drain: the stages from 2 on lie where the accumulator of the previous item was, so their
// first use waits until all warps have read it (acc_empty, phase `drain_parity`).  false = aborted.
template <bool REFINED, int RC, int BK, class Mid>
__device__ __forceinline__ bool decode_strip(const ProjPlanes& P, const StripRef& sr, int C, int NS, int lane, int group,
                                             uint32_t tmem_a, uint32_t ring, PfShared* sh, int nstages, uint32_t& par_a, bool drain,
                                             uint32_t drain_parity, Mid& mid)
{
    // per-unit scalars of this warp's chunks, one chunk (group + kPfGroups * lane) per lane: ring signs and, for refined units,
    // the block word with its fp16 multiplier / addend (computed once here instead of by every lane of every unit)
    uint32_t var_b = 0, ac = 0, mbn = 0;
    {
        const int ch = group + kPfGroups * lane;
        if (ch < C)
        {
            if (P.var) var_b = __ldg(P.var + sr.unit0 + ch);
            if constexpr (REFINED)
                if (chunk_refined(sr, ch))
                {
                    mbn = __ldg(P.d4 + sr.res0 + refined_before(sr, ch)) & 0xFFFFu;
                    ac = block_multipliers(mbn);
                }
        }
    }
    RecordCursor<BK> cb;
    cb.init(P.base, (size_t)NS * C * 32, sr.unit0, lane);
    RecordCursor<RC> cr;
    if constexpr (REFINED) cr.init(P.p4, sr.res_nrec, sr.res0, lane);
    auto issue = [&](int ch, uint32_t st) {
        cb.copy(st, ch, lane);
        if constexpr (REFINED)
            if (chunk_refined(sr, ch)) cr.copy(st + kStageBase, refined_before(sr, ch), lane);
    };
#pragma unroll
    for (int d = 0; d < kPfRingDepth - 1; ++d)
    {
        if (group + kPfGroups * d < C) issue(group + kPfGroups * d, ring + d * kStageBytes);
        cp_async_commit();
    }
    int slot = 0, slot_in = kPfRingDepth - 1, i = 0, stage = group;
    bool ok = true;
    for (int ch = group; ch < C; ch += kPfGroups, ++i)
    {
        if (ch + kPfGroups * (kPfRingDepth - 1) < C) issue(ch + kPfGroups * (kPfRingDepth - 1), ring + slot_in * kStageBytes);
        cp_async_commit();
        cp_async_wait<kPfRingDepth - 1>();
        const uint32_t st = ring + slot * kStageBytes;
        slot = slot + 1 == kPfRingDepth ? 0 : slot + 1;
        slot_in = slot_in + 1 == kPfRingDepth ? 0 : slot_in + 1;
        const uint32_t sign2 = sign_mask(__shfl_sync(0xffffffffu, var_b, i), lane);
        uint32_t wb[Pattern<BK>::kWords + 2], wr[Pattern<RC>::kWords + 2];
        RecordCursor<BK>::read(wb, st, lane);
        uint32_t frag[16];
        if (drain && i > 0 && ch < nstages && ok) ok = mbar_wait_warp(saddr(&sh->acc_empty), drain_parity, &sh->waits);
        const UnitSink sink{tmem_a - (uint32_t)stage * (2 * kPfACols), sh, (uint32_t)stage, (par_a >> stage) & 1u, nstages > kPfGroups, lane, &ok, frag};
        par_a ^= 1u << stage;
        stage = stage + kPfGroups >= nstages ? group : stage + kPfGroups;
        bool refined = false;
        if constexpr (REFINED) refined = chunk_refined(sr, ch);
        if (refined)
        {
            const uint32_t acw = __shfl_sync(0xffffffffu, ac, i), mb = __shfl_sync(0xffffffffu, mbn, i);
            RecordCursor<RC>::read(wr, st + kStageBase, lane);
            decode_unit<true, RC, BK>(wb, wr, consts_level4(acw, mb, sign2), lane, sink);
        }
        else
            decode_unit<false, 0, BK>(wb, wr, consts_level2(sign2), lane, sink);
        if (i == 0 && ch + kPfGroups < C) mid();      // the previous item's epilogue, once this item's first tiles are on their way
    }
    cp_async_wait<0>();
    return ok;
}

template <class Mid>
__device__ __forceinline__ bool decode_item(const ProjPlanes& P, int level, int rc, int bk, int strip, int C, int NS, int nm, int lane, int group,
                                            uint32_t tmem_a, uint8_t* ring, PfShared* sh, int nstages, uint32_t& par_a, bool drain,
                                            uint32_t drain_parity, Mid& mid)
{
    const StripRef sr = locate_strip(P, strip, C, NS, nm, level >= 4);
    bool ok = true;
#define NQ_RUN(REF, RCV, BKV) ok = decode_strip<REF, RCV, BKV>(P, sr, C, NS, lane, group, tmem_a, smem_addr(ring), sh, nstages, par_a, drain, drain_parity, mid)
    NQ_WITH_CODES(level >= 4, rc, bk, 0x3FF, NQ_RUN);
#undef NQ_RUN
    return ok;
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// The planes' first lines of an item to L2, an item ahead (by one warp, lane i holding word i of the expert's table row): what a decode
// warp reads before its first unit (flags, signs, block words, two units' records of the widest sub-arrays) is a chain of dependent
// loads that an item of few chunks cannot hide.  Every address lies inside the plane it belongs to.  1 % of a 1,000-token call.
__device__ __forceinline__ void prefetch_item(bool level4, int64_t row_word, int down, int wg, int C, int nm, int lane)
{
    const int o = down ? 5 : 1;
    const char* base = (const char*)__shfl_sync(0xffffffffu, row_word, o);
    const char* p4 = (const char*)__shfl_sync(0xffffffffu, row_word, o + 1);
    const char* d4 = (const char*)__shfl_sync(0xffffffffu, row_word, o + 2);
    const char* flags = (const char*)__shfl_sync(0xffffffffu, row_word, o + 3);
    const char* var = (const char*)__shfl_sync(0xffffffffu, row_word, down ? 13 : 12);
    const int rc = (int)__shfl_sync(0xffffffffu, row_word, 10 + down), bk = (int)(__shfl_sync(0xffffffffu, row_word, 19) >> (8 * down)) & 0xFF;
    // eight strips, four lanes each: 256 bytes of the strip's first 1,024 per lane
    const int strip = wg * 8 + (lane >> 2), part = (lane & 3) * 256;
    const size_t unit0 = (size_t)strip * C;
    if (bk == 0 && C > 1) { prefetch_l2(base + unit0 * 512 + part); prefetch_l2(base + unit0 * 512 + part + 128); }
    if (part == 0 && var) prefetch_l2(var + unit0);
    if (level4)
    {
        const bool compact = flags != nullptr;
        const int refined = compact ? nm : C;
        const size_t res0 = (size_t)strip * refined;
        if (part == 0 && compact) prefetch_l2(flags + (size_t)strip * 8);
        if (refined > 1)
        {
            if (part == 0) prefetch_l2(d4 + res0 * 4);
            if ((kWideCodes >> rc) & 1u) { prefetch_l2(p4 + res0 * 512 + part); prefetch_l2(p4 + res0 * 512 + part + 128); }
        }
    }
}

// A value that is the same in all lanes, as one that the compiler knows to be: what it cannot tell from a lane's own value (anything
// loaded, anything that depends on the thread index) reaches the uniform registers of an MMA or TMA instruction by a move of its own
// in front of every one.
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __reduce_or_sync(0xffffffffu, x); }

// grid = resident CTAs (one per SM), 576 threads
__global__ void __launch_bounds__(kPfThreads, 1) pf_gemm_kernel(const __grid_constant__ CUtensorMap tmap0,
                                                                const __grid_constant__ CUtensorMap tmap1, PfGemmArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* b_tiles = smem;                                  // token tiles [rows][64 k] fp16, 128-byte swizzle (TMA boxes)
    uint8_t* rings = smem + kPfBBoxes * kPfBoxBytes;          // per decode warp: kPfRingDepth plane stages
    PfShared* sh = (PfShared*)(rings + kPfDecodeWarps * kPfRingDepth * kStageBytes);
    const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kPfBStages; ++s) { mbar_init(&sh->full_b[s], 1); mbar_init(&sh->empty_b[s], 1); }
        for (int s = 0; s < kPfUnitStages; ++s) mbar_init(&sh->full_a[s], 8);
        for (int s = 0; s < 2 * kPfUnitStages; ++s) mbar_init(&sh->empty_a[s], 1);
        for (int s = 0; s < 2; ++s) { mbar_init(&sh->head_full[s], 1); mbar_init(&sh->head_empty[s], 1 + kPfDecodeWarps); }
        mbar_init(&sh->acc_full, 1); mbar_init(&sh->acc_empty, kPfDecodeWarps);
        mbar_init(&sh->mma_done, 1);
        sh->waits.aborted = 0; sh->waits.limit_ns = (unsigned long long)a.wait_ns;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1)
    {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&sh->tmem_base)), "r"(kPfTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(sh->tmem_base);

    const int N = a.down ? a.H : 2 * a.I, K = a.down ? a.I : a.H, C = K / 128, NS = N / 16, groups = N / 128;
    const int nitems = (int)uniform(a.plan[0]) * groups;
    const PfPass* passes = (const PfPass*)(a.plan + 4);
    const uint32_t full_a0 = saddr(sh->full_a), empty_a0 = saddr(sh->empty_a), full_b0 = saddr(sh->full_b), empty_b0 = saddr(sh->empty_b);
    // item number n of this CTA: its header slot and the phase of its barriers
    auto wait_head = [&](uint32_t n) { return mbar_wait_warp(saddr(&sh->head_full[n & 1u]), (n >> 1) & 1u, &sh->waits); };
    auto leave_head = [&](uint32_t n) { __syncwarp(); if (lane == 0) mbar_arrive(&sh->head_empty[n & 1u]); };
    // Every role has its own loop over the items; nitem = items handled so far, par_a / par_b bit s = parity of the times unit stage /
    // token-tile stage s was used (how many stages there are changes from pass to pass).
    if (warp == 0)
    {
        // ---- token tiles by TMA, ahead of the MMAs as far as there are stages; pass record and table row of the items, one item ahead
        auto publish = [&](int item, uint32_t n) {
            if (item >= nitems) return true;
            const PfPass* pass = passes + item / groups;
            const int64_t w = lane < kTableWidth ? a.table[(int64_t)pass->expert * kTableWidth + lane] : 0;
            const uint32_t s = n & 1u;
            prefetch_item(__shfl_sync(0xffffffffu, w, 0) >= 4, w, a.down, item % groups, C, a.down ? a.nm_dn : a.nm_gu, lane);
            if (!mbar_wait_warp(saddr(&sh->head_empty[s]), ((n >> 1) & 1u) ^ 1u, &sh->waits)) return false;
            if (lane < kTableWidth) sh->row[s][lane] = w;
            if (lane == 0) sh->pass[s] = *pass;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->head_full[s]);
            return true;
        };
        publish(blockIdx.x, 0);
        uint32_t par_b = 0, nitem = 0;
        int last_sbox = 0;                   // stage size of the previous item
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, ++nitem)
        {
            if (!publish(item + gridDim.x, nitem + 1) || !wait_head(nitem)) break;
            const int wg = item % groups;
            const int nbox = (int)uniform((sh->pass[nitem & 1u].ntok + kPfBoxRows - 1) / kPfBoxRows), row0 = (int)uniform(sh->pass[nitem & 1u].row0);
            const int nb = b_stages(nbox), sbox = b_stage_boxes(nbox);
            const CUtensorMap* map = uniform(!a.down && wg >= a.I / 128) ? &tmap1 : &tmap0;
            bool ok = true;
            if (sbox != last_sbox)
                for (int s = 0; ok && s < kPfBStages; ++s) ok = mbar_wait_warp(empty_b0 + 8 * s, ((par_b >> s) & 1u) ^ 1u, &sh->waits);
            last_sbox = sbox;
            const uint32_t tiles0 = saddr(b_tiles), bytes = (uint32_t)nbox * kPfBoxBytes, step = (uint32_t)sbox * kPfBoxBytes;
            if (stages_one_by_one(nbox))
                for (int kb = 0, s = 0; ok && kb < 2 * C; ++kb, s = s + 1 == nb ? 0 : s + 1)
                {
                    ok = mbar_wait_warp(empty_b0 + 8 * s, ((par_b >> s) & 1u) ^ 1u, &sh->waits);
                    if (!ok) break;
                    par_b ^= 1u << s;
                    tma_load_kblock_elect(tiles0 + s * step, map, kb * 64, row0, nbox, full_b0 + 8 * s);
                }
            else
            for (int c = 0, s = 0; ok && c < C; ++c)
            {
                const int s1 = s + 1 == nb ? 0 : s + 1;
                const uint32_t p0 = ((par_b >> s) & 1u) ^ 1u, p1 = ((par_b >> s1) & 1u) ^ 1u;
                const uint32_t free = mbar_poll(empty_b0 + 8 * s, p0) & mbar_poll(empty_b0 + 8 * s1, p1);
                if (__builtin_expect(!__all_sync(0xffffffffu, free), 0))
                {
                    ok = mbar_wait_slow(empty_b0 + 8 * s, p0, &sh->waits) && mbar_wait_slow(empty_b0 + 8 * s1, p1, &sh->waits);
                    if (!ok) break;
                }
                par_b ^= (1u << s) | (1u << s1);
                const uint32_t d0 = tiles0 + s * step, d1 = tiles0 + s1 * step, f0 = full_b0 + 8 * s, f1 = full_b0 + 8 * s1;
                tma_load_chunk_elect(d0, d1, map, c * 128, row0, f0, f1, bytes);
                for (int j = 1; j < nbox; ++j)
                    tma_load_more_elect(d0 + j * kPfBoxBytes, d1 + j * kPfBoxBytes, map, c * 128, row0 + j * kPfBoxRows, f0, f1);
                s = s1 + 1 == nb ? 0 : s1 + 1;
            }
            if (sh->waits.aborted) break;
        }
        __syncwarp();
        for (int s = 0; s < kPfBStages; ++s) mbar_wait_own(full_b0 + 8 * s, ((par_b >> s) & 1u) ^ 1u);      // loads on their way
    }
    else if (warp == 1)
    {
        // ---- MMA issue
        uint32_t par_a = 0, par_b = 0, nitem = 0;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, ++nitem)
        {
            if (!wait_head(nitem)) break;
            const int ntok = (int)uniform(sh->pass[nitem & 1u].ntok), ntok16 = (ntok + 15) & ~15, nbox = (ntok + kPfBoxRows - 1) / kPfBoxRows;
            const int nb = b_stages(nbox), sbox = b_stage_boxes(nbox), nstages = unit_stages(ntok);
            leave_head(nitem);
            bool ok = mbar_wait_warp(saddr(&sh->acc_empty), (nitem & 1u) ^ 1u, &sh->waits);   // epilogue of the previous item has drained TMEM
            tc_fence_after();
            // N <= 256 per instruction: one MMA per k-step, or two of (nearly) equal width
            const int n0 = ntok16 <= NQ_PF_SPLIT ? ntok16 : ((ntok16 / 2 + 15) & ~15), n1 = ntok16 - n0;
            const uint32_t idesc0 = instr_desc(n0), idesc1 = instr_desc(n1 > 0 ? n1 : 16);
            const uint64_t bdesc0 = smem_desc(saddr(b_tiles), 16, 1024, 2);
            const uint32_t b_lo0 = (uint32_t)bdesc0, b_hi = (uint32_t)(bdesc0 >> 32);
            const uint32_t b_step = (uint32_t)(sbox * (kPfBoxBytes >> 4));
            uint32_t s = 0, b_lo = b_lo0;                 // token-tile stage of this k-block and its descriptor
            if (stages_one_by_one(nbox))
                for (uint32_t kb = 0; ok && kb < 2u * C; ++kb)
                {
                    const uint32_t ua = (kb >> 1) & 1u, h = kb & 1u;           // (two unit stages, two column halves)
                    ok = (h || mbar_wait_warp(full_a0 + 8 * ua, (par_a >> ua) & 1u, &sh->waits)) &&
                         mbar_wait_warp(full_b0 + 8 * s, (par_b >> s) & 1u, &sh->waits);
                    if (!ok) break;
                    par_a ^= h << ua;
                    par_b ^= 1u << s;
                    tc_fence_after();
                    tc_mma_kblock2(tmem, tmem + n0, tmem + kPfTmemCols - 2 * kPfACols - ua * (2 * kPfACols) + h * kPfACols, b_lo, b_lo + (uint32_t)(n0 * 8),
                                   b_hi, idesc0, idesc1, kb, empty_a0 + 16 * ua + 8 * h, empty_b0 + 8 * s);
                    if (++s == (uint32_t)nb) { s = 0; b_lo = b_lo0; } else b_lo += b_step;
                }
            else
            for (int c = 0, ua = 0; ok && c < C; ++c, ua = ua + 1 == nstages ? 0 : ua + 1)
            {
                // the unit and its two token tiles: three polls, one vote, one branch
                const uint32_t s1 = s + 1 == (uint32_t)nb ? 0 : s + 1, b_lo1 = s1 == 0 ? b_lo0 : b_lo + b_step;
                const uint32_t pa = (par_a >> ua) & 1u, p0 = (par_b >> s) & 1u, p1 = (par_b >> s1) & 1u;
                uint32_t ready = mbar_poll(full_a0 + 8 * ua, pa);
                ready &= mbar_poll(full_b0 + 8 * s, p0);
                ready &= mbar_poll(full_b0 + 8 * s1, p1);
                if (__builtin_expect(!__all_sync(0xffffffffu, ready), 0))
                {
                    ok = mbar_wait_slow(full_a0 + 8 * ua, pa, &sh->waits) && mbar_wait_slow(full_b0 + 8 * s, p0, &sh->waits) &&
                         mbar_wait_slow(full_b0 + 8 * s1, p1, &sh->waits);
                    if (!ok) break;
                }
                par_a ^= 1u << ua;
                par_b ^= (1u << s) | (1u << s1);
                tc_fence_after();
                const uint32_t ta = tmem + kPfTmemCols - 2 * kPfACols - ua * (2 * kPfACols), free_a = empty_a0 + 16 * ua;
                if (n1 > 0)
                {
                    const uint32_t half = (uint32_t)(n0 * 8);
                    tc_mma_kblock2(tmem, tmem + n0, ta, b_lo, b_lo + half, b_hi, idesc0, idesc1, (uint32_t)c, free_a, empty_b0 + 8 * s);
                    tc_mma_kblock2(tmem, tmem + n0, ta + kPfACols, b_lo1, b_lo1 + half, b_hi, idesc0, idesc1, 1u, free_a + 8, empty_b0 + 8 * s1);
                }
                else
                {
                    tc_mma_kblock(tmem, ta, b_lo, b_hi, idesc0, (uint32_t)c, free_a, empty_b0 + 8 * s);
                    tc_mma_kblock(tmem, ta + kPfACols, b_lo1, b_hi, idesc0, 1u, free_a + 8, empty_b0 + 8 * s1);
                }
                if (s1 + 1 == (uint32_t)nb) { s = 0; b_lo = b_lo0; } else { s = s1 + 1; b_lo = b_lo1 + b_step; }
            }
            if (ok) tc_commit_elect(&sh->acc_full);
            if (sh->waits.aborted) break;
        }
        __syncwarp();
        tc_commit_elect(&sh->mma_done);
        mbar_wait_own(saddr(&sh->mma_done), 0);
    }
    else
    {
        // ---- decode, then epilogue
        // A warp may touch only the 32 tensor-memory lanes of its quarter (warp % 4): the four decode warps of a
        // quarter take its two strips x the chunk groups.
        const int dw = warp - 2, qd = warp & 3, sub = (dw >> 2) & 1, half = dw >> 3, sidx = 2 * qd + sub;      // half = chunk group
        const uint32_t tmem_a = tmem + ((uint32_t)(32 * qd + 16 * sub) << 16) + kPfTmemCols - 2 * kPfACols;
        uint8_t* ring = rings + dw * kPfRingDepth * kStageBytes;
        const int ld = a.down ? a.H : a.I;
        uint32_t par_a = 0, nitem = 0;
        float* prev_out = nullptr;           // the item whose accumulator this warp has still to write (prev_ntok 0: none)
        int prev_ntok = 0, prev_stages = kPfUnitStages;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, ++nitem)
        {
            if (!wait_head(nitem)) break;
            const int64_t* row = sh->row[nitem & 1u];
            const PfPass ps = sh->pass[nitem & 1u];
            const int level = (int)row[0], wg = item % groups, nstages = unit_stages(ps.ntok);
            const ProjPlanes P = planes_from_row(row, a.down);
            const int rc = (int)row[10 + a.down], nm = a.down ? a.nm_dn : a.nm_gu, bk = (int)(row[19] >> (8 * a.down)) & 0xFF;
            leave_head(nitem);
            // group `half` of 8 warps decodes the chunks c = half (mod kPfGroups): k-blocks 2 c and 2 c + 1.  The epilogue
            // of the previous item runs after this item's first unit is decoded: the MMAs of the previous item's last
            // k-blocks finish meanwhile, and the tensor pipe finds tiles waiting when the accumulator is free again.
            auto mid = [&]() { if (prev_ntok) { write_accumulator_between(sh, tmem, prev_out, ld, prev_ntok, (nitem - 1) & 1u); prev_ntok = 0; } };
            const bool ok = decode_item(P, level, rc, bk, wg * 8 + sidx, C, NS, nm, lane, half, tmem_a, ring, sh, nstages, par_a,
                                        nstages > prev_stages, (nitem - 1) & 1u, mid);
            if (prev_ntok) { write_accumulator(sh, tmem, prev_out, ld, prev_ntok, (nitem - 1) & 1u); prev_ntok = 0; }     // (one unit or none)
            prev_stages = nstages;
            if (ok)
            {
                const bool up = !a.down && wg >= a.I / 128;
                prev_out = (up ? a.out1 : a.out0) + (size_t)ps.row0 * ld + (up ? wg - a.I / 128 : wg) * 128;
                prev_ntok = ps.ntok;
            }
            if (sh->waits.aborted) break;
        }
        if (prev_ntok && !sh->waits.aborted) write_accumulator_between(sh, tmem, prev_out, ld, prev_ntok, (nitem - 1) & 1u);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (sh->waits.aborted && threadIdx.x == 0) atomicExch(a.status, 1);      // every warp is through: none can give up after this look
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPfTmemCols) : "memory");
}

// ---------------------------------------------------------------- pass plan (device side, no host sync)
// A pass = one expert x up to 384 of its pairs (pairs are sorted by expert); experts at level 0 get none.  plan: [0] passes,
// [1] pairs covered, then PfPass records from int 4 on, in expert order.
//   WINDOW = false  from[e] = routed pairs of expert e, in the order of the pair list; the plan covers the whole list
//   WINDOW = true   from[e] = first pair of expert e in the sorted list (from[E] = end of the last expert's pairs); the plan covers
//                   the pairs [pair0, pair0 + npairs) with rows counted from pair0
// One CTA, a thread per expert: sums over the CTA (passes before the expert, pairs before it) place every record.  One thread
// that walks the experts alone pays two dependent loads for each of them.
constexpr int kPlanThreads = 1024;

template <bool WINDOW>
__global__ void __launch_bounds__(kPlanThreads) pf_plan_kernel(const int* __restrict__ from, const int64_t* __restrict__ table, int E,
                                                               int pair0, int npairs, int* plan, int max_passes)
{
    __shared__ int s_warp[kPlanThreads / 32];
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

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// tensor map of a row-major fp16 matrix [rows][cols]: boxes of 64 columns x 64 rows, 128-byte swizzle, zero fill
static int make_tile_map(CUtensorMap* map, const void* base, size_t rows, size_t cols)
{
    static EncodeTiledFn fn = nullptr;
    if (!fn)
    {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || !p)
            return fail(NQ_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
        fn = (EncodeTiledFn)p;
    }
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)kPfBoxRows}, estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(NQ_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return NQ_OK;
}

}  // namespace nq

extern "C" {

int nq_pf_plan_ints(int E, int pairs) { return 4 + 4 * (E + pairs / nq::kPfTokens + 1); }

int nq_pf_plan(const int32_t* counts, const int64_t* table, int E, int pairs, int32_t* plan, int plan_ints, void* stream)
{
    NQ_REQUIRE(counts && table && plan && E > 0 && pairs >= 0, "nq_pf_plan: bad arguments");
    NQ_REQUIRE(plan_ints >= nq_pf_plan_ints(E, pairs), "nq_pf_plan: plan needs %d ints", nq_pf_plan_ints(E, pairs));
    nq::pf_plan_kernel<false><<<1, nq::kPlanThreads, 0, (cudaStream_t)stream>>>(counts, table, E, 0, 0, plan, (plan_ints - 4) / 4);
    return nq::check_launch("nq_pf_plan");
}

int nq_pf_plan_window(const int32_t* start, const int64_t* table, int E, int pair0, int npairs, int32_t* plan, int plan_ints, void* stream)
{
    NQ_REQUIRE(start && table && plan && E > 0 && pair0 >= 0 && npairs >= 0, "nq_pf_plan_window: bad arguments");
    NQ_REQUIRE(plan_ints >= nq_pf_plan_ints(E, npairs), "nq_pf_plan_window: plan needs %d ints", nq_pf_plan_ints(E, npairs));
    nq::pf_plan_kernel<true><<<1, nq::kPlanThreads, 0, (cudaStream_t)stream>>>(start, table, E, pair0, npairs, plan, (plan_ints - 4) / 4);
    return nq::check_launch("nq_pf_plan_window");
}

int nq_pf_gemm_within(const int64_t* table, const int32_t* plan, const void* act0, const void* act1, int pairs, float* out0, float* out1,
                      int H, int I, int nm_gu, int nm_dn, int down, int32_t* status, long long wait_ns, void* stream)
{
    NQ_REQUIRE(wait_ns >= 0, "nq_pf_gemm: wait_ns = %lld", wait_ns);
    NQ_REQUIRE(table && plan && act0 && out0 && status, "nq_pf_gemm: null pointer");
    NQ_REQUIRE(down || (act1 && out1), "nq_pf_gemm: the gate|up projection needs both activation matrices and both outputs");
    NQ_REQUIRE(H > 0 && I > 0 && H % 128 == 0 && I % 128 == 0 && H / 128 <= 64 && I / 128 <= 64, "nq_pf_gemm: H = %d, I = %d", H, I);
    NQ_REQUIRE(pairs >= 0, "nq_pf_gemm: pairs = %d", pairs);
    if (pairs == 0) return NQ_OK;
    NQ_REQUIRE(nq::aligned16(act0) && nq::aligned16(act1) && nq::aligned16(out0), "nq_pf_gemm: matrices must be 16-byte aligned");
    // SM count and the shared-memory opt-in are per device: cached per device ordinal
    static int ctas_of[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nq::fail(NQ_ERR_CUDA, "nq_pf_gemm: no usable current device");
    if (!ctas_of[dev])
    {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaFuncSetAttribute((const void*)nq::pf_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, nq::kPfSmem) != cudaSuccess)
            return nq::fail(NQ_ERR_CUDA, "nq_pf_gemm: cannot reserve %d bytes of shared memory", nq::kPfSmem);
        ctas_of[dev] = sms;
    }
    const int ctas = ctas_of[dev];
    CUtensorMap m0, m1;
    const size_t K = down ? I : H;
    if (int e = nq::make_tile_map(&m0, act0, (size_t)pairs, K)) return e;
    if (int e = nq::make_tile_map(&m1, down ? act0 : act1, (size_t)pairs, K)) return e;
    nq::PfGemmArgs a{};
    a.table = table; a.plan = plan; a.out0 = out0; a.out1 = out1; a.status = status;
    a.H = H; a.I = I; a.nm_gu = nm_gu; a.nm_dn = nm_dn; a.down = down ? 1 : 0; a.wait_ns = wait_ns;
    nq::pf_gemm_kernel<<<ctas, nq::kPfThreads, nq::kPfSmem, (cudaStream_t)stream>>>(m0, m1, a);
    return nq::check_launch("nq_pf_gemm");
}

int nq_pf_gemm(const int64_t* table, const int32_t* plan, const void* act0, const void* act1, int pairs, float* out0, float* out1,
               int H, int I, int nm_gu, int nm_dn, int down, int32_t* status, void* stream)
{
    return nq_pf_gemm_within(table, plan, act0, act1, pairs, out0, out1, H, I, nm_gu, nm_dn, down, status, nq::kPfWaitNs, stream);
}

}  // extern "C"
