// Prefill grouped GEMM with the trellis decode fused in: acc[pair][n] = sum_k act[pair][k] * W_expert(pair)[n][k].
//
// Replaces the reference's prefill sequence pf_decode -> dense fp16 weights in VRAM -> cuBLAS / Triton grouped GEMM
// (sm120/moe.py:303-324, sm120/pf_gemm.py, sm120/nqmoe.cu:1013-1080): the dense weights are never written to HBM.
//
// One work item = (pass, 128-row weight group): a pass is one expert and up to 384 of its tokens.  Per item a CTA
// walks K in blocks of 64:
//   warp 0        TMA: the tokens' activation tiles [ntok x 64] fp16 (SWIZZLE_128B boxes of 64 rows) -> shared memory; the header
//                 of the next item (everything the other warps need to know of it) -> shared memory, the first lines of its planes -> L2
//   warps 2..17   decode: a warp streams every other chunk of one strip, the records of the next unit into registers while it
//                 decodes this one (bit-exact fp16) and stores it with tcgen05.st as two weight tiles [128 x 64] in TENSOR MEMORY
//                 (k-blocks 2 c and 2 c + 1): the m16n8k16-style fragment a lane holds is exactly what the 16x256b
//                 store shape takes, so a tile costs one store per warp and no shared memory at all
//   warps 1, 18   one elected lane issues tcgen05.mma with the A operand in tensor memory (M 128 = weight rows, N =
//                 tokens, K 16) into a [128 x 384] fp32 accumulator, also in tensor memory; one tcgen05.commit per chunk of two
//                 k-blocks frees its weight and token tiles.  Both run 6, 4, 3 or 2 chunks ahead, as many as the accumulator of the pass
//                 and 192 KB of shared memory leave room for.  Passes of up to 64 tokens are multiplied by both warps, wider ones by warp 1
//   warps 2..17   epilogue: tcgen05.ld the accumulator and store fp32 rows acc[pair][128 columns] (coalesced); it runs
//                 after the first units of the CTA's next item have been decoded
// A lane's fragment registers of a k-step hold k = 2 t4 + {0, 1} and 8 + 2 t4 + {0, 1}; stored side by side they make
// the tile's k order inside every 16: position 4 i + {0, 1} = k 2 i + {0, 1}, position 4 i + {2, 3} = k 8 + 2 i + {0, 1}.
// The activation matrices must be in the same order (nq_pf_pre / nq_pf_mid with kperm = 1).
// Each decoded weight is used for every token of the pass, so decode cost is paid once per expert (for up to 384
// tokens).  Tensor-pipe bound by intent; the decode instruction rate is the practical limit: with 31 tokens per expert a unit takes a
// scheduler 777 clocks at level 4, 663 in mask mode and 475 at level 2, borders of items included (gate|up of H 6,144: 613, 523 and 376 instructions,
// at most 0.84 per clock: the half-rate multiply and byte-sum pipe is busy for nine tenths of that); a loop that only decodes and stores takes 662 at
// level 4 and 393 at level 2.  What the two issuing warps spend comes on top of the decode warps of their schedulers, and the slowest scheduler
// paces the others; see mbar_wait_warp, uniform and split_chunks.  H 6,144, I 2,048, us, gate|up / down:
//     experts x tokens    128 x 31       32 x 100     16 x 160     16 x 256     16 x 384
//     level 2             712 / 409      229 / 143    148 / 93     175 / 109    255 / 147 (bound by the token tiles that come from L2)
//     level 4             1,147 / 641    318 / 199    197 / 120    209 / 131    265 / 166
//     mask mode           985 / 583      279 / 183    175 / 113    194 / 125    261 / 159
// Every mbarrier wait is bounded: on time-out the CTA raises status[0], waits for its TMA loads and MMAs in flight, frees its tensor
// memory and returns.
#include <cuda.h>

#include "nq_common.cuh"
#include "nq_plan.cuh"
#include "nq_unit.cuh"

namespace nq {

constexpr int kPfGroups = 2;                         // groups of 8 decode warps; group g takes the chunks c = g (mod 2) of its strips.  (3 groups,
                                                     // 24 decode warps at 72 registers, were slower on narrow passes and no faster on wide ones.)
constexpr int kPfDecodeWarps = 8 * kPfGroups;
constexpr int kPfACols = 32;                         // weight tile [128 lanes x 64 k] fp16 = 32 columns; a unit stage is two of them
constexpr int kPfTmemCols = 512;                     // the accumulator from column 0 on, unit stages from the top down
constexpr int kPfStages = 6;                         // most stages of a pass (chunk_stages)
constexpr int kPfBoxRows = 64;                       // token rows per TMA box
constexpr int kPfBoxBytes = kPfBoxRows * 128;        // [64 rows][64 k] fp16
constexpr int kPfBBoxes = 24;                        // token-tile region: 6, 4, 3 or 2 chunk stages of 2 x 2, 2 x 3, 2 x 4 or 2 x 6 boxes
constexpr int kPfSecondIssuer = 2 + kPfDecodeWarps;      // warp 1 and this one issue MMAs
constexpr int kPfThreads = 32 * (kPfSecondIssuer + 1);
constexpr long long kPfWaitNs = 2000000000ll;             // a wait that lasts 2 s is treated as a hang, unless the caller has another limit

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
__device__ __forceinline__ void mbar_arrive32(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) { mbar_arrive32(saddr(bar)); }
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
// Token boxes of the two k-blocks of a chunk, 64 columns apart, on one election.  first: with what the barrier has to expect.
__device__ __forceinline__ void tma_load_chunk_elect(uint32_t dst0, uint32_t dst1, const CUtensorMap* map, int x, int y, uint32_t bar, uint32_t bytes)
{
    asm volatile("{\n\t.reg .pred e;\n\t.reg .b32 x1;\n\telect.sync _|e, 0xffffffff;\n\tadd.s32 x1, %3, 64;\n\t"
                 "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%5], %6;\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%3, %4}], [%5];\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {x1, %4}], [%5];\n\t}"
                 ::"r"(dst0), "r"(dst1), "l"(map), "r"(x), "r"(y), "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_more_elect(uint32_t dst0, uint32_t dst1, const CUtensorMap* map, int x, int y, uint32_t bar)
{
    asm volatile("{\n\t.reg .pred e;\n\t.reg .b32 x1;\n\telect.sync _|e, 0xffffffff;\n\tadd.s32 x1, %3, 64;\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%3, %4}], [%5];\n\t"
                 "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {x1, %4}], [%5];\n\t}"
                 ::"r"(dst0), "r"(dst1), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit_elect(uint64_t* bar)
{
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(saddr(bar)) : "memory");
}
// The eight K = 16 steps of a chunk and the commit that releases its stage, issued by one elected lane of a converged warp (one election
// for all nine: the warp that issues shares its scheduler with four decode warps, and what it spends per chunk is what paces the
// kernel when passes are narrow).  The weight operand is in tensor memory (8 columns per step), the token operand in shared memory
// (descriptor advances by 32 B, in 16-byte units on the low word: shared-memory addresses fit its 14-bit field; b_kb: from the first
// k-block's tile to the second's).  first == 0: the first MMA overwrites the accumulator.
__device__ __forceinline__ void tc_mma_chunk(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_kb, uint32_t b_hi, uint32_t idesc, uint32_t first,
                                             uint32_t empty)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t.reg .b32 ta, tb;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "mov.b32 tb, %2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %5, p;\n\t"
        "setp.eq.b32 p, %5, %5;\n\t"
        "add.u32 ta, %1, 8;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, %1, 16;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, %1, 24;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, %1, 32;\n\t"
        "add.u32 tb, %2, %3;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, %1, 40;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, %1, 48;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, %1, 56;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
        "}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_kb), "r"(b_hi), "r"(idesc), "r"(first), "r"(empty) : "memory");
}
// The same for a token tile cut into two column halves with their own accumulator columns (alternating chains); half_a is told when the
// first k-block's weight tile has been read.
__device__ __forceinline__ void tc_mma_chunk2(uint32_t tmem_d0, uint32_t tmem_d1, uint32_t tmem_a, uint32_t b_lo, uint32_t b_half, uint32_t b_kb, uint32_t b_hi,
                                              uint32_t idesc0, uint32_t idesc1, uint32_t first, uint32_t half_a, uint32_t empty)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t.reg .b32 ta, tb;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "mov.b32 tb, %2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %5, p;\n\t"
        "add.u32 ta, tb, %9;\n\tmov.b64 db, {ta, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%8], [%1], db, %10, p;\n\t"
        "setp.eq.b32 p, %5, %5;\n\t"
        "add.u32 ta, %1, 8;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, tb, %9;\n\tmov.b64 db, {ta, %4};\n\t"
        "add.u32 ta, %1, 8;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%8], [ta], db, %10, p;\n\t"
        "add.u32 ta, %1, 16;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, tb, %9;\n\tmov.b64 db, {ta, %4};\n\t"
        "add.u32 ta, %1, 16;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%8], [ta], db, %10, p;\n\t"
        "add.u32 ta, %1, 24;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, tb, %9;\n\tmov.b64 db, {ta, %4};\n\t"
        "add.u32 ta, %1, 24;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%8], [ta], db, %10, p;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%11];\n\t"
        "add.u32 ta, %1, 32;\n\t"
        "add.u32 tb, %2, %3;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, tb, %9;\n\tmov.b64 db, {ta, %4};\n\t"
        "add.u32 ta, %1, 32;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%8], [ta], db, %10, p;\n\t"
        "add.u32 ta, %1, 40;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, tb, %9;\n\tmov.b64 db, {ta, %4};\n\t"
        "add.u32 ta, %1, 40;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%8], [ta], db, %10, p;\n\t"
        "add.u32 ta, %1, 48;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, tb, %9;\n\tmov.b64 db, {ta, %4};\n\t"
        "add.u32 ta, %1, 48;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%8], [ta], db, %10, p;\n\t"
        "add.u32 ta, %1, 56;\n\t"
        "add.u32 tb, tb, 2;\n\t"
        "mov.b64 db, {tb, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %5, p;\n\t"
        "add.u32 ta, tb, %9;\n\tmov.b64 db, {ta, %4};\n\t"
        "add.u32 ta, %1, 56;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%8], [ta], db, %10, p;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
        "}"
        ::"r"(tmem_d0), "r"(tmem_a), "r"(b_lo), "r"(b_kb), "r"(b_hi), "r"(idesc0), "r"(first), "r"(empty), "r"(tmem_d1), "r"(b_half), "r"(idesc1), "r"(half_a)
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

// 16 accumulator columns, and the same of the second accumulator; the wait is part of it, so nothing reads the registers in front of it
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                   "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld16_two(uint32_t taddr, uint32_t second, uint32_t (&v)[16], uint32_t (&w)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                   "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                   "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]), "=r"(w[8]), "=r"(w[9]),
                   "=r"(w[10]), "=r"(w[11]), "=r"(w[12]), "=r"(w[13]), "=r"(w[14]), "=r"(w[15])
                 : "r"(taddr), "r"(second) : "memory");
}

// ---------------------------------------------------------------- decode warps
// What the warps need to know of an item, put into shared memory by the producer warp one item ahead: pass record and table row are two
// dependent loads from L2 (~0.7 us), and worked out by every decode warp for itself the rest takes 1,800 clocks of an item of 25,000
// to 80,000 (four warps of a scheduler do it at the same time).
struct PfItem
{
    ProjPlanes P;
    uint32_t nrec, res_nrec;         // records of the base and of the residual plane
    uint32_t unit0, res0;            // first strip of the weight group: its first unit, its first refined unit in the residual plane
    float* out;                      // row of the item's first token, column of the weight group's first row
    int strip0, res_strip;           // number of the first strip; refined units per strip
    int ntok, nst, row0, up, variant;
};
constexpr int kPfCodes = kNumCodes + 2;     // window codes of a decoder function: the residual codes beside base code 0, 3 and 9 beside base code 1
constexpr int kPfHeads = 3;          // this item, the one before it (its epilogue runs in this one) and the next
struct PfShared
{
    // full_a / full_b: weight / token tiles of a chunk are there; empty: the MMAs that read them are through; half_a: those of the first
    // k-block (passes of two stages, i.e. one per group)
    uint64_t full_a[kPfStages], full_b[kPfStages], empty[kPfStages], half_a[kPfGroups], acc_full[2], acc_empty[2];
    uint64_t head_full[kPfHeads], head_empty[kPfHeads], mma_done[2];
    PfItem item[kPfHeads];
    int C, ld;                       // chunks of an item, floats from output row to output row
    uint32_t tmem_base;
    PfWaits waits;
};
constexpr int kPfSmem = kPfBBoxes * kPfBoxBytes + (int)sizeof(PfShared);
static_assert(kPfSmem <= 232448, "shared memory of the prefill GEMM");
extern __shared__ __align__(1024) uint8_t nq_pf_smem[];      // (the token tiles' swizzle needs the alignment; addresses in it are constants of the code)
__device__ __forceinline__ uint8_t* pf_tiles() { return nq_pf_smem; }
__device__ __forceinline__ PfShared* pf_shared() { return (PfShared*)(pf_tiles() + kPfBBoxes * kPfBoxBytes); }
// Chunk stages of a pass: chunk c of an item uses stage c mod chunk_stages, its weight tiles in tensor memory (64 columns a stage, from the
// top down beside the accumulator) and its token tiles in shared memory (2 x 12 / stages boxes).  One set of barriers serves both.  The
// stages of a narrow pass reach into columns that the accumulator of a wide one before it used (see decode_strip), and when the number of
// stages changes between two items of a CTA the new token tiles overlap old ones at other indices, so the producer first waits
// until every stage of the old layout has been released.  Where the chunks of a strip take different times (mask mode) the stages even them
// out: 16 experts, H 6,144, I 2,048, gate|up / down, us, with three / four stages: 160 tokens 177 / 175 and 114 / 112, at level 2 153 / 148 and 94 / 93; 192 tokens
// 181 / 180 and 118 / 115, at level 2 159 / 158 and 99.1 / 98.5; at level 4 the same.
__device__ __forceinline__ int chunk_stages(int ntok) { return ntok <= 128 ? 6 : ntok <= 192 ? 4 : ntok <= 256 ? 3 : 2; }
// Passes of up to 64 tokens: even and odd chunks are multiplied by two warps, each into an accumulator of its own that the epilogue adds up.
// What a chunk costs the warp that issues its MMAs comes on top of the decode warps of its scheduler, and the slowest scheduler paces the
// others: 128 experts x 31 tokens, H 6,144, I 2,048, gate|up / down, with one warp / two, us: level 2 766 / 712 and 426 / 409, level 4 1,183 / 1,147 and
// 666 / 641, mask mode 1,009 / 985 and 601 / 583; strips of two chunks lose by it (I 256, down: 114 / 119, 154 / 156, 158 / 165).  Beyond 64 tokens the second
// accumulator would leave four stages instead of six, which comes out even or a little better (32 x 100 tokens, six stages and one warp / four and
// two: level 2 229 / 221 and 143 / 143, level 4 318 / 311 and 199 / 197, mask mode 279 / 275 and 183 / 183); before the decoders kept clear of
// spills it was 7 to 10 % slower.
__device__ __forceinline__ bool split_chunks(int ntok) { return ntok <= 64; }
// First column of an item's accumulator, and from there to the second one.  Up to 32 tokens the items take turns with two pairs, so the MMAs
// of the next item need not wait for the epilogue.
__device__ __forceinline__ uint32_t acc_column(int ntok, uint32_t acc) { return ntok <= 32 ? 64u * acc : 0u; }
__device__ __forceinline__ uint32_t acc_second(int ntok) { return ntok <= 32 ? 32u : 64u; }
// bit s = parity of the times stage s was used, after an item of C chunks in nst stages
__device__ __forceinline__ uint32_t stage_parities(uint32_t par, int C, int nst)
{
    const int rounds = C / nst;
    return par ^ (rounds & 1 ? (1u << nst) - 1u : 0u) ^ ((1u << (C - rounds * nst)) - 1u);
}

// A unit is decoded whole (8 k-steps) by one warp: k-steps 0..3 fill the weight tile of k-block 2 c, k-steps 4..7 the
// tile of k-block 2 c + 1.  The sink keeps the fragments of four k-steps in registers and hands them over as one 32-column store.
// DEEP (more stages than groups: six or four, of which a group uses its own three or two, or three that both go round): the stage is free before
// the unit is begun, and the 64 weights are one straight run of arithmetic with nothing to wait for in it.  Two stages, one per group: each half
// is waited for when it is to be written.
template <bool DEEP>
struct UnitSink
{
    uint32_t tmem_a;      // tensor-memory address of the stage, at the warp's 16 lanes
    PfShared* sh; uint32_t stage, parity, half_parity; bool first; bool* ok; uint32_t* frag;      // frag: 16 registers
    template <int T>
    __device__ __forceinline__ void operator()(std::integral_constant<int, T>, const uint32_t (&a)[4]) const
    {
        // a[0], a[2]: row g, k = 2 t4 + {0,1} and 8 + 2 t4 + {0,1}; a[1], a[3]: row g + 8
        constexpr int o = 4 * (T & 3), h = T >> 2;
        frag[o] = a[0]; frag[o + 1] = a[2]; frag[o + 2] = a[1]; frag[o + 3] = a[3];
        if constexpr ((T & 3) == 3)
        {
            if constexpr (!DEEP)
            {
                if (h == 0) *ok = mbar_wait_warp(saddr(&sh->half_a[stage]), half_parity, &sh->waits);
                // (first unit of an item: the stage may have been used last by a pass that does not report halves)
                if ((h == 1 || first) && *ok) *ok = mbar_wait_warp(saddr(&sh->empty[stage]), parity, &sh->waits);
                tc_fence_after();
            }
            // (an aborted launch stores too: the columns are this CTA's until the end, the results are discarded)
            tmem_st_16x256b_x4(tmem_a + h * kPfACols, frag);
        }
    }
};

// What a decoder function needs to know beside the item: in one word.
struct PfInfo
{
    uint32_t w;      // bits 0, 1 header slot of the item, 2, 3 of the one before it, 4 whose accumulator is to be written, 5 drain, 6 accumulator
                     // barriers of the one before it, 7 their phase
    __device__ __forceinline__ uint32_t slot() const { return w & 3u; }
    __device__ __forceinline__ uint32_t prev() const { return w >> 2 & 3u; }
    __device__ __forceinline__ bool has_prev() const { return w >> 4 & 1u; }
    __device__ __forceinline__ bool drain() const { return w >> 5 & 1u; }
    __device__ __forceinline__ uint32_t acc() const { return w >> 6 & 1u; }
    __device__ __forceinline__ uint32_t phase() const { return w >> 7 & 1u; }
};
// Units of an item that a warp decodes before it writes the accumulator of the previous item, whose last MMAs finish meanwhile.  128 experts x 31
// tokens, H 6,144, I 2,048, gate|up / down, us, after two units, after one, at once: level 2 712 / 409, 721 / 411, 722 / 415; level 4 1,147 / 641, 1,162 /
// 640, 1,155 / 668; with I 256, whose down strips have one unit per warp, down after it 119, 156 at level 4, at once 130, 180.
__device__ __forceinline__ int units_before_epilogue(int nst, bool drain) { return nst == kPfStages && !drain ? 2 : 1; }

// Decode warps: accumulator [128 weight rows x ntok] of the item before this one -> out.  TMEM lanes 32 q .. 32 q + 31 (the quarter this warp
// may read) are weight rows; the four warps of a quarter take 16-column pieces in turn.
__device__ __forceinline__ void write_accumulator(PfInfo info)
{
    PfShared* sh = pf_shared();
    const PfItem& I = sh->item[info.prev()];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ntok = I.ntok, ld = sh->ld;
    const bool both = split_chunks(ntok) && sh->C > 1;
    const uint32_t tmem = sh->tmem_base + acc_column(ntok, info.acc());
    if (!mbar_wait_warp(saddr(&sh->acc_full[info.acc()]), info.phase(), &sh->waits)) return;
    tc_fence_after();
    const int q = warp & 3, cpart = (warp - 2) >> 2;
    for (int c0 = cpart * 16; c0 < ntok; c0 += 16 * (kPfDecodeWarps / 4))
    {
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + c0;
        uint32_t v[16];
        if (both)
        {
            uint32_t w[16];
            tmem_ld16_two(at, at + acc_second(ntok), v, w);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
        }
        else tmem_ld16(at, v);
        float* o = I.out + (size_t)c0 * ld + q * 32 + lane;
#pragma unroll
        for (int j = 0; j < 16; ++j, o += ld)
            if (c0 + j < ntok) *o = __uint_as_float(v[j]);
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) { mbar_arrive(&sh->acc_empty[info.acc()]); mbar_arrive(&sh->head_empty[info.prev()]); }
}
// Between two units it is a call, because the registers of the decode loop are all taken there; after the last unit it is in line.  A warp
// with one unit per item has no other place for it than after that unit, and every item pays what the call costs: 128 experts x 31
// tokens, H 6,144, down projection of 256 columns, us, call / in line: 126 / 120 at level 2, 170 / 156 at level 4; of 512 columns 164 / 158, 243 / 228.
__device__ __noinline__ void write_accumulator_between(uint32_t info) { write_accumulator(PfInfo{info}); }

// One decode warp, one item: its strip over the chunks c = group, group + 2, ... (the other group of 8 warps takes the other
// parity), i.e. k-blocks 4 i + 2 group and + 1.  MODE 0: level 2, 1: level 4, 2: level 4 in mask mode (chunks without a flag decode as
// level 2).  The records of the next unit are fetched into registers while the current one is decoded.
// par: bit s = parity of the times stage s was used before this item, bit kPfStages the same for half_a of this warp's group.
// false: a wait ran out.
// The epilogue of the previous item runs after this item's first units are decoded: the MMAs of the previous item's last k-blocks finish
// meanwhile, and the tensor pipe finds tiles waiting when the accumulator is free again.  It stands between two runs of the
// unit loop, not in it.  drain: the stages from 2 on lie where the accumulator of the previous item was, so they wait until all warps have
// read it.
template <int MODE, int RC, int BK, bool DEEP>
__device__ __noinline__ bool decode_strip(uint32_t par, uint32_t info_word)
{
    PfShared* sh = pf_shared();
    const PfInfo info{info_word};
    const int warp = (int)(threadIdx.x >> 5), lane = threadIdx.x & 31, group = (warp - 2) >> 3, nxt = ring_successor(lane);
    const int sidx = 2 * (warp & 3) + (((warp - 2) >> 2) & 1);        // strip of the weight group: two to every quarter of the lanes
    const PfItem& I = sh->item[info.slot()];
    const int C = sh->C, n = (C - group + kPfGroups - 1) / kPfGroups;         // units of this warp: at most 32
    if (n <= 0) return true;
    const uint32_t unit0 = I.unit0 + (uint32_t)(sidx * C), res0 = I.res0 + (uint32_t)(sidx * I.res_strip);
    const uint8_t *base = (const uint8_t*)I.P.base, *p4 = I.P.p4;
    const uint32_t nrec = I.nrec, res_nrec = MODE == 1 ? nrec : I.res_nrec;
    uint32_t rec = (unit0 + group) * 32 + lane, res = (MODE == 1 ? unit0 + group : res0) * 32 + lane;       // this unit's records (level 4 without flags: of both planes)
    RecordValues<BK> rb;
    rb.load_at(base, nrec, rec);
    // Zeroed, and taken apart for every unit: a record that holds nothing yet, or is taken apart on refined units only, costs the compiler
    // registers beside the words made of it, 2,480 bytes of spill loads over all decoders without the one, 1,440 without the other, none with both.
    // us, gate|up / down, without both / with: 128 experts x 31 tokens in mask mode 1,074 / 705 -> 984 / 583, level 2 759 / 435 -> 710 / 407,
    // level 4 1,165 / 679 -> 1,146 / 641; 16 x 256 in mask mode 212 / 152 -> 192 / 127; 225 x 244, H 1,792, I 640, 307 / 250 -> 276 / 205.
    RecordValues<RC> rr = {};
    unsigned long long flags = 0;        // refined chunks of the strip
    uint32_t own = 0, other = 0;         // of them this warp's units, and the chunks behind those, from this unit on
    if constexpr (MODE == 1) rr.load_at(p4, nrec, rec);
    if constexpr (MODE == 2)
    {
        flags = (unsigned long long)__ldg((const unsigned long long*)I.P.flags + I.strip0 + sidx);
        if (group) res += (uint32_t)(flags & 1ull) * 32u;
        own = __ballot_sync(0xffffffffu, flags >> group >> (kPfGroups * lane) & 1ull);
        other = __ballot_sync(0xffffffffu, flags >> group >> (kPfGroups * lane) >> 1 & 1ull);
        if (own & 1u) rr.load_at(p4, res_nrec, res);
    }
    // per-unit scalars, one unit per lane: ring signs and block word (meta = word | signs << 16) and the block word's multipliers
    uint32_t meta = 0, ac = 0;
    if (lane < n)
    {
        const int ch = group + kPfGroups * lane;
        if (I.P.var) meta = (uint32_t)__ldg(I.P.var + unit0 + ch) << 16;
        if (MODE == 1 || (MODE == 2 && (flags >> ch & 1ull)))
        {
            const size_t at = res0 + (MODE == 1 ? ch : __popcll(flags & ((1ull << ch) - 1ull)));
            const uint32_t word = __ldg(I.P.d4 + at) & 0xFFFFu;
            meta |= word;
            ac = block_multipliers(word);
        }
    }
    const uint32_t tmem_a = sh->tmem_base + ((uint32_t)(16 * sidx) << 16) + kPfTmemCols - 2 * kPfACols, full_a0 = saddr(sh->full_a), empty0 = saddr(sh->empty);
    const uint32_t nst = DEEP ? (uint32_t)I.nst : 2u;
    const uint32_t half_par = par >> kPfStages;
    uint32_t stage = (uint32_t)group, free = ~par;       // bit s of free: phase of `empty` that frees stage s for this round
    int i = 0, end = info.has_prev() ? min(n, units_before_epilogue((int)nst, info.drain())) : n;
    bool ok = true;
#pragma unroll 1
    for (;;)
    {
#pragma unroll 1
        for (; i < end; ++i)
        {
            uint32_t wb[Pattern<BK>::kWords + 2], wr[Pattern<RC>::kWords + 2];
            const bool refined = MODE == 1 || (MODE == 2 && (own & 1u));
            rb.words(wb, lane);
            if constexpr (MODE > 0) rr.words(wr, lane);      // (mask mode: also of a unit that is not refined, where nothing uses them)
            if (i + 1 < n)
            {
                rec += kPfGroups * 32;
                rb.load_at(base, nrec, rec);
                if constexpr (MODE == 1) rr.load_at(p4, nrec, rec);
                if constexpr (MODE == 2)
                {
                    res += ((own & 1u) + (other & 1u)) * 32u;
                    own >>= 1; other >>= 1;
                    if (own & 1u) rr.load_at(p4, res_nrec, res);
                }
            }
            if constexpr (DEEP)
            {
                if (!mbar_wait_warp(empty0 + 8 * stage, (free >> stage) & 1u, &sh->waits)) return false;
                tc_fence_after();
            }
            continue_stream<Pattern<BK>::kBits>(wb, __shfl_sync(0xffffffffu, wb[0], nxt));
            const uint32_t um = __shfl_sync(0xffffffffu, meta, i), sign2 = sign_mask(um >> 16, lane);
            uint32_t frag[16];
            const UnitSink<DEEP> sink{tmem_a - stage * (2 * kPfACols), sh, stage, (free >> stage) & 1u, (half_par ^ i ^ 1u) & 1u, i == 0, &ok, frag};
            if (MODE > 0 && refined)
            {
                if constexpr (MODE > 0)
                {
                    continue_stream<Pattern<RC>::kBits>(wr, __shfl_sync(0xffffffffu, wr[0], nxt));
                    decode_words<true, RC, BK>(wb, wr, consts_level4(__shfl_sync(0xffffffffu, ac, i), um, sign2), sink);
                }
            }
            else if constexpr (MODE != 1) decode_words<false, 0, BK>(wb, wr, consts_level2(sign2), sink);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if constexpr (!DEEP)
                if (!ok) return false;
            if (lane == 0) mbar_arrive32(full_a0 + 8 * stage);
            stage += kPfGroups;
            if (stage >= nst) { stage -= nst; free = ~free; }
        }
        if (end == n) break;
        write_accumulator_between(info_word);
        if (info.drain() && !mbar_wait_warp(saddr(&sh->acc_empty[info.acc()]), info.phase(), &sh->waits)) return false;
        end = n;
    }
    return true;
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

// grid = resident CTAs (one per SM), 608 threads
__global__ void __launch_bounds__(kPfThreads, 1) pf_gemm_kernel(const __grid_constant__ CUtensorMap tmap0,
                                                                const __grid_constant__ CUtensorMap tmap1, PfGemmArgs a)
{
    uint8_t* b_tiles = pf_tiles();                            // token tiles [rows][64 k] fp16, 128-byte swizzle (TMA boxes)
    PfShared* sh = pf_shared();
    const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (saddr(b_tiles) & 1023u)          // (never: the swizzled tiles would be read from the wrong places)
    {
        grid_dependency_wait();
        if (threadIdx.x == 0) atomicExch(a.status, 1);
        return;
    }

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kPfStages; ++s) { mbar_init(&sh->full_a[s], 8); mbar_init(&sh->full_b[s], 1); mbar_init(&sh->empty[s], 1); }
        for (int s = 0; s < kPfGroups; ++s) mbar_init(&sh->half_a[s], 1);
        for (int s = 0; s < kPfHeads; ++s) { mbar_init(&sh->head_full[s], 1); mbar_init(&sh->head_empty[s], 2 + kPfDecodeWarps); }
        for (int s = 0; s < 2; ++s) { mbar_init(&sh->acc_full[s], 2); mbar_init(&sh->acc_empty[s], kPfDecodeWarps); mbar_init(&sh->mma_done[s], 1); }
        sh->waits.aborted = 0; sh->waits.limit_ns = (unsigned long long)a.wait_ns;
        sh->C = (a.down ? a.I : a.H) / 128; sh->ld = a.down ? a.H : a.I;
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
    grid_dependency_wait();
    const uint32_t tmem = uniform(sh->tmem_base);

    const int N = a.down ? a.H : 2 * a.I, K = a.down ? a.I : a.H, C = K / 128, NS = N / 16, groups = N / 128;
    const int nitems = (int)uniform(a.plan[0]) * groups;
    const PfPass* passes = (const PfPass*)(a.plan + 4);
    const uint32_t full_a0 = saddr(sh->full_a), full_b0 = saddr(sh->full_b), empty0 = saddr(sh->empty), half_a0 = saddr(sh->half_a);
    // header slot of an item of this CTA and the phase of its barriers
    struct Head
    {
        uint32_t slot = 0, phase = 0;
        __device__ __forceinline__ void next() { if (++slot == kPfHeads) { slot = 0; phase ^= 1u; } }
    };
    auto wait_head = [&](const Head& h) { return mbar_wait_warp(saddr(&sh->head_full[h.slot]), h.phase, &sh->waits); };
    // Every role has its own loop over the items; nitem = items handled so far, par bit s = parity of the times stage s was used (how many
    // stages there are changes from pass to pass).
    if (warp == 0)
    {
        // ---- token tiles by TMA, ahead of the MMAs as far as there are stages; the headers of the items, one item ahead: the pass record
        // is fetched two items ahead of that, the table row one
        struct At { int pass, wg; } at0{(int)blockIdx.x / groups, (int)blockIdx.x % groups}, at1, at2;
        const int step_pass = (int)gridDim.x / groups, step_wg = (int)gridDim.x % groups, npass = nitems / groups;
        auto behind = [&](At t) {
            t.pass += step_pass; t.wg += step_wg;
            if (t.wg >= groups) { t.wg -= groups; ++t.pass; }
            return t;
        };
        auto pass_of = [&](const At& t) {
            const PfPass ps = t.pass < npass ? passes[t.pass] : PfPass{0, 0, 0, 0};
            return make_int4(ps.expert, ps.row0, ps.ntok, 0);
        };
        auto row_of = [&](const At& t, const int4& p) { return t.pass < npass && lane < kTableWidth ? a.table[(int64_t)p.x * kTableWidth + lane] : 0; };
        auto publish = [&](const At& t, const int4& p, int64_t w, const Head& h) {
            if (t.pass >= npass) return true;
            auto field = [&](int i) { return __shfl_sync(0xffffffffu, w, i); };
            const int down = a.down, o = down ? 5 : 1, nm = down ? a.nm_dn : a.nm_gu;
            const bool level4 = (int)field(0) >= 4;
            prefetch_item(level4, w, down, t.wg, C, nm, lane);
            const int64_t base = field(o), p4 = field(o + 1), d4 = field(o + 2), flags = field(o + 3), var = field(down ? 13 : 12);
            const int rc = (int)field(10 + down), bk = (int)(field(19) >> (8 * down)) & 0xFF, mode = !level4 ? 0 : flags ? 2 : 1;
            const int code = bk == 1 ? (mode && rc == 9 ? 11 : 10) : mode && rc >= 0 && rc < kNumCodes ? rc : 0;
            const int refined = mode == 2 ? nm : C, nst = chunk_stages(p.z), up = !down && t.wg >= a.I / 128;
            if (!mbar_wait_warp(saddr(&sh->head_empty[h.slot]), h.phase ^ 1u, &sh->waits)) return false;
            if (lane == 0)
            {
                PfItem& I = sh->item[h.slot];
                I.P.base = (const uint4*)base; I.P.p4 = (const uint8_t*)p4; I.P.d4 = (const uint32_t*)d4; I.P.flags = (const uint64_t*)flags;
                I.P.var = (const uint8_t*)var;
                I.nrec = (uint32_t)(NS * C * 32); I.res_nrec = (uint32_t)(NS * refined * 32);
                I.strip0 = t.wg * 8; I.unit0 = (uint32_t)(t.wg * 8 * C); I.res0 = (uint32_t)(t.wg * 8 * refined); I.res_strip = refined;
                I.out = (up ? a.out1 : a.out0) + (size_t)p.y * sh->ld + (up ? t.wg - a.I / 128 : t.wg) * 128;
                I.ntok = p.z; I.nst = nst; I.row0 = p.y; I.up = up; I.variant = (mode * kPfCodes + code) * 2 + (nst > 2);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->head_full[h.slot]);
            return true;
        };
        int4 p0 = pass_of(at0), p1;
        int64_t w1;
        Head head, ahead;
        publish(at0, p0, row_of(at0, p0), ahead);
        at1 = behind(at0); p1 = pass_of(at1); w1 = row_of(at1, p1);
        at2 = behind(at1);
        int4 p2 = pass_of(at2);
        uint32_t par = 0;
        int last_nst = 0;                    // stages of the previous item
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, head.next())
        {
            if (!wait_head(head)) break;
            const PfItem& I = sh->item[head.slot];
            const int ntok = (int)uniform(I.ntok), nbox = (ntok + kPfBoxRows - 1) / kPfBoxRows, row0 = (int)uniform(I.row0);
            const int nst = chunk_stages(ntok);
            const CUtensorMap* map = uniform(I.up) ? &tmap1 : &tmap0;
            bool ok = true;
            if (nst != last_nst)
                for (int s = 0; ok && s < kPfStages; ++s) ok = mbar_wait_warp(empty0 + 8 * s, ((par >> s) & 1u) ^ 1u, &sh->waits);
            last_nst = nst;
            const uint32_t tiles0 = saddr(b_tiles), bytes = 2u * (uint32_t)nbox * kPfBoxBytes, step = (uint32_t)(kPfBBoxes / nst) * kPfBoxBytes;
            uint32_t free = ~par, loaded = par;
            for (int c = 0, s = 0; c < C; ++c)
            {
                ok = ok && mbar_wait_warp(empty0 + 8 * s, (free >> s) & 1u, &sh->waits);
                if (!ok) break;
                loaded ^= 1u << s;
                const uint32_t d0 = tiles0 + s * step, d1 = d0 + step / 2, f = full_b0 + 8 * s;
                tma_load_chunk_elect(d0, d1, map, c * 128, row0, f, bytes);
                for (int j = 1; j < nbox; ++j) tma_load_more_elect(d0 + j * kPfBoxBytes, d1 + j * kPfBoxBytes, map, c * 128, row0 + j * kPfBoxRows, f);
                if (++s == nst) { s = 0; free = ~free; }
            }
            par = loaded;
            if (!ok || sh->waits.aborted) break;
            ahead.next();
            if (!publish(at1, p1, w1, ahead)) break;
            w1 = row_of(at2, p2);
            at1 = at2; p1 = p2;
            at2 = behind(at2); p2 = pass_of(at2);
        }
        __syncwarp();
        for (int s = 0; s < kPfStages; ++s) mbar_wait_own(full_b0 + 8 * s, ((par >> s) & 1u) ^ 1u);      // loads on their way
    }
    else if (warp == 1 || warp == kPfSecondIssuer)
    {
        // ---- MMA issue
        const int who = warp == 1 ? 0 : 1;
        uint32_t par = 0, nitem = 0;
        bool turns_before = true;            // the previous item's accumulators are one of the two pairs
        Head head;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, ++nitem, head.next())
        {
            if (!wait_head(head)) break;
            const int ntok = (int)uniform(sh->item[head.slot].ntok), ntok16 = (ntok + 15) & ~15, nst = chunk_stages(ntok);
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->head_empty[head.slot]);
            // the epilogues that have to be through: that of the item before the previous one, and that of the previous one where the two
            // share columns
            const uint32_t acc = nitem & 1u, phase = (nitem >> 1) & 1u;
            const bool turns = ntok <= 32;
            bool ok = mbar_wait_warp(saddr(&sh->acc_empty[acc]), phase ^ 1u, &sh->waits);
            if (ok && nitem > 0 && !(turns && turns_before)) ok = mbar_wait_warp(saddr(&sh->acc_empty[acc ^ 1u]), ((nitem - 1) >> 1) & 1u, &sh->waits);
            turns_before = turns;
            tc_fence_after();
            const bool split = split_chunks(ntok);
            const int first = split ? who : who ? C : 0, step = split ? 2 : 1;
            const uint32_t tmem_d = tmem + acc_column(ntok, acc) + (who ? acc_second(ntok) : 0u);
            // N <= 256 per instruction: one MMA per k-step, or two of (nearly) equal width
            const int n0 = nst > 2 ? ntok16 : ((ntok16 / 2 + 15) & ~15), n1 = ntok16 - n0;
            const uint32_t idesc0 = instr_desc(n0), idesc1 = instr_desc(n1 > 0 ? n1 : 16);
            const uint64_t bdesc0 = smem_desc(saddr(b_tiles), 16, 1024, 2);
            const uint32_t b_lo0 = (uint32_t)bdesc0, b_hi = (uint32_t)(bdesc0 >> 32);
            const uint32_t b_step = (uint32_t)(kPfBBoxes / nst) * (kPfBoxBytes >> 4), b_kb = b_step / 2;
            uint32_t full = par, s = split ? (uint32_t)who : 0u;
            for (int c = first; ok && c < C; c += step)
            {
                // weight and token tiles: two polls, one vote, one branch
                const uint32_t p = (full >> s) & 1u;
                uint32_t ready = mbar_poll(full_a0 + 8 * s, p);
                ready &= mbar_poll(full_b0 + 8 * s, p);
                if (__builtin_expect(!__all_sync(0xffffffffu, ready), 0))
                {
                    ok = mbar_wait_slow(full_a0 + 8 * s, p, &sh->waits) && mbar_wait_slow(full_b0 + 8 * s, p, &sh->waits);
                    if (!ok) break;
                }
                tc_fence_after();
                const uint32_t b_lo = b_lo0 + s * b_step, ta = tmem + kPfTmemCols - 2 * kPfACols - s * (2 * kPfACols);
                if (nst == 2) tc_mma_chunk2(tmem_d, tmem_d + n0, ta, b_lo, (uint32_t)(n0 * 8), b_kb, b_hi, idesc0, idesc1, (uint32_t)c, half_a0 + 8 * s, empty0 + 8 * s);
                else tc_mma_chunk(tmem_d, ta, b_lo, b_kb, b_hi, idesc0, (uint32_t)(c - first), empty0 + 8 * s);
                s += (uint32_t)step;
                if (s >= (uint32_t)nst) { s -= (uint32_t)nst; full = ~full; }
            }
            if (ok) tc_commit_elect(&sh->acc_full[acc]);
            par = stage_parities(par, C, nst);
            if (sh->waits.aborted) break;
        }
        __syncwarp();
        tc_commit_elect(&sh->mma_done[who]);
        mbar_wait_own(saddr(&sh->mma_done[who]), 0);
    }
    else
    {
        // ---- decode, then epilogue.  A warp may touch only the 32 tensor-memory lanes of its quarter (warp % 4): the four decode warps of a
        // quarter take its two strips x the chunk groups.  Group `half` of 8 warps decodes the chunks c = half (mod kPfGroups).
        const int half = (warp - 2) >> 3, units = (C - half + kPfGroups - 1) / kPfGroups;
        uint32_t par = 0, nitem = 0, info = 0;
        int prev_nst = kPfStages;
        Head head;
        bool left = false;                   // the previous item's accumulator is still to be written
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, ++nitem, head.next())
        {
            if (!wait_head(head)) break;
            const PfItem& I = sh->item[head.slot];
            const int nst = I.nst;
            const bool drain = nst > prev_nst;
            const uint32_t before = nitem - 1;
            info = head.slot | (head.slot ? head.slot - 1 : kPfHeads - 1) << 2 | (uint32_t)left << 4 | (uint32_t)drain << 5 | (before & 1u) << 6 | (before >> 1 & 1u) << 7;
            bool ok = true;
#define NQ_RUN(MODE, CODE, RC, BK) \
    case ((MODE) * kPfCodes + (CODE)) * 2: ok = decode_strip<MODE, RC, BK, false>(par, info); break; \
    case ((MODE) * kPfCodes + (CODE)) * 2 + 1: ok = decode_strip<MODE, RC, BK, true>(par, info); break;
#define NQ_RUN4(MODE) \
    NQ_RUN(MODE, 0, 0, 0) NQ_RUN(MODE, 1, 1, 0) NQ_RUN(MODE, 2, 2, 0) NQ_RUN(MODE, 3, 3, 0) NQ_RUN(MODE, 4, 4, 0) NQ_RUN(MODE, 5, 5, 0) \
    NQ_RUN(MODE, 6, 6, 0) NQ_RUN(MODE, 7, 7, 0) NQ_RUN(MODE, 8, 8, 0) NQ_RUN(MODE, 9, 9, 0) NQ_RUN(MODE, 10, 3, 1) NQ_RUN(MODE, 11, 9, 1)
            switch (I.variant)
            {
                NQ_RUN(0, 0, 0, 0) NQ_RUN(0, 10, 0, 1) NQ_RUN4(1) NQ_RUN4(2)
            }
#undef NQ_RUN4
#undef NQ_RUN
            par = stage_parities(par, C, nst) ^ (nst == 2 ? (units & 1u) << kPfStages : 0u);
            if (left && units <= units_before_epilogue(nst, drain)) write_accumulator(PfInfo{info});     // (the decoder function had no unit left behind it)
            prev_nst = nst;
            left = ok;
            if (!ok || sh->waits.aborted) break;
        }
        if (left && !sh->waits.aborted)
        {
            const uint32_t before = nitem - 1;
            write_accumulator_between((head.slot ? head.slot - 1 : kPfHeads - 1) << 2 | (before & 1u) << 6 | (before >> 1 & 1u) << 7);
        }
    }
    // Not at the start: with CTAs of the next pass waiting beside this one's, whole prefill calls took 7 % longer (geometric mean over 54 of 50 to 1,200 us).
    // It also keeps the chain's scratch safe: no kernel comes up before a GEMM has ended that lies between two uses of an array (zg, zd, y, the
    // pass list and the index arrays are written again call after call), so none can hold a line of its former contents in L1.
    launch_dependents();
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (sh->waits.aborted && threadIdx.x == 0) atomicExch(a.status, 1);      // every warp is through: none can give up after this look
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPfTmemCols) : "memory");
}

// ---------------------------------------------------------------- pass plan (device side, no host sync), see nq_plan.cuh
template <bool WINDOW>
__global__ void __launch_bounds__(kPlanThreads) pf_plan_kernel(const int* from, const int64_t* table, int E,
                                                               int pair0, int npairs, int* plan, int max_passes)
{
    __shared__ int s_warp[kPlanThreads / 32];
    launch_dependents();
    grid_dependency_wait();
    plan_passes<WINDOW>(from, table, E, pair0, npairs, plan, max_passes, s_warp);
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
    nq::launch_dependent(nq::pf_plan_kernel<false>, dim3(1), dim3(nq::kPlanThreads), 0, (cudaStream_t)stream, counts, table, E, 0, 0, plan, (plan_ints - 4) / 4);
    return nq::check_launch("nq_pf_plan");
}

int nq_pf_plan_window(const int32_t* start, const int64_t* table, int E, int pair0, int npairs, int32_t* plan, int plan_ints, void* stream)
{
    NQ_REQUIRE(start && table && plan && E > 0 && pair0 >= 0 && npairs >= 0, "nq_pf_plan_window: bad arguments");
    NQ_REQUIRE(plan_ints >= nq_pf_plan_ints(E, npairs), "nq_pf_plan_window: plan needs %d ints", nq_pf_plan_ints(E, npairs));
    nq::launch_dependent(nq::pf_plan_kernel<true>, dim3(1), dim3(nq::kPlanThreads), 0, (cudaStream_t)stream, start, table, E, pair0, npairs, plan, (plan_ints - 4) / 4);
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
    m1 = m0;
    if (!down)
        if (int e = nq::make_tile_map(&m1, act1, (size_t)pairs, K)) return e;
    nq::PfGemmArgs a{};
    a.table = table; a.plan = plan; a.out0 = out0; a.out1 = out1; a.status = status;
    a.H = H; a.I = I; a.nm_gu = nm_gu; a.nm_dn = nm_dn; a.down = down ? 1 : 0; a.wait_ns = wait_ns;
    nq::launch_dependent(nq::pf_gemm_kernel, dim3(ctas), dim3(nq::kPfThreads), nq::kPfSmem, (cudaStream_t)stream, m0, m1, a);
    return nq::check_launch("nq_pf_gemm");
}

int nq_pf_gemm(const int64_t* table, const int32_t* plan, const void* act0, const void* act1, int pairs, float* out0, float* out1,
               int H, int I, int nm_gu, int nm_dn, int down, int32_t* status, void* stream)
{
    return nq_pf_gemm_within(table, plan, act0, act1, pairs, out0, out1, H, I, nm_gu, nm_dn, down, status, nq::kPfWaitNs, stream);
}

}  // extern "C"
