// The decode of the 64 weights that a lane holds of a 16x128 unit, and the choice of its compiled form.
#pragma once
#include "nq_stream.cuh"

namespace nq {

// ring sign of this lane's ring (bit g of the unit's sign byte) as an fp16x2 xor mask
__device__ __forceinline__ uint32_t sign_mask(uint32_t var_byte, int lane) { return ((var_byte >> (lane >> 2)) & 1u) * 0x80008000u; }

// Decode the lane's 64 weights of a unit whose stream words are in registers (wb: the base record, wr: the residual record,
// each already continued with the ring successor's first word: kWords + 2 words).  sink(integral_constant<T>, a[4])
// receives, for k-step T = 0..7, the m16n8k16 A-fragment registers: a[q] = rows g + 8 (q & 1),
// k = 16 T + 2 t4 + 8 (q >> 1) + {0, 1}.
template <bool RES, int RC, int BK, class Sink>
__device__ __forceinline__ void decode_words(const uint32_t* wb, const uint32_t* wr, const UnitConsts& k, Sink&& sink)
{
    static_for<8>([&](auto tc) {
        uint32_t a[4];
        decode_kstep<RES, RC, BK, decltype(tc)::value>(wb, wr, k, a);
        sink(tc, a);
    });
}
// Base code 1 is built with the residual codes it ships with (3 for gate|up, 9 for down: sm120/NQ_RES_V2.md:9-13).
__host__ __device__ constexpr bool bk1_has_rc(int rc) { return rc == 3 || rc == 9; }

// run-time (level 4?, residual code, base code) -> compile-time: expands X(RES, RC, BK) for the matching combination.
// CODES: bit c set = residual code c is built (others fall back to code 0, as the reference's kernels do for codes they
// were not compiled with, sm120/nqmoe.cu:547-548).  A macro, not a callback: every decoder instance must be inlined into
// the loop that holds its accumulators.
#define NQ_CODE_CASE(CODES, c, X) case c: if constexpr (((CODES) >> c) & 1) { X(true, c, 0); } break;
#define NQ_WITH_CODES(level4, rc, bk, CODES, X)                                                  \
    do {                                                                                         \
        if ((bk) == 1)                                                                           \
        {                                                                                        \
            if (!(level4)) { X(false, 0, 1); }                                                   \
            else if ((rc) == 9) { X(true, 9, 1); }                                               \
            else { X(true, 3, 1); }                                                              \
        }                                                                                        \
        else if (!(level4)) { X(false, 0, 0); }                                                  \
        else                                                                                     \
            switch ((((CODES) >> (rc)) & 1) ? (rc) : 0)                                          \
            {                                                                                    \
                NQ_CODE_CASE(CODES, 1, X) NQ_CODE_CASE(CODES, 2, X) NQ_CODE_CASE(CODES, 3, X)     \
                NQ_CODE_CASE(CODES, 4, X) NQ_CODE_CASE(CODES, 5, X) NQ_CODE_CASE(CODES, 6, X)     \
                NQ_CODE_CASE(CODES, 7, X) NQ_CODE_CASE(CODES, 8, X) NQ_CODE_CASE(CODES, 9, X)     \
                default: X(true, 0, 0); break;                                                   \
            }                                                                                    \
    } while (0)

}  // namespace nq
