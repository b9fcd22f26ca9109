// Streams of packed planes, straight into registers: a warp that decodes a unit for ~1 us between two loads needs no deeper pipeline than the
// records of the next unit, and no copies through shared memory.
//
// Plane layout (sm120/moe.py:36-49): a record of BITS bits is cut into pieces - BITS / 128 pieces of 128 bits, then a
// 64-, a 32- and a 16-bit piece as the binary digits of BITS % 128 say, then a tail of BITS % 16 bits - and every piece
// kind is stored as its own array over all records of the plane (the tail bit-packed, followed by a 4-byte pad).  The
// base plane of window code 0 is the special case of one 128-bit piece.  32 records make a unit, so every piece array advances by a
// fixed number of bytes per unit.
#pragma once
#include "nq_format.cuh"

namespace nq {

// Shared-memory operands are 32-bit shared-space addresses (smem_addr of a pointer), so that every piece is an immediate offset from one register.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint4 lds128(uint32_t a)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
// pieces of a record of window code CODE
template <int CODE>
struct RecordLayout
{
    static constexpr int kBits = Pattern<CODE>::kBits;
    static constexpr int n128 = kBits / 128, rem = kBits % 128, T = kBits % 16;
    static constexpr bool has64 = (rem & 64) != 0, has32 = (rem & 32) != 0, has16 = (rem & 16) != 0;
    static constexpr bool tail2 = T != 0 && (32 % (T ? T : 1)) != 0;          // a lane's tail can straddle two words
    static_assert(n128 <= 1, "a record has one 128-bit piece at most");
    // the tail lands in the upper half of the 16-bit piece's word when the pieces before it end on a half word
    static constexpr bool tail_joins = T != 0 && ((kBits - T) & 31) == 16;
};

// Window codes (bit c = code c) whose records have a 128-bit piece: the first sub-array of their planes has 16 bytes per record, that of the
// others 8.
template <int... C>
constexpr uint32_t codes_with_128(std::integer_sequence<int, C...>) { return (0u | ... | ((uint32_t)(RecordLayout<C>::n128 != 0) << C)); }
constexpr uint32_t kWideCodes = codes_with_128(std::make_integer_sequence<int, 10>{});

// Plane bytes are used once: they bypass L1, which holds the token rows.
__device__ __forceinline__ uint4 ldg_stream128(const void* p)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ldg_stream64(const void* p)
{
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg_stream32(const void* p)
{
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg_stream16(const void* p)
{
    uint16_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

template <int CODE>
struct RecordValues
{
    using L = RecordLayout<CODE>;
    uint4 v128; uint2 v64, vtail; uint32_t v32, v16;      // pieces in flight

    // fetch record r of a plane of nrec records.  One index and one address for all pieces, where the reader below keeps an address per
    // piece: the prefill GEMM has no registers for up to six of them.  Offset: uint32_t for planes below 4 GB.
    template <class Offset = uint32_t>
    __device__ __forceinline__ void load_at(const uint8_t* plane, uint32_t nrec, uint32_t r)
    {
        constexpr uint32_t b64 = 16 * L::n128, b32 = b64 + (L::has64 ? 8 : 0), b16 = b32 + (L::has32 ? 4 : 0), bt = b16 + (L::has16 ? 2 : 0);
        if constexpr (L::n128) v128 = ldg_stream128(plane + (size_t)r * 16);
        if constexpr (L::has64) v64 = ldg_stream64(plane + ((Offset)nrec * b64 + (Offset)r * 8));
        if constexpr (L::has32) v32 = ldg_stream32(plane + ((Offset)nrec * b32 + (Offset)r * 4));
        if constexpr (L::has16) v16 = ldg_stream16(plane + ((Offset)nrec * b16 + (Offset)r * 2));
        if constexpr (L::T != 0)
        {
            const uint8_t* p = plane + ((Offset)nrec * bt + (((Offset)r * L::T) >> 5) * 4);
            vtail.x = ldg_stream32(p);
            if constexpr (L::tail2) vtail.y = ldg_stream32(p + 4);
        }
    }
    // the fetched record as stream words w[0 .. kWords), bits past the record zero
    __device__ __forceinline__ void words(uint32_t* w, int lane) const
    {
        int k = 0;
        if constexpr (L::n128) { w[k++] = v128.x; w[k++] = v128.y; w[k++] = v128.z; w[k++] = v128.w; }
        if constexpr (L::has64) { w[k++] = v64.x; w[k++] = v64.y; }
        if constexpr (L::has32) w[k++] = v32;
        if constexpr (L::has16) w[k++] = v16;
        if constexpr (L::T != 0)
        {
            const int sh = (lane * L::T) & 31;
            uint32_t v = L::tail2 ? __funnelshift_r(vtail.x, vtail.y, sh) : vtail.x >> sh;
            v &= (1u << L::T) - 1u;
            if constexpr (L::tail_joins) w[k - 1] |= v << 16;
            else w[k++] = v;
        }
    }
};
template <int CODE>
struct RecordReader : RecordValues<CODE>
{
    using L = RecordLayout<CODE>;
    using V = RecordValues<CODE>;
    const uint8_t *p128, *p64, *p32, *p16, *ptail;

    __device__ __forceinline__ void init(const void* plane, size_t nrec, size_t unit0, int lane)
    {
        const uint8_t* p = (const uint8_t*)plane;
        if constexpr (L::n128) { p128 = p + unit0 * 512 + lane * 16; p += nrec * 16; }
        if constexpr (L::has64) { p64 = p + unit0 * 256 + lane * 8; p += nrec * 8; }
        if constexpr (L::has32) { p32 = p + unit0 * 128 + lane * 4; p += nrec * 4; }
        if constexpr (L::has16) { p16 = p + unit0 * 64 + lane * 2; p += nrec * 2; }
        if constexpr (L::T != 0) ptail = p + unit0 * (4 * L::T) + ((lane * L::T) >> 5) * 4;
    }
    // fetch the unit at the read position and move on
    __device__ __forceinline__ void fetch()
    {
        if constexpr (L::n128) { V::v128 = ldg_stream128(p128); p128 += 512; }
        if constexpr (L::has64) { V::v64 = ldg_stream64(p64); p64 += 256; }
        if constexpr (L::has32) { V::v32 = ldg_stream32(p32); p32 += 128; }
        if constexpr (L::has16) { V::v16 = ldg_stream16(p16); p16 += 64; }
        if constexpr (L::T != 0)
        {
            V::vtail.x = ldg_stream32(ptail);
            if constexpr (L::tail2) V::vtail.y = ldg_stream32(ptail + 4);
            ptail += 4 * L::T;
        }
    }
};

}  // namespace nq
