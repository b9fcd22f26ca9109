// Warp-level pieces of the layer math around the GEMVs / GEMMs: the 128-point Hadamard rotation and fp16 <-> fp32
// vector access.  A warp holds a 128-vector as 4 consecutive elements per lane (element 4 * lane + i).
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace nq {

// normalised Sylvester-Hadamard transform of order 128 (reference: H128 in sm120/moe.py:168-172; the kernel-side
// butterfly it matches is sm120/nqmoe.cu:337-349)
__device__ __forceinline__ void wht128(float (&v)[4], int lane)
{
    const float a = v[0] + v[1], b = v[0] - v[1], c = v[2] + v[3], d = v[2] - v[3];
    v[0] = a + c; v[1] = b + d; v[2] = a - c; v[3] = b - d;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1)
    {
        const float s = (lane & m) ? -1.f : 1.f;       // o - v or v + o as one fma (exact either way)
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = fmaf(v[i], s, __shfl_xor_sync(0xffffffffu, v[i], m));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] *= 0.08838834764831845f;   // 1 / sqrt(128)
}
__device__ __forceinline__ void load4h(const __half* p, float (&f)[4])
{
    const uint2 u = *(const uint2*)p;
    const __half2 a = *(const __half2*)&u.x, b = *(const __half2*)&u.y;
    f[0] = __low2float(a); f[1] = __high2float(a); f[2] = __low2float(b); f[3] = __high2float(b);
}
__device__ __forceinline__ void store4h(__half* p, const float (&v)[4])
{
    const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    uint2 u; u.x = *(const uint32_t*)&a; u.y = *(const uint32_t*)&b;
    *(uint2*)p = u;
}

// Two fp32 values per register pair and instruction (each rounded on its own, like the scalar instruction)
__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpack2(uint64_t p, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// The same transform for eight 128-vectors per warp: lanes 4 v .. 4 v + 3 hold vector v, 32 elements each (lane bits
// and register bits are index bits of the vector, see the maps below).  Five of the seven butterfly stages stay inside a
// lane; two cross lanes (8 shuffles per vector instead of 20).  The passes that use it are bound by issue slots, so all but
// the first stage work on pairs of registers: 208 instead of 320 instructions, the same sums in the same order
// (b * -1 + a is a - b, rounded once).  Whole prefill calls are faster by less than their times spread (0.6 %).
__device__ __forceinline__ void wht128_x8(float (&v)[32], int lane)
{
    uint64_t w[16];
    const uint64_t minus = pack2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = pack2(v[2 * i] + v[2 * i + 1], v[2 * i] - v[2 * i + 1]);
#pragma unroll
    for (int h = 1; h < 16; h <<= 1)
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (!(i & h))
            {
                const uint64_t a = w[i], b = w[i | h];
                w[i] = add2(a, b); w[i | h] = fma2(b, minus, a);
            }
#pragma unroll
    for (int m = 1; m < 4; m <<= 1)
    {
        const float s = (lane & m) ? -1.f : 1.f;       // o - v or v + o as one fma (exact either way)
        const uint64_t s2 = pack2(s, s);
#pragma unroll
        for (int i = 0; i < 16; ++i)
        {
            float lo, hi;
            unpack2(w[i], lo, hi);
            w[i] = fma2(w[i], s2, pack2(__shfl_xor_sync(0xffffffffu, lo, m), __shfl_xor_sync(0xffffffffu, hi, m)));
        }
    }
    const uint64_t r = pack2(0.08838834764831845f, 0.08838834764831845f);
#pragma unroll
    for (int i = 0; i < 16; ++i) unpack2(mul2(w[i], r), v[2 * i], v[2 * i + 1]);
}
// Which 32 elements of its vector a lane holds is free (any assignment of the 7 index bits to 5 register bits and 2
// lane bits gives the same transform), so it is chosen for coalescing: the 4 lanes of a vector access adjacent pieces.
//   map H (fp16 arrays, 16-byte accesses; fp32 arrays, 32-byte accesses):
//                                          register 8 j + e of lane q = element 32 j + 8 q + e   (j < 4, e < 8)
//   map W (fp16 arrays, 32-byte accesses): register 16 j + e of lane q = element 64 j + 16 q + e (j < 2, e < 16)
// With 32 bytes per lane the four lanes of a vector cover one 128-byte line per access; with 16 (or 8) an access of the warp touches
// eight lines and half (or a quarter) of each.  WIDE: the array is aligned to 32 bytes; else the same elements go as two 16-byte pieces.
// 65,536 pairs of 6,144 (2,048) columns, us, 16 or 8 bytes per lane / 32: first pass 573 / 525 (it also writes the GEMM's k order without
// an exchange between lanes), middle pass 455 / 412, last pass 435 / 421.
// p points at the vector's first element, q = lane & 3.
template <bool WIDE>
__device__ __forceinline__ void load32b(const void* p, uint32_t* w)
{
    if constexpr (WIDE)
        asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"      // volatile, memory: stays behind a barrier or a wait in front of it
                     : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(p) : "memory");
    else
    {
        const uint4 a = ((const uint4*)p)[0], b = ((const uint4*)p)[1];
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    }
}
template <bool WIDE>
__device__ __forceinline__ void store32b(void* p, const uint32_t* w)
{
    if constexpr (WIDE)
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                     ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
    else
    {
        ((uint4*)p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        ((uint4*)p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}
template <bool WIDE>
__device__ __forceinline__ void load32f_mapH(const float* p, int q, float (&f)[32])
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        uint32_t w[8];
        load32b<WIDE>(p + 32 * j + 8 * q, w);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[8 * j + e] = __uint_as_float(w[e]);
    }
}
template <bool WIDE>
__device__ __forceinline__ void store32f_mapH(float* p, int q, const float (&v)[32])
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(v[8 * j + e]);
        store32b<WIDE>(p + 32 * j + 8 * q, w);
    }
}
template <bool WIDE>
__device__ __forceinline__ void load16w_mapW(const __half* p, int q, uint32_t (&w)[16])
{
#pragma unroll
    for (int j = 0; j < 2; ++j) load32b<WIDE>(p + 64 * j + 16 * q, w + 8 * j);
}
// kperm: the k order of the fused prefill GEMM (below); a lane holds whole groups of 16, so it is a choice of words
template <bool WIDE>
__device__ __forceinline__ void store32h_mapW(__half* p, int q, const float (&v)[32], bool kperm)
{
#pragma unroll
    for (int j = 0; j < 2; ++j)
    {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
        {
            const __half2 h = __floats2half2_rn(v[16 * j + 2 * i], v[16 * j + 2 * i + 1]);
            w[i] = *(const uint32_t*)&h;
        }
        const uint32_t o[8] = {w[0], kperm ? w[4] : w[1], kperm ? w[1] : w[2], kperm ? w[5] : w[3],
                               kperm ? w[2] : w[4], kperm ? w[6] : w[5], kperm ? w[3] : w[6], w[7]};
        store32b<WIDE>(p + 64 * j + 16 * q, o);
    }
}
__device__ __forceinline__ void store32h_mapH(__half* p, int q, const float (&v)[32])
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const __half2 h = __floats2half2_rn(v[8 * j + 2 * i], v[8 * j + 2 * i + 1]);
            w[i] = *(const uint32_t*)&h;
        }
        *(uint4*)(p + 32 * j + 8 * q) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
// k-permuted fp16 stores for the fused prefill GEMM, whose decode warps write weight fragments to tensor memory in
// their register order: inside every group of 16 consecutive k, position 4 i + {0, 1} holds k = 2 i + {0, 1} and
// position 4 i + {2, 3} holds k = 8 + 2 i + {0, 1} (i = 0 .. 3).
// map H: lane q holds 8 consecutive k of a 16-group (first half for even q, second for odd q); the two lanes of a pair
// swap two packed words so that each still writes 16 contiguous bytes.
__device__ __forceinline__ void store32h_mapH_kperm(__half* p, int q, const float (&v)[32], bool live)
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const __half2 h = __floats2half2_rn(v[8 * j + 2 * i], v[8 * j + 2 * i + 1]);
            w[i] = *(const uint32_t*)&h;
        }
        const bool odd = q & 1;
        // even lane (k 0..7 of the group) keeps words 0, 1 and needs the partner's words 0, 1 (k 8..11);
        // odd lane (k 8..15) keeps words 2, 3 and needs the partner's words 2, 3 (k 4..7)
        const uint32_t s0 = __shfl_xor_sync(0xffffffffu, odd ? w[0] : w[2], 1), s1 = __shfl_xor_sync(0xffffffffu, odd ? w[1] : w[3], 1);
        const uint4 o = odd ? make_uint4(s0, w[2], s1, w[3]) : make_uint4(w[0], s0, w[1], s1);
        // group base = 32 j + 16 (q >> 1); even lane writes positions 0..7, odd lane positions 8..15
        if (live) *(uint4*)(p + 32 * j + 16 * (q >> 1) + 8 * (q & 1)) = o;      // every lane takes part in the exchange above
    }
}
// the same permutation for a lane holding 4 consecutive k (element 4 * lane + i of a 128-vector)
__device__ __forceinline__ void store4h_kperm(__half* vec, int lane, const float (&v)[4])
{
    const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    const int q = lane & 3, half = q >> 1, i0 = (2 * q) & 3;
    uint32_t* g = (uint32_t*)(vec + 16 * (lane >> 2));
    g[2 * i0 + half] = *(const uint32_t*)&a;
    g[2 * (i0 + 1) + half] = *(const uint32_t*)&b;
}

// fused forms (no staging array): v = x * s for packed fp16 x (map H); v *= s, v += z * s, sum v * s for an fp16 vector s (map H,
// aligned to 8 bytes)
__device__ __forceinline__ void load16w_mapH(const __half* p, int q, uint32_t (&w)[16])
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        const uint4 u = *(const uint4*)(p + 32 * j + 8 * q);
        w[4 * j] = u.x; w[4 * j + 1] = u.y; w[4 * j + 2] = u.z; w[4 * j + 3] = u.w;
    }
}
// the same words from a vector that is aligned to 8 bytes only
__device__ __forceinline__ void load16w_mapH_align8(const __half* p, int q, uint32_t (&w)[16])
{
#pragma unroll
    for (int j = 0; j < 8; ++j)
    {
        const uint2 u = *(const uint2*)(p + 32 * (j >> 1) + 8 * q + 4 * (j & 1));
        w[2 * j] = u.x; w[2 * j + 1] = u.y;
    }
}
// v = x * s for the lane's 32 elements, both given as packed fp16 words of one map (fp32 products)
__device__ __forceinline__ void mul32w(const uint32_t (&xw)[16], const uint32_t (&sw)[16], float (&v)[32])
{
#pragma unroll
    for (int i = 0; i < 16; ++i)
    {
        const __half2 a = *(const __half2*)&xw[i], b = *(const __half2*)&sw[i];
        v[2 * i] = __low2float(a) * __low2float(b); v[2 * i + 1] = __high2float(a) * __high2float(b);
    }
}
template <class F>
__device__ __forceinline__ void each32h_mapH(const __half* p, int q, F&& f)
{
#pragma unroll
    for (int j = 0; j < 8; ++j)
    {
        const uint2 u = *(const uint2*)(p + 32 * (j >> 1) + 8 * q + 4 * (j & 1));
        const __half2 a = *(const __half2*)&u.x, b = *(const __half2*)&u.y;
        f(4 * j, __low2float(a)); f(4 * j + 1, __high2float(a)); f(4 * j + 2, __low2float(b)); f(4 * j + 3, __high2float(b));
    }
}
__device__ __forceinline__ void scale32h_mapH(const __half* p, int q, float (&v)[32]) { each32h_mapH(p, q, [&](int i, float s) { v[i] *= s; }); }
__device__ __forceinline__ void axpy32h_mapH(const __half* p, int q, float z, float (&v)[32]) { each32h_mapH(p, q, [&](int i, float s) { v[i] += z * s; }); }
__device__ __forceinline__ float dot32h_mapH(const __half* p, int q, const float (&v)[32])
{
    float d = 0.f;
    each32h_mapH(p, q, [&](int i, float s) { d += v[i] * s; });
    return d;
}

__device__ __forceinline__ float silu(float g) { return g / (1.f + __expf(-g)); }

}  // namespace nq
