// Dense decode of whole experts to fp16 matrices (loaders, checks).  HBM-bound by the fp16 output (2 B per weight written against
// 0.25-0.52 B per weight read).
//
// A warp takes a run of up to four consecutive units (16 rows x 128 k) of one projection, 24 warps on an SM: the records of the next unit
// are fetched into registers while the current one is decoded, its fragments go to shared memory with stmatrix (they are laid out like
// the operand that it stores) and from there to memory in 256-byte row segments.  us, one unit per warp through cp.async and 32 plain
// stores to shared memory / this: 4 experts of H 6,144, I 2,048 at level 2 70.2 / 59.0 (5.1 TB/s written), level 4 86.8 / 67.8, mixed
// 80.6 / 66.3; one expert at level 4 25.1 / 20.4; one of H 1,024, I 512 11.0 / 10.5.  Mixed with runs of 8 units 72.6, 16 warps of 128
// registers 79.3, bulk stores 79.8.  Back to back, a launch starts while the one before it drains: 68.4 -> 66.3, the smallest 11.3 -> 10.5.
#include "nq_common.cuh"
#include "nq_unit.cuh"

namespace nq {

constexpr int kDenseWarps = 8, kDenseCtas = 3;       // per CTA and per SM: 80 registers a thread
constexpr int kDenseRow = 272;                       // bytes from tile row to tile row: 256 and a 16-byte step, the eight rows of an stmatrix
                                                     // matrix fall on different banks
constexpr int kDenseTile = 16 * kDenseRow;
constexpr int kDenseRun = 4;                         // most units of a run (a lane holds the scalars of one: at most 32)
struct DenseJob
{
    ProjPlanes P;
    uint32_t nrec, res_nrec;         // records of the base and of the residual plane
    __half* out;                     // [N][K]
    int C, nm, unit, n;              // chunks per strip, refined ones of a masked strip, first unit, units
};
struct DenseShared { uint8_t tile[kDenseWarps][kDenseTile]; DenseJob job[kDenseWarps]; };
static_assert(sizeof(DenseShared) <= 48 * 1024, "more than a launch may ask for without opting in");
extern __shared__ __align__(128) uint8_t nq_dense_smem[];

__device__ __forceinline__ void stmatrix_x4(uint32_t addr, const uint32_t (&a)[4])
{
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]) : "memory");
}
// k-step T of a unit: matrices rows 0..7 and 8..15 at k 16 T, the same at k 16 T + 8; at = the address this lane supplies for T = 0
struct TileSink
{
    uint32_t at;
    template <int T>
    __device__ __forceinline__ void operator()(std::integral_constant<int, T>, const uint32_t (&a)[4]) const { stmatrix_x4(at + T * 32, a); }
};
// The tile to rows of out; the warp may fill it again afterwards.
__device__ __forceinline__ void store_tile(uint32_t tile, __half* out, size_t K, int lane)
{
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j)
    {
        const int r = 2 * j + (lane >> 4), c8 = lane & 15;      // two rows x 16 segments of 8 halves
        *(uint4*)(out + (size_t)r * K + c8 * 8) = lds128(tile + r * kDenseRow + c8 * 16);
    }
    __syncwarp();
}

// This warp's run.  MODE 0: level 2, 1: level 4, 2: level 4 in mask mode, 3: level 0 (zeros).
template <int MODE, int RC, int BK>
__device__ __noinline__ void dense_run()
{
    DenseShared& S = *(DenseShared*)nq_dense_smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nxt = ring_successor(lane);
    const DenseJob& J = S.job[warp];
    const int C = J.C, n = J.n;
    const uint8_t *base = (const uint8_t*)J.P.base, *p4 = J.P.p4;
    uint32_t rec = (uint32_t)J.unit * 32u + lane;
    RecordValues<BK> rb;
    RecordValues<RC> rr;
    if constexpr (MODE < 3) rb.template load_at<size_t>(base, J.nrec, rec);
    if constexpr (MODE == 1) rr.template load_at<size_t>(p4, J.res_nrec, rec);
    // scalars of unit J.unit + lane: ring signs and block word (meta = word | signs << 16), the block word's multipliers, mask mode: residual record
    uint32_t meta = 0, ac = 0, res = 0, refined = 0;
    if (MODE < 3 && lane < n)
    {
        const int u = J.unit + lane, s = u / C, ch = u - s * C;
        uint32_t at = (uint32_t)u;
        bool on = MODE == 1;
        if constexpr (MODE == 2)     // chunk ch is refined iff bit ch of flags[strip]; refined chunks are stored compactly, nm per strip (sm120/nqmoe.cu:202-206)
        {
            const unsigned long long flags = (unsigned long long)__ldg((const unsigned long long*)J.P.flags + s);
            on = flags >> ch & 1ull;
            at = (uint32_t)(s * J.nm + __popcll(flags & ((1ull << ch) - 1ull)));
        }
        if (J.P.var) meta = (uint32_t)__ldg(J.P.var + u) << 16;
        if (on)
        {
            const uint32_t word = __ldg(J.P.d4 + at) & 0xFFFFu;
            meta |= word;
            ac = block_multipliers(word);
        }
        res = at;
        refined = on;
    }
    if constexpr (MODE == 2)
    {
        refined = __ballot_sync(0xffffffffu, refined);
        const uint32_t r = __shfl_sync(0xffffffffu, res, 0);
        if (refined & 1u) rr.template load_at<size_t>(p4, J.res_nrec, r * 32u + lane);
    }
    int ch = J.unit % C;
    const size_t K = (size_t)C * 128;
    __half* out = J.out + (size_t)(J.unit / C) * 16 * K + (size_t)ch * 128;
    const uint32_t tile = smem_addr(S.tile[warp]), corner = ((lane & 7) + 8 * (lane >> 3 & 1)) * kDenseRow + 16 * (lane >> 4);
#pragma unroll 1
    for (int i = 0; i < n; ++i)
    {
        if constexpr (MODE < 3)
        {
            uint32_t wb[Pattern<BK>::kWords + 2], wr[Pattern<RC>::kWords + 2];
            const bool on = MODE == 1 || (MODE == 2 && (refined >> i & 1u));
            rb.words(wb, lane);
            if constexpr (MODE > 0)
                if (on) rr.words(wr, lane);
            if (i + 1 < n)
            {
                rec += 32;
                rb.template load_at<size_t>(base, J.nrec, rec);
                if constexpr (MODE == 1) rr.template load_at<size_t>(p4, J.res_nrec, rec);
                if constexpr (MODE == 2)
                {
                    const uint32_t r = __shfl_sync(0xffffffffu, res, i + 1);
                    if (refined >> i >> 1 & 1u) rr.template load_at<size_t>(p4, J.res_nrec, r * 32u + lane);
                }
            }
            continue_stream<Pattern<BK>::kBits>(wb, __shfl_sync(0xffffffffu, wb[0], nxt));
            const uint32_t um = __shfl_sync(0xffffffffu, meta, i), sign2 = sign_mask(um >> 16, lane);
            const TileSink sink{tile + corner};
            if (MODE > 0 && on)
            {
                if constexpr (MODE > 0)
                {
                    continue_stream<Pattern<RC>::kBits>(wr, __shfl_sync(0xffffffffu, wr[0], nxt));
                    decode_words<true, RC, BK>(wb, wr, consts_level4(__shfl_sync(0xffffffffu, ac, i), um, sign2), sink);
                }
            }
            else if constexpr (MODE != 1) decode_words<false, 0, BK>(wb, wr, consts_level2(sign2), sink);
        }
        else
        {
            const uint32_t zero[4] = {0u, 0u, 0u, 0u};
            for (int T = 0; T < 8; ++T) stmatrix_x4(tile + corner + T * 32, zero);
        }
        store_tile(tile, out, K, lane);
        if (++ch == C) { ch = 0; out += 15 * K; }
        out += 128;
    }
}

// grid (ceil(units / (8 run)), n_experts, 2 = gate|up / down); run = units of a run
__global__ void __launch_bounds__(32 * kDenseWarps, kDenseCtas) pf_decode_kernel(const int64_t* table, const int32_t* experts,
                                                                                __half* Wgu, __half* Wdn, int H, int I, int nm_gu, int nm_dn,
                                                                                int force_level, int run)
{
    launch_dependents();
    grid_dependency_wait();
    DenseShared& S = *(DenseShared*)nq_dense_smem;
    const int down = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __half* W = down ? Wdn : Wgu;
    const int N = down ? H : 2 * I, K = down ? I : H, C = K / 128, NS = N / 16, units = NS * C, nm = down ? nm_dn : nm_gu;
    const int unit = ((int)blockIdx.x * kDenseWarps + warp) * run;
    if (!W || unit >= units) return;     // warp-uniform
    const int64_t* row = table + (int64_t)experts[blockIdx.y] * kTableWidth;
    int level = (int)row[0];
    if (force_level > 0 && level > 0) level = force_level;
    const ProjPlanes P = planes_from_row(row, down);
    const int rc = (int)row[10 + down], bk = (int)(row[19] >> (8 * down)) & 0xFF, mode = level < 4 ? 0 : P.flags ? 2 : 1;
    if (lane == 0)
    {
        DenseJob& J = S.job[warp];
        J.P = P;
        J.nrec = (uint32_t)units * 32u; J.res_nrec = (uint32_t)(NS * (mode == 2 ? nm : C)) * 32u;
        J.out = W + (size_t)blockIdx.y * N * K;
        J.C = C; J.nm = nm; J.unit = unit; J.n = units - unit < run ? units - unit : run;
    }
    __syncwarp();
    if (level <= 0) dense_run<3, 0, 0>();
    else
    {
#define NQ_RUN(RES, RCV, BKV) do { if (RES && mode == 2) dense_run<RES ? 2 : 0, RCV, BKV>(); else dense_run<RES ? 1 : 0, RCV, BKV>(); } while (0)
        NQ_WITH_CODES(mode > 0, rc, bk, 0x3FF, NQ_RUN);
#undef NQ_RUN
    }
}

}  // namespace nq

extern "C" int nq_pf_decode(const int64_t* table, const int32_t* experts, int n_experts, void* Wgu, void* Wdn,
                            int H, int I, int nm_gu, int nm_dn, int force_level, void* stream)
{
    NQ_REQUIRE(table && experts, "nq_pf_decode: null table or expert list");
    NQ_REQUIRE(n_experts >= 0, "nq_pf_decode: n_experts = %d", n_experts);
    // gate|up is [2I][H] (K = H), down is [H][I] (K = I): K must be whole 128-wide chunks (at most 64 per strip, the width
    // of a flags word), row counts whole 16-row strips
    NQ_REQUIRE(H > 0 && I > 0 && H % 128 == 0 && H / 128 <= 64 && I % 8 == 0, "nq_pf_decode: H = %d, I = %d", H, I);
    NQ_REQUIRE(!Wdn || (I % 128 == 0 && I / 128 <= 64), "nq_pf_decode: I = %d must be a multiple of 128, at most 64 * 128", I);
    NQ_REQUIRE(nq::aligned16(Wgu) && nq::aligned16(Wdn), "nq_pf_decode: outputs must be 16-byte aligned");
    NQ_REQUIRE(force_level == 0 || force_level == 2 || force_level == 4, "nq_pf_decode: force_level = %d", force_level);
    if (n_experts == 0 || (!Wgu && !Wdn)) return NQ_OK;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nq::fail(NQ_ERR_CUDA, "nq_pf_decode: no usable current device");
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int ugu = Wgu ? (2 * I / 16) * (H / 128) : 0, udn = Wdn ? (H / 16) * (I / 128) : 0, units = ugu > udn ? ugu : udn;
    // Runs of more than one unit once every resident warp gets two of them (one expert of H 6,144, I 2,048: runs of 1 26.7, of 2 21.0 us).
    const long long want = (long long)n_experts * (ugu + udn) / ((long long)(sms > 0 ? sms : 148) * nq::kDenseCtas * nq::kDenseWarps * 2);
    const int run = want < 1 ? 1 : want > nq::kDenseRun ? nq::kDenseRun : (int)want;
    nq::launch_dependent(nq::pf_decode_kernel, dim3((units + nq::kDenseWarps * run - 1) / (nq::kDenseWarps * run), n_experts, 2), dim3(32 * nq::kDenseWarps),
                         sizeof(nq::DenseShared), (cudaStream_t)stream, table, experts, (__half*)Wgu, (__half*)Wdn, H, I, nm_gu, nm_dn, force_level, run);
    return nq::check_launch("nq_pf_decode");
}
