// A whole prefill call: sort, pass list, and chunk by chunk the two GEMMs with the passes around them, enqueued by one call of the host.
// The reference's host side (sm120/moe.py:282-327) makes one call per kernel; from Python those take 92 to 94 us, more than the GPU needs for a short
// prompt on a small layer.  A call per kernel / this, the same kernels, us back to back: 75 tokens, 64 experts, H 1,024, I 512: 94.3 / 80.3;
// 110 tokens, 25 experts, H 768, I 640: 92.4 / 51.8.
#include "nq_common.cuh"

namespace nq {
int sort_pairs(const int64_t* sel, const void* rw, const int64_t* table, int T, int topk, int E, int32_t* pe, int32_t* pt, int32_t* pos, int32_t* start,
               int32_t* hits, int32_t* scratch, int scratch_ints, int32_t* plan, int plan_ints, void* stream);
}

extern "C" int nq_prefill(const NqPrefill* p, void* stream)
{
    NQ_REQUIRE(p, "nq_prefill: null arguments");
    NQ_REQUIRE(p->T >= 0 && p->topk >= 1 && (long long)p->T * p->topk <= 0x7fffffffLL, "nq_prefill: T = %d, topk = %d", p->T, p->topk);
    const int P = p->T * p->topk;
    if (P == 0) return NQ_OK;
    NQ_REQUIRE(p->R >= 1 && p->xg && p->xu && p->y && p->acc_g && p->acc_u && p->h && p->zg && p->zd && p->plan && p->status && p->start,
               "nq_prefill: null scratch or R = %d", p->R);
    NQ_REQUIRE(!p->hits || p->hit_counts, "nq_prefill: hits without hit_counts");
    NQ_REQUIRE(p->world <= 0 || (p->peer_x && (long long)p->world * p->tokens_per_rank >= p->T), "nq_prefill: %d tokens on %d ranks of %d", p->T, p->world,
               p->tokens_per_rank);      // (a token behind them would be looked for in a buffer that is not there)
    const int H = p->H, I = p->I, E = p->E, R = p->R < P ? p->R : P;
    NQ_REQUIRE(E >= 1 && p->plan_ints >= nq_pf_plan_ints(E, R), "nq_prefill: plan needs %d ints", nq_pf_plan_ints(E, R));
    if (p->hits && cudaMemsetAsync(p->hit_counts, 0, sizeof(int32_t) * E, (cudaStream_t)stream) != cudaSuccess)
        return nq::fail(NQ_ERR_CUDA, "nq_prefill: memset failed");
    // one chunk: the sort writes the pass list too
    if (int e = nq::sort_pairs(p->sel, p->rw, p->table, p->T, p->topk, E, p->pe, p->pt, p->pos, p->start, p->hits ? p->hit_counts : nullptr, p->sort_scratch,
                               p->sort_scratch_ints, R == P ? p->plan : nullptr, p->plan_ints, stream))
        return e;
    if (p->hits)
        if (int e = nq_pf_hits(p->hit_counts, p->hits, E, stream)) return e;
    for (int c0 = 0, n; c0 < P; c0 += n)
    {
        n = P - c0 < R ? P - c0 : R;
        if (R < P)
            if (int e = nq_pf_plan_window(p->start, p->table, E, c0, n, p->plan, p->plan_ints, stream)) return e;
        const int32_t *pt = p->pt + c0, *pe = p->pe + c0;
        if (int e = p->world > 0 ? nq_pf_pre_ep(p->peer_x, p->world, p->tokens_per_rank, pt, pe, n, p->table, E, p->xg, p->xu, p->zg, H, I, 1, stream)
                                 : nq_pf_pre(p->x, pt, pe, n, p->table, E, p->xg, p->xu, p->zg, H, I, 1, stream))
            return e;
        if (int e = nq_pf_gemm(p->table, p->plan, p->xg, p->xu, n, p->acc_g, p->acc_u, H, I, p->nm_gu, p->nm_dn, 0, p->status, stream)) return e;
        if (int e = nq_pf_mid(p->acc_g, p->acc_u, p->zg, pe, n, p->table, E, p->h, p->zd, H, I, 1, stream)) return e;
        if (int e = nq_pf_gemm(p->table, p->plan, p->h, nullptr, n, p->y, nullptr, H, I, p->nm_gu, p->nm_dn, 1, p->status, stream)) return e;
        if (int e = nq_pf_combine(p->y, p->zd, p->pos, p->sel, p->rw, p->T, p->topk, p->table, E, p->out, H, I, c0, n, c0 > 0, stream)) return e;
    }
    return NQ_OK;
}
