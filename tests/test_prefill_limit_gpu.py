"""Launches of the fused prefill GEMM whose waits run out: they end by themselves, say so in the status word, leave nothing of theirs in
flight, and the next launch finds tensor memory and buffers as it should."""
import pytest
import torch

from nestquant_b200 import ext, moe
from nestquant_b200.capi import check, current_stream, lib

pytestmark = pytest.mark.gpu


def _launch(down, E, H, I, tokens):
    """a GEMM over E experts of `tokens` pairs each -> (run(limit in ns, None: the usual one) -> status word, outputs).  The planes lie
    in pinned host memory, where every read takes its time: the token tiles are there long before the first weight tile, and the waits
    for weights last tens of us."""
    L = moe.MoELayer(E, H, I, Bmax=1, topk=1)
    exs = [moe.Expert(H, I, seed=70 + e, rk_gu=0, rk_dn=7, var=True, sv=0.02) for e in range(E)]
    for e, ex in enumerate(exs):
        for p in (ex.gu, ex.dn):
            p.base, p.p4, p.d4, p.var = (t.cpu().pin_memory() for t in (p.base, p.p4, p.d4, p.var))
        L.set(e, ex, (4, 2)[e % 2])
    pairs, K, N = E * tokens, (I if down else H), (H if down else I)
    gen = torch.Generator(device="cuda").manual_seed(3)
    act = [torch.randn(pairs, K, generator=gen, device="cuda").half() for _ in range(1 if down else 2)]
    out = [torch.empty(pairs, N, device="cuda") for _ in act]
    plan = torch.empty(ext.pf_plan_ints(E, pairs), dtype=torch.int32, device="cuda")
    ext.pf_plan(torch.full((E,), tokens, dtype=torch.int32, device="cuda"), L.table, plan, pairs)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(limit):
        status.zero_()
        for o in out:
            o.fill_(float("nan"))
        args = [L.table.data_ptr(), plan.data_ptr(), act[0].data_ptr(), None if down else act[1].data_ptr(), pairs, out[0].data_ptr(),
                None if down else out[1].data_ptr(), H, I, 0, 0, int(down), status.data_ptr()]
        if limit is None:
            check(lib().nq_pf_gemm(*args, current_stream()), "pf_gemm")
        else:
            check(lib().nq_pf_gemm_within(*args, limit, current_stream()), "pf_gemm_within")
        torch.cuda.synchronize()
        return int(status)

    run.keep = (L, exs, act, plan)
    return run, out


CASES = [(True, 2, 8192, 512, 16),        # 128 items, one per CTA: a CTA's loads are all issued at the start
         (False, 6, 1024, 2048, 384)]     # 192 items of the widest passes: loads and MMAs in flight throughout


@pytest.mark.parametrize("down,E,H,I,tokens", CASES)
def test_launch_that_gives_up_leaves_nothing_behind(down, E, H, I, tokens):
    run, out = _launch(down, E, H, I, tokens)
    assert run(None) == 0
    ref = [o.clone() for o in out]
    assert all(bool(torch.isfinite(r).all()) for r in ref)
    gave_up = 0
    for limit in (0, 5000, 10000, 20000, 40000, 80000) * 3:
        run(limit)
        gave_up += not all(torch.equal(o, r) for o, r in zip(out, ref))
        assert run(None) == 0
        assert all(torch.equal(o, r) for o, r in zip(out, ref)), f"after a launch with a limit of {limit} ns"
    assert gave_up > 0


@pytest.mark.parametrize("down,E,H,I,tokens", CASES)
def test_launch_that_gives_up_says_so(down, E, H, I, tokens):
    """whichever warp gives up, and whenever: with one item per CTA the warp that loads the tokens is long through by then"""
    run, out = _launch(down, E, H, I, tokens)
    assert run(None) == 0
    ref = [o.clone() for o in out]
    raised = 0
    for limit in (0, 5000, 10000, 20000, 40000, 80000) * 3:
        status = run(limit)
        raised += status
        assert status == 1 or all(torch.equal(o, r) for o, r in zip(out, ref)), f"limit {limit} ns: outputs missing, status 0"
    assert raised > 0
