"""How the decode kernel cuts a call into shares and jobs, at the places where a cut can go wrong.  The outputs have to be those of
the oracle, and bit for bit the same however many of the kernel's CTAs find an SM at once."""
import random

import pytest
import torch

from tests.test_moe_layer_gpu import _routing

pytestmark = pytest.mark.gpu


def _layer(H, I, NE, levels, Bmax, topk, rk_gu=0, rk_dn=7):
    from nestquant_b200 import moe
    exs = [moe.Expert(H, I, seed=900 + i, rk_gu=rk_gu, rk_dn=rk_dn, var=True, sv=0.02, gen_device="cuda") for i in range(NE)]
    L = moe.MoELayer(NE, H, I, Bmax=Bmax, topk=topk)
    for e in range(NE):
        L.set(e, exs[e], levels[e])
    return L, exs


@pytest.mark.parametrize("H,I,NE,topk,B,level", [(6144, 2048, 8, 8, 1, 2), (6144, 2048, 12, 8, 3, 4), (2048, 1024, 24, 4, 32, 2)])
def test_same_bits_when_other_work_holds_sms(H, I, NE, topk, B, level):
    """The call beside a long kernel that holds some of the SMs: CTAs that start late find their shares drawn by the others, which
    then work on several shares of a list, whose rows must not touch those of the next list."""
    L, exs = _layer(H, I, NE, [level] * NE, B, topk)
    rng = random.Random(H + B)
    side = torch.cuda.Stream()
    for held, rows in ((1, 12000), (20, 12000), (75, 8000), (130, 6000)):
        sel, rw = (t.cuda() for t in _routing(B, NE, topk, rng))
        x = torch.randn(B, H, device="cuda").bfloat16().half()
        alone = L(x, sel, rw).clone()
        work, out = torch.ones(rows, 512 * held, device="cuda"), torch.empty(rows, 512 * held, device="cuda")
        torch.cumsum(work, 0, out=out)
        torch.cuda.synchronize()
        ends = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
        with torch.cuda.stream(side):
            ends[0].record()
            torch.cumsum(work, 0, out=out)      # a column per thread, row after row: one CTA of 512 threads per 512 columns
            ends[1].record()
        ends[2].record()
        y = L(x, sel, rw)
        ends[3].record()
        torch.cuda.synchronize()
        assert ends[0].elapsed_time(ends[3]) < ends[0].elapsed_time(ends[1]), "the call did not run beside the other kernel"
        assert L.status() == 0
        assert torch.equal(alone, y), (held, int((alone != y).sum()), float((alone - y).abs().max()))
        for t in (L.cnt_gu, L.cnt_d, L.wq):
            assert int(t.abs().sum()) == 0
