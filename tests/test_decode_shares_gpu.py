"""How the decode kernel cuts a call into shares and jobs, at the places where a cut can go wrong.  The outputs have to be those of
the oracle, and bit for bit the same however many of the kernel's CTAs find an SM at once."""
import random

import pytest
import torch

from tests.test_moe_layer_gpu import _check, _routing
from tests.util import expert_to_oracle

pytestmark = pytest.mark.gpu


def _layer(H, I, NE, levels, Bmax, topk, rank=0, had=128):
    from nestquant_b200 import moe
    gen = torch.Generator().manual_seed(NE)
    exs = [moe.Expert(H, I, seed=900 + i, rk_gu=0, rk_dn=7, var=True, sv=0.02, gen_device="cuda") for i in range(NE)]
    for ex in exs:
        ex.had_dn = had
        if rank:
            ex.set_lr(*[torch.randn(rank, n, generator=gen) * 0.02 for n in (H, I, I, I, I, I, H, H)])
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


# A CTA has room for 9 token rows at H = 6144, 13 at 4096, 6 at 8192 (of 272 bytes per 128 elements, beside 23 KB of routing and
# 20 KB of partial sums), and one expert's tokens make a run of up to 8, 16 or 32 of them, as many as fit.
@pytest.mark.parametrize("H,I,NE,topk,B,mode,rank,had", [
    (6144, 128, 40, 8, 32, "rand", 0, 128),     # 207 units per CTA, 6 tokens per expert: a share over two runs' halves takes two jobs
    (6144, 256, 4, 2, 32, "same", 0, 128),      # 32 tokens of one expert: runs of 8
    (8192, 128, 8, 8, 8, "same", 0, 128),       # 8 tokens of one expert, rows for 6
    (4096, 512, 6, 3, 17, "rand", 2, 512),      # runs of two column tiles, low rank, 512-wide rotation: finishers in two steps
    (768, 512, 16, 8, 32, "rand", 1, 128),      # runs of up to 32 tokens, four column tiles
    (128, 8192, 8, 8, 32, "same", 0, 128),      # 110 finishers per CTA and list: more than the queue holds
    (1024, 1024, 3, 2, 2, "same", 3, 512),      # the smallest call that shares its finishers
])
def test_cuts_against_the_oracle(H, I, NE, topk, B, mode, rank, had):
    levels = [(4, 2, 4, 4)[e % 4] for e in range(NE)]
    L, exs = _layer(H, I, NE, levels, B, topk, rank, had)
    rng = random.Random(NE + B)
    sel, rw = _routing(B, NE, topk, rng, mode)
    x = torch.randn(B, H, generator=torch.Generator().manual_seed(B)).bfloat16().half()
    _check(L, [expert_to_oracle(e) for e in exs], levels, x, sel, rw, (H, I, B, mode))
    assert L.status() == 0


@pytest.mark.parametrize("B", [1, 4])
def test_scale_vectors_aligned_to_8_bytes(B):
    """a decode call asks 8 bytes of the scale vectors, which may be views into a larger array: same bits as from aligned ones"""
    H, I, NE, topk = 1024, 512, 6, 3
    L, exs = _layer(H, I, NE, [4, 2] * 3, B, topk)
    sel, rw = (t.cuda() for t in _routing(B, NE, topk, random.Random(B)))
    x = torch.randn(B, H, device="cuda").bfloat16().half()
    want = L(x, sel, rw).clone()
    for e, ex in enumerate(exs):
        room = torch.zeros(ex.signs.numel() + 8, dtype=torch.float16, device="cuda")
        ex.signs = room[4:4 + ex.signs.numel()].copy_(ex.signs)
        assert ex.signs.data_ptr() % 16 == 8
        L.set(e, ex, (4, 2)[e % 2])
    assert torch.equal(L(x, sel, rw), want)
