"""The fused prefill GEMM changes its layout with the width of a pass (2, 3, 4 or 6 stages beside the accumulator; up to 64 tokens two accumulators,
up to 32 two pairs of them in turn): passes of every width one after the other on the same CTAs, for few and odd numbers of chunks, experts of
every mode (level 2, level 4, mask mode) and both base codes among them."""
import pytest
import torch

from nestquant_b200 import moe
from tests.prefill_lib import prefill_library
from tests.util import layer_errors

pytestmark = pytest.mark.gpu

# pairs of the experts, in expert order: edges of the layouts (128, 256), of the passes (384) and of the token boxes (64)
COUNTS = [384, 1, 128, 300, 129, 64, 256, 65, 385, 20, 257, 0, 127, 383, 16]


# gate|up has 15 passes x I / 64 items of H / 128 chunks, down 15 x H / 128 items of I / 128.  `turns`: the projection whose CTAs take three
# items or more, so that a layout follows another one twice; with three chunks or more it then also uses the unit stages that lie where
# the accumulator before it was, which one and two chunks leave out.
@pytest.mark.parametrize("H,I,turns", [(128, 2048, "gate|up"), (256, 2048, "gate|up"), (384, 2048, "gate|up"), (640, 2048, "gate|up"),
                                       (1152, 1664, "gate|up"), (2048, 1664, "gate|up"), (2048, 128, None), (2048, 256, None),
                                       (2560, 384, "down"), (2560, 640, "down")])
def test_passes_of_every_width_in_turn(H, I, turns):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    passes = sum((c + 383) // 384 for c in COUNTS)
    assert passes == 15 and (turns is None or passes * (I // 64 if turns == "gate|up" else H // 128) > 2 * sms)
    _check(COUNTS, H, I)


# Narrow passes in a row, with a wide one between: accumulators in turn and not, one chunk (nothing for the second issuing warp) to seven.
NARROW = [31, 1, 32, 16, 33, 5, 32, 64, 2, 30, 65, 8, 31, 384, 17, 32, 129, 24]


@pytest.mark.parametrize("H,I", [(128, 2048), (256, 2048), (384, 2048), (896, 2048), (2048, 128), (2560, 256), (2560, 640)])
def test_narrow_passes_in_a_row(H, I):
    _check(NARROW, H, I)


# Every layout behind every other one, at both ends of the four-stage widths.
MIDDLE = [192, 129, 193, 160, 384, 144, 16, 191, 128, 130, 257, 192, 256, 40, 384, 193, 65, 300, 8, 256, 176]


@pytest.mark.parametrize("H,I", [(128, 2048), (384, 2048), (640, 2048), (1152, 1664), (2560, 640)])
def test_four_stage_passes_in_turn(H, I):
    _check(MIDDLE, H, I)


def _check(counts, H, I):
    nm = [max(1, k // 256) for k in (H, I)]
    exs, levels = [], []
    for e in range(len(counts)):
        masked, base = e % 5 in (1, 3), int(e % 5 == 4 or e % 10 == 3)
        exs.append(moe.Expert(H, I, seed=60 + e, nm_gu=nm[0] if masked else None, nm_dn=nm[1] if masked else None, rk_gu=3 if base else (0, 6)[e % 2],
                              rk_dn=9 if base else 7, var=True, sv=0.02, bk_gu=base, bk_dn=base))
        levels.append(4 if masked else (4, 4, 2)[e % 3])
    _compare(counts, H, I, exs, levels, nm)


# Every residual code in mask mode and with either base code, in passes of two stages, of three and of six with an odd number of chunks.
@pytest.mark.parametrize("rk,base", [(rk, 0) for rk in range(10)] + [(3, 1), (9, 1)])
def test_every_code_in_wide_passes(rk, base):
    H, I, nm = 640, 384, (2, 1)
    exs = [moe.Expert(H, I, seed=300 + 10 * rk + e, nm_gu=nm[0] if e % 2 == 0 else None, nm_dn=nm[1] if e % 2 == 0 else None, rk_gu=rk, rk_dn=rk, var=e != 2,
                      sv=0.02, bk_gu=base, bk_dn=base) for e in range(6)]
    _compare([384, 300, 257, 200, 30, 250], H, I, exs, [4] * 6, nm)


def _compare(counts, H, I, exs, levels, nm):
    E, T = len(counts), sum(counts)
    L = moe.MoELayer(E, H, I, *nm, Bmax=1, topk=1)
    for e in range(E):
        L.set(e, exs[e], levels[e])
    gen = torch.Generator().manual_seed(7)
    sel = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T, generator=gen)].view(T, 1).cuda()
    x = torch.randn(T, H, generator=gen).bfloat16().half().cuda()
    rw = torch.rand(T, 1, generator=gen).half().cuda()
    ref = prefill_library(L, x, sel, rw)
    y, y2 = L.prefill(x, sel, rw), L.prefill(x, sel, rw)
    torch.cuda.synchronize()
    assert torch.equal(y, y2)
    # the same fp16 operands multiplied in fp32 by both: what differs is the order of the sums (2^-24 per addition) and, where that moves
    # the SwiGLU output across a rounding to fp16, half a unit of 2^-11 of single elements
    assert layer_errors(y.cpu().numpy(), ref.cpu().numpy())[1] <= 1e-4
    assert L.prefill_status() == 0
