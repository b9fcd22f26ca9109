"""The fused prefill GEMM changes its tensor-memory layout with the width of a pass (2, 4 or 6 unit stages beside the accumulator): passes of
every width one after the other on the same CTAs, for few and odd numbers of chunks."""
import pytest
import torch

from nestquant_b200 import moe
from tests.prefill_lib import prefill_library
from tests.util import layer_errors

pytestmark = pytest.mark.gpu

# pairs of the experts, in expert order: edges of the layouts (128, 256), of the passes (384) and of the token boxes (64)
COUNTS = [384, 1, 128, 300, 129, 64, 256, 65, 385, 20, 257, 0, 127, 383, 16]


@pytest.mark.parametrize("H,I", [(128, 2048), (256, 2048), (384, 2048), (2048, 128), (2048, 256), (2048, 1664)])
def test_passes_of_every_width_in_turn(H, I):
    E, T = len(COUNTS), sum(COUNTS)
    # 16 passes x 32 (or 16) weight groups of a projection: every CTA takes several items, of passes that lie apart in the list
    exs = [moe.Expert(H, I, seed=60 + e, rk_gu=(0, 6)[e % 2], rk_dn=7, var=True, sv=0.02) for e in range(E)]
    L = moe.MoELayer(E, H, I, Bmax=1, topk=1)
    for e in range(E):
        L.set(e, exs[e], (4, 4, 2)[e % 3])
    gen = torch.Generator().manual_seed(7)
    sel = torch.repeat_interleave(torch.arange(E), torch.tensor(COUNTS))[torch.randperm(T, generator=gen)].view(T, 1).cuda()
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
