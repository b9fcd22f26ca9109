"""Runs of the dense decode kernel: lists long enough that a warp takes 2, 3 or 4 units in a row - runs that cross strips and end short -
with experts of every level side by side, dense and mask mode, both base codes, against the CPU oracle bit for bit."""
import numpy as np
import pytest
import torch

from oracle import nq_oracle as O
from tests.util import f16_bits, proj_to_oracle, same_fp16_bits

pytestmark = pytest.mark.gpu


# units per matrix: 85 | 80, 40 | 240, 120 | 40; run length by the units of the whole call (a shorter list: runs of one)
@pytest.mark.parametrize("H,I,gu,dn,n", [(640, 136, True, False, 420), (640, 128, True, True, 200), (640, 384, True, True, 41), (640, 128, False, True, 760),
                                         (640, 384, True, True, 3)])
def test_mixed_lists_vs_oracle(H, I, gu, dn, n):
    from nestquant_b200 import ext, moe
    gen = torch.Generator().manual_seed(H + I + n)
    nm = 2 if I != 128 else 1
    table, want, keep = torch.zeros(6, 20, dtype=torch.int64), [[], []], []
    for e, (level, masked, bk) in enumerate([(0, False, 0), (2, False, 0), (4, False, 0), (4, True, 0), (4, True, 1), (2, False, 1)]):
        table[e, 0] = level
        for d, (use, N, K) in enumerate([(gu, 2 * I, H), (dn, H, I)]):
            if not use:
                continue
            p = proj_to_oracle(moe.Proj(N, K, gen, nm=nm if masked else None, rk=(9 if d else 3) if bk else (7 if d else e), mbn=("exh", 900 * e), var=e % 2 == 0, bk=bk))
            want[d].append(f16_bits(torch.zeros(N, K, dtype=torch.float16)) if level == 0 else O.decode_proj(p, level))
            for col, a in [(1, p.base), (2, p.p4), (3, p.d4), (4, p.flags), (12, p.var)]:
                if a is not None:
                    keep.append(torch.from_numpy(np.ascontiguousarray(a).copy()).cuda())
                    table[e, col + (d if col == 12 else 4 * d)] = keep[-1].data_ptr()
            table[e, 10 + d] = p.rk
            table[e, 19] |= bk << (8 * d)
    lst = torch.randint(0, 6, (n,), generator=gen, dtype=torch.int32)
    lst[-1] = 4
    out = [torch.full((n, *s), float("nan"), dtype=torch.float16, device="cuda") if u else None for u, s in [(gu, (2 * I, H)), (dn, (H, I))]]
    ext.pf_decode(table.cuda(), lst.cuda(), out[0], out[1], H, I, nm, nm, 0)
    torch.cuda.synchronize()
    for d in (0, 1):
        if out[d] is not None:
            got = f16_bits(out[d]).reshape(n, -1)
            for i, e in enumerate(lst.tolist()):
                assert same_fp16_bits(got[i].reshape(want[d][e].shape), want[d][e]) == 0, (d, i, e)
