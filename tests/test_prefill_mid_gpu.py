"""The middle pass of the prefill on its own, from accumulators to the down GEMM's rows: row widths on both sides of the one up to which a
warp takes several pairs, experts of different levels, ranks and rotation widths beside each other, pairs without an expert, pair
counts that leave the last warp part of its pairs; against fp64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _wht(v, width):
    n = v.shape[-1] // width
    h = torch.ones(1, 1, dtype=torch.float64)
    while h.shape[0] < width:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    return (v.reshape(-1, n, width) @ h).reshape(v.shape) / width ** 0.5


@pytest.mark.parametrize("I,R,kperm", [(128, 1, True), (128, 77, True), (256, 50, False), (256, 33, True), (384, 29, True), (512, 41, True), (512, 30, False), (640, 13, True)])
def test_mid_pass_vs_fp64(I, R, kperm):
    from nestquant_b200 import ext
    H, E = 128, 6
    gen = torch.Generator().manual_seed(I + R)
    rnd = lambda *s: (torch.rand(*s, generator=gen) - 0.5)
    table, keep, ex = torch.zeros(E, 20, dtype=torch.int64), [], []
    for e, (level, rg, rd, wide, four) in enumerate([(2, 0, 0, 0, 0), (4, 4, 1, 1, 1), (0, 0, 0, 0, 0), (2, 1, 4, 0, 1), (4, 3, 3, 0, 1), (4, 2, 0, 1, 0)]):
        hw = 512 if wide and I % 512 == 0 else 256 if wide and I % 256 == 0 else 128
        sc = (rnd(3 * H + 3 * I) * 2).half()
        lr, lr4 = rnd(rg * H + 2 * rg * I + rd * I + rd * H).half(), rnd(2 * rg * I + rd * H).half()
        d = [t.cuda() for t in (sc, lr, lr4)]
        keep += d
        table[e, 0], table[e, 9], table[e, 18] = level, d[0].data_ptr(), hw
        if rg or rd:
            table[e, 14], table[e, 15], table[e, 16], table[e, 17] = d[1].data_ptr(), d[2].data_ptr() if four else 0, rg, rd
        ex.append((level, rg, rd, hw, sc.double(), lr.double(), lr4.double() if four and level == 4 else None))
    pe = torch.randint(-1, E + 1, (R,), generator=gen, dtype=torch.int32)      # -1 and E: no expert
    pe[0] = 1
    ag, au, zg = rnd(R, I) * 4, rnd(R, I) * 4, rnd(R, 4)
    h = torch.full((R, I), 7.0, dtype=torch.float16, device="cuda")
    zd = torch.full((R, 4), 7.0, device="cuda")
    ext.pf_mid(ag.cuda(), au.cuda(), zg.cuda(), pe.cuda(), table.cuda(), h, zd, H, I, kperm=kperm)
    h, zd = h.cpu().double(), zd.cpu().double()
    order = [16 * (k // 16) + (2 * (k % 16 // 4) + k % 4 if k % 4 < 2 else 8 + 2 * (k % 16 // 4) + k % 4 - 2) for k in range(I)] if kperm else list(range(I))
    for p in range(R):
        e = int(pe[p])
        if not 0 <= e < E or ex[e][0] == 0:
            assert (h[p] == 7).all() and (zd[p] == 7).all(), p
            continue
        level, rg, rd, hw, sc, lr, lr4 = ex[e]
        u2 = lr[rg * H:].clone()
        if lr4 is not None:
            u2[:2 * rg * I] += lr4[:2 * rg * I]
        g, u = (_wht(a[p].double(), 128) * sc[H + i * I:H + (i + 1) * I] + sum((zg[p, r].double() * u2[(i * rg + r) * I:(i * rg + r + 1) * I] for r in range(rg)), torch.zeros(I))
                for i, a in enumerate((ag, au)))
        m = g * torch.sigmoid(g) * u
        z = torch.tensor([float(m @ lr[rg * H + 2 * rg * I + r * I:rg * H + 2 * rg * I + (r + 1) * I]) if r < rd else 0.0 for r in range(4)], dtype=torch.float64)
        t = m * sc[H + 2 * I:H + 3 * I]
        want = _wht(t, hw)[order]
        # fp32 sums of up to 512 terms of size <= |t| (2^-24 per step, < 40 steps with the expf) before the fp16 rounding (2^-11, subnormals 2^-25)
        slack = 64 * 2.0 ** -24 * float(t.norm() + m.norm())
        assert ((h[p] - want).abs() <= want.abs() * 2.0 ** -11 + slack + 2.0 ** -25).all(), (p, e)
        assert ((zd[p] - z).abs() <= slack * 4).all(), (p, e)
