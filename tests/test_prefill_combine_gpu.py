"""The last pass of the prefill on its own: picks per token on both sides of a warp's 32, picks that add nothing (no expert, not resident,
weight zero, outside the window of pairs), row widths that leave lanes without columns; against fp64, and window by window."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("topk,H", [(1, 128), (3, 1152), (8, 640), (32, 256), (33, 256), (70, 1024)])
def test_combine_vs_fp64(topk, H):
    from nestquant_b200 import ext
    T, E, I = 13, 5, 128
    gen = torch.Generator().manual_seed(topk + H)
    rnd = lambda *s: torch.rand(*s, generator=gen) - 0.5
    table, keep, ex = torch.zeros(E, 20, dtype=torch.int64), [], []
    for e, (level, rd) in enumerate([(2, 0), (0, 0), (4, 3), (2, 4), (4, 0)]):
        sc, lr, lr4 = (rnd(3 * H + 3 * I) * 2).half(), rnd(rd * I + rd * H).half(), rnd(rd * H).half()
        keep += [t.cuda() for t in (sc, lr, lr4)]
        table[e, 0], table[e, 9], table[e, 18] = level, keep[-3].data_ptr(), 128
        if rd:
            table[e, 14], table[e, 15], table[e, 17] = keep[-2].data_ptr(), keep[-1].data_ptr(), rd
        ex.append((level, rd, sc.double(), lr.double()[rd * I:] + (lr4.double() if level == 4 else 0.0)))
    P = T * topk
    sel = torch.randint(-1, E + 1, (T, topk), generator=gen)      # -1 and E: no expert
    pos = torch.randperm(P, generator=gen).view(T, topk).int()
    rw = rnd(T, topk).half()
    rw[::2, 0] = 0
    y, zd = rnd(P, H), rnd(P, 4)
    h = torch.ones(1, 1, dtype=torch.float64)
    while h.shape[0] < 128:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    want, size = torch.zeros(T, H, dtype=torch.float64), torch.zeros(T, 1, dtype=torch.float64)
    for t in range(T):
        for k in range(topk):
            e, p, w = int(sel[t, k]), int(pos[t, k]), float(rw[t, k])
            if 0 <= e < E and ex[e][0] and w:
                _, rd, sc, u2 = ex[e]
                v = (y[p].double().view(-1, 128) @ h / 128 ** 0.5).reshape(H) * sc[2 * H + 3 * I - H:3 * H + 3 * I - H]
                v = v + sum((float(zd[p, r]) * u2[r * H:(r + 1) * H] for r in range(rd)), torch.zeros(H, dtype=torch.float64))
                want[t] += w * v
                size[t] += abs(w) * (float(y[p].view(-1, 128).norm(dim=1).max()) + 2.0 * rd)
    out = torch.full((T, H), 7.0, device="cuda")
    d = [a.cuda() for a in (y, zd, pos, sel, rw, table)]
    ext.pf_combine(*d, out, I)
    # fp32 throughout: fewer than 20 roundings of 2^-24 on a term, then one per pick on the sum
    assert ((out.cpu().double() - want).abs() <= (20 + topk) * 2.0 ** -24 * size + 1e-30).all()
    parts, at = torch.full((T, H), 7.0, device="cuda"), P // 3
    ext.pf_combine(d[0][:at].clone(), d[1][:at].clone(), *d[2:], parts, I, pair0=0, npairs=at, accumulate=False)
    ext.pf_combine(d[0][at:].clone(), d[1][at:].clone(), *d[2:], parts, I, pair0=at, npairs=P - at, accumulate=True)
    assert ((parts.cpu().double() - want).abs() <= (24 + topk) * 2.0 ** -24 * size + 1e-30).all()
