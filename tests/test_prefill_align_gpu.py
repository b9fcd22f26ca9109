"""The elementwise passes of the prefill read and write 32 bytes per lane where their arrays are aligned to 32 and 16 where they are not:
the same elements in the same lanes, so the results have to be the same bits."""
import pytest
import torch

from nestquant_b200 import ext, moe

pytestmark = pytest.mark.gpu


def _at(shape, dtype, offset):
    """a tensor whose first element lies `offset` bytes after a boundary of 256"""
    n = 1
    for d in shape:
        n *= d
    size = torch.empty(0, dtype=dtype).element_size()
    flat = torch.zeros(n + 256 // size, dtype=dtype, device="cuda")
    lead = (offset - flat.data_ptr()) % 256 // size
    t = flat[lead:lead + n].view(shape)
    assert t.data_ptr() % 256 == offset
    return t


@pytest.mark.parametrize("H,I,had,rank", [(128, 128, 128, 0), (1152, 512, 512, 2), (2048, 1152, 128, 1)])
@pytest.mark.parametrize("kperm", [False, True])
def test_passes_do_not_depend_on_the_alignment(H, I, had, rank, kperm):
    E, T, topk = 3, 5, 2
    L = moe.MoELayer(E, H, I, topk=topk)
    exs = [moe.Expert(H, I, seed=5 + e, rk_gu=0, rk_dn=7, var=True, sv=0.02) for e in range(E)]
    gen = torch.Generator(device="cuda").manual_seed(1)
    for e, lv in enumerate((2, 4, 0)):
        exs[e].had_dn = had
        if rank:
            exs[e].rg = exs[e].rd = rank
            exs[e].lr = (torch.randn(rank * (2 * H + 3 * I), generator=gen, device="cuda") * 0.02).half()
            exs[e].lr4 = (torch.randn(rank * (2 * I + H), generator=gen, device="cuda") * 0.01).half()
        L.set(e, exs[e], lv)
    x0 = torch.randn(T, H, generator=gen, device="cuda").half()
    sel = torch.randint(0, E, (T, topk), generator=gen, device="cuda")
    rw = torch.rand(T, topk, generator=gen, device="cuda").half()
    order = sel.flatten().argsort(stable=True)
    pos = torch.empty_like(order).scatter_(0, order, torch.arange(T * topk, device="cuda")).int()
    pe, pt, R = sel.flatten()[order].int(), (order // topk).int(), T * topk
    acc = torch.randn(2, R, I, generator=gen, device="cuda")
    y0 = torch.randn(R, H, generator=gen, device="cuda")

    def passes(offset):
        x, xg, xu = _at((T, H), torch.float16, offset), _at((R, H), torch.float16, offset), _at((R, H), torch.float16, offset)
        ag, au, h = _at((R, I), torch.float32, offset), _at((R, I), torch.float32, offset), _at((R, I), torch.float16, offset)
        y, out = _at((R, H), torch.float32, offset), _at((T, H), torch.float32, offset)
        zg, zd = torch.zeros(R, 4, device="cuda"), torch.zeros(R, 4, device="cuda")
        x.copy_(x0), ag.copy_(acc[0]), au.copy_(acc[1]), y.copy_(y0)
        ext.pf_pre(x, pt, pe, L.table, xg, xu, zg, I, kperm=kperm)
        ext.pf_mid(ag, au, zg, pe, L.table, h, zd, H, I, kperm=kperm)
        ext.pf_combine(y, zd, pos, sel, rw, L.table, out, I)
        return xg.clone(), xu.clone(), h.clone(), zd, out.clone()

    a, b = passes(0), passes(16)
    assert float(a[0].abs().max()) > 0 and float(a[2].abs().max()) > 0 and float(a[4].abs().max()) > 0
    for s, t in zip(a, b):
        assert torch.equal(s, t)


def test_rows_of_other_ranks_and_windows_of_pairs():
    """the first pass with one buffer per rank (one that is aligned to 16 only is enough to leave the wide accesses), the last pass window by
    window, adding to what is there"""
    E, H, I, Tl, W, topk = 4, 1152, 512, 7, 3, 2
    T, R = W * Tl, W * Tl * topk
    L = moe.MoELayer(E, H, I, topk=topk)
    exs = [moe.Expert(H, I, seed=9 + e, rk_gu=0, rk_dn=7, var=True, sv=0.02) for e in range(E)]
    for e, lv in enumerate((2, 4, 0, 4)):
        L.set(e, exs[e], lv)
    gen = torch.Generator(device="cuda").manual_seed(2)
    x0 = torch.randn(T, H, generator=gen, device="cuda").half()
    sel = torch.randint(0, E, (T, topk), generator=gen, device="cuda")
    rw = torch.rand(T, topk, generator=gen, device="cuda").half()
    order = sel.flatten().argsort(stable=True)
    pos = torch.empty_like(order).scatter_(0, order, torch.arange(R, device="cuda")).int()
    pe, pt = sel.flatten()[order].int(), (order // topk).int()
    y0 = torch.randn(R, H, generator=gen, device="cuda")
    cut = R // 3

    def passes(x_at, row_at, y_at, out_at):
        xs = [_at((Tl, H), torch.float16, o) for o in x_at]
        for r in range(W):
            xs[r].copy_(x0[r * Tl:(r + 1) * Tl])
        xg, xu, out = _at((R, H), torch.float16, row_at), _at((R, H), torch.float16, row_at), _at((T, H), torch.float32, out_at)
        ext.pf_pre_ep([x.data_ptr() for x in xs], Tl, H, pt, pe, L.table, xg, xu, torch.zeros(R, 4, device="cuda"), I, kperm=True)
        for a, b in ((0, cut), (cut, R)):
            y = _at((b - a, H), torch.float32, y_at)
            y.copy_(y0[a:b])
            ext.pf_combine(y, torch.zeros(b - a, 4, device="cuda"), pos, sel, rw, L.table, out, I, pair0=a, npairs=b - a, accumulate=a > 0)
        return xg.clone(), xu.clone(), out.clone()

    ref = passes((0, 0, 0), 0, 0, 0)
    assert all(float(t.abs().max()) > 0 for t in ref)
    for at in (((16, 16, 16), 16, 16, 16), ((0, 0, 16), 0, 0, 16), ((0, 0, 0), 16, 16, 0), ((32, 32, 32), 32, 32, 32)):
        for s, t in zip(ref, passes(*at)):
            assert torch.equal(s, t), at
