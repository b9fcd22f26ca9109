"""nq_prefill: one host call for a whole prefill, its kernels launched one on the heels of the other."""
import pytest
import torch

from nestquant_b200 import moe
from nestquant_b200.capi import NestQuantError
from tests.prefill_lib import prefill_library
from tests.util import layer_errors

pytestmark = pytest.mark.gpu


def _layer(E, topk, H=256, I=128, seed=5):
    L = moe.MoELayer(E, H, I, Bmax=1, topk=topk)
    exs = [moe.Expert(H, I, seed=seed + e, rk_gu=0, rk_dn=7, var=True, sv=0.02) for e in range(min(E, 6))]
    for e in range(E):
        L.set(e, exs[e % len(exs)], (4, 2, 0 if e % 7 == 5 else 4)[e % 3])
    return L, exs


def _inputs(E, topk, T, H, gen):
    sel = torch.rand(T, E, generator=gen, device="cuda").topk(topk, 1).indices
    return torch.randn(T, H, generator=gen, device="cuda").half(), sel, torch.rand(T, topk, generator=gen, device="cuda").half()


# pairs and experts on both sides of what the one-kernel sort takes (8,192 picks, 369 experts), in one chunk (the sort writes the pass list)
# and in several (a kernel of its own writes it)
@pytest.mark.parametrize("E,topk,T,R", [(16, 4, 33, None), (16, 4, 33, 131), (16, 4, 33, 1), (16, 4, 2048, None), (16, 4, 2049, None), (369, 2, 50, None),
                                        (370, 2, 50, None), (370, 2, 50, 99), (16, 4, 2049, 4096)])
def test_chunks_and_sort_paths(E, topk, T, R):
    L, exs = _layer(E, topk)
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, sel, rw = _inputs(E, topk, T, 256, gen)
    ref = prefill_library(L, x, sel, rw)
    y = L.prefill(x, sel, rw, R=R)
    torch.cuda.synchronize()
    # fp32 sums of the same fp16 operands in another order (2^-24 an addition), single h elements half a unit of 2^-11 apart
    assert layer_errors(y.cpu().numpy(), ref.cpu().numpy())[1] <= 1e-4
    assert L.prefill_status() == 0


def test_calls_in_a_row_see_their_own_inputs():
    """a kernel may be launched while its predecessor runs: what it reads must be what that one (and the one before it) wrote, call after call
    over the same scratch, whatever an SM still holds in its L1"""
    L, exs = _layer(16, 4, H=512, I=256)
    gen = torch.Generator(device="cuda").manual_seed(2)
    ins = [_inputs(16, 4, T, 512, gen) for T in (40, 700, 3, 2100, 129)]
    want = []
    for a in ins:
        want.append(L.prefill(*a))
        torch.cuda.synchronize()
    for _ in range(10):
        got = [L.prefill(*a) for a in ins]
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for g, w in zip(got, want))
    # chunks of one call follow one another the same way
    small = L.prefill(*ins[3], R=512)
    for _ in range(5):
        assert torch.equal(L.prefill(*ins[3], R=512), small)
    assert L.prefill_status() == 0


def test_refused_inputs():
    L, exs = _layer(16, 4)
    gen = torch.Generator(device="cuda").manual_seed(3)
    x, sel, rw = _inputs(16, 4, 40, 256, gen)
    for bad in (x[:, :128].contiguous(), x[:39], x.cpu(), x[:, ::2]):
        with pytest.raises(NestQuantError):
            L.prefill(bad, sel, rw)
    with pytest.raises(NestQuantError):
        L.prefill(x, sel, rw, out=torch.empty(39, 256, device="cuda"))


def test_table_of_more_experts_than_the_layer_is_refused():
    """also where an earlier, larger call has left scratch that would be large enough for it"""
    L, exs = _layer(16, 4)
    gen = torch.Generator(device="cuda").manual_seed(4)
    L.prefill(*_inputs(16, 4, 8192, 256, gen))
    x, sel, rw = _inputs(16, 4, 10, 256, gen)
    with pytest.raises(NestQuantError):
        L.prefill(x, sel, rw, table=L.table.repeat(19, 1)[:300].contiguous())
    fewer = L.prefill(x, sel % 12, rw, table=L.table[:12].contiguous())
    torch.cuda.synchronize()
    assert torch.equal(fewer, L.prefill(x, sel % 12, rw))


def test_calls_in_a_row_over_arrays_aligned_to_16_bytes():
    """the forms of the passes for arrays that are not aligned to 32 bytes, call after call in several chunks"""
    L, exs = _layer(16, 4, H=512, I=256)
    gen = torch.Generator(device="cuda").manual_seed(5)
    ins = [_inputs(16, 4, T, 512, gen) for T in (300, 77, 513)]
    want = [L.prefill(*a, R=200) for a in ins]
    torch.cuda.synchronize()

    def shifted(t):
        n = 16 // t.element_size()
        return torch.empty(t.numel() + n, dtype=t.dtype, device="cuda")[n:].view(t.shape)

    sc = L._prefill_scratch(200, torch.device("cuda", torch.cuda.current_device()))
    sc.update({n: shifted(sc[n]) for n in ("acc_g", "acc_u", "h", "xg", "xu", "y")})
    sc["plan"] = torch.empty(sc["plan"].numel() + 1, dtype=torch.int32, device="cuda")[1:]      # (4 bytes: any int array will do)
    ins = [(shifted(x).copy_(x), sel, rw) for x, sel, rw in ins]
    outs = [shifted(w) for w in want]
    for _ in range(10):
        for a, o in zip(ins, outs):
            L.prefill(*a, R=200, out=o.fill_(7.0))
        torch.cuda.synchronize()
        assert all(torch.equal(o, w) for o, w in zip(outs, want))
    assert L.prefill_status() == 0


@pytest.mark.parametrize("R", [None, 200])
def test_captured_calls(R):
    """replays over other inputs, beside larger and smaller eager calls that replace the layer's scratch, against eager calls; the first call of
    a layer may be the captured one, and a raised status word outlives replays"""
    L, exs = _layer(16, 4, H=512, I=256)
    gen = torch.Generator(device="cuda").manual_seed(6)
    ins = [_inputs(16, 4, 130, 512, gen) for _ in range(3)]
    big = _inputs(16, 4, 900, 512, gen)
    _layer(16, 4, H=512, I=256)[0].prefill(*ins[0])      # (the kernels are loaded)
    x, sel, rw = (t.clone() for t in ins[0])
    out = torch.empty(130, 512, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        L.prefill(x, sel, rw, out=out, R=R)
    want = [L.prefill(*a, R=R) for a in ins]
    large = L.prefill(*big)
    spare = [torch.full((n,), 3.0, device="cuda") for n in (1 << 14, 1 << 17, 1 << 20) for _ in range(4)]      # where freed scratch would have been
    for i in (1, 0, 2, 1):
        for dst, src in zip((x, sel, rw), ins[i]):
            dst.copy_(src)
        out.fill_(7.0)
        graph.replay()
        assert torch.equal(L.prefill(*big), large)
        assert torch.equal(L.prefill(*ins[i], R=R), want[i])
        torch.cuda.synchronize()
        assert torch.equal(out, want[i])
    assert all((t == 3.0).all() for t in spare)
    assert L.prefill_status() == 0
    L._pf_status.fill_(1)
    graph.replay()
    assert L.prefill_status() == 1
    del graph
