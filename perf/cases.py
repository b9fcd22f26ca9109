"""Performance cases of the quantized MoE layer: what a serving program has it do, through the public entry points.

listed() names the cases, draw() gives more of the same ranges, prepare() builds what the program holds before a call (the
layer with its experts' planes on the GPU, the step's tokens and routing, the captured graph), run() is one pass.

A case is
  op        call        MoELayer.__call__, up to 32 tokens (a decode step launched from Python)
            graph       one replay of MoELayer.capture with a mailbox in front (a decode step of a serving engine)
            host graph  the same without a mailbox, inputs and outputs copied from / to pinned host memory
            prefill     MoELayer.prefill
            dense       ext.pf_decode of T experts to fp16 matrices (loaders and checks that want dense weights)
  E, topk, H, I, T   experts, picks per token, hidden and intermediate width, tokens
  four      share of the experts at level 4, the most routed ones; the rest is at level 2
  masked    share of the level-4 experts that refine half of their chunks only (mask mode)
  resident  share of the experts on this GPU (expert parallelism); the others' picks are skipped
  skew      weight of a Zipf(1.1) popularity law in the routing logits (0.3: about 63 % of the picks hit the first 30 %)
  gu, dn, base       residual window codes of gate|up and down, base window code of both
  rank      rank of the low-rank plane (0: none)
  had       width of the down projection's input rotation (128 or 512)

The planes are random packed words, which is what packed trellis streams look like; block words, scales, tokens and routing
follow nestquant_b200.synth.
"""
import types

import torch

from nestquant_b200 import ext, moe


def _case(name, op, T, E=256, topk=8, H=6144, I=2048, four=0.3, masked=0.0, resident=1.0, skew=0.3, gu=0, dn=7, base=0, rank=0, had=128):
    return dict(name=name, op=op, T=T, E=E, topk=topk, H=H, I=I, four=four, masked=masked, resident=resident, skew=skew, gu=gu,
                dn=dn, base=base, rank=rank, had=had)


def listed():
    return [
        # one decode step of a small layer, launched from Python: nothing but latency
        _case("small decode 1", "call", 1, E=64, topk=4, H=1024, I=512, four=0.75, masked=0.33, skew=0.0),
        # the same layer with a batch of decode streams
        _case("small decode 16", "call", 16, E=64, topk=4, H=1024, I=512, four=0.75, masked=0.33, skew=0.0),
        # one token through the full layer: interactive decoding on one GPU
        _case("decode 1", "call", 1),
        # one token through one of eight tensor-parallel shards, copies from and to the host included
        _case("decode 1 of a shard", "host graph", 1, I=256),
        # four tokens: verification of speculated tokens, captured, with the level mailbox in front
        _case("decode 4", "graph", 4),
        # a full decode batch
        _case("decode 32", "call", 32),
        # the 1.75-bit base with its residual codes, low-rank plane and wide rotation: a layer with every option of the format
        _case("decode 3 all options", "call", 3, E=128, topk=6, H=4096, I=1536, four=0.5, gu=3, dn=9, base=1, rank=3, had=512),
        # a short prompt on the small layer
        _case("small prefill 75", "prefill", 75, E=64, topk=4, H=1024, I=512, four=0.75, masked=0.33, skew=0.0),
        # a prompt chunk on the full layer, mixed levels: few tokens per expert
        _case("prefill 1000", "prefill", 1000, four=0.75, masked=0.33),
        # a ragged window on one of four expert-parallel ranks
        _case("prefill 3001 of a rank", "prefill", 3001, four=0.5, resident=0.25, rank=2),
        # a full prefill window, every expert at level 4
        _case("prefill 8192", "prefill", 8192, four=1.0, skew=0.0),
        # dense matrices of a few experts
        _case("dense 4", "dense", 4, E=4, four=0.75, masked=0.33),
    ]


def _log_between(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["call", "call", "graph", "host graph", "prefill", "prefill", "prefill", "dense"])
    H = 128 * _log_between(rng, 6, 48)
    I = 128 * _log_between(rng, 2, 16)
    E = _log_between(rng, 16, 256)
    topk = rng.randint(2, 8)
    T = _log_between(rng, 1, 32)
    if op == "prefill":
        T = _log_between(rng, 33, 8192)
        while T * topk * H * I > 65536 * 6144 * 2048:
            T = T * 3 // 4
    if op == "dense":
        E = T = rng.randint(1, 8)
        topk = 1
    base = 1 if rng.random() < 0.15 else 0
    gu, dn = (3, 9) if base else rng.choice([(0, 7), (0, 7), (0, 7), (3, 9), (6, 8), (5, 1), (4, 2)])
    c = _case("", op, T, E=E, topk=topk, H=H, I=I, four=rng.choice([0.0, 0.3, 0.5, 0.75, 1.0]), masked=rng.choice([0.0, 0.0, 0.33, 1.0]),
              resident=rng.choice([1.0, 1.0, 1.0, 0.5, 0.25]) if op in ("call", "prefill") else 1.0, skew=rng.choice([0.0, 0.3, 0.6]),
              gu=gu, dn=dn, base=base, rank=rng.choice([0, 0, 0, 1, 4]), had=512 if I % 512 == 0 and rng.random() < 0.2 else 128)
    del c["name"]
    return c


# ---------------------------------------------------------------- the layer
def _chunks_refined(K):
    return max(1, K // 128 // 2)


def _placement(c):
    """level of every expert (0 = not resident) and whether it is in mask mode; expert 0 is the most routed one"""
    E, n4 = c["E"], round(c["four"] * c["E"])
    every = max(1, round(1 / c["resident"]))
    levels = [(4 if e < n4 else 2) if e % every == 0 else 0 for e in range(E)]
    step = round(1 / c["masked"]) if c["masked"] > 0 else 0
    return levels, [bool(step and levels[e] == 4 and (e // every) % step == 0) for e in range(E)]


def _proj(N, K, n, nm, rk, bk, gen):
    """planes of n experts' N x K projection: one allocation per plane, a view per expert"""
    z = moe.proj_sizes(N, K, nm, rk, bk)
    units, dev = z["S"] * z["C"], gen.device
    refined = z["nrec_r"] // 32

    def words(nbytes):
        stride = (nbytes + 15) // 16 * 4
        return torch.randint(-2**31, 2**31 - 1, (n, stride), generator=gen, dtype=torch.int32, device=dev)

    base, p4 = words(z["base"]), words(z["p4"])
    if moe.rbits(rk) % 16:
        p4.view(torch.uint8)[:, z["p4"] - 4:z["p4"]] = 0
    # block words: Mb in [120, 255], N up to 0.8 Mb, one in twenty from the whole valid range
    mb = torch.randint(120, 256, (n, refined), generator=gen, device=dev)
    nn = (torch.rand(n, refined, generator=gen, device=dev) * 0.8 * mb).round().long()
    wild = torch.rand(n, refined, generator=gen, device=dev) < 0.05
    mw = torch.randint(1, 256, (n, refined), generator=gen, device=dev)
    nw = (torch.rand(n, refined, generator=gen, device=dev) * (torch.clamp(257 - mw, max=255) + 1)).floor().long()
    mb, nn = torch.where(wild, mw, mb), torch.where(wild, nw, nn)
    d4 = (mb | (torch.minimum(nn, 257 - mb) << 8)).to(torch.int32)
    var = torch.randint(0, 256, (n, units), generator=gen, dtype=torch.int64, device=dev).to(torch.uint8)
    flags = None
    if nm is not None:
        host = torch.Generator().manual_seed(int(torch.randint(0, 2**31 - 1, (1,), generator=gen, device=dev)))
        flags = torch.stack([moe.make_flags(z["S"], z["C"], nm, host)[0] for _ in range(n)]).to(dev)
    return [types.SimpleNamespace(N=N, K=K, rk=rk, bk=bk, z=z, base=base[i], p4=p4[i, :(z["p4"] + 3) // 4], d4=d4[i], var=var[i],
                                  flags=None if flags is None else flags[i]) for i in range(n)]


def _experts(c, ids, masked, gen):
    H, I, n, dev = c["H"], c["I"], len(ids), gen.device
    gus = _proj(2 * I, H, n, _chunks_refined(H) if masked else None, c["gu"], c["base"], gen)
    dns = _proj(H, I, n, _chunks_refined(I) if masked else None, c["dn"], c["base"], gen)
    # scales: +-1 on the inputs, |N(0, 0.02)| on the outputs
    sc = (torch.randint(0, 2, (n, 3 * H + 3 * I), generator=gen, device=dev) * 2 - 1).half()
    for lo, hi in ((H, H + 2 * I), (H + 3 * I, 2 * H + 3 * I)):
        sc[:, lo:hi] = (torch.randn(n, hi - lo, generator=gen, device=dev) * 0.02).abs().half()
    r = c["rank"]
    if r:
        lr = (torch.randn(n, r * (2 * H + 3 * I), generator=gen, device=dev) * 0.02).half()
        lr4 = (torch.randn(n, r * (2 * I + H), generator=gen, device=dev) * 0.01).half()
    return {e: types.SimpleNamespace(gu=gus[i], dn=dns[i], H=H, I=I, signs=sc[i], rg=r, rd=r, lr=lr[i] if r else None,
                                     lr4=lr4[i] if r else None, had_dn=c["had"]) for i, e in enumerate(ids)}


def _routing(c, gen):
    rank = torch.arange(1, c["E"] + 1, device=gen.device, dtype=torch.float32)
    bias = torch.log(rank.pow(-1.1) / rank.pow(-1.1).sum())
    logits = torch.randn(c["T"], c["E"], generator=gen, device=gen.device).bfloat16().float() + c["skew"] * bias
    top, sel = logits.topk(c["topk"], dim=1)
    return sel, torch.softmax(top, 1).half()


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    H, I, E, T = c["H"], c["I"], c["E"], c["T"]
    levels, masked = _placement(c)
    any_masked = any(masked)
    nm_gu, nm_dn = (_chunks_refined(H), _chunks_refined(I)) if any_masked else (0, 0)
    decode = c["op"] in ("call", "graph", "host graph")
    L = moe.MoELayer(E, H, I, nm_gu, nm_dn, Bmax=T if decode else 1, topk=c["topk"], dev=dev, share=c["resident"])
    experts = _experts(c, [e for e in range(E) if levels[e] and not masked[e]], False, gen)
    if any_masked:
        experts.update(_experts(c, [e for e in range(E) if masked[e]], True, gen))
    for e, ex in experts.items():
        L.set(e, ex, levels[e])
    s = types.SimpleNamespace(op=c["op"], L=L, experts=experts)
    if c["op"] == "dense":
        s.ids = torch.randperm(E, generator=gen, device=dev)[:T].to(torch.int32)
        s.Wgu = torch.empty(T, 2 * I, H, dtype=torch.float16, device=dev)
        s.Wdn = torch.empty(T, H, I, dtype=torch.float16, device=dev)
        return s
    s.sel, s.rw = _routing(c, gen)
    s.x = torch.randn(T, H, generator=gen, device=dev).bfloat16().half()
    if c["op"] == "graph":
        s.box = moe.Mailbox(L)
        s.G = L.capture(T, with_mailbox=s.box)
        s.G.x.copy_(s.x), s.G.sel.copy_(s.sel), s.G.rw.copy_(s.rw)
    elif c["op"] == "host graph":
        s.G = L.capture(T, host_io=True)
        s.G.x_host.copy_(s.x), s.G.sel_host.copy_(s.sel), s.G.rw_host.copy_(s.rw)
    return s


def run(s):
    if s.op == "call":
        return s.L(s.x, s.sel, s.rw)
    if s.op == "graph":
        return s.G.replay()
    if s.op == "host graph":
        s.G.replay()
        return s.G.out_host
    if s.op == "prefill":
        return s.L.prefill(s.x, s.sel, s.rw)
    L = s.L
    ext.pf_decode(L.table, s.ids, s.Wgu, s.Wdn, L.H, L.I, L.nm_gu, L.nm_dn)
    return s.Wgu, s.Wdn


def work(case):
    """planes and scales of the distinct experts that the tokens reach (of one routing with these odds), tokens in, rows out"""
    c = dict(case)
    H, I, T, topk = c["H"], c["I"], c["T"], c["topk"]
    levels, masked = _placement(c)
    if c["op"] == "dense":
        hit, pairs = list(range(T)), 0
        moved = T * 3 * H * I * 2
    else:
        sel = _routing(c, torch.Generator().manual_seed(1))[0]
        live = torch.tensor([lv > 0 for lv in levels])[sel]
        hit, pairs = sorted(set(sel[live].tolist())), int(live.sum())
        moved = T * H * (2 + 4) + T * topk * 10
    for e in hit:
        for N, K, rk in ((2 * I, H, c["gu"]), (H, I, c["dn"])):
            z = moe.proj_sizes(N, K, _chunks_refined(K) if masked[e] else None, rk, c["base"])
            moved += z["base"] + z["S"] * z["C"] + (z["p4"] + z["d4"] + z["flags"] if levels[e] == 4 else 0)
        if c["op"] != "dense":
            moved += 6 * (H + I) + 2 * c["rank"] * (2 * H + 3 * I + (2 * I + H if levels[e] == 4 else 0))
    return {"bytes": moved, "flops": 2 * pairs * 3 * H * I}


def tolerance(case):
    # dense weights are defined bit for bit; layer outputs have two roundings to fp16 on the way (the rotated input and the
    # SwiGLU output), half a unit of 2^-10 each, everything else in fp32
    return "exact" if case["op"] == "dense" else {"rel": 5e-4}
