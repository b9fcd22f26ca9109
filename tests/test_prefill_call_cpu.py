"""What a prefill call refuses before anything is enqueued: sizes that do not fit one another.  The checks look at shapes only, so CPU
tensors and a library that records what reaches it do."""
import ctypes as C

import pytest
import torch

from nestquant_b200 import capi, ext
from nestquant_b200.capi import NestQuantError


class _Recorder:
    def __init__(s):
        s.calls = 0

    def nq_prefill(s, args, stream):
        s.calls += 1
        return 0


@pytest.fixture
def library(monkeypatch):
    lib = _Recorder()
    monkeypatch.setattr(ext, "lib", lambda: lib)
    monkeypatch.setattr(ext, "_need", lambda *a: None)
    monkeypatch.setattr(ext, "current_stream", lambda: 0)
    return lib


def _call(E=16, rows=None, T=10, topk=4, H=256, I=128, R=40, P=40, **over):
    """a call on arrays for E experts, P pairs and chunks of R, with a table of `rows` experts"""
    i32, f16, f32 = torch.int32, torch.float16, torch.float32
    big = 100000                             # plan and sort scratch of an earlier, larger call
    perm = dict(P=P, pe=torch.empty(P, dtype=i32), pt=torch.empty(P, dtype=i32), pos=torch.empty(P, dtype=i32), start=torch.empty(E + 2, dtype=i32),
                hit=torch.empty(E, dtype=i32), scratch=torch.empty(big, dtype=i32))
    sc = dict(R=R, y=torch.empty(R, H), xg=torch.empty(R, H, dtype=f16), xu=torch.empty(R, H, dtype=f16), acc_g=torch.empty(R, I), acc_u=torch.empty(R, I),
              h=torch.empty(R, I, dtype=f16), zg=torch.empty(R, 4), zd=torch.empty(R, 4), plan=torch.empty(big, dtype=i32), status=torch.zeros(1, dtype=i32))
    a = dict(x=torch.empty(T, H, dtype=f16), sel=torch.zeros(T, topk, dtype=torch.int64), rw=torch.empty(T, topk, dtype=f16),
             table=torch.zeros(rows or E, 20, dtype=torch.int64), out=torch.empty(T, H, dtype=f32), hits_ptr=0)
    a.update({k: v for k, v in over.items() if k in a})
    perm.update({k: v for k, v in over.items() if k in perm})
    sc.update({k: v for k, v in over.items() if k in sc and k != "R"})
    ext.prefill(a["x"], a["sel"], a["rw"], a["table"], a["out"], perm, sc, over.get("chunk", R), I, 1, 1, a["hits_ptr"])


def test_fitting_sizes_reach_the_library(library):
    _call()
    _call(hits_ptr=4096)
    _call(rows=3)                            # a table of fewer experts than the layer
    _call(out=torch.empty(12, 256))          # rows to spare
    _call(chunk=7)
    assert library.calls == 5


@pytest.mark.parametrize("over", [
    dict(rows=300),                                                    # a table of more experts than the index arrays are for
    dict(rows=17),
    dict(rows=17, start=torch.empty(19, dtype=torch.int32), hits_ptr=4096),      # only the hit counters are too short
    dict(out=torch.empty(20, 128)),                                    # as many elements, rows of another width
    dict(out=torch.empty(5, 512)),
    dict(out=torch.empty(2560)),
    dict(out=torch.empty(9, 256)),
    dict(rw=torch.empty(9, 4, dtype=torch.float16)),
    dict(T=11),
    dict(chunk=41),
    dict(acc_g=torch.empty(40, 64)),
], ids=lambda o: ",".join(o))
def test_sizes_that_do_not_fit_are_refused(library, over):
    with pytest.raises(NestQuantError):
        _call(**over)
    assert library.calls == 0


@pytest.mark.skipif(torch.cuda.is_available(), reason="the arguments are not device addresses")
@pytest.mark.parametrize("world,per,T", [(2, 20, 41), (8, 5, 100), (4, 0, 1), (4, -3, 12)])
def test_tokens_that_no_rank_has_are_refused(world, per, T):
    """before anything is enqueued: an argument error, where a call that reached the device would fail for want of one"""
    a = capi.NqPrefill()
    for n, t in capi.NqPrefill._fields_:
        setattr(a, n, 4096 if t is C.c_void_p else 0)
    a.hits = a.hit_counts = None
    a.T, a.topk, a.E, a.H, a.I, a.nm_gu, a.nm_dn, a.R = T, 4, 16, 256, 128, 1, 1, 400
    a.plan_ints = a.sort_scratch_ints = 1 << 20
    peers = (C.c_void_p * 8)(*[4096] * 8)
    a.peer_x, a.world, a.tokens_per_rank = C.addressof(peers), world, per
    assert capi.lib().nq_prefill(C.byref(a), None) == -1          # NQ_ERR_ARG
    assert b"ranks" in capi.lib().nq_last_error()
