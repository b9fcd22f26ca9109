"""Which scratch a prefill call gets: the layer's own, kept between calls, or - under capture - tensors of the graph's."""
import pytest
import torch

from nestquant_b200 import moe


@pytest.fixture
def layer(monkeypatch):
    L = moe.MoELayer(8, 256, 128, Bmax=1, topk=2, dev="cpu")
    L.captured = False
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: L.captured)
    return L


CPU = torch.device("cpu")


def test_captured_calls_neither_use_nor_replace_what_is_kept(layer):
    L = layer
    sc, pm = L._prefill_scratch(64, CPU), L._prefill_perm(64, CPU)
    L.captured = True
    a, b = L._prefill_scratch(64, CPU), L._prefill_scratch(500, CPU)
    pa = L._prefill_perm(64, CPU)
    mine = {t.data_ptr() for t in (*sc.values(), *pm.values()) if isinstance(t, torch.Tensor)} - {sc["status"].data_ptr()}
    for d in (a, b, pa):
        assert not mine & {t.data_ptr() for t in d.values() if isinstance(t, torch.Tensor)}
    assert a["status"] is sc["status"] and b["status"] is sc["status"]      # one word, made with the layer: no replay clears it
    L.captured = False
    assert L._prefill_scratch(64, CPU) is sc and L._prefill_perm(64, CPU) is pm
    assert L._prefill_scratch(65, CPU)["R"] == 65
    assert L._prefill_scratch(65, CPU)["status"] is a["status"]


def test_first_call_under_capture_leaves_nothing_behind(layer):
    L = layer
    L.captured = True
    a = L._prefill_scratch(64, CPU)
    L._prefill_perm(64, CPU)
    assert a["status"].item() == 0 and L.prefill_status() == 0
    a["status"].fill_(1)
    L.captured = False
    assert L._prefill_scratch(64, CPU) is not a and L.prefill_status() == 1


def test_a_smaller_limit_gives_memory_back(layer):
    L = layer
    big = L._prefill_scratch(4096, CPU)
    assert L._prefill_scratch(100, CPU) is big                      # no limit named: kept
    assert L._prefill_scratch(100, CPU, 4096) is big
    small = L._prefill_scratch(100, CPU, 1024)                      # a call of 100 pairs that names 1,024
    assert small["R"] == 100 and small["y"].shape == (100, 256)
    assert L._prefill_scratch(1024, CPU, 1024)["R"] == 1024
    assert L._prefill_scratch(5, CPU, 1024)["R"] == 1024


def test_layers_that_share_scratch(layer):
    other = moe.MoELayer(8, 256, 128, Bmax=1, topk=2, dev="cpu")
    other.share_prefill_scratch(layer)
    assert other._prefill_scratch(64, CPU, 64) is layer._prefill_scratch(64, CPU)
    assert other._prefill_perm(9, CPU) is layer._prefill_perm(9, CPU)
    layer._pf_status.fill_(1)
    assert other.prefill_status() == 1
