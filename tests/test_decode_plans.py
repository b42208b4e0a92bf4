"""How attention is planned (kernels/ops.py): which kernel runs, in how many splits, for how many SMs, on the CPU with a library that records."""
import pytest
import torch

from transformers_neuronx_b200.kernels import ops


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append((name, args)) or 0


@pytest.fixture
def recorded(monkeypatch):
    lib = Recorder()
    monkeypatch.setattr(ops, "_lib", lambda *a: lib)
    monkeypatch.setattr(ops, "_need", lambda *a, **k: None)
    monkeypatch.setattr(ops, "_state", lambda device: {"sms": 148})
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "_check", lambda *a: None)
    return lib


def _grouped_call(lib, rows, heads, kv, d, pages, **kw):
    q = torch.zeros(rows, heads * d, dtype=torch.bfloat16)
    i32 = torch.zeros(rows, dtype=torch.int32)
    cache = torch.zeros(1, 2, kv, 16, d, dtype=torch.bfloat16)
    ops.attention_decode(q, cache, torch.zeros(rows, pages, dtype=torch.int32), i32, i32, q.clone(), heads, 0.1, max_kv_len=16 * pages,
                         grouped=True, **kw)
    name, args = lib.calls[-1]
    assert name == "tnx_attention_decode_grouped"
    return args[17].value                               # the splits, after the scale


@pytest.mark.parametrize("rows,heads,kv,d,pages", [(2, 32, 8, 128, 33), (1, 32, 2, 128, 25), (4, 12, 12, 64, 33), (8, 16, 1, 128, 25), (3, 32, 8, 128, 9)])
def test_grouped_decode_runs_the_planned_splits(recorded, rows, heads, kv, d, pages):
    """A row's own pages are cut into as many parts as the plan says, also where that does not divide the bound on them."""
    per_block = ops.grouped_decode_heads(heads, kv, d)
    planned = ops.grouped_decode_plan(rows * kv * -(-(heads // kv) // per_block), 148, per_block, pages, d)[1]
    assert planned > 1 and pages % planned              # (a plan that was rounded: 8 to 7, 6 to 5, 4 to 3)
    assert _grouped_call(recorded, rows, heads, kv, d, pages) == planned


def test_grouped_decode_runs_the_splits_asked_for(recorded):
    assert [_grouped_call(recorded, 2, 8, 2, 64, 44, n_splits=n, warps=4) for n in (1, 3, 7, 8, 20)] == [1, 3, 7, 8, 8]
    assert _grouped_call(recorded, 2, 8, 2, 64, 3, n_splits=7, warps=4) == 3


@pytest.mark.parametrize("heads,rows,pages,grouped", [(12, 32, 2, False), (12, 32, 4, False), (32, 64, 4, False), (32, 16, 2, False),
                                                      (32, 8, 2, True), (12, 32, 12, True), (32, 64, 12, True), (32, 64, 128, True)])
def test_many_short_contexts_of_112_dims_go_a_head_a_block(heads, rows, pages, grouped):
    assert ops.grouped_decode_takes(rows, heads, heads, 112, 148, pages) == grouped
    assert ops.grouped_decode_takes(rows, heads, heads, 96, 148, pages)
    assert ops.grouped_decode_takes(rows, heads, heads // 4, 112, 148, pages)


def test_32_bit_attention_lays_its_blocks_out_for_the_devices_sms(recorded, monkeypatch):
    monkeypatch.setattr(ops, "_sm_count", lambda device: 132)
    q, i32 = torch.zeros(70, 32 * 64), torch.zeros(70, dtype=torch.int32)
    ops.attention_simt(q, torch.zeros(1, 2, 32, 16, 64), torch.zeros(1, 8, dtype=torch.int32), i32, i32, q.clone(), 32, 0.1)
    assert recorded.calls[-1][1][-2].value == 132        # before the stream
