"""What the runner chooses for a decode step before it looks for a CUDA graph: how attention is cut, and the rows of the graph."""
import types

import pytest

from zse_b200.models.decoder import DecoderModel
from zse_b200.models.hybrid import HybridModel
from zse_b200.runtime.runner import ModelRunner


def _splits(seqs, max_len, tokens=None, kv_heads=4, head_dim=128, most=16, sms=148):
    model = types.SimpleNamespace(plan=types.SimpleNamespace(num_kv_heads=kv_heads),
                                  config=types.SimpleNamespace(head_dim=head_dim))
    return DecoderModel.attention_splits(model, seqs, max_len, most, sms, tokens)


@pytest.mark.parametrize("seqs", [1, 8, 64, 160])
def test_a_batch_size_has_two_ways_to_cut(seqs):
    """Contexts grow from nothing to 32768 tokens: whole items first, then equal shares; never a third CUDA graph, and no way back."""
    seen = [_splits(seqs, n, tokens) for n in range(1, 32769, 61) for tokens in (seqs * n,)]
    assert set(seen) <= {1, 16} and seen == sorted(seen)


@pytest.mark.parametrize("seqs,max_len,tokens,kv_heads,cut", [
    (1, 300, 300, 4, False), (1, 1000, 1000, 4, True), (17, 100, 1700, 4, False), (32, 300, 9600, 4, False),
    (17, 3000, 26350, 4, True), (100, 900, 48200, 4, False), (16, 2300, 19424, 8, True), (64, 2300, 77696, 8, False),
    (5, 20011, 65030, 4, True), (160, 1100, 93120, 4, False), (160, 20011, 80000, 4, True)])
def test_cut_where_the_longest_sequence_decides(seqs, max_len, tokens, kv_heads, cut):
    assert _splits(seqs, max_len, tokens, kv_heads) == (16 if cut else 1)


def test_bounds_of_the_cut():
    assert _splits(1, 20000, 20000, most=1) == 1 and _splits(1, 20000, 20000, most=8) == 8
    assert _splits(4, 3000) == _splits(4, 3000, 12000)


def test_models_without_paged_heads_take_the_number_of_tokens_too():
    assert HybridModel.attention_splits(types.SimpleNamespace(heads_specs=[]), 1, 100, 16, 148, 100) == 1


@pytest.mark.parametrize("sharded,rows", [(False, {1: 1, 5: 8, 65: 96, 96: 96, 97: 128, 130: 160, 161: 192, 193: 256, 256: 256}),
                                          (True, {1: 1, 5: 8, 65: 128, 96: 128, 97: 128, 130: 256, 161: 256, 256: 256})])
def test_rows_of_the_graph(sharded, rows):
    """A sharded model's step keeps the rows, and so the exchange, of the next power of two."""
    runner = types.SimpleNamespace(model=types.SimpleNamespace(comm=object() if sharded else None), max_batch_seqs=256,
                                   DECODE_BUCKETS=ModelRunner.DECODE_BUCKETS, SHARDED_BUCKETS=ModelRunner.SHARDED_BUCKETS)
    assert {n: ModelRunner._graph_rows(runner, n) for n in rows} == rows
    runner.max_batch_seqs = 80
    assert ModelRunner._graph_rows(runner, 70) == 80
