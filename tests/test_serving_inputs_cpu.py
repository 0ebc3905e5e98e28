"""Inputs of prompt portions and decode steps as they are packed on the host."""
import numpy as np
import pytest
import torch


def _model():
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    from litetorch_b200.models.registry import new_serving
    cfg = LlamaConfig(vocab_size=64, n_layers=1, d_model=64, n_heads=2, n_kv_heads=1, head_dim=32, ffn=64, max_seq=256)
    return new_serving(LlamaEngine(cfg, "cpu", seed=1), num_blocks=40, block_size=4, max_num_seqs=4)


def test_prompt_inputs():
    m = _model()
    for start, n in ((0, 1), (0, 9), (3, 5), (8, 4)):
        blocks = [7, 3, 30, 11, 2][:(start + n + 3) // 4 + 1]
        tok, pos, slots, table = m._prompt_inputs(list(range(10, 10 + n)), start, blocks)
        assert tok.tolist() == list(range(10, 10 + n)) and pos.tolist() == list(range(start, start + n))
        assert slots.tolist() == [blocks[p // 4] * 4 + p % 4 for p in range(start, start + n)] and table.tolist() == blocks[:(start + n + 3) // 4]
        assert all(t.dtype == torch.int32 for t in (tok, pos, slots, table))


def test_decode_inputs():
    m = _model()
    seen = []
    m._decode_body = lambda d, S, width: seen.append((d, S, width)) or (torch.zeros(S, 64), torch.zeros(S))
    tables = [[5], [9, 1, 8, 12, 13], (4, 6, 20)]         # the second is longer than its sequence
    m._run_decode([3, 1, 2], [2, 11, 8], tables, [7, 0, 5])
    d, S, width = seen[0]
    assert (S, width) == (3, 3) and d.shape == (8, 3) and d.dtype == torch.int32
    assert d[:5].tolist() == [[3, 1, 2], [2, 11, 8], [22, 35, 80], [3, 12, 9], [7, 0, 5]]
    assert d[5:].t().tolist() == [[5, 0, 0], [9, 1, 8], [4, 6, 20]]


def test_runs_of_rows():
    m = _model()
    assert m._run_of([5]) == slice(5, 6) and m._run_of(range(2, 6)) == slice(2, 6)
    assert m._run_of([]) is None and m._run_of([1, 3]) is None and m._run_of([2, 1]) is None and m._run_of([-1]) is None
    x = torch.randn(8, 64, generator=torch.Generator().manual_seed(6))
    # other rows beside a row may change the order of its 32-bit sums: 64 terms, 64 x 2^-24 of the sum of their sizes, which is at most
    # |normalised row| |weights of a column| = 8 x 0.3
    near = dict(rtol=0, atol=64 * 2.0 ** -24 * 8 * 0.3)
    assert float(m.e.w.p("lm_head").float().norm(dim=1).max()) < 0.3
    assert torch.allclose(m._logits(x, [3, 4]), m._logits(x)[3:5], **near) and torch.allclose(m._logits(x, [4, 1]), m._logits(x)[[4, 1]], **near)


def _family(name):
    """(serving model, vocabulary) of a small model."""
    import os
    import sys
    sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
    if name == "llama":
        return _model(), 64
    suite = __import__(name + "_suite")
    cfg = suite.CONFIGS["odd"]
    from decoder_suite import server
    return server(suite.engine(cfg, suite.weights(cfg), "cpu", torch.float32), block_size=4)[0], cfg["vocab"]


@pytest.mark.parametrize("name", ["llama", "ravenex", "safuvik"])
def test_rows_that_are_not_there_are_refused(name):
    m, vocab = _family(name)
    tokens, table = [3, 1, 4], [7, 2]
    every = m.score_chunk(tokens, 0, table, [0, 1, 2])
    assert every.shape == (3, vocab)
    for rows in ([2, 3], [3], [1, 5], [-4], [-4, -3], range(1, 4)):
        with pytest.raises(IndexError):
            m.score_chunk(tokens, 0, table, rows)
    for rows in ([1, 2], [2], [-1], [-3, -2], [2, 0], (1,), range(0, 2), torch.tensor([1, 2]), np.array([0, 2])):
        at = [int(r) for r in rows]
        assert torch.allclose(m.score_chunk(tokens, 0, table, rows), every[at], atol=1e-5)
    assert m.score_chunk(tokens, 0, table, []).shape == (0, vocab)


def test_inputs_that_are_tensors_and_tokens_past_32_bits():
    m = _model()
    tables = [[5, 9, 2], [1, 3, 8]]
    for t in tables:
        m.prefill_chunk(list(range(6)), 0, t, False)
    want = m.decode_logits([7, 63], [6, 6], tables)
    for tok, pos, bt in ((torch.tensor([7, 63]), torch.tensor([6, 6]), [torch.tensor(t) for t in tables]),
                         ((np.int64(7), 63), np.array([6, 6]), [np.array(t) for t in tables]),
                         ([torch.tensor(7), torch.tensor(63)], (6, 6), tables), ([7, 1 << 40], [6, 6], tables)):
        assert torch.equal(m.decode_logits(tok, pos, bt, slots=torch.tensor([0, 0])), want)
    one = m.score_chunk([1, 63], 0, tables[0], [1])
    assert torch.equal(m.score_chunk(torch.tensor([1, 63]), 0, torch.tensor(tables[0]), [1]), one)
    assert torch.equal(m.score_chunk([1, 1 << 40], 0, tables[0], [1]), one)
    assert torch.equal(m.score_chunk([1, -1 << 40], 0, tables[0], [1]), m.score_chunk([1, -3], 0, tables[0], [1]))
