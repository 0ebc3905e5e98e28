"""Decode steps and prompt portions whose inputs come from the device."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(graphs=True):
    from litetorch_b200.models import registry
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    cfg = LlamaConfig(vocab_size=512, n_layers=2, d_model=128, n_heads=4, n_kv_heads=2, head_dim=64, ffn=256, max_seq=256)
    return registry.new_serving(LlamaEngine(cfg, "cuda", seed=2), num_blocks=64, block_size=16, max_num_seqs=4, graphs=graphs)


@pytest.mark.parametrize("graphs", [False, True])
def test_tokens_and_positions_on_the_device(graphs):
    """What a step returns can be handed to the next one as it is."""
    m = _model(graphs)
    tables = [[5, 9, 2, 30], [1, 3, 8, 7]]
    for t in tables:
        m.prefill_chunk(list(range(20)), 0, t, False)
    want = m.decode_logits([7, 300], [20, 20], tables)
    tok, pos = torch.tensor([7, 300], device="cuda"), torch.tensor([20, 20], device="cuda")
    for dt in (torch.int64, torch.int32):
        assert torch.equal(m.decode_logits(tok.to(dt), pos.to(dt), tables), want)
    assert torch.equal(m.decode_logits(list(tok), [20, 20], [torch.tensor(t, device="cuda") for t in tables]), want)
    one = m.score_chunk(torch.arange(20, device="cuda"), 0, torch.tensor(tables[0], device="cuda"), [3])
    assert torch.equal(one, m.score_chunk(list(range(20)), 0, tables[0], [3]))
    # a token beyond 32 bits is the vocabulary's last one, as any other beyond it
    assert torch.equal(m.decode_logits([1 << 40, 300], [20, 20], tables), m.decode_logits([511, 300], [20, 20], tables))
    assert torch.equal(m.score_chunk([1, 1 << 40], 0, tables[0], [1]), m.score_chunk([1, 600], 0, tables[0], [1]))
