"""Recording of decode steps when memory is short, and inputs that come from the device."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(graphs=True):
    from litetorch_b200.models import registry
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    cfg = LlamaConfig(vocab_size=512, n_layers=2, d_model=128, n_heads=4, n_kv_heads=2, head_dim=64, ffn=256, max_seq=256)
    return registry.new_serving(LlamaEngine(cfg, "cuda", seed=2), num_blocks=64, block_size=16, max_num_seqs=4, graphs=graphs)


def test_recording_gives_cached_memory_back_when_none_is_left():
    """Memory that is cached on another stream cannot be used while a step is recorded: it is given back, and the step recorded once more."""
    prompt, table = list(range(40)), [5, 9, 2, 30]
    ref, m = _model(False), _model()
    want = [x.prefill_chunk(prompt, 0, table, True) and x.decode_logits([7], [40], [table]) for x in (ref, m)]      # (the second one records)
    m._graphs.clear()
    torch.cuda.empty_cache()
    real, calls = m._decode_body, []

    def body(*a):
        calls.append(torch.cuda.is_current_stream_capturing())
        out = real(*a)
        if not calls[-1]:
            # a free block that only this stream may use, and no room for another one
            del_me = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
            del del_me
            total = torch.cuda.get_device_properties(0).total_memory
            torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / total)
        return out

    m._decode_body = body
    try:
        got = m.decode_logits([7], [40], [table])
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert calls == [False, True, True]
    assert torch.equal(got, want[1])
    assert torch.equal(m.decode_logits([7], [40], [table]), want[1]) and len(calls) == 3
    # a step that needs more than there is still says so
    m._graphs.clear()

    def greedy(*a):
        if torch.cuda.is_current_stream_capturing():
            raise torch.cuda.OutOfMemoryError("none left")
        return real(*a)

    m._decode_body = greedy
    with pytest.raises(torch.cuda.OutOfMemoryError):
        m.decode_logits([7], [40], [table])
    m._decode_body = real
    assert torch.equal(m.decode_logits([7], [40], [table]), want[1])


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
