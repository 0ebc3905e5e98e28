"""A later portion of a prompt reads keys and values back from the cache; attention takes heads that lie side by side."""
import pytest
import torch


@pytest.mark.parametrize("portions,bs", [([5, 6], 16), ([1, 15], 16), ([3, 2, 7], 16), ([9, 20], 16), ([16, 1], 16)])
def test_portions_within_a_block(portions, bs, monkeypatch):
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    from litetorch_b200.models.llama_serving import LlamaKVModel
    from litetorch_b200.ops import kernels_ref
    eng = LlamaEngine(LlamaConfig.tiny(), "cpu", seed=0)
    flash, seen = kernels_ref.flash_fwd, []

    def checked(q, k, v, **kw):
        seen.append(k.shape[1])
        for t in (q, k, v):
            assert t.stride(3) == 1 and (t.shape[2] == 1 or t.stride(2) == t.shape[3]), (t.shape, t.stride())
        return flash(q, k, v, **kw)

    monkeypatch.setattr(eng.K, "flash_fwd", checked)
    model = LlamaKVModel(eng, num_blocks=8, block_size=bs)
    prompt = torch.randint(0, eng.cfg.vocab_size, (sum(portions),), generator=torch.Generator().manual_seed(1)).tolist()
    at = 0
    for n in portions:
        got = model.score_chunk(prompt[at:at + n], at, list(range(8)), [n - 1])
        at += n
    whole = LlamaKVModel(eng, num_blocks=8, block_size=bs).score_chunk(prompt, 0, list(range(8)), [len(prompt) - 1])
    assert max(seen) == len(prompt)
    # the same sums in the order of other shapes, activations in 16 bits
    assert float((got.float() - whole.float()).norm() / whole.float().norm()) < 0.02
