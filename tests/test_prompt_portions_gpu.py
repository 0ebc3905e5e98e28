"""A prompt in portions gives the logits of the whole prompt, also where a later portion still lies in the first block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kv", [torch.bfloat16, torch.float8_e4m3fn])
@pytest.mark.parametrize("portions,bs", [([5, 6], 16), ([1, 15], 16), ([3, 2, 7], 16), ([16, 1], 16), ([10, 100], 64)])
def test_portions_against_the_whole(portions, bs, kv):
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    from litetorch_b200.models.llama_serving import LlamaKVModel
    from litetorch_b200.ops import kernels as K
    eng = LlamaEngine(LlamaConfig.tiny(), "cuda", seed=0)
    prompt = torch.randint(0, eng.cfg.vocab_size, (sum(portions),), generator=torch.Generator().manual_seed(1)).tolist()
    model, at = LlamaKVModel(eng, num_blocks=8, block_size=bs, kv_dtype=kv), 0
    for n in portions:
        got = model.score_chunk(prompt[at:at + n], at, list(range(8)), [n - 1])
        at += n
    whole = LlamaKVModel(eng, num_blocks=8, block_size=bs, kv_dtype=kv).score_chunk(prompt, 0, list(range(8)), [len(prompt) - 1])
    # activations of two layers in 16 bits; an 8-bit cache is read back by later portions only, and rounds to 2^-4
    assert float((got.float() - whole.float()).norm() / whole.float().norm()) < (0.02 if kv == torch.bfloat16 else 0.06)
    assert K.status_fetch() == 0
