"""Greedy tokens of logits, tokens of 32 bits, and later portions whose context is gathered in one launch."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,V", [(1, 1), (3, 7), (2, 1024), (5, 4097), (3, 8192), (40, 16390), (1, 32000), (7, 32003), (70, 32001), (200, 9000), (2, 128256)])
@pytest.mark.parametrize("odd", [False, True])
def test_argmax(dtype, rows, V, odd):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(V)
    room = torch.randn(rows, V + 3, device="cuda", generator=g).to(dtype)
    x = room[:, 1:V + 1] if odd else room[:, :V].contiguous()
    assert torch.equal(K.argmax_rows(x), x.float().argmax(-1))
    x[:, V // 2] = 100.0
    x[:, V - 1] = 100.0                             # of equals the first
    assert bool((K.argmax_rows(x) == V // 2).all())
    x.fill_(-math.inf)
    assert bool((K.argmax_rows(x) == 0).all())
    x[-1, V - 1] = math.nan
    assert torch.equal(K.argmax_rows(x), x.float().argmax(-1)) and int(K.argmax_rows(x)[-1]) == V - 1
    assert K.status_fetch() == 0


def test_tokens_of_32_bits():
    from litetorch_b200.ops import kernels as K
    table = torch.randn(77, 64, device="cuda").bfloat16()
    idx = torch.tensor([0, 76, 5, -3, 1000], device="cuda")
    want = table[idx.clamp(0, 76)]
    assert torch.equal(K.embedding_fwd(idx, table), want) and torch.equal(K.embedding_fwd(idx.to(torch.int32), table), want)


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_tokens_and_targets_that_do_not_lie_side_by_side(dtype):
    """Columns, every other one and repeats of one token, and their targets: the kernels read a dense list."""
    from litetorch_b200.ops import kernels as K
    V, D = 77, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    table = torch.randn(V, D, device="cuda", generator=g).bfloat16()
    room = torch.randint(0, V, (40, 6), device="cuda", generator=g).to(dtype)
    for idx in (room[:, 1:2], room[::2, 0], room[:, ::3], room[5, 2].expand(7, 3), room.t()):
        flat = [int(i) for i in idx.reshape(-1).tolist()]
        assert torch.equal(K.embedding_fwd(idx, table), table[flat])
        n = len(flat)
        dout = torch.randint(0, 2, (n, D), device="cuda", generator=g).bfloat16()
        want = torch.zeros(V, D, device="cuda").index_add_(0, torch.tensor(flat, device="cuda"), dout.float())
        got = torch.zeros_like(table)
        K.embedding_bwd(idx, dout, got)
        assert torch.equal(got.float(), want)                           # whole numbers up to 240: bf16 holds them and every sum on the way
        logits = torch.randn(n, V, device="cuda", generator=g).bfloat16()
        dense = torch.tensor(flat, device="cuda")
        tgt = idx.reshape(-1) if idx.dim() < 2 or idx.shape[1] == 1 else idx.flatten()
        stats = K.ce_stats(logits, tgt)
        assert torch.equal(stats, K.ce_stats(logits, dense))
        a, b = logits.clone(), logits.clone()
        assert torch.equal(K.ce_finish(a, tgt, stats), K.ce_finish(b, dense, stats)) and torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_logits_and_loss_of_columns(dtype):
    """One token of every sequence out of a longer batch, as `tokens[:, at : at + 1]` gives it."""
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    eng = LlamaEngine(LlamaConfig(vocab_size=256, n_layers=1, d_model=128, n_heads=2, n_kv_heads=1, head_dim=64, ffn=256, max_seq=64), "cuda", seed=4)
    tokens = torch.randint(0, 256, (5, 9), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).to(dtype)
    part, target = tokens[:, 3:4], tokens[:, 4:5]
    assert torch.equal(eng.forward_logits(part), eng.forward_logits(part.long().contiguous()))
    assert torch.equal(eng.eval_loss(part, target), eng.eval_loss(part.long().contiguous(), target.long().contiguous()))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [1, 400])
@pytest.mark.parametrize("V", [31, 255, 257, 2047, 2048, 2049, 4095, 4096, 4098, 16384, 16388])
def test_argmax_of_few_and_many_threads(dtype, rows, V):
    from litetorch_b200.ops import kernels as K
    x = torch.randn(rows, V, device="cuda", generator=torch.Generator(device="cuda").manual_seed(V)).to(dtype)
    x[:, V - 1] = 9.0
    assert bool((K.argmax_rows(x) == V - 1).all())
    x[:, V // 3] = 9.0
    assert bool((K.argmax_rows(x) == V // 3).all())
    assert K.status_fetch() == 0
