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
