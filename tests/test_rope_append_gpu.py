"""Rotation with the cache write in one launch, against the separate kernels bit for bit; the merge of more splits than a warp has lanes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("n,H,G,D,bs", [(1, 4, 1, 64, 16), (33, 32, 8, 128, 16), (7, 12, 3, 8, 5), (300, 6, 6, 64, 32)])
def test_rope_append(n, H, G, D, bs, in_place, fp8):
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(n)
    blocks, ld = (n + bs - 1) // bs + 2, (H + 2 * G) * D + 8
    qkv = torch.randn(n, ld, device="cuda").bfloat16()[:, :ld - 8]
    cos, sin = (torch.randn(1000, D // 2, device="cuda") for _ in range(2))
    pos = torch.randint(0, 1000, (n,), device="cuda").int()
    slots = torch.randperm(blocks * bs, device="cuda")[:n].int()
    if n > 1:
        slots[n // 2] = -1                                # not cached
    dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
    caches = [[torch.zeros(blocks, G, bs, D, device="cuda").to(dt) for _ in range(2)] for _ in range(2)]
    x, y = qkv.clone(), qkv.clone()
    K.rope_(x, cos, sin, 1, H, D, positions=pos)
    K.rope_(x, cos, sin, 1, G, D, col_offset=H * D, positions=pos)
    k, v = (x[:, a * D:(a + G) * D].reshape(n, G, D).contiguous() for a in (H, H + G))
    K.kv_append(k, v, *caches[0], slots, bs, fp8, 0.5, 0.25)
    wide, far = pos.long(), torch.stack([slots.long(), slots.long()], 1)[:, 0]           # other types and strides of whole numbers mean the same
    q = K.rope_append(y, cos, sin, wide, far, H, G, D, *caches[1], bs, fp8, 0.5, 0.25, in_place=in_place)
    assert torch.equal(q, x[:, :H * D].reshape(n, H, D))
    assert torch.equal(y, x if in_place else qkv)
    for a, b in zip(*caches):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


@pytest.mark.parametrize("D,splits", [(64, 31), (64, 33), (128, 32), (128, 70)])
def test_merge_of_many_splits(D, splits):
    """Some splits hold no keys.  Rounding to bf16 on both sides (2^-8 of the value each) and of the weights inside every split (2^-8 of
    the largest value)."""
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(splits)
    kc, vc = (torch.randn(100, 2, 16, D, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(2, 8, D, device="cuda").bfloat16()
    bt = torch.randperm(100, device="cuda").int()[:100].view(2, 50).contiguous()
    ctx = torch.tensor([790, 45], dtype=torch.int32, device="cuda")
    one, many = (K.paged_decode(q, kc, vc, bt, ctx, 16, s, D ** -0.5) for s in (1, splits))
    assert ((one.float() - many.float()).abs() <= 2 ** -7 * one.float().abs() + 2 ** -7 * vc.float().abs().max() * 0.25).all()
    assert torch.isfinite(many).all()
