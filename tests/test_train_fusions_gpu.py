"""Parts of a training step that share a launch: gate, up and their product from one product; attention gradients turned back by the rotary angles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,F,Kd", [(1, 64, 64), (128, 136, 64), (129, 8, 64), (256, 128, 72), (1000, 1000, 256), (2000, 5632, 2048)])
def test_gates_and_their_product(M, F, Kd):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + F)
    x = torch.randn(M, Kd, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * F, Kd, device="cuda", generator=g) * 2 * Kd ** -0.5).bfloat16()
    gu, h = K.gemm_swiglu(x, w)
    want = x.double() @ w.double().t()
    # a rounding to bf16 and 32-bit sums; the product, of rounded gates and ups with few rows, two of their roundings more
    assert ((gu.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-4).all()
    ref = torch.nn.functional.silu(want[:, :F]) * want[:, F:]
    assert ((h.double() - ref).abs() <= 3 * ref.abs() * 2.0 ** -8 + 1e-3).all()
    assert K.status_fetch() == 0


@pytest.mark.parametrize("B,T,H,G,D", [(1, 1, 2, 1, 64), (2, 129, 4, 2, 128), (1, 300, 8, 2, 64), (1, 640, 24, 8, 128), (2, 257, 40, 8, 64)])
@pytest.mark.parametrize("odd", [False, True])
def test_gradients_turned_back(B, T, H, G, D, odd):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(T + H)
    q, k, v, do = (torch.randn(B, T, h, D, device="cuda", generator=g).bfloat16() for h in (H, G, G, H))
    o, lse = K.flash_fwd(q, k, v, causal=True)
    ang = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * 1e4 ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)[None]
    cos, sin = ang.cos().float().contiguous(), ang.sin().float().contiguous()
    # rows of dq that lie 8 bytes past a 16-byte boundary, too
    room = torch.zeros(B, T, H * D + 8, device="cuda", dtype=torch.bfloat16)
    dq = room[:, :, 4:4 + H * D].unflatten(2, (H, D)) if odd else None
    plain = [t.clone() for t in K.flash_bwd(q, k, v, o, lse, do, causal=True)]
    turned = K.flash_bwd(q, k, v, o, lse, do, causal=True, dq=dq, rope=(cos, sin))
    for a, b in zip(plain[:2], turned[:2]):
        ref = a.clone().view(B * T, -1)
        K.rope_(ref, cos, sin, T, ref.shape[1] // D, D, backward=True)
        # both are rounded to bf16, one of them twice; dq is summed in any order
        size = a.float().abs().max() * 2.0 ** -7
        assert ((b.reshape(B * T, -1).float() - ref.float()).abs() <= ref.float().abs() * 2.0 ** -7 + size).all()
        err = (b.reshape(B * T, -1).double() - ref.double()).norm() / ref.double().norm()
        assert float(err) < 4e-3
    assert torch.equal(plain[2], turned[2]) and (room[:, :, :4] == 0).all() and (room[:, :, 4 + H * D:] == 0).all()
    assert K.status_fetch() == 0
