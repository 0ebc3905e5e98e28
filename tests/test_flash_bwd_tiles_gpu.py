"""FlashAttention backward at the edges of its query and key blocks, over one and several waves of thread blocks, against 64-bit
arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -8 * 1.02                                      # rounding to bf16


@pytest.mark.parametrize("B,Tq,Tk,H,G,D,causal", [
    (1, 1, 1, 2, 2, 64, True), (1, 127, 127, 4, 2, 64, True), (2, 129, 129, 4, 4, 128, True), (1, 128, 320, 2, 1, 128, True),
    (1, 65, 257, 3, 1, 64, False), (2, 385, 130, 4, 2, 128, False), (1, 700, 700, 8, 1, 64, True), (1, 1000, 1000, 8, 2, 128, True),
    (4, 1100, 1100, 16, 16, 64, True), (4, 1100, 1100, 16, 16, 128, False),
])
def test_backward_against_64_bits(B, Tq, Tk, H, G, D, causal):
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(Tq + Tk + D)
    q, k, v, do = (torch.randn(B, t, h, D, device="cuda").bfloat16() for t, h in ((Tq, H), (Tk, G), (Tk, G), (Tq, H)))
    o, lse = K.flash_fwd(q, k, v, causal=causal)
    dq, dk, dv = K.flash_bwd(q, k, v, o, lse, do, causal=causal)
    scale, R = D ** -0.5, H // G
    hidden = ((torch.arange(Tq, device="cuda") + Tk - Tq)[:, None] < torch.arange(Tk, device="cuda")[None]) & causal
    for b in range(B):
        for g in range(G):
            kk, vv = k[b, :, g].double(), v[b, :, g].double()
            sums = [torch.zeros(Tk, D, device="cuda").double() for _ in range(4)]
            for h in range(g * R, (g + 1) * R):
                qq, dd = q[b, :, h].double(), do[b, :, h].double()
                p = torch.softmax((qq @ kk.t() * scale).masked_fill(hidden, -torch.inf), -1)
                oo = p @ vv
                ds = p * (dd @ vv.t() - (oo * dd).sum(-1, keepdim=True)) * scale
                # weights and their gradients are rounded for the products; the row term comes from the rounded output
                ep = (U + 1e-5) * p
                es = (U + 1e-4) * ds.abs() + p * scale * (U * (p @ vv.abs() * dd.abs()).sum(-1, keepdim=True) * 2 + 1e-4)
                want = ds @ kk
                assert ((dq[b, :, h].double() - want).abs() <= es @ kk.abs() + U * want.abs() + 1e-6).all()
                for s, x in zip(sums, (p.t() @ dd, ep.t() @ dd.abs(), ds.t() @ qq, es.t() @ qq.abs())):
                    s += x
            assert ((dv[b, :, g].double() - sums[0]).abs() <= sums[1] + U * sums[0].abs() + 1e-6).all()
            assert ((dk[b, :, g].double() - sums[2]).abs() <= sums[3] + U * sums[2].abs() + 1e-6).all()
    again = K.flash_bwd(q, k, v, o, lse, do, causal=causal)
    assert torch.equal(again[1], dk) and torch.equal(again[2], dv)              # dQ is summed in any order
    assert K.status_fetch() == 0
