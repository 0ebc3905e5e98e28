"""FlashAttention forward at the edges of its query tiles and key blocks, with masks that cut through blocks, many rescales of the
output and several waves of thread blocks, against 64-bit arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(q, k, v, causal, window):
    """-> o [Tq, H, D], p @ |v|, lse [H, Tq] of one batch entry."""
    Tq, H, D = q.shape
    Tk, G = k.shape[:2]
    gap = (torch.arange(Tq, device=q.device) + Tk - Tq)[:, None] - torch.arange(Tk, device=q.device)[None]
    hidden = (gap < 0) & causal
    if window:
        hidden = hidden | (gap >= window)
    o, mag, lse = torch.zeros(Tq, H, D, device=q.device).double(), torch.zeros(Tq, H, D, device=q.device).double(), []
    for h in range(H):
        s = (q[:, h].double() @ k[:, h // (H // G)].double().t() * D ** -0.5).masked_fill(hidden, -torch.inf)
        p = torch.softmax(s, -1).nan_to_num(0.0)                      # a row that sees nothing is zero
        o[:, h], mag[:, h] = p @ v[:, h // (H // G)].double(), p @ v[:, h // (H // G)].double().abs()
        lse.append(torch.logsumexp(s, -1))
    return o, mag, torch.stack(lse)


@pytest.mark.parametrize("B,Tq,Tk,H,G,D,causal,window,grow", [
    (1, 1, 1, 4, 4, 64, True, 0, 1),
    (2, 127, 127, 4, 2, 64, True, 0, 1),
    (1, 129, 128, 4, 4, 128, True, 0, 1),            # the first query sees nothing
    (1, 65, 193, 3, 1, 128, True, 0, 1),
    (1, 64, 63, 4, 4, 64, False, 0, 1),
    (2, 257, 65, 4, 2, 128, False, 0, 1),
    (1, 300, 1000, 4, 4, 64, True, 1, 1),            # a window of the own position
    (1, 300, 700, 4, 2, 128, True, 65, 1),
    (1, 513, 513, 8, 1, 64, True, 128, 1),
    (1, 640, 640, 4, 4, 64, True, 0, 40),            # later keys ever larger: the maximum moves in every block
    (1, 640, 640, 4, 4, 128, True, 0, 40),
    (2, 2048, 2048, 32, 8, 128, True, 0, 1),         # several waves
    (2, 2048, 2048, 32, 4, 64, True, 0, 1),
])
def test_forward_against_64_bits(B, Tq, Tk, H, G, D, causal, window, grow):
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(Tq + Tk + D)
    q, k, v = (torch.randn(B, t, h, D, device="cuda") for t, h in ((Tq, H), (Tk, G), (Tk, G)))
    if grow > 1:
        k = k * torch.linspace(0.1, grow, Tk, device="cuda")[None, :, None, None]
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    o, lse = K.flash_fwd(q, k, v, causal=causal, window=window)
    for b in range(B):
        ref, mag, lref = reference(q[b], k[b], v[b], causal, window)
        # weights are rounded to bf16 and so is the result (8 bits: up to 2^-8 each, of p |v| and of |o| <= p |v|); scores in 32 bits are off
        # by up to D 2^-24 of the sum of their terms' sizes, and every weight by as much again
        terms = D ** 0.5 * 3 * max(1.0, 3.0 * grow)
        slack = 2 * D * 2.0 ** -24 * terms + 1e-6
        assert ((o[b].double() - ref).abs() <= (2.0 ** -7 * 1.01 + slack) * mag + 1e-30).all()
        live = torch.isfinite(lref)
        assert ((lse[b].double() - lref).abs()[live] <= slack * (1 + lref[live].abs())).all()
        assert (lse[b][~live] == -torch.inf).all()
    again, _ = K.flash_fwd(q, k, v, causal=causal, window=window)
    assert torch.equal(o, again)
    assert K.status_fetch() == 0


@pytest.mark.parametrize("Tq,Tk,D,causal,window", [(200, 200, 64, True, 0), (200, 265, 64, True, 0), (200, 200, 128, True, 0), (300, 365, 128, True, 0),
                                                   (300, 300, 64, True, 70), (300, 400, 128, True, 33), (100, 300, 128, False, 0)])
@pytest.mark.parametrize("scale", [-0.05, 0.0])
def test_negative_and_zero_scale(Tq, Tk, D, causal, window, scale):
    """Masked keys stay out whatever the sign of the scale, also where a row sees nothing of a whole block."""
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(0)
    q, k, v = (torch.randn(1, t, 2, D, device="cuda").bfloat16() for t in (Tq, Tk, Tk))
    o, lse = K.flash_fwd(q, k, v, causal=causal, scale=scale, window=window)
    gap = (torch.arange(Tq, device="cuda") + Tk - Tq)[:, None] - torch.arange(Tk, device="cuda")[None]
    hidden = ((gap < 0) & causal) | ((gap >= window) if window else False)
    for h in range(2):
        s = (q[0, :, h].double() @ k[0, :, h].double().t() * scale).masked_fill(hidden, -torch.inf)
        p = torch.softmax(s, -1)
        # weights and result are rounded to bf16
        assert ((o[0, :, h].double() - p @ v[0, :, h].double()).abs() <= 2.0 ** -7 * 1.01 * (p @ v[0, :, h].double().abs())).all()
        # scores and the logarithm of their sum in 32 bits
        assert ((lse[0, h].double() - torch.logsumexp(s, -1)).abs() <= 1e-5).all()
    assert K.status_fetch() == 0
