"""RMSNorm over many rows (several warps a row, the next row fetched ahead) against 64 bits, at the edges of its range of rows and widths."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [295, 296, 297, 1337])
@pytest.mark.parametrize("D", [256, 512, 1024, 1536, 3072, 4096, 5120, 8192])
def test_rows_against_64_bits(M, D):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + D)
    x, dy, dres = (torch.randn(M, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(D, device="cuda", generator=g)).bfloat16()
    y, _, _, rstd = K.norm_fwd(x, w, eps=1e-5)
    x64, w64, dy64 = x.double(), w.double(), dy.double()
    r = torch.rsqrt((x64 ** 2).mean(-1, keepdim=True) + 1e-5)
    xh = x64 * r

    def close(got, ref, size):
        # a rounding to bf16 of the result (2^-9 of it), and 32-bit sums of D terms of the given size
        assert ((got.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + size * 1e-5).all()

    close(y, xh * w64, 1.0)
    assert ((rstd.double() - r[:, 0]).abs() <= 1e-5 * r[:, 0]).all()
    gw = dy64 * w64
    dx_ref = r * (gw - xh * (gw * xh).mean(-1, keepdim=True))
    dw_ref = (dy64 * xh).sum(0)
    for res in (None, dres):
        for accumulate in (False, True):
            dw = torch.full((D,), 3.0, device="cuda", dtype=torch.bfloat16)
            dx, dw, _ = K.norm_bwd(dy, x, w, None, rstd, dres=res, dw=dw, accumulate=accumulate)
            close(dx, dx_ref + (0 if res is None else res.double()), 4.0)
            close(dw, dw_ref + (3.0 if accumulate else 0.0), M ** 0.5)
