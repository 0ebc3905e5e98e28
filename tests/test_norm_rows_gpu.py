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


@pytest.mark.parametrize("T,W", [(296, 256), (701, 512), (400, 768), (1337, 1792), (600, 2048), (4099, 2048), (513, 4096)])
@pytest.mark.parametrize("y_norm,norm,embed,pick", [(1, 1, 0, 0), (0, 1, 0, 0), (1, 0, 0, 1), (1, 1, 1, 0), (0, 0, 1, 1)])
def test_residual_of_many_rows(T, W, y_norm, norm, embed, pick):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(T + W)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, y, gy, gh = rand(T, W), rand(T, W + 8).bfloat16()[:, :W], 1 + 0.1 * rand(W), 1 + 0.1 * rand(W)
    table, tokens = rand(50, W).bfloat16(), torch.randint(0, 50, (T,), device="cuda", generator=g, dtype=torch.int32)
    rows = torch.randperm(T, device="cuda", generator=g)[:T - 3 if T > 300 else T].int() if pick else None
    opt = dict(dtype=torch.bfloat16, mult=0.6, y=y, y_norm=gy if y_norm else None, norm=gh if norm else None, rows=rows)
    if embed:
        opt.update(tokens=tokens, embed=table)
    rms = lambda v, w: v / (v.square().mean(1, keepdim=True) + 1e-5).sqrt() * w.double()
    base = table[tokens.long()].double() if embed else x.double()
    want = base + 0.6 * (rms(y.double(), gy) if y_norm else y.double())
    at = rows.long() if pick else torch.arange(T, device="cuda")
    out = rms(want, gh) if norm else want
    keep = x.clone()
    h = K.residual_norm(x, 1e-5, **opt)
    # 32 bits: W products summed, a root, a quotient; h is rounded to bf16 once
    err = (W ** 0.5 + 16) * 2.0 ** -24
    assert ((x[at].double() - want[at]).abs() <= (want[at].abs() + base[at].abs() + 1) * err).all()
    assert ((h.double() - out[at]).abs() <= out[at].abs() * (2.0 ** -8 + err) + 4 * err).all()
    untouched = torch.ones(T, dtype=torch.bool, device="cuda")
    untouched[at] = False
    assert torch.equal(x[untouched], keep[untouched])
    again = keep.clone()
    assert torch.equal(K.residual_norm(again, 1e-5, write=False, **opt), h) and torch.equal(again, keep)
