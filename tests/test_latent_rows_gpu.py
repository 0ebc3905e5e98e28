"""Rotation, norm and cache write of latent rows, and the gate of a token's own input, at the edges of what is loaded at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,d,r,rot,rank,c", [(1, 6, 2, 2, 1, 2), (1, 8, 8, 8, 8, 8), (16, 128, 64, 64, 512, 512), (17, 64, 64, 62, 511, 512), (33, 8, 64, 64, 1024, 1032),
                                             (16, 64, 64, 56, 504, 512), (2, 6, 200, 198, 1301, 1400)])
@pytest.mark.parametrize("odd", [0, 1])
def test_latent_rows(dtype, H, d, r, rot, rank, c, odd):
    from litetorch_b200.ops import kernels as K
    N, bs = 5, 16
    g = torch.Generator(device="cuda").manual_seed(H + rank)
    q_cols = H * (d + r) + odd
    ld = q_cols + rank + rot
    proj = torch.randn(N, ld + -ld % 8, device="cuda", generator=g).to(dtype)
    proj[3, q_cols:q_cols + rank] = 0                           # its norm is zero over the root of eps
    w = torch.randn(rank, device="cuda", generator=g)
    freq = torch.tensor([500.0 ** (-2.0 * i / rot) for i in range(rot // 2)], dtype=torch.float64, device="cuda")
    pos = torch.tensor([0, 3, 64, 5000, 100001], dtype=torch.int32, device="cuda")
    slots = torch.tensor([7, 0, 31, 16, 33], dtype=torch.int32, device="cuda")
    cache, before = torch.full((3, 1, bs, c + r), 7.0, dtype=dtype, device="cuda"), proj.clone().double()
    K.latent_rope(proj, H, d, r, rot, pos, slots, freq=freq, c_off=q_cols, rank=rank, c_norm=w, eps=1e-6, cache=cache)
    a = pos.double()[:, None] * freq
    def turn(x):
        t = a.view(N, *[1] * (x.dim() - 2), -1)
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * t.cos() - v * t.sin(), v * t.cos() + u * t.sin()], -1).flatten(-2)
    def close(got, want, size):
        # two 32-bit products of the angle's cosine and sine (2 ulp), one rounding to the type
        err = 2.0 ** -20 * size + (want.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0)
        assert ((got.double() - want).abs() <= err).all()
    heads = before[:, :H * (d + r)].view(N, H, d + r)
    got = proj[:, :H * (d + r)].view(N, H, d + r)
    close(got[..., d:d + rot], turn(heads[..., d:d + rot]), 8.0)
    assert torch.equal(got[..., :d].double(), heads[..., :d]) and not bool(got[..., d + rot:].any())
    rows = cache[slots.long() // bs, 0, slots.long() % bs]
    lat = before[:, q_cols:q_cols + rank]
    want = lat / (lat.square().mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
    close(rows[:, :rank], want, want.abs() * 8)
    close(rows[:, c:c + rot], turn(before[:, q_cols + rank:q_cols + rank + rot]), 8.0)
    assert not bool(rows[:, rank:c].any()) and not bool(rows[:, c + rot:].any())
    assert int((cache != 7.0).any(-1).sum()) <= N


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,F,dim,off,width", [(1, 8, 8, 0, 8), (300, 64, 56, 104, 160), (300, 64, 56, 101, 160), (4096, 256, 256, 8, 1544), (7, 20, 16, 8, 64)])
def test_gates(dtype, N, F, dim, off, width):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(N + F)
    x, table = 2 * torch.randn(N, F, device="cuda", generator=g).to(dtype), torch.randn(11, width, device="cuda", generator=g).to(dtype)
    tok = torch.randint(0, 11, (N,), device="cuda", generator=g, dtype=torch.int32)
    o = K.token_gate(x, tok, table, off, dim)
    t = table[tok.long(), off:off + dim].double()
    want = torch.nn.functional.gelu(x[:, :dim].double(), approximate="tanh") * t
    err = want.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0
    assert ((o[:, :dim].double() - want).abs() <= err + 2.0 ** -20 * t.abs() * (1 + x[:, :dim].double().abs())).all()
    assert not bool(o[:, dim:].any())


@pytest.mark.parametrize("H,rank,w,window", [(4, 128, 192, 0), (17, 512, 576, 0), (16, 512, 576, 300)])
@pytest.mark.parametrize("splits", [1, 2, 7])
def test_not_a_number_in_latent_attention(H, rank, w, window, splits):
    """A NaN in a query makes its head's results NaN, one in a row that is seen those of all heads, and no others."""
    from litetorch_b200.ops import kernels as K
    bs, lens = 16, [700, 33, 501]
    g = torch.Generator(device="cuda").manual_seed(w + splits)
    width = (max(lens) + bs - 1) // bs
    tables = torch.randperm(len(lens) * width, generator=torch.Generator().manual_seed(w)).to(torch.int32).view(len(lens), width).cuda()
    cache = torch.randn(len(lens) * width, 1, bs, w, device="cuda", generator=g).bfloat16()
    q = torch.randn(len(lens), H, w, device="cuda", generator=g).bfloat16()
    ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")

    def run(q, cache):
        return K.latent_decode(q, cache, tables, ctx, rank=rank, window=window, scale=w ** -0.5, max_keys=max(lens), splits=splits)

    base = run(q, cache)
    assert bool(torch.isfinite(base.float()).all())
    q, cache = q.clone(), cache.clone()
    q[2, 3, 5] = float("nan")
    at = lens[0] - 100                                      # its place among the keys, not the values
    cache[int(tables[0, at // bs]), 0, at % bs, w - 1] = float("nan")
    want = torch.zeros_like(base, dtype=torch.bool)
    want[0] = True
    want[2, 3] = True
    got = run(q, cache)
    assert torch.equal(torch.isnan(got), want) and torch.equal(got[~want], base[~want])
    assert K.status_fetch() == 0
