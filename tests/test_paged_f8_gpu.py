"""Decode attention over e4m3 caches on the tensor-core kernel, against 64-bit arithmetic over sizes at the edges of its chunks, copies,
groups and splits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(q, kc, vc, tables, ctx, bs, scale, ks, vs, window):
    S, H, D = q.shape
    G = kc.shape[1]
    out = torch.zeros(S, H, D, dtype=torch.float64, device=q.device)
    for s in range(S):
        n = int(ctx[s])
        lo = max(0, n - window) if window else 0
        if n == lo:
            continue
        at = torch.arange(lo, n, device=q.device)
        k = kc[tables[s].long()[at // bs], :, at % bs].double() * ks                 # [keys, G, D]
        v = vc[tables[s].long()[at // bs], :, at % bs].double() * vs
        k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
        p = torch.softmax(torch.einsum("hd,khd->hk", q[s].double(), k) * scale, -1)
        out[s] = torch.einsum("hk,khd->hd", p, v)
    return out


@pytest.mark.parametrize("D,H,G,bs,window,contexts,splits", [
    (64, 8, 8, 8, 0, [1, 31, 32, 33], 1),
    (128, 8, 2, 16, 0, [1, 127, 128, 129, 1000], 3),
    (128, 32, 2, 32, 0, [4095, 17], 8),                  # 16 query heads to a key head
    (64, 12, 4, 64, 0, [63, 64, 65, 700], 2),            # blocks longer than a chunk, 3 heads to a key head
    (128, 16, 4, 16, 100, [5, 99, 100, 101, 131, 2000], 4),
    (64, 4, 4, 16, 33, [32, 33, 34, 500], 1),
    (64, 4, 4, 16, 1701, [2011, 1702, 1718], 1),         # a window that starts inside a chunk, in a stage that is filled several times
    (128, 8, 2, 32, 1701, [2011, 1719], 1),
])
def test_e4m3_decode_against_64_bits(D, H, G, bs, window, contexts, splits):
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(D + H + bs)
    S, ks, vs = len(contexts), 0.05, 0.07
    width = (max(contexts) + bs - 1) // bs + 1
    n_blocks = S * width
    kc, vc = (torch.randn(n_blocks, G, bs, D, device="cuda").mul_(20).to(torch.float8_e4m3fn) for _ in range(2))
    tables = torch.randperm(n_blocks, device="cuda").int().view(S, width).contiguous()
    q = torch.randn(S, H, D, device="cuda").to(torch.bfloat16)
    q[0, 0] *= 1e-6                                       # a head far below fp16's range as it stands, and one above it (see test_queries_of_any_size)
    q[0, -1] *= 1e6
    ctx = torch.tensor(contexts, dtype=torch.int32, device="cuda")
    # what lies past a sequence's end, or before its window, must not matter
    for s, n in enumerate(contexts):
        rows = list(range(n, width * bs)) + (list(range(0, n - window)) if window else [])
        for r in rows:
            for t in (kc, vc):
                t.view(torch.uint8)[tables[s, r // bs].long(), :, r % bs] = 0x7F      # NaN
    out = K.paged_decode(q, kc, vc, tables, ctx, bs, splits, D ** -0.5, ks, vs, window=window)
    ref = reference(q, kc, vc, tables, ctx, bs, D ** -0.5, ks, vs, window)
    assert torch.isfinite(out).all()
    # the result is rounded to bf16 (2^-9); scores of the row times 1e6 are in the millions, where 32-bit products are off by up to
    # 2^-24 of them times the length of the dot product, so that row may weigh two keys of nearly equal score differently: left out
    keep = torch.ones(S, H, dtype=torch.bool, device="cuda")
    keep[0, -1] = False
    err = (out.double() - ref)[keep].abs().max()
    assert err <= 2 ** -8 * ref[keep].abs().max(), float(err)
    assert K.status_fetch() == 0


def test_e4m3_decode_propagates_nan_keys():
    """A NaN inside the context is not hidden by the conversion of 8-bit values."""
    from litetorch_b200.ops import kernels as K
    kc, vc = (torch.randn(4, 1, 16, 64, device="cuda").to(torch.float8_e4m3fn) for _ in range(2))
    vc.view(torch.uint8)[1, 0, 3, 5] = 0x7F
    q = torch.randn(1, 2, 64, device="cuda").to(torch.bfloat16)
    out = K.paged_decode(q, kc, vc, torch.arange(4, device="cuda").int().view(1, 4), torch.tensor([60], dtype=torch.int32, device="cuda"), 16, 1, 0.125)
    assert torch.isnan(out[0, :, 5]).all() and torch.isfinite(out[0, :, 6]).all()


@pytest.mark.parametrize("fp8,D,bs,window", [(True, 64, 16, 0), (True, 128, 16, 40), (False, 128, 16, 0), (False, 64, 16, 33), (False, 64, 4, 0)])
@pytest.mark.parametrize("at", [1, 2, 3, 4])
def test_queries_at_any_address(fp8, D, bs, window, at):
    """Queries that start at any element (a packed view into a larger tensor) go to a kernel that reads them as they lie."""
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(at + D)
    kc, vc = (torch.randn(12, 2, bs, D, device="cuda").to(torch.float8_e4m3fn if fp8 else torch.bfloat16) for _ in range(2))
    tables = torch.randperm(12, device="cuda").int().view(2, 6).contiguous()
    ctx = torch.tensor([6 * bs - 1, 2 * bs + 1], dtype=torch.int32, device="cuda")
    room = torch.randn(2 * 8 * D + 8, device="cuda").to(torch.bfloat16)
    q = room[at:at + 2 * 8 * D].view(2, 8, D)
    out = K.paged_decode(q, kc, vc, tables, ctx, bs, 2, D ** -0.5, window=window)
    ref = reference(q, kc, vc, tables, ctx, bs, D ** -0.5, 1.0, 1.0, window)
    # 16-bit caches: weights and result are rounded to bf16 (2^-8 of the largest value each); 8-bit caches: the result alone
    assert (out.double() - ref).abs().max() <= 2 ** -7 * ref.abs().max()
    assert K.status_fetch() == 0


@pytest.mark.parametrize("D,n,splits", [(64, 4096, 1), (128, 16384, 1), (128, 16384, 32)])
def test_partial_sums_in_32_bits(D, n, splits):
    """The splits' outputs, as they go to the merge, over more chunks than a cut-off addition could take."""
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(n)
    H, G, bs = 8, 2, 16
    kc, vc = (torch.randn(n // bs, G, bs, D, device="cuda").to(torch.float8_e4m3fn) for _ in range(2))
    q, tables = torch.randn(1, H, D, device="cuda").bfloat16(), torch.randperm(n // bs, device="cuda").int().view(1, -1).contiguous()
    ctx, part = torch.tensor([n], dtype=torch.int32, device="cuda"), torch.empty(H, splits, D + 2, device="cuda")
    o = torch.empty(1, H, D, dtype=torch.bfloat16, device="cuda")
    assert K._fn("lt_paged_decode")(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), tables.data_ptr(), ctx.data_ptr(), part.data_ptr(), o.data_ptr(), 1, H, G, D,
                                    bs, n // bs, n // bs, splits, D ** -0.5, 1, 1.0, 1.0, K._stream()) == 0
    p = part.double()
    w = p[..., D + 1] * torch.exp(p[..., D] - p[..., D].amax(-1, keepdim=True))
    out = (w[..., None] * p[..., :D]).sum(1) / w.sum(1, keepdim=True)
    ref = reference(q, kc, vc, tables, ctx, bs, D ** -0.5, 1.0, 1.0, 0)[0]
    # a warp adds up to n / 128 chunks, each addition rounded to 2^-24 of a sum that is at most some times the result's size (values of
    # both signs), in either direction: (n / 128) ** 0.5 of them; scores of some units in 32 bits move weights by as much again
    assert float((out - ref).norm() / ref.norm()) <= 2 * 2.0 ** -24 * (n / 128) ** 0.5 / 3 ** 0.5 + 3e-7


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("up", [-80, -30, -14, 14, 30, 80])
def test_queries_of_any_size(D, up):
    """Queries far outside fp16's range, with the scale that brings the scores back: powers of two change nothing, bit for bit.  Heads of
    very different sizes side by side."""
    from litetorch_b200.ops import kernels as K
    torch.manual_seed(D)
    kc, vc = (torch.randn(40, 2, 16, D, device="cuda").to(torch.float8_e4m3fn) for _ in range(2))
    tables = torch.randperm(40, device="cuda").int().view(2, 20).contiguous()
    ctx = torch.tensor([317, 40], dtype=torch.int32, device="cuda")
    q = torch.randn(2, 8, D, device="cuda").bfloat16()
    q[:, 1] *= 2.0 ** -5
    q[:, 2] *= 4
    plain = K.paged_decode(q, kc, vc, tables, ctx, 16, 2, D ** -0.5)
    ref = reference(q, kc, vc, tables, ctx, 16, D ** -0.5, 1.0, 1.0, 0)
    assert ((plain.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * ref.abs().max()).all()      # rounded to bf16; 32-bit sums of values of both signs
    assert torch.equal(K.paged_decode(q * 2.0 ** up, kc, vc, tables, ctx, 16, 2, D ** -0.5 * 2.0 ** -up), plain)
    assert K.status_fetch() == 0
