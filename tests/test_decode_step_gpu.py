"""Attention of a decode step in one launch (rotation, cache write, splits merged in a cluster) against the launches it stands in for and against 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(S, G, Hkv, D, bs, longest, fp8, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    H = G * Hkv
    ctx = [longest] + [1 + (longest - 1) * (37 * s % 101) // 101 for s in range(1, S)]
    width = (longest + bs - 1) // bs + 1
    order = torch.randperm(S * width + 3, generator=torch.Generator().manual_seed(seed)).tolist()
    bt = torch.tensor(order[:S * width], dtype=torch.int32).view(S, width)
    dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
    kc, vc = (torch.randn(S * width + 3, Hkv, bs, D, device="cuda", generator=g).bfloat16().to(dt) for _ in range(2))
    pos = torch.tensor([c - 1 for c in ctx], dtype=torch.int32)
    slots = torch.tensor([int(bt[s, (c - 1) // bs]) * bs + (c - 1) % bs for s, c in enumerate(ctx)], dtype=torch.int32)
    qkv = torch.randn(S, (H + 2 * Hkv) * D + 8, device="cuda", generator=g).bfloat16()[:, :(H + 2 * Hkv) * D]
    ang = torch.arange(longest + 1, device="cuda", dtype=torch.float64)[:, None] * 1e4 ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)[None]
    return qkv, ang.cos().float().contiguous(), ang.sin().float().contiguous(), pos.cuda(), slots.cuda(), kc, vc, bt.cuda(), torch.tensor(ctx, dtype=torch.int32).cuda(), ctx


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("S,G,Hkv,D,bs", [(1, 8, 4, 64, 16), (3, 4, 2, 128, 16), (5, 1, 3, 64, 8), (2, 16, 1, 128, 32), (4, 9, 2, 64, 64)])
@pytest.mark.parametrize("longest,splits", [(1, 1), (2, 8), (31, 1), (32, 2), (33, 3), (128, 1), (129, 4), (700, 8), (1500, 5), (3000, 32), (300, 0), (3000, 0), (4500, 0)])
def test_step_against_its_parts(S, G, Hkv, D, bs, longest, splits, fp8):
    from litetorch_b200.ops import kernels as K
    H = G * Hkv
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(S, G, Hkv, D, bs, longest, fp8, longest + S)
    ks, vs = (0.5, 2.0) if fp8 else (1.0, 1.0)
    k1, v1, k2, v2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
    keep = qkv.clone()
    o = K.decode_step(qkv, cos, sin, pos, slots, H, Hkv, D, k1, v1, bt, ctx, bs, splits, ks, vs)
    assert torch.equal(qkv, keep)
    q = K.rope_append(qkv, cos, sin, pos, slots, H, Hkv, D, k2, v2, bs, fp8, ks, vs)
    want = K.paged_decode(q, k2, v2, bt, ctx, bs, max(1, splits), D ** -0.5, ks, vs)
    bits = torch.uint8 if fp8 else torch.int16
    assert torch.equal(k1.view(bits), k2.view(bits)) and torch.equal(v1.view(bits), v2.view(bits))
    assert ((o.float() - want.float()).abs() <= want.float().abs() * 2.0 ** -7 + 2e-3).all()
    # 64 bits, from the rotated queries and the caches
    for s, n in enumerate(lens):
        at = bt[s].long()[torch.arange(n, device="cuda") // bs], torch.arange(n, device="cuda") % bs
        kk, vv = (t[at[0], :, at[1]].double() * f for t, f in ((k1, ks), (v1, vs)))                    # [n, Hkv, D]
        p = torch.softmax(torch.einsum("hgd,nhd->hgn", q[s].double().view(Hkv, G, D), kk) * D ** -0.5, -1)
        ref = torch.einsum("hgn,nhd->hgd", p, vv).reshape(H, D)
        # a rounding of the result; of the 16-bit kernel's weights too, each within 2^-9 of itself
        size = torch.einsum("hgn,nhd->hgd", p, vv.abs()).reshape(H, D)
        assert ((o[s].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + size * 2.0 ** -8 + 1e-4).all()
    assert K.status_fetch() == 0


def test_splits_by_size():
    from litetorch_b200.ops import kernels as K
    sms = K.sm_count()
    seen = set()
    for pairs in (1, 4, 8, 9, 24, 64, 96, 128, 160, 256, 512):
        for keys in (16, 300, 1000, 4096, 16384, 70000):
            for D in (64, 128):
                for fp8 in (False, True):
                    how, n = K._decode_splits(pairs, keys, D, fp8)
                    seen.add(how)
                    assert n >= 1 and (how != "cluster" or n <= 16) and (n == 1 or keys // n >= 100)
                    assert how != "cluster" or n == 1 or n <= 8 or (D == 64 and pairs * n <= sms)
    assert seen == {"cluster", "part"}


def test_tokens_without_a_slot_and_caches_it_does_not_take():
    from litetorch_b200.ops import kernels as K
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(4, 4, 2, 64, 16, 200, False, 1)
    none = slots.clone()
    none[1:] = -1
    k1, v1, k2, v2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
    a = K.decode_step(qkv, cos, sin, pos, slots, 8, 2, 64, k1, v1, bt, ctx, 16, 4)
    b = K.decode_step(qkv, cos, sin, pos, none, 8, 2, 64, k2, v2, bt, ctx, 16, 4)
    assert torch.equal(a, b)                        # the newest row comes from the product, not from the cache
    assert torch.equal(k2[[i for i in range(k2.shape[0]) if i != int(slots[0]) // 16]], kc[[i for i in range(k2.shape[0]) if i != int(slots[0]) // 16]])
    # blocks of four keys go through the parts
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(4, 4, 2, 64, 4, 200, False, 1)
    k1, v1, k2, v2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
    a = K.decode_step(qkv, cos, sin, pos, slots, 8, 2, 64, k1, v1, bt, ctx, 4, 3)
    b = K.paged_decode(K.rope_append(qkv, cos, sin, pos, slots, 8, 2, 64, k2, v2, 4, False), k2, v2, bt, ctx, 4, 3, 64 ** -0.5)
    assert torch.equal(a, b) and torch.equal(k1.view(torch.int16), k2.view(torch.int16))
    assert K.status_fetch() == 0


def test_not_a_number_past_the_context():
    """What lies in a block past the newest row, and in the newest row's place, is not seen."""
    from litetorch_b200.ops import kernels as K
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(3, 4, 2, 128, 16, 45, False, 7)
    a = K.decode_step(qkv, cos, sin, pos, slots, 8, 2, 128, kc.clone(), vc.clone(), bt, ctx, 16, 2)
    for s, n in enumerate(lens):
        for t in (kc, vc):
            t[int(bt[s, (n - 1) // 16]), :, (n - 1) % 16:] = math.nan
    b = K.decode_step(qkv, cos, sin, pos, slots, 8, 2, 128, kc, vc, bt, ctx, 16, 2)
    assert torch.equal(a, b) and bool(torch.isfinite(b.float()).all())


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("G,Hkv,D,bs", [(4, 2, 64, 16), (9, 2, 128, 32), (4, 2, 128, 4), (12, 2, 64, 4)])
@pytest.mark.parametrize("longest,splits", [(20, 0), (20, 2), (700, 0), (700, 1), (700, 8), (3000, 0)])
def test_not_a_number_inside_the_context(G, Hkv, D, bs, longest, splits, fp8):
    """A NaN in a query makes its head's results NaN, one in a key that is seen those of the key's group, however the keys are cut into splits and
    whichever kernel takes the shape; the other results stay as they are."""
    from litetorch_b200.ops import kernels as K
    H = G * Hkv
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(3, G, Hkv, D, bs, longest, fp8, longest + D)
    run = lambda q, k, v: K.decode_step(q, cos, sin, pos, slots, H, Hkv, D, k, v, bt, ctx, bs, splits)                       # noqa: E731
    parts = lambda q, k, v: K.paged_decode(K.rope_append(q.clone(), cos, sin, pos, slots, H, Hkv, D, k, v, bs, fp8), k, v, bt, ctx, bs,   # noqa: E731
                                           max(1, splits), D ** -0.5)
    for attend in (run, parts):
        base = attend(qkv, kc.clone(), vc.clone())
        assert bool(torch.isfinite(base.float()).all())
        q = qkv.clone()
        q[1, 2 * D + 5] = math.nan                                      # head 2 of sequence 1
        want = torch.zeros_like(base, dtype=torch.bool)
        want[1, 2] = True
        got = attend(q, kc.clone(), vc.clone())
        assert torch.equal(torch.isnan(got), want) and torch.equal(got[~want], base[~want])
        # an older key of sequence 0's second group, and the newest of sequence 2's first
        k = kc.clone()
        at = lens[0] // 2
        k[int(bt[0, at // bs]), 1, at % bs, 3] = math.nan
        q = qkv.clone()
        q[2, H * D + 7] = math.nan
        want = torch.zeros_like(base, dtype=torch.bool)
        want[0, G:] = True
        want[2, :G] = True
        got = attend(q, k, vc.clone())
        assert torch.equal(torch.isnan(got), want) and torch.equal(got[~want], base[~want])
    assert K.status_fetch() == 0


@pytest.mark.parametrize("D,bs", [(64, 16), (128, 16), (128, 4)])
@pytest.mark.parametrize("longest,splits", [(700, 0), (700, 8), (3000, 0)])
def test_scores_of_minus_infinity(D, bs, longest, splits):
    """Keys whose scores are too far below zero for 32 bits have weights of zero, chunks of nothing else included."""
    from litetorch_b200.ops import kernels as K
    G, Hkv = 4, 2
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(2, G, Hkv, D, bs, longest, False, longest + D)
    cos.fill_(1.0)
    sin.zero_()
    qkv[:, :G * Hkv * D].abs_().add_(0.5)
    n, dead = lens[0], 256
    at = torch.arange(n, device="cuda")
    cells = bt[0].long()[at // bs], at % bs
    kc[cells[0][:dead], :, cells[1][:dead]] = -3e38
    o = K.decode_step(qkv, cos, sin, pos, slots, G * Hkv, Hkv, D, kc, vc, bt, ctx, bs, splits)
    kk, vv = kc[cells[0], :, cells[1]].double(), vc[cells[0], :, cells[1]].double()
    p = torch.softmax(torch.einsum("hgd,nhd->hgn", qkv[0, :G * Hkv * D].double().view(Hkv, G, D), kk) * D ** -0.5, -1)
    assert float(p[..., :dead].abs().max()) == 0.0
    ref, size = (torch.einsum("hgn,nhd->hgd", p, v).reshape(G * Hkv, D) for v in (vv, vv.abs()))
    # roundings of the result and of the weights, each within 2^-9 of itself
    assert ((o[0].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + size * 2.0 ** -8 + 1e-4).all()
    assert K.status_fetch() == 0


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("G,Hkv,D", [(8, 4, 64), (4, 8, 128)])
def test_rows_cached_by_the_kernel_in_front(G, Hkv, D, fp8):
    """A step right behind the launch that caches the rows it attends to, and, with the cached rows complete before the step's embedding, behind that
    and a product: both start while the kernel in front of them runs."""
    from litetorch_b200.ops import kernels as K
    H, bs, n, S = G * Hkv, 16, 6000, 2
    g = torch.Generator(device="cuda").manual_seed(D)
    dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
    blocks = n // bs + 1
    kc, vc = (torch.zeros(S * blocks, Hkv, bs, D, device="cuda", dtype=torch.bfloat16).to(dt) for _ in range(2))
    bt = torch.arange(S * blocks, dtype=torch.int32, device="cuda").view(S, blocks)
    ang = torch.arange(n + 1, device="cuda", dtype=torch.float64)[:, None] * 1e4 ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)[None]
    cos, sin = ang.cos().float().contiguous(), ang.sin().float().contiguous()
    rows = torch.randn(S * n, (H + 2 * Hkv) * D, device="cuda", generator=g).bfloat16()          # the earlier tokens of both sequences
    at = torch.arange(n, dtype=torch.int32, device="cuda").repeat(S)
    cells = torch.cat([torch.arange(n, dtype=torch.int32, device="cuda") + s * blocks * bs for s in range(S)])
    pos = torch.full((S,), n, dtype=torch.int32, device="cuda")
    slots = torch.tensor([s * blocks * bs + n for s in range(S)], dtype=torch.int32, device="cuda")
    tok = torch.tensor([3, 1], dtype=torch.int32, device="cuda")
    table = torch.randn(5, 256, device="cuda", generator=g).bfloat16()
    w = torch.randn((H + 2 * Hkv) * D, 256, device="cuda", generator=g).bfloat16() / 16
    step = K.product_of_constants(K.embedding_fwd(tok, table), w)
    ctx = pos + 1
    K.rope_append(rows, cos, sin, at, cells, H, Hkv, D, kc, vc, bs, fp8)
    torch.cuda.synchronize()
    want = K.decode_step(step, cos, sin, pos, slots, H, Hkv, D, kc, vc, bt, ctx, bs)
    assert bool(want.float().abs().max() > 0)
    for _ in range(5):
        for t in (kc, vc):
            t.view(torch.uint8).zero_()
        K.rope_append(rows, cos, sin, at, cells, H, Hkv, D, kc, vc, bs, fp8)
        o = K.decode_step(step, cos, sin, pos, slots, H, Hkv, D, kc, vc, bt, ctx, bs)
        assert torch.equal(o, want)
        for t in (kc, vc):
            t.view(torch.uint8).zero_()
        K.rope_append(rows, cos, sin, at, cells, H, Hkv, D, kc, vc, bs, fp8)
        qkv = K.product_of_constants(K.embedding_fwd(tok, table), w)
        o = K.decode_step(qkv, cos, sin, pos, slots, H, Hkv, D, kc, vc, bt, ctx, bs, early=True)
        assert torch.equal(o, want)
    assert K.status_fetch() == 0


def test_early_reads_are_asked_for(monkeypatch):
    """`early` is off unless the caller says so; the served model does."""
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    from litetorch_b200.models.registry import new_serving
    from litetorch_b200.ops import kernels as K
    real, seen = K._fn, []

    def fn(name):
        return (lambda *a: seen.append(a[-2]) or real(name)(*a)) if name == "lt_paged_decode_step" else real(name)

    monkeypatch.setattr(K, "_fn", fn)
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(2, 4, 2, 64, 16, 40, False, 3)
    K.decode_step(qkv, cos, sin, pos, slots, 8, 2, 64, kc, vc, bt, ctx, 16)
    m = new_serving(LlamaEngine(LlamaConfig(vocab_size=64, n_layers=2, d_model=128, n_heads=2, n_kv_heads=1, head_dim=64, ffn=256, max_seq=64), "cuda", seed=1),
                    num_blocks=4, block_size=16, max_num_seqs=1, graphs=False)
    m.decode_logits([3], [0], [[2]])
    assert seen == [0, 1, 1]


def test_launches_are_counted():
    from litetorch_b200.ops import kernels as K
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(2, 4, 2, 64, 16, 600, False, 3)
    for splits, launches in ((0, 1), (1, 1), (4, 2)):           # splits that meet in a cluster, one, and a merge kernel
        before = K.launch_count()
        K.decode_step(qkv, cos, sin, pos, slots, 8, 2, 64, kc, vc, bt, ctx, 16, splits)
        assert K.launch_count() - before == launches


@pytest.mark.parametrize("S,longest,bs", [(1, 6000, 4), (2, 3000, 12), (40, 600, 4)])
def test_splits_of_caches_that_go_through_the_parts(S, longest, bs, monkeypatch):
    """As many as a merge kernel takes, not as a cluster holds."""
    from litetorch_b200.ops import kernels as K
    real, seen = K.paged_decode, []
    monkeypatch.setattr(K, "paged_decode", lambda *a: seen.append(a[6]) or real(*a))
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(S, 4, 2, 64, bs, longest, False, 5)
    k2, v2 = kc.clone(), vc.clone()
    o = K.decode_step(qkv, cos, sin, pos, slots, 8, 2, 64, kc, vc, bt, ctx, bs)
    many = max(1, min(32, bt.shape[1] * bs // 256, -(-4 * K.sm_count() // (2 * S))))
    assert seen == [many]
    q = K.rope_append(qkv, cos, sin, pos, slots, 8, 2, 64, k2, v2, bs, False)
    assert torch.equal(o, real(q, k2, v2, bt, ctx, bs, many, 64 ** -0.5)) and K.status_fetch() == 0


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("S,longest", [(37, 250), (38, 250), (75, 256), (75, 270)])
def test_many_short_contexts(S, longest, fp8, monkeypatch):
    """Both sides of the line beyond which queries are turned and rows cached by a launch of their own."""
    from litetorch_b200.ops import kernels as K
    seen, real = [], K._fn
    monkeypatch.setattr(K, "_fn", lambda name: seen.append(name) or real(name))
    G, Hkv, D, bs = 2, 4, 128, 16
    qkv, cos, sin, pos, slots, kc, vc, bt, ctx, lens = _case(S, G, Hkv, D, bs, longest, fp8, S)
    bt = bt[:, :(longest + bs - 1) // bs].contiguous()
    k2, v2 = kc.clone(), vc.clone()
    o = K.decode_step(qkv, cos, sin, pos, slots, G * Hkv, Hkv, D, kc, vc, bt, ctx, bs)
    apart = S * Hkv > K._decode_places(0, D, fp8, 1) and bt.shape[1] * bs <= 256
    assert ("lt_paged_decode_step" in seen) == (not apart) and apart == (longest <= 256 and S * Hkv > K.sm_count() * (2 if fp8 else 1))
    q = K.rope_append(qkv, cos, sin, pos, slots, G * Hkv, Hkv, D, k2, v2, bs, fp8)
    want = K.paged_decode(q, k2, v2, bt, ctx, bs, 1, D ** -0.5)
    bits = torch.uint8 if fp8 else torch.int16
    assert torch.equal(kc.view(bits), k2.view(bits)) and torch.equal(vc.view(bits), v2.view(bits))
    assert ((o.float() - want.float()).abs() <= want.float().abs() * 2.0 ** -7 + 2e-3).all() and K.status_fetch() == 0


def test_one_round_of_clusters():
    """Clusters are as large as they all find places at once, parts as many as fill one round."""
    from litetorch_b200.ops import kernels as K
    for D in (64, 128):
        for fp8 in (False, True):
            for pairs in (1, 4, 8, 16, 24, 32, 48, 64, 96, 128, 256):
                for keys in (256, 1024, 2048, 8192, 32768):
                    how, n = K._decode_splits(pairs, keys, D, fp8)
                    if how == "cluster" and n > 1:
                        assert pairs <= K._decode_places(0, D, fp8, n)
                        assert n >= 8 or keys // (n + 1) < 128 or pairs > K._decode_places(0, D, fp8, n + 1)
                    if how == "part" and pairs <= K._decode_places(0, D, fp8, 2):
                        assert pairs * n <= K._decode_places(0, D, fp8, 1)
