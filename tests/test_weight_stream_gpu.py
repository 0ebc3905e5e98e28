"""Products of a few rows with a weight matrix, over sizes at the edges of tiles, stages and row blocks, against 64-bit arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def bound(ref, mag, K):
    """Rounding to bf16 (2^-8 of the result), and of every 32-bit addition, which a tensor core may cut off (2^-23 of the sum of sizes each)."""
    return 2.0 ** -8 * ref.abs() + (K + 16) * 2.0 ** -23 * mag + 1e-30


@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (1, 17, 2056), (2, 2367, 64), (3, 2369, 72), (8, 4737, 136), (8, 9473, 520), (7, 31, 14336), (8, 20001, 64)])
def test_gemv_rows(M, N, K):
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(N + K)
    x, w, r = (torch.randn(*s, device="cuda").bfloat16() for s in ((M, K), (N, K), (M, N)))
    for res in (None, r):
        y = KK.gemm(x, w, residual=res)
        ref = x.double() @ w.double().t() + (0 if res is None else res.double())
        mag = x.double().abs() @ w.double().abs().t() + (0 if res is None else res.double().abs())
        assert ((y.double() - ref).abs() <= bound(ref, mag, K)).all()
    assert torch.equal(KK.gemm(x, w, residual=r), y)
    assert KK.status_fetch() == 0


@pytest.mark.parametrize("M", [9, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("N,K", [(8, 32), (2368, 96), (2376, 64), (4736, 544), (4744, 2048), (9480, 128), (28672, 64)])
def test_skinny_rows(M, N, K):
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(M + N + K)
    x, w, r = (torch.randn(*s, device="cuda").bfloat16() for s in ((M, K), (N, K), (M, N)))
    y = KK.gemm(x, w, residual=r)
    ref = x.double() @ w.double().t() + r.double()
    assert ((y.double() - ref).abs() <= bound(ref, x.double().abs() @ w.double().abs().t() + r.double().abs(), K)).all()
    assert KK.status_fetch() == 0


@pytest.mark.parametrize("act", ["gelu", "silu"])
@pytest.mark.parametrize("M,F,K", [(1, 8, 32), (8, 1184, 64), (9, 1192, 96), (16, 2376, 64), (17, 520, 544), (32, 5632, 64), (64, 1000, 96)])
def test_gated(M, F, K, act):
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(M + F)
    x, gu = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(2 * F, K, device="cuda") * K ** -0.5).bfloat16()
    down = torch.eye(F, device="cuda").bfloat16()                     # hands the gated values through
    y = KK.glu_mlp(x, gu, down, act)
    g, u = (x.double() @ gu.double().t()).chunk(2, -1)
    a = torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")
    mag = (x.double().abs() @ gu.double().abs().t())
    slack = (K + 16) * 2.0 ** -23 * 1.2 * (mag[:, :F] * u.abs() + mag[:, F:] * a.abs())      # both factors' sums; the slopes of the activations are below 1.2
    assert ((y.double() - a * u).abs() <= 2.0 ** -7 * (a * u).abs() + slack + 1e-5 * u.abs()).all()
    assert KK.status_fetch() == 0


def test_rows_that_overlap():
    """Expanded and sliding views take the general kernels."""
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(0)
    base = torch.randn(4096, device="cuda").bfloat16()
    x = base[:256].expand(4, 256)                                     # pitch 0
    w = base.as_strided((64, 256), (8, 1))                            # pitch below the row's length
    plain = torch.randn(64, 256, device="cuda").bfloat16()
    for a, b in ((x, plain), (plain[:4], w), (x, w)):
        ref = a.double() @ b.double().t()
        assert ((KK.gemm(a, b).double() - ref).abs() <= bound(ref, a.double().abs() @ b.double().abs().t(), 256)).all()


@pytest.mark.parametrize("M", [1, 17, 64])
def test_products_that_start_early(M):
    """A chain of products behind norms and each other, recorded and replayed: the same as one after another, also when x has just been
    overwritten."""
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(M)
    W, F = 1024, 2816
    x = torch.randn(M, W, device="cuda").bfloat16()
    n = torch.ones(W, device="cuda").bfloat16()
    ws = [tuple((torch.randn(*s, device="cuda") * s[1] ** -0.5).bfloat16() for s in ((W, W), (2 * F, W), (W, F))) for _ in range(4)]

    def chain(x, product, gated):
        for a, gu, down in ws:
            x = product(KK.norm_fwd(x, n, eps=1e-5)[0], a, x)
            x = product(gated(KK.norm_fwd(x, n, eps=1e-5)[0], gu), down, x)
        return x

    early = lambda x: chain(x, lambda h, w, r: KK.product_of_constants(h, w, residual=r), lambda h, w: KK.product_of_constants(h, w, act="silu"))  # noqa: E731
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        early(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = early(x)
    for seed in range(5):
        x.copy_(torch.randn(M, W, generator=torch.Generator().manual_seed(seed)).bfloat16())
        graph.replay()
        ref = chain(x.clone(), lambda h, w, r: KK.gemm(h, w, residual=r), lambda h, w: KK.glu_rows(h, w, "silu"))
        assert torch.equal(out, ref)
    assert KK.status_fetch() == 0


@pytest.mark.parametrize("M,N,K", [(1, 4096, 14336), (8, 1024, 14336), (3, 2048, 5632), (8, 28672, 4096)])
def test_few_rows_add_in_32_bits(M, N, K):
    """Sums of one sign: what every addition cuts off would add up."""
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(N + K)
    x, w = torch.randn(M, K, device="cuda").abs().bfloat16(), (torch.randn(N, K, device="cuda").abs() * K ** -0.5).bfloat16()
    y = KK.gemm(x, w)
    ref = x.double() @ w.double().t()
    ulp = torch.exp2(torch.floor(torch.log2(ref)) - 7)
    # beyond half a unit of the 16-bit result by as much as the 32-bit sum was off.  A stage's four instructions cut off up to 2^-23 of its
    # part each (2^-23 of the whole, at most, as parts add up); then come K / 512 + 8 rounded additions, 2^-24 each at most, in either
    # direction: three standard deviations (2^-24 / sqrt 3 each) of them
    slack = 4 * 2.0 ** -23 + 3 * (K / 512 + 8) ** 0.5 * 2.0 ** -24 / 3 ** 0.5
    assert (((y.double() - ref).abs() - 0.5 * ulp) / ref).max() <= slack


@pytest.mark.parametrize("M", [1, 8, 20, 64, 100, 200])
def test_silu_of_far_negative_gates(M):
    """Gates between -88.8 and -87.3, where the sigmoid's divisor passes 2^126."""
    from litetorch_b200.ops import kernels as KK
    K, F = 64, 256
    x = torch.zeros(M, K, device="cuda").bfloat16()
    x[:, 0], x[:, 1] = 1.0, 2.0 ** 100
    gu = torch.zeros(2 * F, K, device="cuda").bfloat16()
    gu[:F, 0] = torch.linspace(-88.5, -86.0, F, device="cuda").bfloat16()
    gu[F:, 1] = 1.0
    y = KK.glu_rows(x, gu, "silu").double()
    ref = torch.nn.functional.silu(gu[:F, 0].double())[None].expand(M, F) * 2.0 ** 100
    # __expf of 88 is off by 88 2^-23 (its argument is multiplied by log2 e in 32 bits) and a little; the result is rounded to bf16
    assert ((y - ref).abs() <= (2.0 ** -8 + 88 * 2.0 ** -22) * ref.abs()).all()


@pytest.mark.parametrize("M", [65, 79, 81, 113, 127, 128])
@pytest.mark.parametrize("N,K", [(8, 8192), (40, 16416), (2056, 8224), (2048, 544), (1000, 14336)])
def test_split_of_k_beyond_64_rows(M, N, K):
    """K over several CTAs of a column group, as it is by default and as far as it goes; plain and gated."""
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(M + N + K)
    x, w, r = (torch.randn(*s, device="cuda").bfloat16() for s in ((M, K), (N, K), (M, N)))
    ref = x.double() @ w.double().t()
    mag = x.double().abs() @ w.double().abs().t()
    gated = torch.nn.functional.silu(ref[:, :N // 2]) * ref[:, N // 2:]
    room = (K + 16) * 2.0 ** -23 * 1.2 * (mag[:, :N // 2] * ref[:, N // 2:].abs() + mag[:, N // 2:] * ref[:, :N // 2].abs())    # as in test_gated
    for target in ((1, 16), (8, 1)):
        KK.gemm_skinny_set_target(*target)
        try:
            y, again, g = KK.gemm(x, w, residual=r), KK.gemm(x, w, residual=r), KK.glu_rows(x, w, "silu")
        finally:
            KK.gemm_skinny_set_target()
        assert torch.equal(y, again)
        assert ((y.double() - ref - r.double()).abs() <= bound(ref + r.double(), mag + r.double().abs(), K)).all()
        assert ((g.double() - gated).abs() <= 2.0 ** -7 * gated.abs() + room + 1e-5 * ref[:, N // 2:].abs()).all()
    assert KK.status_fetch() == 0


@pytest.mark.parametrize("M", [9, 17, 64, 65])
def test_more_rows_that_overlap(M):
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(M)
    base = torch.randn(4096, device="cuda").bfloat16()
    x, w = base.as_strided((M, 256), (8, 1)), (torch.randn(48, 256, device="cuda") / 16).bfloat16()
    ref, mag = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert ((KK.gemm(x, w).double() - ref).abs() <= bound(ref, mag, 256)).all()
    v = base.as_strided((48, 256), (8, 1))
    rv, mv = w[:1].expand(M, 256).double() @ v.double().t(), w[:1].expand(M, 256).double().abs() @ v.double().abs().t()
    assert ((KK.gemm(w[:1].expand(M, 256), v).double() - rv).abs() <= bound(rv, mv, 256)).all()
    a, u = ref.chunk(2, -1)
    want = torch.nn.functional.silu(a) * u
    assert ((KK.glu_rows(x, w, "silu").double() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-3).all()
    assert KK.status_fetch() == 0


@pytest.mark.parametrize("act", ["gelu", "silu"])
@pytest.mark.parametrize("M,F,K", [(129, 1000, 2048), (1025, 1000, 4096), (1337, 14336, 4096), (2050, 2824, 1024)])
def test_gated_prompts(M, F, K, act):
    from litetorch_b200.ops import kernels as KK
    torch.manual_seed(M + F)
    x, gu = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(2 * F, K, device="cuda") * K ** -0.5).bfloat16()
    g, u = (x.double() @ gu.double().t()).chunk(2, -1)
    want = (torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * u
    # rounded to bf16; sums of K products of size 1 / sqrt(K) in 32 bits, cut off
    assert ((KK.glu_rows(x, gu, act).double() - want).abs() <= 2.0 ** -8 * want.abs() + K * 2.0 ** -23 * 2 * (1 + u.abs() + g.abs())).all()
    assert KK.status_fetch() == 0
