"""Products of a few rows that are normalised on the way, and those with 32-bit results, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("N,Kd", [(2, 8), (100, 72), (2048, 2048), (2560, 2048), (18, 4096), (9472, 264), (33, 8192)])
@pytest.mark.parametrize("act", ["", "silu"])
def test_normalised_products(M, N, Kd, act):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + N + Kd)
    x = (torch.randn(M, Kd + 8, device="cuda", generator=g) * torch.logspace(-3, 3, M, device="cuda")[:, None]).bfloat16()[:, :Kd]
    gain = (1 + 0.1 * torch.randn(Kd, device="cuda", generator=g)).bfloat16()
    w = (torch.randn((2 if act else 1) * N, Kd, device="cuda", generator=g) * Kd ** -0.5).bfloat16()
    res = None if act else torch.randn(M, N, device="cuda", generator=g).bfloat16()
    y = K.product_of_constants(x, w, res, act, norm=(gain, 1e-5))
    x64 = x.double()
    xh = x64 * torch.rsqrt((x64 ** 2).mean(-1, keepdim=True) + 1e-5) * gain.double()
    z, size = xh @ w.double().t(), xh.abs() @ w.double().abs().t()      # a factor is rounded to bf16 (2^-9), as is the result; sums are of 32 bits
    if act:
        # |d silu(a) b| <= 1.1 |b| da + |silu(a)| db
        a, b, da, db = z[:, :N], z[:, N:], size[:, :N] * 2.0 ** -8, size[:, N:] * 2.0 ** -8
        want, bound = torch.nn.functional.silu(a) * b, 1.1 * b.abs() * da + a.abs() * db + da * db
    else:
        want, bound = z + res.double(), size * 2.0 ** -8
    assert ((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + bound + 1e-5).all()
    assert float((y.double() - want).norm() / want.norm()) < 6e-3
    # what it stands in for, whose normalised rows are rounded alike
    h = K.norm_fwd(x.contiguous(), gain, eps=1e-5)[0]
    z = K.product_of_constants(h, w, res, act)
    assert float((y.double() - z.double()).norm() / want.norm()) < 6e-3
    assert K.status_fetch() == 0


def test_more_rows_or_columns_are_normalised_first():
    from litetorch_b200.ops import kernels as K
    for M, Kd in ((17, 256), (200, 256), (2, 8200)):
        x = torch.randn(M, Kd, device="cuda").bfloat16()
        gain, w = (1 + 0.1 * torch.randn(Kd, device="cuda")).bfloat16(), (torch.randn(64, Kd, device="cuda") * Kd ** -0.5).bfloat16()
        assert torch.equal(K.product_of_constants(x, w, norm=(gain, 1e-6)), K.product_of_constants(K.norm_fwd(x, gain, eps=1e-6)[0], w))


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,Kd", [(3, 8), (32000, 2048), (1001, 264)])
def test_32_bit_results(M, N, Kd):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + N + Kd)
    x = torch.randn(M, Kd, device="cuda", generator=g).bfloat16()
    w = torch.randn(N, Kd, device="cuda", generator=g).bfloat16()
    y = K.linear(x, w, out_dtype=torch.float32)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert y.dtype == torch.float32 and ((y.double() - want).abs() <= size * 2.0 ** -20).all()
    assert K.status_fetch() == 0


@pytest.mark.parametrize("M,N,Kd", [(1, 1, 8), (1, 1000, 72), (7, 129, 1024), (17, 96, 200), (64, 257, 512), (65, 96, 512)])
@pytest.mark.parametrize("strided", [False, True])
def test_products_with_constant_matrices(M, N, Kd, strided):
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, Kd + (24 if strided else 0), device="cuda", generator=g).bfloat16()[:, :Kd]
    w = (torch.randn(2 * N, Kd, device="cuda", generator=g) * Kd ** -0.5).bfloat16()
    want = x.double() @ w.double().t()
    # 32-bit sums of exact products, one rounding to bf16
    slack = (x.double().abs() @ w.double().abs().t()) * (Kd * 2.0 ** -24)
    for dtype, unit in ((torch.bfloat16, 2.0 ** -8), (torch.float32, 2.0 ** -23)):
        got = K.linear(x, w, out_dtype=dtype, constant=True).double()
        assert ((got - want).abs() <= want.abs() * unit + slack).all()
    gate, up = want[:, :N], want[:, N:]
    for act, f in (("silu", torch.nn.functional.silu), ("gelu", lambda v: torch.nn.functional.gelu(v, approximate="tanh"))):
        got = K.glu_rows(x, w, act, constant=True).double()
        # 1.13: the steepest that either gate is; more than 64 rows round gate and up to bf16 first
        e = (2.0 ** -8 if M > 64 else 0) + 2.0 ** -18
        assert ((got - f(gate) * up).abs() <= (f(gate) * up).abs() * 2.0 ** -8 + 1.13 * (gate.abs() * up.abs() * 2 * e + slack[:, :N] * up.abs() + slack[:, N:] * gate.abs()) + 1e-6).all()
    assert K.status_fetch() == 0


@pytest.mark.parametrize("M,Kd", [(8, 512), (9, 512), (16, 2048), (1, 7808), (8, 7816), (1, 8192), (9, 8192)])
@pytest.mark.parametrize("N,act", [(7104, "silu"), (7112, "silu"), (40000, ""), (40002, "")])
def test_norm_on_the_way_or_in_front(M, Kd, N, act):
    """Both sides of the lines between them, against 64 bits."""
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + Kd + N)
    x = torch.randn(M, Kd, device="cuda", generator=g).bfloat16()
    gain = (1 + 0.1 * torch.randn(Kd, device="cuda", generator=g)).bfloat16()
    w = torch.empty((2 if act else 1) * N, Kd, device="cuda").normal_(0.0, Kd ** -0.5, generator=g).bfloat16()
    y = K.product_of_constants(x, w, None, act, norm=(gain, 1e-5))
    x64 = x.double()
    z = (x64 * torch.rsqrt((x64 ** 2).mean(-1, keepdim=True) + 1e-5) * gain.double()) @ w.double().t()
    want = torch.nn.functional.silu(z[:, :N]) * z[:, N:] if act else z
    assert float((y.double() - want).norm() / want.norm()) < 6e-3            # factors and result rounded to bf16, as above
    first = K.product_of_constants(K.norm_fwd(x, gain, eps=1e-5)[0], w, None, act)
    assert float((first.double() - want).norm() / want.norm()) < 6e-3
    if not K._norm_on_the_way(M, N, Kd, bool(act)):
        assert torch.equal(y, first)
    assert K.status_fetch() == 0


@pytest.mark.parametrize("M,N,Kd,act", [(3, 40, 256, ""), (17, 40, 256, ""), (200, 512, 256, "silu"), (9, 7112, 512, "silu"), (2, 40, 8200, "")])
def test_rows_with_a_pitch(M, N, Kd, act):
    """Rows out of a wider matrix give what dense ones give."""
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, Kd + 24, device="cuda", generator=g).bfloat16()[:, 8:Kd + 8]
    gain, w = torch.ones(Kd, device="cuda").bfloat16(), torch.randn((2 if act else 1) * N, Kd, device="cuda", generator=g).bfloat16()
    assert torch.equal(K.product_of_constants(x, w, None, act, norm=(gain, 1e-6)), K.product_of_constants(x.contiguous(), w, None, act, norm=(gain, 1e-6)))
    assert K.status_fetch() == 0
