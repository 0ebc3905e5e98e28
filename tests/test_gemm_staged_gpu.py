"""Products whose bf16 results leave through shared memory and TMA, on CTA pairs and one CTA a tile, at edges of tiles and with K cut for few tiles, in every
operand layout, with a residual, into a sum, and with rows of C apart, against 64 bits; gates in the epilogue likewise."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, Kd, am, bm):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + Kd)
    a = torch.randn((M, Kd) if am == 0 else (Kd, M), device="cuda", generator=g).bfloat16()
    b = torch.randn((N, Kd) if bm == 0 else (Kd, N), device="cuda", generator=g).bfloat16()
    want = (a.double() if am == 0 else a.double().t()) @ (b.double().t() if bm == 0 else b.double())
    return a, b, want, torch.randn(M, N, device="cuda", generator=g).bfloat16()


def _close(got, want, Kd):
    # one rounding to bf16 (2^-9 of the result) and 32-bit sums of Kd products of unit size
    assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + Kd * 2.0 ** -22).all()


@pytest.mark.parametrize("M,N,Kd", [(136, 8, 64), (256, 256, 64), (264, 264, 72), (520, 2056, 2048), (2000, 2560, 520), (144, 2048, 11264), (1336, 4096, 4096),
                                    (4096, 2048, 256)])
@pytest.mark.parametrize("am,bm", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_layouts_and_additions(M, N, Kd, am, bm):
    from litetorch_b200.ops import kernels as K
    a, b, want, res = _operands(M, N, Kd, am, bm)
    _close(K.gemm(a, b, a_major=am, b_major=bm), want, Kd)
    _close(K.gemm(a, b, a_major=am, b_major=bm, residual=res, alpha=0.5), 0.5 * want + res.double(), Kd)
    wide = torch.full((M, N + 24), 7.0, device="cuda", dtype=torch.bfloat16)
    c = wide[:, 8:N + 8]
    c.copy_(res)
    first = K.gemm(a, b, a_major=am, b_major=bm, out=c, accumulate=True).clone()
    _close(first, want + res.double(), Kd)
    assert (wide[:, :8] == 7).all() and (wide[:, N + 8:] == 7).all()
    c.copy_(res)
    assert torch.equal(K.gemm(a, b, a_major=am, b_major=bm, out=c, accumulate=True), first)      # the same sums in the same order
    assert K.status_fetch() == 0


@pytest.mark.parametrize("M,F,Kd", [(129, 8, 64), (256, 128, 64), (257, 136, 2048), (1337, 1000, 520), (600, 5632, 2048)])
@pytest.mark.parametrize("act", ["gelu", "silu"])
def test_gates(M, F, Kd, act):
    from litetorch_b200.ops import kernels as K
    a, b, want, _ = _operands(M, 2 * F, Kd, 0, 0)
    b = b * (2 * Kd ** -0.5)
    want = a.double() @ b.double().t()
    f = torch.nn.functional.silu if act == "silu" else lambda z: torch.nn.functional.gelu(z, approximate="tanh")
    ref = f(want[:, :F]) * want[:, F:]
    # a rounding of the result and approximations of the exponential (about 2^-20) and 32-bit sums before it
    assert ((K.glu_rows(a, b, act).double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 2e-4).all()
    assert K.status_fetch() == 0
