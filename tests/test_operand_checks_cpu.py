"""Operands that a kernel would read past their end, or as another type, are refused before anything is launched."""
import pytest
import torch


def _t(*shape, dtype=torch.bfloat16):
    return torch.zeros(*shape, dtype=dtype)


@pytest.mark.parametrize("x,w,residual,act", [
    (_t(2, 64), _t(16, 32), None, ""),                                    # a weight of another width
    (_t(2, 64), _t(16, 72), None, ""),
    (_t(2, 64), _t(16, 64, dtype=torch.float32), None, ""),
    (_t(2, 64), _t(16, 64), _t(2, 8), ""),
    (_t(2, 64), _t(16, 64), _t(1, 16), ""),
    (_t(2, 64), _t(16, 64), _t(2, 16, dtype=torch.float32), ""),
    (_t(2, 64), _t(16, 64), _t(16, 2).t(), ""),
    (_t(64, 2).t(), _t(16, 64), None, ""),
    (_t(2, 64), _t(64, 16).t(), None, ""),
    (_t(2, 64), _t(17, 64), None, "silu"),                                # no two halves
    (_t(2, 64), _t(16, 64), _t(2, 8), "silu"),
])
def test_product_of_constants(x, w, residual, act):
    from litetorch_b200.ops import kernels as K
    with pytest.raises(AssertionError):
        K.product_of_constants(x, w, residual=residual, act=act)


@pytest.mark.parametrize("change", [
    dict(qkv=_t(3, 4 * 64)),                                              # too few columns for the heads
    dict(qkv=_t(3, 6 * 64, dtype=torch.float32)),
    dict(qkv=_t(6 * 64, 3).t()),
    dict(positions=torch.zeros(2, dtype=torch.int32)),
    dict(slots=torch.zeros(4, dtype=torch.int32)),
    dict(cos=_t(9, 64, dtype=torch.float32)),
    dict(sin=_t(9, 32)),
    dict(fp8=True),                                                       # 16-bit caches written as bytes
    dict(k_cache=_t(5, 1, 16, 64)),
    dict(v_cache=_t(5, 8, 16, 64)[:, ::8]),
])
def test_rope_append(change):
    from litetorch_b200.ops import kernels as K
    args = dict(qkv=_t(3, 8 * 64), cos=_t(9, 32, dtype=torch.float32), sin=_t(9, 32, dtype=torch.float32), positions=torch.zeros(3, dtype=torch.int32),
                slots=torch.zeros(3, dtype=torch.int32), k_cache=_t(5, 2, 16, 64), v_cache=_t(5, 2, 16, 64), fp8=False)
    args.update(change)
    with pytest.raises(AssertionError):
        K.rope_append(heads=4, kv_heads=2, head_dim=64, block_size=16, **args)
