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
