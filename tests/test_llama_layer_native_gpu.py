"""A layer of a training step as one native call: the same launches, and so the same bits, as the schedule step by step."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,hd,heads,kv", [(1, 129, 64, 4, 2), (3, 100, 64, 4, 4), (2, 256, 128, 2, 1)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_layer_against_its_steps(B, T, hd, heads, kv, accumulate):
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    from litetorch_b200.ops import kernels as K
    cfg = LlamaConfig(vocab_size=64, n_layers=2, d_model=256, n_heads=heads, n_kv_heads=kv, head_dim=hd, ffn=264, max_seq=512)
    eng = LlamaEngine(cfg, "cuda", seed=3)
    g = torch.Generator(device="cuda").manual_seed(T)
    x, dx2 = (torch.randn(B * T, 256, device="cuda", generator=g).bfloat16() for _ in range(2))
    got = {}
    for way in ("native", "steps"):
        eng.w.flat_g.fill_(0.5)
        fwd, bwd = (eng._layer_fwd, eng._layer_bwd) if way == "native" else (eng._layer_fwd_steps, eng._layer_bwd_steps)
        n = K.launch_count()
        x2, ctx = fwd(1, x, B, T)
        dx = bwd(1, dx2, ctx, B, T, accumulate)
        got[way] = (x2, dx, eng.w.flat_g.clone(), K.launch_count() - n, len(ctx))
    assert got["native"][4] == 2 and got["steps"][4] > 2 and got["native"][3] == got["steps"][3]
    assert torch.equal(got["native"][0], got["steps"][0])
    # dQ is summed in any order
    for a, b in zip(got["native"][1:3], got["steps"][1:3]):
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 2e-3
    K.check_status()


def test_few_rows_take_the_steps():
    from litetorch_b200.models.llama import LlamaConfig, LlamaEngine
    cfg = LlamaConfig(vocab_size=64, n_layers=1, d_model=128, n_heads=2, n_kv_heads=1, head_dim=64, ffn=128, max_seq=128)
    eng = LlamaEngine(cfg, "cuda", seed=3)
    assert eng._native_layer(0, 1, 128) is None and eng._native_layer(0, 2, 65) is not None and eng._native_layer(0, 1, 129) is None
