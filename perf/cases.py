"""The work this framework is used for, as cases that can be timed and compared: training steps of Llama-shaped models
(`Trainer.step`), prompts and decode steps of served models (`registry.new_serving`: Llama and Ravenex), and a decoder block
built by a user from the differentiable operators.  Shapes are those of the repository's benchmarks and configurations, with
fewer layers where the whole model would not leave room for several copies; `draw` gives further cases of the same ranges.

Ravenex models have dense feed-forwards here: with experts, two scores that lie close may be ranked differently after a rounding
elsewhere, and whole tokens then differ between equally good implementations.

`exact` states every computation in plain torch at 64 bits.
"""
import math
import zlib

import torch
from torch.utils.checkpoint import checkpoint

F64 = torch.float64
DEV = "cuda"

# vocabulary, width, query heads, key heads, head size, feed-forward, rotary base
SHAPES = {
    "tiny": (512, 256, 4, 2, 64, 512, 1e4),
    "1.1b": (32000, 2048, 32, 4, 64, 5632, 1e4),
    "8b": (32000, 4096, 32, 8, 128, 14336, 5e5),              # the vocabulary of the serving benchmarks
    "8b-train": (128256, 4096, 32, 8, 128, 14336, 5e5),
}
LIMIT = {"train": 0.03, "prefill": 0.03, "decode": 0.03, "block": 0.028, "latent-prefill": 0.026, "latent-decode": 0.026}
BS = 16                                                      # tokens of a cache block


def listed():
    return [
        # the two-layer model of the benchmark's probe: launches and host work are all there is
        {"name": "train-tiny", "kind": "train", "model": "tiny", "layers": 2, "batch": 4, "seq": 256, "micro": 1},
        # the 1.1B configuration as benchmarked on one GPU
        {"name": "train-1.1b", "kind": "train", "model": "1.1b", "layers": 22, "batch": 4, "seq": 2048, "micro": 1},
        # the headline shape (long sequence, large vocabulary), 4 of its 32 layers
        {"name": "train-8b-layers", "kind": "train", "model": "8b-train", "layers": 4, "batch": 1, "seq": 8192, "micro": 1},
        # gradient accumulation over sequences that fill no tile
        {"name": "train-ragged", "kind": "train", "model": "1.1b", "layers": 8, "batch": 4, "seq": 1000, "micro": 2},
        # a prompt of the serving benchmark
        {"name": "prefill-1.1b", "kind": "prefill", "model": "1.1b", "layers": 22, "start": 0, "tokens": 4096},
        # a later portion of a long prompt, of an odd size
        {"name": "prefill-8b-later", "kind": "prefill", "model": "8b", "layers": 6, "start": 4100, "tokens": 1337},
        # interactive use: one sequence
        {"name": "decode-1.1b", "kind": "decode", "model": "1.1b", "layers": 22, "batch": 1, "context": 4096, "kv": "bf16"},
        # a loaded server
        {"name": "decode-8b-batch", "kind": "decode", "model": "8b", "layers": 6, "batch": 32, "context": 4096, "kv": "bf16"},
        # 8-bit cache, sequences of unequal length
        {"name": "decode-fp8-cache", "kind": "decode", "model": "8b", "layers": 6, "batch": 8, "context": 9000, "kv": "fp8"},
        # a model written on the differentiable operators: full (not causal) attention, odd length
        {"name": "block-operators", "kind": "block", "batch": 2, "seq": 1111, "width": 2048, "heads": 16, "kv_heads": 16, "dim": 128, "ff": 5632,
         "causal": False},
        # the other kind of attention that is served: keys and values made from latents
        {"name": "latent-prefill", "kind": "latent-prefill", "layers": 6, "tokens": 4096},
        {"name": "latent-decode", "kind": "latent-decode", "layers": 6, "batch": 16, "context": 4096},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["train", "train", "prefill", "prefill", "decode", "decode", "block", "latent-prefill", "latent-decode"])
    if kind == "train":
        model = rng.choice(["tiny", "1.1b", "1.1b", "8b-train"])
        seq = _log(rng, 64, {"tiny": 2048, "1.1b": 4096, "8b-train": 8192}[model])
        micro = rng.choice([1, 1, 2])
        batch = micro * _log(rng, 1, max(1, min(8, 8192 // seq // micro)))
        return {"kind": kind, "model": model, "layers": rng.randint(1, {"tiny": 2, "1.1b": 12, "8b-train": 2}[model]), "batch": batch, "seq": seq,
                "micro": micro}
    if kind == "prefill":
        return {"kind": kind, "model": rng.choice(["1.1b", "8b"]), "layers": rng.randint(2, 6), "start": rng.choice([0, 0, _log(rng, 16, 8192)]),
                "tokens": _log(rng, 16, 8192)}
    if kind == "decode":
        batch = _log(rng, 1, 64)
        return {"kind": kind, "model": rng.choice(["1.1b", "8b"]), "layers": rng.randint(2, 6), "batch": batch,
                "context": _log(rng, 32, min(16384, 131072 // batch)), "kv": rng.choice(["bf16", "bf16", "fp8"])}
    if kind == "block":
        dim = rng.choice([64, 128])
        heads = rng.choice([8, 16, 32])
        kv = heads // rng.choice([1, 2, 4, 8])
        return {"kind": kind, "batch": rng.randint(1, 4), "seq": _log(rng, 48, 2048), "width": rng.choice([1024, 2048]), "heads": heads,
                "kv_heads": kv, "dim": dim, "ff": rng.choice([2816, 5632]), "causal": rng.random() < 0.5}
    if kind == "latent-prefill":
        return {"kind": kind, "layers": rng.randint(2, 6), "tokens": _log(rng, 32, 6000)}
    batch = _log(rng, 1, 48)
    return {"kind": kind, "layers": rng.randint(2, 6), "batch": batch, "context": _log(rng, 32, min(12000, 98304 // batch))}


# ------------------------------------------------------------------------------------------------ values made from the seed
def _gen(seed, name):
    return torch.Generator(device=DEV).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)


def _normal(seed, name, shape, std=1.0):
    return torch.empty(shape, dtype=torch.float32, device=DEV).normal_(0.0, std, generator=_gen(seed, name))


def _ints(seed, name, shape, hi):
    g = torch.Generator().manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
    return torch.randint(0, hi, shape, generator=g)


def _llama_shapes(case):
    V, W, H, G, D, F, _ = SHAPES[case["model"]]
    out = [("embed", (V, W))]
    for i in range(case["layers"]):
        p = "layers.%d." % i
        out += [(p + "attn_norm", (W,)), (p + "wqkv", ((H + 2 * G) * D, W)), (p + "wo", (W, H * D)), (p + "mlp_norm", (W,)),
                (p + "w_gu", (2 * F, W)), (p + "w_down", (W, F))]
    return out + [("final_norm", (W,)), ("lm_head", (V, W))]


def _llama_tensor(case, seed, name, shape):
    """Embeddings of unit size and products back into the residual scaled by the depth, as in a model some way into its training."""
    if len(shape) == 1:
        return 1.0 + _normal(seed, name, shape, 0.1)
    return _normal(seed, name, shape, 1.0 if name == "embed" else 0.02 / math.sqrt(2 * case["layers"]) if name.endswith(("wo", "w_down")) else 0.02)


def _llama_config(case, max_seq):
    from litetorch_b200.models.llama import LlamaConfig
    V, W, H, G, D, F, base = SHAPES[case["model"]]
    return LlamaConfig(vocab_size=V, n_layers=case["layers"], d_model=W, n_heads=H, n_kv_heads=G, head_dim=D, ffn=F, rope_theta=base,
                       max_seq=max_seq, name="llama-" + case["model"])


def _load(weights, case, seed):
    weights.load_parameters(_llama_tensor(case, seed, n, s) for n, s in _llama_shapes(case))


def _contexts(case, seed):
    """Cached tokens of every sequence: between half of the case's and all of them, the first sequence all."""
    c, b = case["context"], case["batch"]
    return [c] + [c - c * int(x) // 2000 for x in _ints(seed, "contexts", (b - 1,), 1000)] if b > 1 else [c]


def _tables(case, seed, positions):
    """Block tables in an order of their own, as a server that has run for a while has them, and the size of its pool."""
    need = [(p + BS) // BS for p in positions]
    pool = len(need) * max(need)
    order = torch.randperm(pool, generator=torch.Generator().manual_seed(seed + 77)).tolist()
    tables, at = [], 0
    for n in need:
        tables.append(order[at:at + n])
        at += n
    return tables, pool


def _cache_values(seed, case, layer, what, blocks, heads, dim):
    x = _normal(seed, "cache.%d.%s" % (layer, what), (blocks, heads, BS, dim)).to(torch.bfloat16)
    return x.to(torch.float8_e4m3fn) if case.get("kv") == "fp8" else x


# latent attention: 1b-like width, heads of 128 + 64, latents of 512, every other layer reads the latents of the one before
LW, LH, LD, LR, LE, LC, LF, LV, LWIN, LSIDE = 2048, 16, 128, 64, 128, 512, 5632, 32000, 1024, 256


def _latent_config(case):
    layers = []
    for i in range(case["layers"]):
        m = {"heads": LH, "dim": LD, "rot_dim": LR, "vdim": LE, "kv_rank": LC, "mask": {"size": LWIN}, "scale": (LD + LR) ** -0.5,
             "rot": {"base": 5e5, "dims": LR}}
        if i % 2:
            m["kv_from"] = i - 1
        layers.append({"type": "latent_attention", "mixer": m, "mlp": {"kind": "dense", "ff": LF}})
    return {"architecture": "Ravenex", "vocab": LV, "width": LW, "norm": {"eps": 1e-6}, "residual_mult": 0.6, "token_side": {"dim": LSIDE},
            "layers": layers}


def _latent_shapes(case):
    n = case["layers"]
    t = {"embed": (LV, LW), "side.embed": (LV, LSIDE * n), "final.norm": (LW,), "head": (LV, LW)}
    for i in range(n):
        p = "l%d." % i
        t.update({p + k: (LW,) for k in ("norm1", "norm1b", "norm2", "norm2b", "side.norm")})
        t.update({p + "mix.q": (LH * (LD + LR), LW), p + "mix.uk": (LH * LD, LC), p + "mix.uv": (LH * LE, LC), p + "mix.o": (LW, LH * LE),
                  p + "mlp.gate": (LF, LW), p + "mlp.up": (LF, LW), p + "mlp.down": (LW, LF), p + "side.gate": (LSIDE, LW),
                  p + "side.proj": (LW, LSIDE)})
        if i % 2 == 0:
            t.update({p + "mix.dkv": (LC + LR, LW), p + "mix.dkv.norm": (LC,)})
    return t


def _latent_tensor(seed, name, shape):
    if len(shape) == 1:
        return (1.0 + _normal(seed, name, shape, 0.1)).to(torch.bfloat16)
    return _normal(seed, name, shape, 1.0 if name.endswith("embed") else shape[-1] ** -0.5).to(torch.bfloat16)


# ------------------------------------------------------------------------------------------------ state and one pass
def prepare(case, seed):
    from litetorch_b200.models import registry
    kind = case["kind"]
    if kind == "train":
        from litetorch_b200.trainer import Trainer
        tr = Trainer(_llama_config(case, case["seq"]), parallel="none", micro_batches=case["micro"])
        _load(tr.engine.w, case, seed)
        ids = _ints(seed, "tokens", (case["batch"], case["seq"] + 1), SHAPES[case["model"]][0])
        return {"kind": kind, "trainer": tr, "tokens": ids[:, :-1].contiguous().pin_memory(), "targets": ids[:, 1:].contiguous().pin_memory()}
    if kind == "block":
        B, T, W, H, G, D, F = (case[k] for k in ("batch", "seq", "width", "heads", "kv_heads", "dim", "ff"))
        leaf = lambda n, s, std, one=0.0: (one + _normal(seed, n, s, std)).to(torch.bfloat16).requires_grad_()  # noqa: E731
        ang = torch.arange(T, device=DEV, dtype=F64)[:, None] * (1e4 ** (-torch.arange(0, D, 2, device=DEV, dtype=F64) / D))[None]
        w = {"n1": leaf("n1", (W,), 0.1, 1.0), "qkv": leaf("qkv", ((H + 2 * G) * D, W), W ** -0.5), "o": leaf("o", (W, H * D), (H * D) ** -0.5),
             "n2": leaf("n2", (W,), 0.1, 1.0), "gu": leaf("gu", (2 * F, W), W ** -0.5), "down": leaf("down", (W, F), F ** -0.5)}
        return {"kind": kind, "case": dict(case), "x": leaf("x", (B, T, W), 1.0), "dy": _normal(seed, "dy", (B, T, W)).to(torch.bfloat16), "w": w,
                "cos": ang.cos().float(), "sin": ang.sin().float()}
    if kind in ("prefill", "decode"):
        from litetorch_b200.models.llama import LlamaEngine
        G, D = SHAPES[case["model"]][3:5]
        last = [case["start"] + case["tokens"] - 1] if kind == "prefill" else _contexts(case, seed)
        tables, blocks = _tables(case, seed, last)
        eng = LlamaEngine(_llama_config(case, max(last) + 1), DEV)
        _load(eng.w, case, seed)
        model = registry.new_serving(eng, num_blocks=blocks, block_size=BS, max_num_seqs=len(last),
                                     kv_dtype=torch.float8_e4m3fn if case.get("kv") == "fp8" else None)
        if kind == "decode" or case["start"]:
            for i in range(case["layers"]):
                model.cache.k[i].copy_(_cache_values(seed, case, i, "k", blocks, G, D))
                model.cache.v[i].copy_(_cache_values(seed, case, i, "v", blocks, G, D))
        V = SHAPES[case["model"]][0]
    else:
        from litetorch_b200.models.ravenex import RavenexConfig, RavenexEngine
        last = [case["tokens"] - 1] if kind == "latent-prefill" else _contexts(case, seed)
        tables, blocks = _tables(case, seed, last)
        shapes = _latent_shapes(case)
        eng = RavenexEngine(RavenexConfig.parse(_latent_config(case)), lambda n: _latent_tensor(seed, n, shapes[n]))
        model = registry.new_serving(eng, num_blocks=blocks, block_size=BS, max_num_seqs=len(last))
        if kind == "latent-decode":
            for i in range(0, case["layers"], 2):
                model.cache.k[i].copy_(_cache_values(seed, case, i, "k", blocks, 1, LC + LR))
        V = LV
    n = case["tokens"] if "tokens" in case else case["batch"]
    return {"kind": kind, "model": model, "tokens": _ints(seed, "tokens", (n,), V).tolist(), "tables": tables, "positions": last,
            "start": case.get("start", 0)}


def _cache_out(model):
    # 8-bit caches go out as whole numbers
    return [t.view(torch.uint8) if t.dtype == torch.float8_e4m3fn else t for t in model.cache.k + model.cache.v if t is not None]


def run(state):
    kind = state["kind"]
    if kind == "train":
        tr = state["trainer"]
        loss = tr.step(state["tokens"], state["targets"])
        return {"loss": loss, "gradient": tr.engine.w.flat_g, "weights": tr.engine.w.master}
    if kind == "block":
        from litetorch_b200.ops import functional as LF_
        c, w, x = state["case"], state["w"], state["x"]
        B, T, W, H, G, D = (c[k] for k in ("batch", "seq", "width", "heads", "kv_heads", "dim"))
        qkv = LF_.linear(LF_.rms_norm(x, w["n1"]), w["qkv"]).view(B, T, H + 2 * G, D)
        q, k = LF_.rope_bthd(qkv[:, :, :H], state["cos"], state["sin"]), LF_.rope_bthd(qkv[:, :, H:H + G], state["cos"], state["sin"])
        o = LF_.flash_attention_bthd(q, k, qkv[:, :, H + G:], causal=c["causal"])
        x1 = x + LF_.linear(o.reshape(B, T, H * D), w["o"])
        y = x1 + LF_.linear(LF_.swiglu(LF_.linear(LF_.rms_norm(x1, w["n2"]), w["gu"])), w["down"])
        leaves = [x] + [w[k] for k in sorted(w)]
        return {"y": y.detach(), "gradients": list(torch.autograd.grad(y, leaves, state["dy"]))}
    model = state["model"]
    if kind.endswith("prefill"):
        out = model.score_chunk(state["tokens"], state["start"], state["tables"][0], [len(state["tokens"]) - 1])
    else:
        out = model.decode_logits(state["tokens"], state["positions"], state["tables"])
    return {"logits": out, "cache": _cache_out(model)}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "block":
        B, T, W, H, G, D, F = (case[k] for k in ("batch", "seq", "width", "heads", "kv_heads", "dim", "ff"))
        mats = (H + 2 * G) * D * W + W * H * D + 3 * F * W
        pairs = T * (T + 1) / 2 if case["causal"] else T * T
        return {"bytes": 2.0 * (2 * (mats + 2 * W) + 4 * B * T * W), "flops": 6.0 * mats * B * T + 3 * 4.0 * B * H * D * pairs}
    if kind.startswith("latent"):
        n = case["layers"]
        mats = n * (LH * (LD + LR) * LW + LW * LH * LE + 3 * LF * LW + 2 * LSIDE * LW) + (n + 1) // 2 * (LC + LR) * LW
        unroll, head = n * LH * (LD + LE) * LC, LV * LW
        rows = case["tokens"] if kind == "latent-prefill" else case["batch"]
        if kind == "latent-prefill":
            pairs = sum(min(i + 1, LWIN) for i in range(rows))
            flops = 2.0 * ((mats + unroll) * rows + head) + n * 2.0 * LH * (LD + LR + LE) * pairs
            kept = rows
        else:
            seen = case["batch"] * min(0.75 * case["context"], LWIN)     # unequal lengths, about three quarters on average
            flops = 2.0 * (mats + unroll + head) * rows + n * 2.0 * LH * (2 * LC + LR) * seen
            kept = seen * 2                                              # every layer reads a cache of its own or another's
        return {"bytes": 2.0 * (mats + unroll + head) + 2.0 * kept * (n + 1) // 2 * (LC + LR) + 2.0 * rows * (LW + LSIDE * n) + 4.0 * LV, "flops": flops}
    V, W, H, G, D, F, _ = SHAPES[case["model"]]
    n = case["layers"]
    mats = n * ((H + 2 * G) * D * W + W * H * D + 3 * F * W)
    if kind == "train":
        B, T = case["batch"], case["seq"]
        params = mats + 2 * V * W + (2 * n + 1) * W
        # fp32 masters and moments read and written, 16-bit weights read and written, gradients written
        return {"bytes": 30.0 * params + 16.0 * B * T,
                "flops": 6.0 * (mats + V * W) * B * T + n * 3 * 4.0 * B * H * D * T * (T + 1) / 2}
    if kind == "prefill":
        s, t = case["start"], case["tokens"]
        return {"bytes": 2.0 * (mats + V * W + t * W) + n * 4.0 * (s + t) * G * D, "flops": 2.0 * (mats * t + V * W) + n * 4.0 * H * D * (s * t + t * (t + 1) / 2)}
    seen = case["context"] * (1 + 0.75 * (case["batch"] - 1))
    size = 1 if case["kv"] == "fp8" else 2
    return {"bytes": 2.0 * (mats + V * W) + n * 2.0 * size * seen * G * D + 4.0 * V * case["batch"],
            "flops": 2.0 * (mats + V * W) * case["batch"] + n * 4.0 * H * D * seen}


def tolerance(case):
    # 16-bit weights and activations through several layers, 32-bit sums: against 64 bits the results are 0.004 (two layers) to
    # 0.015 (22 layers, gradients) off, and two implementations may differ by a few times that.  Single values may lie a few
    # roundings of the largest off.  Whole numbers are the bytes of an 8-bit cache, of which one pass writes few.
    return {"rel": LIMIT[case["kind"]], "max": 0.9, "differ": 0.002}


# ------------------------------------------------------------------------------------------------ 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, pos, base):
    """x [T, heads, D]: the pair (2i, 2i + 1) turns by position * base^(-2i / D)."""
    D = x.shape[-1]
    a = (pos.to(F64)[:, None] * base ** (-torch.arange(0, D, 2, device=DEV, dtype=F64) / D))[:, None]
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()], -1).flatten(-2)


def _attend(q, k, v, scale, first=None, window=0):
    """q [Tq, H, D], k / v [Tk, G, .]; `first`: position of the first query among the keys (None: every key is seen).  One head
    after another, a portion of the queries at a time."""
    H, G, Tq, Tk = q.shape[1], k.shape[1], q.shape[0], k.shape[0]
    part = max(1, min(Tq, (1 << 27) // Tk))

    def rows(qh, kh, vh, at):
        s = qh @ kh.t() * scale
        if first is not None:
            gap = (torch.arange(qh.shape[0], device=DEV) + first + at)[:, None] - torch.arange(Tk, device=DEV)[None]
            s = s.masked_fill((gap < 0) | ((gap >= window) if window else False), -math.inf)
        return torch.softmax(s, -1) @ vh

    heads = []
    for h in range(H):
        g = h // (H // G)
        got = [checkpoint(rows, q[a:a + part, h], k[:, g], v[:, g], a, use_reentrant=False) if q.requires_grad else rows(q[a:a + part, h], k[:, g], v[:, g], a)
               for a in range(0, Tq, part)]
        heads.append(torch.cat(got))
    return torch.stack(heads, 1)


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(z):
    return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))


def _llama_layer(x, n1, wqkv, wo, n2, wgu, wdown, heads, attend):
    """attend(q, k, v) of the unrotated projections [rows, heads, D] -> [rows, H D]."""
    H, G, D = heads
    qkv = (_rms(x, n1, 1e-5) @ wqkv.t()).unflatten(-1, (H + 2 * G, D))
    x = x + attend(qkv[:, :H], qkv[:, H:H + G], qkv[:, H + G:]) @ wo.t()
    gate, up = (_rms(x, n2, 1e-5) @ wgu.t()).chunk(2, -1)
    return x + (_silu(gate) * up) @ wdown.t()


def _exact_train(case, seed):
    V, W, H, G, D, F, base = SHAPES[case["model"]]
    B, T = case["batch"], case["seq"]
    names = _llama_shapes(case)
    master = {n: _llama_tensor(case, seed, n, s) for n, s in names}
    w = {n: t.to(torch.bfloat16).to(F64).requires_grad_() for n, t in master.items()}
    ids = _ints(seed, "tokens", (B, T + 1), V).to(DEV)
    pos = torch.arange(T, device=DEV)

    def attend(q, k, v):
        return _attend(_turn(q, pos, base), _turn(k, pos, base), v, D ** -0.5, 0).flatten(1)

    def layer(x, *ws):
        return torch.cat([_llama_layer(x[b * T:(b + 1) * T], *ws, (H, G, D), attend) for b in range(B)])

    def loss_rows(x, norm, head, target):
        return torch.nn.functional.cross_entropy(_rms(x, norm, 1e-5) @ head.t(), target, reduction="sum")

    x = w["embed"][ids[:, :-1].reshape(-1)]
    for i in range(case["layers"]):
        ws = [w["layers.%d.%s" % (i, k)] for k in ("attn_norm", "wqkv", "wo", "mlp_norm", "w_gu", "w_down")]
        x = checkpoint(layer, x, *ws, use_reentrant=False)
    target = ids[:, 1:].reshape(-1)
    loss = sum(checkpoint(loss_rows, x[a:a + 2048], w["final_norm"], w["lm_head"], target[a:a + 2048], use_reentrant=False)
               for a in range(0, B * T, 2048)) / (B * T)
    loss.backward()
    grads, weights = [], []
    order = [n for n, s in names if len(s) == 2] + [n for n, s in names if len(s) == 1]        # matrices first, then vectors
    for n in order:
        g = w[n].grad
        decay = 0.1 if g.dim() == 2 else 0.0
        # the first AdamW step: both corrected moments are the gradient and its square
        weights.append((master.pop(n).to(F64) * (1 - 3e-4 * decay) - 3e-4 * g / (g.abs() + 1e-8)).reshape(-1))
        grads.append(g.reshape(-1))
    return {"loss": float(loss), "gradient": torch.cat(grads), "weights": torch.cat(weights)}


def _exact_block(case, seed):
    s = prepare(case, seed)
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    pos = torch.arange(case["seq"], device=DEV)
    w = {k: t.detach().to(F64).requires_grad_() for k, t in s["w"].items()}
    x = s["x"].detach().to(F64).requires_grad_()

    def attend(q, k, v):
        return _attend(_turn(q, pos, 1e4), _turn(k, pos, 1e4), v, D ** -0.5, 0 if case["causal"] else None).flatten(1)

    y = torch.stack([_llama_layer(x[b], w["n1"], w["qkv"], w["o"], w["n2"], w["gu"], w["down"], (H, G, D), attend) for b in range(case["batch"])])
    return {"y": y.detach(), "gradients": list(torch.autograd.grad(y, [x] + [w[k] for k in sorted(w)], s["dy"].to(F64)))}


def _cells(table, n):
    """(block, offset) of positions 0 .. n - 1 of a sequence."""
    p = torch.arange(n, device=DEV)
    return torch.tensor(table, device=DEV)[p // BS], p % BS


def _exact_llama_serving(case, seed):
    V, W, H, G, D, F, base = SHAPES[case["model"]]
    prefill = case["kind"] == "prefill"
    last = [case["start"] + case["tokens"] - 1] if prefill else _contexts(case, seed)
    tables, blocks = _tables(case, seed, last)
    n = case["tokens"] if prefill else case["batch"]
    tok = _ints(seed, "tokens", (n,), V).to(DEV)
    shapes = dict(_llama_shapes(case))
    get = lambda name: _llama_tensor(case, seed, name, shapes[name]).to(torch.bfloat16).to(F64)  # noqa: E731
    x, ks, vs = get("embed")[tok], [], []
    fp8 = case.get("kv") == "fp8"
    for i in range(case["layers"]):
        if prefill and not case["start"]:
            kc, vc = (torch.zeros(blocks, G, BS, D, dtype=F64, device=DEV) for _ in range(2))
        else:
            kc, vc = (_cache_values(seed, case, i, c, blocks, G, D).to(F64) for c in "kv")

        def attend(q, k, v):
            pos = torch.arange(case["start"], case["start"] + n, device=DEV) if prefill else torch.tensor(last, device=DEV)
            q, k = _turn(q, pos, base), _turn(k, pos, base)
            out = []
            for s, p in enumerate(last):
                at, off = _cells(tables[s], p + 1)
                own = slice(0, n) if prefill else slice(s, s + 1)
                first = case["start"] if prefill else p
                # what a pass caches it reads back at the cache's precision
                kc[at[first:], :, off[first:]] = k[own].to(torch.float8_e4m3fn).to(F64) if fp8 else k[own]
                vc[at[first:], :, off[first:]] = v[own].to(torch.float8_e4m3fn).to(F64) if fp8 else v[own]
                out.append(_attend(q[own], kc[at, :, off], vc[at, :, off], D ** -0.5, first))
            return torch.cat(out).flatten(1)

        x = _llama_layer(x, *(get("layers.%d.%s" % (i, k)) for k in ("attn_norm", "wqkv", "wo", "mlp_norm", "w_gu", "w_down")), (H, G, D), attend)
        ks.append(None if fp8 else kc)
        vs.append(None if fp8 else vc)
    x = x[-1:] if prefill else x
    return {"logits": _rms(x, get("final_norm"), 1e-5) @ get("lm_head").t(), "cache": ks + vs}


def _exact_latent(case, seed):
    prefill = case["kind"] == "latent-prefill"
    last = [case["tokens"] - 1] if prefill else _contexts(case, seed)
    tables, blocks = _tables(case, seed, last)
    n = case["tokens"] if prefill else case["batch"]
    tok = _ints(seed, "tokens", (n,), LV).to(DEV)
    pos = torch.arange(n, device=DEV) if prefill else torch.tensor(last, device=DEV)
    shapes = _latent_shapes(case)
    get = lambda name: _latent_tensor(seed, name, shapes[name]).to(F64)  # noqa: E731
    eps, mult = 1e-6, 0.6
    x, side, caches = get("embed")[tok], get("side.embed")[tok], []
    for i in range(case["layers"]):
        p = "l%d." % i
        h = _rms(x, get(p + "norm1"), eps)
        if i % 2 == 0:
            y = h @ get(p + "mix.dkv").t()
            row = torch.cat([_rms(y[:, :LC], get(p + "mix.dkv.norm"), eps), _turn(y[:, None, LC:], pos, 5e5)[:, 0]], 1)
            kc = torch.zeros(blocks, 1, BS, LC + LR, dtype=F64, device=DEV) if prefill else _cache_values(seed, case, i, "k", blocks, 1, LC + LR).to(F64)
            for s, q_at in enumerate(last):
                at, off = _cells(tables[s], q_at + 1)
                own = slice(0, n) if prefill else slice(s, s + 1)
                kc[at[0 if prefill else q_at:], 0, off[0 if prefill else q_at:]] = row[own]
            caches.append(kc)
        kc = caches[-1]
        q = (h @ get(p + "mix.q").t()).view(n, LH, LD + LR)
        q = torch.cat([q[..., :LD], _turn(q[..., LD:], pos, 5e5)], -1)
        uk, uv, out = get(p + "mix.uk"), get(p + "mix.uv"), []
        for s, q_at in enumerate(last):
            lo = 0 if prefill else max(0, q_at + 1 - LWIN)
            at, off = _cells(tables[s], q_at + 1)
            seen = kc[at[lo:], 0, off[lo:]]
            c, rot = seen[:, :LC], seen[:, LC:]
            k = torch.cat([(c @ uk.t()).view(-1, LH, LD), rot[:, None].expand(-1, LH, -1)], -1)
            own = slice(0, n) if prefill else slice(s, s + 1)
            out.append(_attend(q[own], k, (c @ uv.t()).view(-1, LH, LE), (LD + LR) ** -0.5, 0 if prefill else q_at - lo, LWIN))
        x = x + mult * _rms(torch.cat(out).flatten(1) @ get(p + "mix.o").t(), get(p + "norm1b"), eps)
        h = _rms(x, get(p + "norm2"), eps)
        y = (_gelu(h @ get(p + "mlp.gate").t()) * (h @ get(p + "mlp.up").t())) @ get(p + "mlp.down").t()
        x = x + mult * _rms(y, get(p + "norm2b"), eps)
        y = (_gelu(x @ get(p + "side.gate").t()) * side[:, i * LSIDE:(i + 1) * LSIDE]) @ get(p + "side.proj").t()
        x = x + mult * _rms(y, get(p + "side.norm"), eps)
    x = x[-1:] if prefill else x
    return {"logits": _rms(x, get("final.norm"), eps) @ get("head").t(), "cache": caches}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "block":
        return _exact_block(case, seed)
    with torch.no_grad():
        return _exact_llama_serving(case, seed) if kind in ("prefill", "decode") else _exact_latent(case, seed)
