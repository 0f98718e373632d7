"""The work the framework is timed and compared on: single layers and blocks through their module calls, and one whole decode step.

Every case is a plain dict (``kind`` names the module) of sizes that the configurations, tests and benchmark of this repository use, or
generic ones.  ``prepare`` builds what a program has in hand before the call -- quantized modules, caches, states, inputs on the GPU --
and ``run`` makes the call.  ``exact`` recomputes the same outputs in 64 bits with plain torch, without the package.
"""
from __future__ import annotations

import math
from typing import Any, Dict, List, Optional, Tuple

import torch
import torch.nn.functional as F

F64 = torch.float64
DEV = "cuda"

# (width, heads, key-value groups, feed-forward) of the decoder shapes in lit_gpt_b200/config.py that the benchmark runs
SHAPES = {
    "7b": (4096, 32, 32, 11008),      # Llama-2-7b-hf
    "13b": (5120, 40, 40, 13824),     # Llama-2-13b-hf
    "7b-gqa": (4096, 32, 8, 14336),   # Mistral-7B
}


def listed() -> List[Dict[str, Any]]:
    return [
        # one token of batch-1 decoding through one quantized projection (the fused q/k/v projection of the 7B shape)
        dict(name="linear-nf4-1", kind="linear", mode="nf4", rows=1, n_in=4096, n_out=12288, bias=False),
        # batched decoding: sixteen sequences through the 13B feed-forward
        dict(name="mlp-int4-16", kind="mlp", mode="int4", rows=16, shape="13b"),
        # an ordinary chat prompt (ragged length) through a feed-forward
        dict(name="mlp-nf4-203", kind="mlp", mode="nf4", rows=203, shape="7b"),
        # a long prompt through a feed-forward: the largest dense work of a prefill
        dict(name="mlp-int4-4096", kind="mlp", mode="int4", rows=4096, shape="7b-gqa"),
        # LLM.int8(): a prompt with outlier columns through one projection, fp16
        dict(name="linear-int8-777", kind="linear", mode="int8", rows=777, n_in=4096, n_out=11008, bias=True),
        # one decode step of eight sequences over a long context, grouped-query attention layer
        dict(name="attn-decode-8x3000", kind="attention", mode="int4", shape="7b-gqa", batch=8, start=3000, rows=1),
        # a long prompt through a grouped-query attention layer
        dict(name="attn-prompt-4096", kind="attention", mode="int4", shape="7b-gqa", batch=1, start=0, rows=4096),
        # a later portion of a prompt over cached positions, one key-value head per query head
        dict(name="attn-portion-613", kind="attention", mode="nf4", shape="7b", batch=1, start=1500, rows=613),
        # two prompts packed into one step of a sliding-window layer (convolution, rotation, sink, grouped heads)
        dict(name="window-prompt-2048", kind="window", dtype="bf16", rows=2048, seqs=2, width=2048, heads=16, kv_heads=4, dim=128, window=1024),
        # a prompt through a gated delta rule with one decay per head and key channel
        dict(name="delta-channel-2048", kind="delta", dtype="bf16", rows=2048, seqs=1, width=2048, heads=16, kv_heads=16, dim=128, channel=True),
        # a prompt through decaying linear attention with one decay per head and key channel
        dict(name="linear-channel-2048", kind="decay", dtype="bf16", rows=2048, seqs=1, width=2048, heads=8, dim=128, channel=True),
        # a whole decode step of a shortened 7B model, captured as a serving loop captures it; returns the logits
        dict(name="step-nf4-300", kind="step", mode="nf4", shape="7b", layers=4, batch=1, start=300, vocab=32000),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> Dict[str, Any]:
    kind = rng.choice(["linear", "linear", "mlp", "mlp", "attention", "attention", "window", "delta", "decay", "step"])
    if kind == "linear":
        mode = rng.choice(["nf4", "int4", "int8"])
        n_in, n_out = rng.choice([(4096, 12288), (4096, 4096), (11008, 4096), (5120, 15360), (4096, 6144), (2048, 5632), (2560, 7680)])
        return dict(kind=kind, mode=mode, rows=_log(rng, 1, 1024 if mode == "int8" else 4096), n_in=n_in, n_out=n_out, bias=rng.random() < 0.3)
    if kind == "mlp":
        return dict(kind=kind, mode=rng.choice(["nf4", "int4"]), rows=_log(rng, 1, 3000), shape=rng.choice(list(SHAPES)))
    if kind == "attention":
        shape, mode = rng.choice(list(SHAPES)), rng.choice(["nf4", "int4"])
        if rng.random() < 0.3:
            return dict(kind=kind, mode=mode, shape=shape, batch=rng.choice([1, 2, 5, 8]), start=_log(rng, 16, 4000), rows=1)
        rows = _log(rng, 2, 3600)
        return dict(kind=kind, mode=mode, shape=shape, batch=rng.choice([1, 1, 2]) if rows < 1500 else 1,
                    start=rng.choice([0, 0, rng.randrange(1, 2500)]) if rows < 3000 else 0, rows=rows)
    heads = rng.choice([4, 8, 16])
    rows, seqs = _log(rng, 64, 2048), rng.choice([1, 1, 2, 3])
    dtype = rng.choice(["bf16", "bf16", "fp32"])
    dim = rng.choice([64, 128])
    if kind == "window":
        return dict(kind=kind, dtype=dtype if rows < 1000 else "bf16", rows=rows, seqs=seqs, width=1024, heads=heads, kv_heads=heads // rng.choice([1, 2, 4]), dim=dim,
                    window=rng.choice([256, 500, 1024]))
    if kind == "delta":
        return dict(kind=kind, dtype=dtype, rows=rows, seqs=seqs, width=1024, heads=heads, kv_heads=heads // rng.choice([1, 2]), dim=dim,
                    channel=rng.random() < 0.5)
    if kind == "decay":
        return dict(kind=kind, dtype=dtype, rows=rows, seqs=seqs, width=1024, heads=heads, dim=dim, channel=rng.random() < 0.5)
    return dict(kind=kind, mode=rng.choice(["nf4", "int4"]), shape=rng.choice(["7b", "7b-gqa"]), layers=rng.choice([2, 4]), batch=rng.choice([1, 1, 3, 16]),
                start=_log(rng, 8, 2000), vocab=32000)


# ---- inputs ------------------------------------------------------------------------------------------------------------------------
class _Maker:
    """Tensors from a seed, in the order they are asked for."""

    def __init__(self, seed: int) -> None:
        self.gen = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape: int, std: float = 1.0, dtype: torch.dtype = torch.bfloat16) -> torch.Tensor:
        return torch.empty(shape, device=DEV, dtype=torch.float32).normal_(0.0, std, generator=self.gen).to(dtype)

    def uniform(self, lo: float, hi: float, *shape: int, dtype: torch.dtype = torch.bfloat16) -> torch.Tensor:
        return torch.empty(shape, device=DEV, dtype=torch.float32).uniform_(lo, hi, generator=self.gen).to(dtype)

    def integers(self, n: int, *shape: int) -> torch.Tensor:
        return torch.randint(0, n, shape, device=DEV, generator=self.gen)


def _dtype(case: Dict[str, Any]) -> torch.dtype:
    return torch.float32 if case["dtype"] == "fp32" else torch.bfloat16


def _lengths(case: Dict[str, Any]) -> List[int]:
    """`seqs` unequal prompt lengths that add up to `rows`."""
    rows, n = case["rows"], case["seqs"]
    parts = [max(1, rows * (i + 1) // (n * (n + 1) // 2)) for i in range(n)]
    parts[-1] += rows - sum(parts)
    return parts


def _linear_data(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    m = _Maker(seed)
    dt = torch.float16 if case["mode"] == "int8" else torch.bfloat16
    x = m.normal(case["rows"], case["n_in"], dtype=torch.float32).clamp_(-5.5, 5.5)
    if case["mode"] == "int8":
        x[:, m.integers(case["n_in"], 6)] *= 12.0   # a few columns carry outliers, as activations of large models do
    return dict(x=x.to(dt), w=m.normal(case["n_out"], case["n_in"], std=0.02, dtype=dt),
                b=m.normal(case["n_out"], std=0.1, dtype=dt) if case["bias"] else None)


def _mlp_weights(m: _Maker, d: int, ff: int) -> Tuple[torch.Tensor, ...]:
    return m.normal(ff, d, std=0.02), m.normal(ff, d, std=0.02), m.normal(d, ff, std=0.02)


def _attn_weights(m: _Maker, d: int, H: int, G: int) -> Tuple[torch.Tensor, ...]:
    hs = d // H
    return m.normal((H + 2 * G) * hs, d, std=0.02), m.normal(d, d, std=0.02)


def _cache(m: _Maker, batch: int, G: int, start: int, total: int, hs: int) -> Tuple[torch.Tensor, torch.Tensor]:
    k, v = (torch.zeros((batch, G, total, hs), device=DEV, dtype=torch.bfloat16) for _ in range(2))
    if start:
        k[:, :, :start], v[:, :, :start] = m.normal(batch, G, start, hs), m.normal(batch, G, start, hs)
    return k, v


def _rope(total: int, hs: int, dtype: torch.dtype) -> Tuple[torch.Tensor, torch.Tensor]:
    theta = 1.0 / (10000 ** (torch.arange(0, hs, 2, device=DEV, dtype=dtype) / hs))
    ang = torch.outer(torch.arange(total, device=DEV, dtype=dtype), theta).repeat(1, 2)
    return torch.cos(ang), torch.sin(ang)


def _attention_data(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    m = _Maker(seed)
    d, H, G, _ = SHAPES[case["shape"]]
    wqkv, wo = _attn_weights(m, d, H, G)
    k, v = _cache(m, case["batch"], G, case["start"], case["start"] + case["rows"] + 5, d // H)
    return dict(x=m.normal(case["batch"], case["rows"], d), wqkv=wqkv, wo=wo, k=k, v=v)


def _window_data(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    m, dt = _Maker(seed), _dtype(case)
    H, G, hs, d = case["heads"], case["kv_heads"], case["dim"], case["width"]
    cols = (H + 2 * G) * hs
    return dict(h=m.normal(case["rows"], d, dtype=dt), w_qkv=m.normal(cols, d, std=d ** -0.5, dtype=dt), b_qkv=m.normal(cols, std=0.1, dtype=dt),
                conv=m.normal(cols, 4, std=0.5, dtype=dt), sink=m.normal(H, dtype=dt), w_o=m.normal(d, H * hs, std=(H * hs) ** -0.5, dtype=dt),
                b_o=m.normal(d, std=0.1, dtype=dt))


def _delta_data(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    m, dt = _Maker(seed), _dtype(case)
    H, G, hs, d, rank = case["heads"], case["kv_heads"], case["dim"], case["width"], 64
    conv_cols = 2 * G * hs + H * hs
    res = dict(h=m.normal(case["rows"], d, dtype=dt), conv=m.normal(conv_cols, 4, std=0.5, dtype=dt), a_log=m.uniform(-1.0, 1.5, H, dtype=dt),
               norm=m.uniform(0.5, 1.5, hs, dtype=dt), w_o=m.normal(d, H * hs, std=(H * hs) ** -0.5, dtype=dt))
    if case["channel"]:
        res.update(w_in=m.normal(conv_cols + 2 * rank + H, d, std=d ** -0.5, dtype=dt), w_gate2=m.normal(H * hs, rank, std=rank ** -0.5, dtype=dt),
                   w_decay2=m.normal(H * hs, rank, std=rank ** -0.5, dtype=dt), dt_bias=m.uniform(-5.0, -1.0, H * hs, dtype=dt))
    else:
        res.update(w_in=m.normal(conv_cols + H * hs + 2 * H, d, std=d ** -0.5, dtype=dt), dt_bias=m.uniform(-5.0, -1.0, H, dtype=dt))
    return res


def _decay_data(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    m, dt = _Maker(seed), _dtype(case)
    H, hs, d, rank = case["heads"], case["dim"], case["width"], 16
    cols = 4 * H * hs + (rank if case["channel"] else 0)
    res = dict(h=m.normal(case["rows"], d, dtype=dt), w_in=m.normal(cols, d, std=d ** -0.5, dtype=dt),
               norm=m.uniform(0.5, 1.5, hs if case["channel"] else H * hs, dtype=dt), w_o=m.normal(d, H * hs, std=(H * hs) ** -0.5, dtype=dt))
    if case["channel"]:
        res.update(w_decay2=m.normal(H * hs, rank, std=rank ** -0.5, dtype=dt), decay_bias=m.uniform(0.0, 4.0, H * hs, dtype=dt))
    return res


def _decays(heads: int) -> List[float]:
    return [1.0 - 2.0 ** (-5.0 - 4.0 * i / heads) for i in range(heads)]


def _step_data(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    m = _Maker(seed)
    d, H, G, ff = SHAPES[case["shape"]]
    total = case["start"] + 4
    layers = []
    for _ in range(case["layers"]):
        layers.append(dict(zip(("wqkv", "wo", "w1", "w2", "w3"), _attn_weights(m, d, H, G) + _mlp_weights(m, d, ff)), n1=m.uniform(0.5, 1.5, d),
                           n2=m.uniform(0.5, 1.5, d), kv=_cache(m, case["batch"], G, case["start"], total, d // H)))
    return dict(layers=layers, wte=m.normal(case["vocab"], d), head=m.normal(case["vocab"], d, std=0.02), nf=m.uniform(0.5, 1.5, d),
                idx=m.integers(case["vocab"], case["batch"], 1))


# ---- the framework's side ------------------------------------------------------------------------------------------------------------
def _qlinear(w: torch.Tensor, mode: str, bias: Optional[torch.Tensor] = None):
    from lit_gpt_b200.quant import QLinear

    lin = torch.nn.Linear(w.shape[1], w.shape[0], bias=bias is not None, device="meta")
    lin.weight = torch.nn.Parameter(w, requires_grad=False)
    if bias is not None:
        lin.bias = torch.nn.Parameter(bias, requires_grad=False)
    return QLinear.from_linear(lin, mode, w.dtype)


def _fill(module: torch.nn.Module, data: Dict[str, torch.Tensor]) -> None:
    for name, p in module.named_parameters():
        if name == "w_in" and p.shape[0] > data[name].shape[0]:
            p.data.zero_()
        p.data[: data[name].shape[0]].copy_(data[name])


def _ragged(case: Dict[str, Any]):
    from lit_gpt_b200.ragged import state_batch

    return state_batch([(i, 0, n) for i, n in enumerate(_lengths(case))], torch.device(DEV), positions=True)[0]


def _config(case: Dict[str, Any], **more: Any):
    from lit_gpt_b200.config import Config

    d, H, G, ff = SHAPES[case["shape"]]
    return Config(block_size=8192, n_embd=d, n_head=H, n_query_groups=G, intermediate_size=ff, rotary_percentage=1.0, parallel_residual=False,
                  bias=False, _norm_class="RMSNorm", norm_eps=1e-5, _mlp_class="LLaMAMLP", **{"vocab_size": 32000, "padded_vocab_size": 32000, "n_layer": 1, **more})


@torch.inference_mode()
def prepare(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    kind = case["kind"]
    if kind == "linear":
        D = _linear_data(case, seed)
        return dict(kind=kind, layer=_qlinear(D["w"], case["mode"], D["b"]), x=D["x"])
    if kind == "mlp":
        from lit_gpt_b200.model import LLaMAMLP

        m = _Maker(seed)
        d, _, _, ff = SHAPES[case["shape"]]
        with torch.device("meta"):
            mlp = LLaMAMLP(_config(case))
        mlp.fc_1, mlp.fc_2, mlp.proj = (_qlinear(w, case["mode"]) for w in _mlp_weights(m, d, ff))
        return dict(kind=kind, layer=mlp, x=m.normal(case["rows"], d))
    if kind == "attention":
        from lit_gpt_b200.model import CausalSelfAttention, KVCache

        D = _attention_data(case, seed)
        with torch.device("meta"):
            attn = CausalSelfAttention(_config(case))
        attn.attn, attn.proj = _qlinear(D["wqkv"], case["mode"]), _qlinear(D["wo"], case["mode"])
        attn.kv_cache = KVCache(D["k"].shape, D["v"].shape, device=DEV, dtype=torch.bfloat16, gqa_native=True)
        attn.kv_cache.k.copy_(D["k"])
        attn.kv_cache.v.copy_(D["v"])
        pos = torch.arange(case["start"], case["start"] + case["rows"], device=DEV)
        cos, sin = _rope(D["k"].shape[2], D["k"].shape[3], torch.float32)
        return dict(kind=kind, layer=attn, x=D["x"], cos=cos[pos], sin=sin[pos], pos=pos)
    if kind == "step":
        return _prepare_step(case, seed)
    batch, slots = _ragged(case), case["seqs"]
    if kind == "window":
        from lit_gpt_b200.config import RotarySpec, WindowMixerSpec
        from lit_gpt_b200.window import WindowAttention

        D = _window_data(case, seed)
        layer = WindowAttention(case["width"], WindowMixerSpec(case["heads"], case["kv_heads"], case["dim"], case["dim"], 4, case["window"], 2.0 * case["dim"] ** -0.5,
                                                               RotarySpec(case["dim"] // 2, 10000.0)), 1e-6)
    elif kind == "delta":
        from lit_gpt_b200.config import DeltaMixerSpec
        from lit_gpt_b200.delta import GatedDeltaRule

        D = _delta_data(case, seed)
        rank = 64 if case["channel"] else 0
        layer = GatedDeltaRule(case["width"], DeltaMixerSpec(case["heads"], case["kv_heads"], case["dim"], case["dim"], 4, case["channel"], rank, rank), 1e-6)
    else:
        from lit_gpt_b200.config import LinearMixerSpec
        from lit_gpt_b200.linear import DecayLinearAttention

        D = _decay_data(case, seed)
        layer = DecayLinearAttention(case["width"], LinearMixerSpec(case["heads"], case["dim"], case["dim"], None if case["channel"] else _decays(case["heads"]),
                                                                    16.0, 16 if case["channel"] else 0), 1e-6)
    layer = layer.to(device=DEV, dtype=_dtype(case))
    _fill(layer, D)
    return dict(kind=kind, layer=layer, x=D["h"], batch=batch, state=layer.build_state(slots, torch.device(DEV), _dtype(case)))


def _prepare_step(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    from lit_gpt_b200.model import GPT

    D = _step_data(case, seed)
    with torch.device("meta"):
        model = GPT(_config(case, n_layer=case["layers"], vocab_size=case["vocab"], padded_vocab_size=case["vocab"]))
    param = lambda t: torch.nn.Parameter(t, requires_grad=False)   # noqa: E731
    model.transformer.wte.weight, model.transformer.ln_f.weight = param(D["wte"]), param(D["nf"])
    model.lm_head = _qlinear(D["head"], case["mode"])
    for block, L in zip(model.transformer.h, D["layers"]):
        block.norm_1.weight, block.norm_2.weight = param(L["n1"]), param(L["n2"])
        block.attn.attn, block.attn.proj = _qlinear(L["wqkv"], case["mode"]), _qlinear(L["wo"], case["mode"])
        block.mlp.fc_1, block.mlp.fc_2, block.mlp.proj = (_qlinear(L[w], case["mode"]) for w in ("w1", "w2", "w3"))
    model.max_seq_length = case["start"] + 4
    model.cos, model.sin = _rope(case["start"] + 4, model.config.head_size, torch.float32)
    model.set_kv_cache(case["batch"], device=torch.device(DEV), dtype=torch.bfloat16)
    for block, L in zip(model.transformer.h, D["layers"]):
        block.attn.kv_cache.k.copy_(L["kv"][0])
        block.attn.kv_cache.v.copy_(L["kv"][1])
    pos = torch.tensor([case["start"]], device=DEV)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            model(D["idx"], pos)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        logits = model(D["idx"], pos)
    return dict(kind="step", model=model, graph=graph, logits=logits, idx=D["idx"], pos=pos, caches=[b.attn.kv_cache for b in model.transformer.h])


@torch.inference_mode()
def run(state: Dict[str, Any]) -> Any:
    kind = state["kind"]
    if kind in ("linear", "mlp"):
        return state["layer"](state["x"])
    if kind == "attention":
        y = state["layer"](state["x"], state["cos"], state["sin"], None, state["pos"])
        return y, state["layer"].kv_cache.k, state["layer"].kv_cache.v
    if kind == "step":
        state["graph"].replay()
        return (state["logits"],) + tuple(t for c in state["caches"] for t in (c.k, c.v))
    y = state["layer"](state["x"], state["batch"], state["state"])
    return (y,) + tuple(state["state"].tensors())


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------------
def _weight_bytes(mode: str, n: int) -> float:
    return n * {"nf4": 0.5625, "int4": 0.5 + 4.0 / 128, "int8": 1.0}[mode]


def work(case: Dict[str, Any]) -> Dict[str, float]:
    kind = case["kind"]
    if kind == "linear":
        r, n = case["rows"], case["n_in"] * case["n_out"]
        return dict(bytes=_weight_bytes(case["mode"], n) + 2 * r * (case["n_in"] + case["n_out"]), flops=2 * r * n)
    if kind == "step":
        d, H, G, ff = SHAPES[case["shape"]]
        n = case["layers"] * ((H + 2 * G) * (d // H) * d + d * d + 3 * d * ff) + case["vocab"] * d
        kv = case["layers"] * case["batch"] * 2 * G * (d // H) * 2 * (case["start"] + 2)
        return dict(bytes=_weight_bytes(case["mode"], n) + kv + 2 * case["batch"] * (case["vocab"] + d), flops=2 * case["batch"] * n)
    r = case["rows"]
    if kind == "mlp":
        d, _, _, ff = SHAPES[case["shape"]]
        return dict(bytes=_weight_bytes(case["mode"], 3 * d * ff) + 4 * r * d, flops=6 * r * d * ff)
    if kind == "attention":
        d, H, G, _ = SHAPES[case["shape"]]
        hs, B, s = d // H, case["batch"], case["start"]
        n = (H + 2 * G) * hs * d + d * d
        return dict(bytes=_weight_bytes(case["mode"], n) + 4 * B * r * d + 4 * B * G * hs * (s + 2 * r),
                    flops=2 * B * r * n + 4 * B * H * hs * (r * s + r * (r + 1) // 2))
    H, hs, d = case["heads"], case["dim"], case["width"]
    size = 4 if case["dtype"] == "fp32" else 2
    if kind == "window":
        G = case["kv_heads"]
        n = d * ((H + 2 * G) * hs + H * hs)
        pairs = sum(sum(min(i + 1, case["window"]) for i in range(t)) for t in _lengths(case))
        return dict(bytes=size * (n + 2 * r * d + 2 * min(r, case["window"] * case["seqs"]) * G * hs), flops=2 * r * n + 4 * H * hs * pairs)
    if kind == "delta":
        G = case["kv_heads"]
        n = d * (2 * G * hs + H * hs + (128 + H if case["channel"] else H * hs + 2 * H)) + d * H * hs + (128 * H * hs if case["channel"] else 0)
        return dict(bytes=size * (n + 2 * r * d) + 4 * case["seqs"] * H * hs * hs, flops=2 * r * n + 8 * r * H * hs * hs)
    n = d * 4 * H * hs + d * H * hs + (16 * (d + H * hs) if case["channel"] else 0)
    return dict(bytes=size * (n + 2 * r * d) + 4 * case["seqs"] * H * hs * hs, flops=2 * r * n + 5 * r * H * hs * hs)


def tolerance(case: Dict[str, Any]) -> Any:
    kind = case["kind"]
    if kind == "linear":
        return {"rel": 2e-3 if case["mode"] == "int8" else 1e-2}   # int8: exact products, the result rounded to fp16 in steps
    if kind in ("mlp", "attention"):
        return {"rel": 2e-2 if kind == "mlp" else 2.5e-2}
    if kind == "step":
        return {"rel": 5e-2}
    return {"rel": 1.5e-5 if case["dtype"] == "fp32" else 1.6e-2}


# ---- the same outputs in 64 bits -------------------------------------------------------------------------------------------------------
_NF4 = [-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334, -0.09105003625154495, 0.0,
        0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224, 0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0]


def _quantized(w: torch.Tensor, mode: str) -> torch.Tensor:
    """The values that the stored 4-bit codes of w stand for."""
    w = w.float()
    if mode == "nf4":   # blocks of 64: the code next to w / absmax
        blocks = w.reshape(-1, 64)
        absmax = blocks.abs().amax(1, keepdim=True)
        code = torch.tensor(_NF4, device=w.device)
        picked = code[torch.bucketize(blocks * (1.0 / absmax), (code[1:] + code[:-1]) / 2)]
        return (picked.to(F64) * absmax.to(F64)).reshape(w.shape)
    groups = w.reshape(w.shape[0], -1, 128)   # int4: scale and zero point per row and 128 columns
    lo, hi = groups.amin(2).clamp(max=0.0), groups.amax(2).clamp(min=0.0)
    scale = ((hi - lo) / 15.0).half().float().unsqueeze(2)
    zero = torch.round(-lo.unsqueeze(2) / scale).clamp(0, 15)
    q = (torch.round(groups / scale) + zero).clamp(0, 15)
    return (scale.to(F64) * (q - zero).to(F64)).reshape(w.shape)


def _exact_int8(D: Dict[str, Any]) -> torch.Tensor:
    x, w = D["x"].float(), D["w"].float()
    outlier = (x.abs() >= 6.0).any(0)
    scb = w.abs().amax(1, keepdim=True)
    cb = torch.round(w * (127.0 / scb))
    xin = torch.where(outlier, torch.zeros_like(x), x)
    sca = xin.abs().amax(1, keepdim=True)
    ca = torch.round(xin * (127.0 / sca))
    y = (ca.to(F64) @ cb.to(F64).T) * (sca.to(F64) * scb.to(F64).T / (127.0 * 127.0))
    y += x[:, outlier].to(F64) @ (cb[:, outlier].to(F64) * (scb.to(F64) / 127.0)).T
    return y if D["b"] is None else y + D["b"].to(F64)


def _turn(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
    half = x.shape[-1] // 2
    return x * cos + torch.cat((-x[..., half:], x[..., :half]), -1) * sin


def _exact_attention(x: torch.Tensor, wqkv: torch.Tensor, wo: torch.Tensor, k: torch.Tensor, v: torch.Tensor, start: int, H: int, G: int):
    B, T, d = x.shape
    hs = d // H
    cos, sin = _rope(start + T, hs, F64)
    cos, sin = cos[start:], sin[start:]
    qkv = (x @ wqkv.T).view(B, T, G, H // G + 2, hs)
    q = _turn(qkv[:, :, :, : H // G].reshape(B, T, H, hs).transpose(1, 2), cos, sin)
    k, v = k.to(F64), v.to(F64)
    k[:, :, start : start + T] = _turn(qkv[:, :, :, -2].transpose(1, 2), cos, sin)
    v[:, :, start : start + T] = qkv[:, :, :, -1].transpose(1, 2)
    hidden = torch.arange(start + T, device=x.device)[None, :] > torch.arange(start, start + T, device=x.device)[:, None]
    y = torch.empty_like(q)
    for b in range(B):
        for h in range(H):
            g = h // (H // G)
            s = (q[b, h] @ k[b, g, : start + T].T) * hs ** -0.5
            y[b, h] = torch.softmax(s.masked_fill_(hidden, float("-inf")), -1) @ v[b, g, : start + T]
    return y.transpose(1, 2).reshape(B, T, d) @ wo.T, k, v


def _exact_mlp(x: torch.Tensor, w1: torch.Tensor, w2: torch.Tensor, w3: torch.Tensor) -> torch.Tensor:
    return (F.silu(x @ w1.T) * (x @ w2.T)) @ w3.T


def _rms(x: torch.Tensor, eps: float) -> torch.Tensor:
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _exact_step(case: Dict[str, Any], seed: int):
    D = _step_data(case, seed)
    d, H, G, _ = SHAPES[case["shape"]]
    deq = lambda w: _quantized(w, case["mode"])   # noqa: E731
    x = D["wte"][D["idx"]].to(F64)
    out: List[torch.Tensor] = []
    for L in D["layers"]:
        y, k, v = _exact_attention(_rms(x, 1e-5) * L["n1"].to(F64), deq(L["wqkv"]), deq(L["wo"]), *L["kv"], case["start"], H, G)
        x = x + y
        x = x + _exact_mlp(_rms(x, 1e-5) * L["n2"].to(F64), deq(L["w1"]), deq(L["w2"]), deq(L["w3"]))
        out += [k, v]
    return ((_rms(x, 1e-5) * D["nf"].to(F64)) @ deq(D["head"]).T, *out)


def _causal_conv(u: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    taps = w.shape[1]
    padded = torch.cat((u.new_zeros(taps - 1, u.shape[1]), u))
    return sum(padded[j : j + u.shape[0]] * w[:, j] for j in range(taps))


def _tail(u: torch.Tensor, taps: int) -> torch.Tensor:
    return torch.cat((u.new_zeros(taps - 1, u.shape[1]), u))[u.shape[0] :]


def _exact_window(case: Dict[str, Any], seed: int):
    D = {k: t.to(F64) for k, t in _window_data(case, seed).items()}
    H, G, hs, W = case["heads"], case["kv_heads"], case["dim"], case["window"]
    rd = hs // 2
    ys, tails, krings, vrings, first = [], [], [], [], 0
    for T in _lengths(case):
        u = D["h"][first : first + T] @ D["w_qkv"].T + D["b_qkv"]
        first += T
        c = _causal_conv(u, D["conv"])
        q, k, v = c[:, : H * hs].view(T, H, hs), c[:, H * hs : (H + G) * hs].view(T, G, hs), c[:, (H + G) * hs :].view(T, G, hs)
        ang = torch.outer(torch.arange(T, device=DEV, dtype=F64), 10000.0 ** (-torch.arange(0, rd, 2, device=DEV, dtype=F64) / rd))[:, None]
        cos, sin = torch.cos(ang), torch.sin(ang)

        def turned(t: torch.Tensor) -> torch.Tensor:
            t = t.clone()
            a, b = t[..., 0:rd:2].clone(), t[..., 1:rd:2].clone()
            t[..., 0:rd:2], t[..., 1:rd:2] = a * cos - b * sin, b * cos + a * sin
            return _rms(t, 1e-6)

        q, k = turned(q), turned(k)
        i = torch.arange(T, device=DEV)
        seen = (i[None, :] <= i[:, None]) & (i[None, :] > i[:, None] - W)
        y = torch.empty(T, H, hs, device=DEV, dtype=F64)
        for h in range(H):
            s = ((q[:, h] @ k[:, h // (H // G)].T) * 2.0 * hs ** -0.5).masked_fill_(~seen, float("-inf"))
            s = torch.cat((s, D["sink"][h].expand(T, 1)), 1)
            y[:, h] = torch.softmax(s, -1)[:, :T] @ v[:, h // (H // G)]
        ys.append(y.reshape(T, H * hs) @ D["w_o"].T + D["b_o"])
        tails.append(_tail(u, 4))
        for rings, t in ((krings, k), (vrings, v)):
            ring = torch.zeros(W, G * hs, device=DEV, dtype=F64)
            keep = i[max(0, T - W) :]
            ring[keep % W] = t.reshape(T, G * hs)[keep]
            rings.append(ring)
    return torch.cat(ys), torch.stack(tails), torch.stack(krings), torch.stack(vrings)


def _exact_delta(case: Dict[str, Any], seed: int):
    D = {k: t.to(F64) for k, t in _delta_data(case, seed).items()}
    H, G, hs, rank = case["heads"], case["kv_heads"], case["dim"], 64
    cc = 2 * G * hs + H * hs
    lanes = 4 if hs <= 64 else 8   # the stored order of a state: keys in runs of `lanes`, columns between the runs
    ys, tails, states, first = [], [], [], 0
    for T in _lengths(case):
        u = D["h"][first : first + T] @ D["w_in"].T
        first += T
        c = F.silu(_causal_conv(u[:, :cc], D["conv"]))
        q, k, v = c[:, : G * hs].view(T, G, hs), c[:, G * hs : 2 * G * hs].view(T, G, hs), c[:, 2 * G * hs :].view(T, H, hs)
        q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * hs ** -0.5).repeat_interleave(H // G, 1)
        k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
        beta = torch.sigmoid(u[:, -H:])
        if case["channel"]:
            z, gate = u[:, cc + rank : cc + 2 * rank] @ D["w_decay2"].T, torch.sigmoid(u[:, cc : cc + rank] @ D["w_gate2"].T)
            z = (z + D["dt_bias"]).view(T, H, hs)
        else:
            z, gate = (u[:, cc + H * hs : cc + H * hs + H] + D["dt_bias"]).view(T, H, 1), F.silu(u[:, cc : cc + H * hs])
        g = torch.exp(-torch.exp(D["a_log"])[:, None] * F.softplus(z))
        S = torch.zeros(H, hs, hs, device=DEV, dtype=F64)
        o = torch.empty(T, H, hs, device=DEV, dtype=F64)
        for t in range(T):
            S = S * g[t, :, :, None]
            w = beta[t, :, None] * (v[t] - torch.einsum("hij,hi->hj", S, k[t]))
            S = S + k[t, :, :, None] * w[:, None, :]
            o[t] = torch.einsum("hij,hi->hj", S, q[t])
        y = _rms(o, 1e-6) * D["norm"] * gate.view(T, H, hs)
        ys.append(y.reshape(T, H * hs) @ D["w_o"].T)
        tails.append(_tail(u[:, :cc], 4))
        states.append(S.view(H, hs // lanes, lanes, hs).transpose(2, 3).reshape(-1))
    return torch.cat(ys), torch.stack(tails), torch.stack(states)


def _exact_decay(case: Dict[str, Any], seed: int):
    D = {k: t.to(F64) for k, t in _decay_data(case, seed).items()}
    H, hs, rank = case["heads"], case["dim"], 16
    ys, states, first = [], [], 0
    for T in _lengths(case):
        u = D["h"][first : first + T] @ D["w_in"].T
        first += T
        q, k, v, gate = (u[:, i * H * hs : (i + 1) * H * hs] for i in range(4))
        if case["channel"]:
            q = q * hs ** -0.5
            g = torch.sigmoid(u[:, 4 * H * hs : 4 * H * hs + rank] @ D["w_decay2"].T + D["decay_bias"]).pow(1.0 / 16.0).view(T, H, hs)
        else:
            q, k, v = F.silu(q), F.silu(k), F.silu(v)
            g = torch.tensor(_decays(H), device=DEV, dtype=F64).view(1, H, 1).expand(T, H, 1)
        q, k, v = q.view(T, H, hs), k.view(T, H, hs), v.view(T, H, hs)
        S = torch.zeros(H, hs, hs, device=DEV, dtype=F64)
        o = torch.empty(T, H, hs, device=DEV, dtype=F64)
        for t in range(T):
            S = S * g[t, :, :, None] + k[t, :, :, None] * v[t, :, None, :]
            o[t] = torch.einsum("hij,hi->hj", S, q[t])
        if case["channel"]:
            y = (_rms(o, 1e-6) * D["norm"]).reshape(T, H * hs) * F.silu(gate)
        else:
            y = _rms(o.reshape(T, H * hs), 1e-6) * D["norm"] * torch.sigmoid(gate)
        ys.append(y @ D["w_o"].T)
        states.append(S.reshape(-1))
    return torch.cat(ys), torch.stack(states)


@torch.inference_mode()
def exact(case: Dict[str, Any], seed: int) -> Optional[Any]:
    kind = case["kind"]
    if kind == "linear":
        D = _linear_data(case, seed)
        if case["mode"] == "int8":
            return _exact_int8(D)
        y = D["x"].to(F64) @ _quantized(D["w"], case["mode"]).T
        return y if D["b"] is None else y + D["b"].to(F64)
    if kind == "mlp":
        m = _Maker(seed)
        d, _, _, ff = SHAPES[case["shape"]]
        w = [_quantized(t, case["mode"]) for t in _mlp_weights(m, d, ff)]
        return _exact_mlp(m.normal(case["rows"], d).to(F64), *w)
    if kind == "attention":
        D = _attention_data(case, seed)
        _, H, G, _ = SHAPES[case["shape"]]
        return _exact_attention(D["x"].to(F64), _quantized(D["wqkv"], case["mode"]), _quantized(D["wo"], case["mode"]), D["k"], D["v"], case["start"], H, G)
    if kind == "step":
        return _exact_step(case, seed)
    return {"window": _exact_window, "delta": _exact_delta, "decay": _exact_decay}[kind](case, seed)
