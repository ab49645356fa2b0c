"""The performance cases of the framework: what a program that serves models with it calls, and with which sizes.

Shapes are those of the benchmark (bench.py) and of the tests: a small layer, the Mixtral-8x7B, DeepSeek-V3 and
Qwen3-30B-A3B MoE layers with random weights N(0, 0.02) in FP8 e4m3 with 128x128 block scales, activations N(0, 1).

A case is one of
  layer    FusedMoE: router, routing, experts and weighted combine.  `graph` = the captured form that a decode loop
           replays (up to 1024 tokens, as in the benchmark), else the plain call that a prefill makes.  `act` is the
           arithmetic: "w8a8" (FP8 tensor cores) or "w8a16" (the reference's: bf16 activations).
  experts  torch.ops.my_ops.fused_moe_fused_experts, the reference's op: routing done by the caller, per-slot rows out.
           `weights` is "fp8" (with fp32 block scales, as checkpoints ship them) or "bf16" (scales = None).
  mlp      torch.ops.my_ops.mlp_w8a8_quant_forward / mlp_w8a16_dq_forward: the dense FP8 MLP of a shared expert.
  linear   torch.ops.my_ops.mm_w8a16_dq_forward: one FP8 block-scaled projection.
"""
import math

import numpy as np
import torch

import torch_tpu_b200
from torch_tpu_b200 import lib as L
from torch_tpu_b200 import weights as W
from torch_tpu_b200.layer import FusedMoE, MoEConfig

DEV = "cuda:0"
GRAPH_TOKENS = 1024  # largest batch that is replayed as a CUDA graph (bench.py does the same)

SHAPES = {
    "small": dict(H=1024, I=512, E=8, k=2, score="softmax"),
    "mixtral": dict(H=4096, I=14336, E=8, k=2, score="softmax"),
    "deepseek": dict(H=7168, I=2048, E=256, k=8, score="sigmoid", groups=8, topk_groups=4, scale=2.5, shared=2048),
    "qwen": dict(H=2048, I=768, E=128, k=8, score="softmax", zipf=True),
}


def _layer(name, shape, tokens, act="w8a8", graph=True):
    return {"name": name, "path": "layer", "shape": shape, "tokens": tokens, "act": act,
            "graph": graph and tokens <= GRAPH_TOKENS}


def listed():
    return [
        _layer("small_16", "small", 16),              # the smallest layer: launches and latency are all there is
        _layer("mixtral_1", "mixtral", 1),            # one user's decode step: two experts' weights are streamed
        _layer("mixtral_32", "mixtral", 32),          # a served decode batch: every expert has a handful of rows
        _layer("mixtral_512", "mixtral", 512),        # a large decode batch or one chunk of a chunked prefill
        _layer("mixtral_4096", "mixtral", 4096),      # prefill of a few thousand tokens: the FP8 tensor cores' case
        _layer("deepseek_64", "deepseek", 64),        # decode over 256 fine experts, grouped routing, shared expert
        _layer("deepseek_2048", "deepseek", 2048),    # prefill over 256 fine experts: 64 rows each on average
        _layer("qwen_8192", "qwen", 8192),            # prefill with heavy-tailed expert loads and short K loops
        _layer("mixtral_333_w8a16", "mixtral", 333, "w8a16"),  # the reference's arithmetic on a ragged batch
        # the reference's op as its callers use it: uncaptured, routing outside, un-weighted rows out, an odd batch
        {"name": "experts_777", "path": "experts", "shape": "qwen", "tokens": 777, "weights": "fp8"},
        # the same op with unquantised experts
        {"name": "experts_bf16_201", "path": "experts", "shape": "qwen", "tokens": 201, "weights": "bf16"},
        # a dense FP8 projection on a prefill chunk of odd length
        {"name": "linear_1001", "path": "linear", "tokens": 1001, "K": 4096, "N": 6144},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    while True:
        c = _draw(rng)
        if all({**c, "name": l["name"]} != l for l in listed()):  # another case than the listed ones
            return c


def _draw(rng):
    r = rng.random()
    if r < 0.55:
        shape = rng.choice(["small", "mixtral", "mixtral", "deepseek", "qwen"])
        most = {"small": 4096, "mixtral": 4096, "deepseek": 2048, "qwen": 8192}[shape]
        c = _layer("", shape, _log_int(rng, 1, most), graph=rng.random() < 0.75)
    elif r < 0.65:
        c = _layer("", rng.choice(["small", "mixtral", "qwen"]), _log_int(rng, 1, 1024), "w8a16")
    elif r < 0.80:
        c = {"path": "experts", "shape": rng.choice(["small", "qwen", "qwen"]), "tokens": _log_int(rng, 1, 2048),
             "weights": rng.choice(["fp8", "fp8", "bf16"])}
    elif r < 0.90:
        c = {"path": "mlp", "H": rng.choice([2048, 4096, 7168]), "I": 128 * rng.randint(4, 48),
             "tokens": _log_int(rng, 1, 2048), "act": rng.choice(["w8a8", "w8a16"])}
    else:
        c = {"path": "linear", "K": 128 * rng.randint(8, 56), "N": 64 * rng.randint(16, 128),
             "tokens": _log_int(rng, 1, 4096)}
    c.pop("name", None)
    return c


# ---- inputs ------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, *size):
    return torch.randn(*size, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)


def _zipf_bias(E, seed):
    """3 * log of Zipf(1.2) popularity with a random assignment of ranks to experts: heavy-tailed expert loads."""
    ranks = np.random.RandomState(seed % (1 << 31)).permutation(E) + 1.0
    p = ranks ** -1.2
    return 3.0 * np.log(p / p.sum())


def _layer_parts(c, seed):
    s = SHAPES[c["shape"]]
    g = _gen(seed)
    T, E = c["tokens"], s["E"]
    wr = (torch.randn(E, s["H"], generator=g, device=DEV) * 0.02).to(torch.bfloat16)
    bias = torch.randn(E, generator=g, device=DEV) * 0.01 if s["score"] == "sigmoid" else None
    logit_bias = torch.from_numpy(_zipf_bias(E, seed)).float().to(DEV) if s.get("zipf") else None
    shared = W.random_experts(1, s["H"], s["shared"], DEV, seed=seed + 777) if s.get("shared") else None
    return _normal(g, T, s["H"]), wr, bias, logit_bias, W.random_experts(E, s["H"], s["I"], DEV, seed=seed), shared


def _prepare_layer(c, seed):
    s, T = SHAPES[c["shape"]], c["tokens"]
    x, wr, bias, logit_bias, experts, shared = _layer_parts(c, seed)
    cfg = MoEConfig(s["H"], s["I"], s["E"], s["k"], s["score"], s.get("groups", 1), s.get("topk_groups", 1), True,
                    s.get("scale", 1.0), s.get("shared", 0))
    layer = FusedMoE(cfg, wr, *experts, bias=bias, shared=shared, logit_bias=logit_bias, max_tokens=T,
                     act_mode=L.ACT_W8A8 if c["act"] == "w8a8" else L.ACT_W8A16)
    if c["graph"]:
        layer.capture(T)
    return {"call": layer.forward_graph if c["graph"] else layer.forward, "args": (x,)}


def _prepare_experts(c, seed):
    s = SHAPES[c["shape"]]
    g = _gen(seed)
    T, H, I, E, k = c["tokens"], s["H"], s["I"], s["E"], s["k"]
    if c["weights"] == "bf16":
        w = [(torch.randn(E, I, H, generator=g, device=DEV) * 0.02).to(torch.bfloat16) for _ in range(3)]
        scales = (None, None, None)
    else:
        parts = W.random_experts(E, H, I, DEV, seed=seed)
        w, scales = parts[:3], parts[3:]
    weight, ids = torch.randn(T, E, generator=g, device=DEV).softmax(-1).topk(k, dim=-1)
    weight = (weight / weight.sum(-1, keepdim=True)).to(torch.bfloat16)
    out = torch.empty(T, k, H, dtype=torch.bfloat16, device=DEV)
    args = (out, _normal(g, T, H), None, None, *w, *scales, ids.to(torch.int32), weight, None, None, None, 128, E, k,
            False, 1, 1, None, None, None, False)
    return {"call": torch.ops.my_ops.fused_moe_fused_experts, "args": args}


def _prepare_mlp(c, seed):
    H, I, T = c["H"], c["I"], c["tokens"]
    w = [t.squeeze(0) for t in W.random_experts(1, H, I, DEV, seed=seed)]
    op = torch.ops.my_ops.mlp_w8a8_quant_forward if c["act"] == "w8a8" else torch.ops.my_ops.mlp_w8a16_dq_forward
    x = _normal(_gen(seed), T, H)
    return {"call": op, "args": (x, *w, torch.empty_like(x), 128)}


def _prepare_linear(c, seed):
    g = _gen(seed)
    M, K, N = c["tokens"], c["K"], c["N"]
    q, scale = W.quantize_blockwise(torch.randn(N, K, generator=g, device=DEV) * 0.02)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    return {"call": torch.ops.my_ops.mm_w8a16_dq_forward, "args": (_normal(g, M, K), q, scale, out, 128)}


def prepare(case, seed):
    torch_tpu_b200.load_ops()
    return {"layer": _prepare_layer, "experts": _prepare_experts, "mlp": _prepare_mlp,
            "linear": _prepare_linear}[case["path"]](case, int(seed) % (1 << 31))


def run(state):
    return state["call"](*state["args"])


# ---- the same arithmetic in 64 bits ---------------------------------------------------------------------------------
# Roundings that belong to the arithmetic are kept (e4m3 activations with one scale per row and 128 columns; in w8a16
# bf16 weights and bf16 intermediate results); every product, sum and activation between them is formed in 64 bits.
def _q8(v):
    """What a row means to the FP8 tensor cores: e4m3 values times a scale per 128 columns."""
    g = v.unflatten(-1, (-1, 128))
    amax = g.abs().amax(-1, keepdim=True).clamp_min(1e-12)
    q = (g.float() * (448.0 / amax.float())).to(torch.float8_e4m3fn).double()
    return (q * (amax.float() / 448.0).double()).flatten(-2)


def _r16(v):
    return v.to(torch.bfloat16).double()


def _dequant(w, s):
    return w.double() * s.double().repeat_interleave(128, 0)[:w.shape[0]].repeat_interleave(128, 1)


def _exact_mlp(x, w, act):
    """x [n,H] float64 -> [n,H]; w = gate, up, down [I,H] and their scales (None: bf16 weights)."""
    if w[3] is None:
        wg, wu, wd = (t.double() for t in w[:3])
    else:
        wg, wu, wd = (_dequant(t, sc) for t, sc in zip(w[:3], w[3:]))
    if act == "w8a8":
        x = _q8(x)
        g, u = x @ wg.t(), x @ wu.t()
        return _q8(g * torch.sigmoid(g) * u) @ wd
    wg, wu, wd = _r16(wg), _r16(wu), _r16(wd)
    g, u = _r16(x @ wg.t()), _r16(x @ wu.t())
    return _r16(_r16(_r16(g * torch.sigmoid(g)) * u) @ wd)


def _exact_slots(x, ids, experts, act):
    T, k = ids.shape
    out = torch.zeros(T, k, x.shape[1], dtype=torch.float64, device=DEV)
    for e in torch.unique(ids).tolist():
        t, j = (ids == e).nonzero(as_tuple=True)
        out[t, j] = _exact_mlp(x[t], [w if w is None else w[e] for w in experts], act)
    return out


def _exact_layer(c, seed):
    s = SHAPES[c["shape"]]
    x, wr, bias, logit_bias, experts, shared = _layer_parts(c, seed)
    x = x.double()
    logits = x @ wr.double().t()
    if logit_bias is not None:
        logits = logits + logit_bias.double()
    score = logits.softmax(-1) if s["score"] == "softmax" else logits.sigmoid()
    sel = score if bias is None else score + bias.double()
    if s.get("groups", 1) > 1:
        g = sel.unflatten(-1, (s["groups"], -1))
        keep = g.topk(2, -1).values.sum(-1).topk(s["topk_groups"], -1).indices
        mask = torch.zeros_like(g[..., 0]).scatter_(-1, keep, 1.0).bool()
        sel = g.masked_fill(~mask.unsqueeze(-1), -math.inf).flatten(-2)
    ids = sel.topk(s["k"], -1).indices
    w = score.gather(-1, ids)
    w = w / w.sum(-1, keepdim=True) * s.get("scale", 1.0)
    out = (w.unsqueeze(-1) * _exact_slots(x, ids, experts, c["act"])).sum(1)
    return out if shared is None else out + _exact_mlp(x, [t[0] for t in shared], c["act"])


def exact(case, seed):
    c = case
    seed = int(seed) % (1 << 31)
    if c["path"] == "layer":
        return _exact_layer(c, seed)
    args = prepare(c, seed)["args"]
    if c["path"] == "experts":  # args: out, x, -, -, three weights, three scales, ids, ...
        return _exact_slots(args[1].double(), args[10], args[4:10], "w8a16" if c["weights"] == "bf16" else "w8a8")
    if c["path"] == "mlp":
        return _exact_mlp(args[0].double(), args[1:7], c["act"])
    x, w, scale = args[:3]
    return _q8(x.double()) @ _dequant(w, scale).t()


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def _activated(s, T):
    """Experts that T tokens activate.  Even routing: its expectation.  Skewed routing: counted on a sample of logits
    of the case's own distribution (router outputs of N(0,1) inputs have a standard deviation of 0.02 * sqrt(H))."""
    E, k = s["E"], s["k"]
    if not s.get("zipf"):
        return E * (1.0 - (1.0 - k / E) ** T)
    n = min(T, 2048)
    rs = np.random.RandomState(1)
    logits = rs.standard_normal((n, E)) * 0.02 * math.sqrt(s["H"]) + _zipf_bias(E, 1)
    return float(len(np.unique(np.argpartition(-logits, k, axis=1)[:, :k])))


def work(case):
    T = case["tokens"]
    if case["path"] == "linear":
        K, N = case["K"], case["N"]
        return {"bytes": N * K + 4 * -(-N // 128) * (K // 128) + 2 * T * (K + N), "flops": 2.0 * T * N * K}
    if case["path"] == "mlp":
        H, I = case["H"], case["I"]
        return {"bytes": 3 * H * I + 12 * (H // 128) * (I // 128) + 4 * T * H, "flops": 6.0 * T * H * I}
    s = SHAPES[case["shape"]]
    H, I, E, k, Is = s["H"], s["I"], s["E"], s["k"], s.get("shared", 0)
    flops = 6.0 * T * k * H * I + 6.0 * T * H * Is
    if case["path"] == "experts":  # routing given, even; per-slot rows out
        act = E * (1.0 - (1.0 - k / E) ** T)
        per = 6 * H * I if case["weights"] == "bf16" else 3 * H * I + 12 * (H // 128) * (I // 128)
        return {"bytes": act * per + 2 * T * H + 2 * T * k * H + 6 * T * k, "flops": flops}
    per = 3 * H * I + 12 * (H // 128) * (I // 128)
    shared = 3 * H * Is + 12 * (H // 128) * (Is // 128)
    return {"bytes": _activated(s, T) * per + shared + 4 * T * H + 2 * E * H, "flops": flops + 2.0 * T * E * H}


def tolerance(case):
    """Measured against the same arithmetic in 64 bits (inputs of one seed, e4m3 / bf16 roundings kept where the
    arithmetic has them): FP8 projection rel 0.003 and max 0.03 (a 128-deep FP8 product is summed by the tensor core
    with fewer than 24 bits); a whole FP8 expert 0.006 to 0.0138 and 0.05 to 0.16 (such a difference moves a hidden
    value across an e4m3 step of 1/16 now and then); W8A16 0.0011 and 0.016; bf16 weights 0.0005 and 0.011.  Stated:
    about four times that, and 0.03 where that would be more."""
    if case["path"] == "linear":
        return {"rel": 1.2e-2, "max": 0.12}
    if case.get("act") == "w8a16" or case.get("weights") == "bf16":
        return {"rel": 4.5e-3, "max": 0.065}
    return {"rel": 3e-2, "max": 0.6}
