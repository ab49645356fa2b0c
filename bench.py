"""Benchmark of the FP8 fused-MoE layer (route -> permute -> gate/up GEMM + SiLU*up -> down GEMM -> combine).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--workload mixtral|deepseek|qwen|small] [--tokens T]
    python bench.py --impl reference ...     # the reference's CPU arithmetic (oracle port) on the host cores

One "step" is one pass of the layer over one batch of T synthetic tokens per GPU.  Prints ONE JSON line:
  value      tokens/s with inputs resident in HBM (whole job, all GPUs); the K-step timed region is repeated
             ``--repeats`` times and ``ms_per_step`` is the median region (``repeat_ms`` lists them all)
  e2e        tokens/s through forward_host: pinned host x -> H2D -> layer -> D2H of the result, every step
  roofline   the dominant kernel (gate/up GEMM) timed alone with CUDA events, algorithmic FLOPs or bytes / time / peak
  sweep      the same layer at the other token counts of the workload (decode sizes are HBM-bound)
  configs    (1 GPU) headline numbers of the other benchmark shapes; ep_configs (N GPUs) the expert-parallel ones
  parity     a seeded sample of the last step's tokens recomputed by the CPU oracle (outside the timed region)
  cpu_baseline  the CPU oracle on a bounded sample, host cores stated (the like-for-like CPU figure is --impl reference)
Inputs are seeded synthetic tensors of the named model shape (no datasets or checkpoints are involved).
Weights (>= 0.6 GB) are far larger than the 126 MB L2, so consecutive steps cannot be served from cache.
"""
import argparse
import hashlib
import json
import os
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOADS = {
    # name: H, I, E, k, routing, tokens (headline first), shared I
    "small": dict(H=1024, I=512, E=8, k=2, score="softmax", tokens=[16], desc="T16 H1024 I512 E8 top2"),
    "mixtral": dict(H=4096, I=14336, E=8, k=2, score="softmax", tokens=[4096, 1, 32, 512],
                    desc="Mixtral-8x7B-shaped layer"),
    "deepseek": dict(H=7168, I=2048, E=256, k=8, score="sigmoid", groups=8, topk_groups=4, scale=2.5, shared=2048,
                     tokens=[2048, 1, 64], desc="DeepSeek-V3-shaped layer (256 routed + 1 shared expert)"),
    "qwen": dict(H=2048, I=768, E=128, k=8, score="softmax", zipf=True, tokens=[8192],
                 desc="Qwen3-30B-A3B-shaped layer, Zipf(1.2)-skewed routing"),
}
METRIC = "fp8_fused_moe_layer_tokens_per_s"


def config_of(name, wl, T, world, ep):
    """The ``config`` object of the JSON line: identical in the b200 arm and the reference arm."""
    return {"workload": f"{name}: {wl['desc']}, {T} tokens/GPU", "H": wl["H"], "I": wl["I"], "E": wl["E"],
            "top_k": wl["k"], "parallelism": f"ep{world} ({ep})" if world > 1 else "single",
            "l2": "weights >> 126 MB L2, 4 rotating input batches"}


def load_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return dict(hbm=d["hbm_gbs"], bf16=d["bf16_tflops"], bf16_sus=d.get("bf16_tflops_sustained", d["bf16_tflops"]),
                    src="measured")
    return dict(hbm=6650.0, bf16=1590.0, bf16_sus=1400.0, src="fallback")


def ncu_traffic(workload, T):
    """DRAM read + write bytes of one launch of the gate/up GEMM from the committed ncu record - valid only for the
    kernel source it was captured from: the record carries the SHA-256 of csrc/gemm_tc.cu, and a stale record
    yields None instead of a number that no longer describes the kernel."""
    rec = os.path.join(ROOT, "profiles", "ncu_dram_traffic.json")
    src = os.path.join(ROOT, "torch-tpu_b200", "csrc", "gemm_tc.cu")
    if not (os.path.exists(rec) and os.path.exists(src)):
        return None, "no ncu record"
    d = json.load(open(rec))
    sha = hashlib.sha256(open(src, "rb").read()).hexdigest()
    for e in d.get("entries", []):
        if e["workload"] == workload and e["tokens"] == T:
            if e["source_sha256"] != sha:
                return None, "ncu record is older than the kernel source"
            return float(e["dram_bytes_per_launch"]), e.get("note", "ncu dram__bytes_read.sum + dram__bytes_write.sum")
    return None, "size not captured"


class ClockSampler:
    """Samples SM clock, power and throttle reasons through NVML every 5 ms while the timed regions run."""

    def __init__(self, index, period=0.005):
        self.samples, self.power, self.reasons, self.stop, self.max_mhz = [], [], set(), False, None
        self.period = period
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM)
        except Exception:
            self.nv = None
        self.t = threading.Thread(target=self._run, daemon=True)

    def _run(self):
        nv = self.nv
        names = {"hw_slowdown": 0x8, "sw_power_cap": 0x4, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40,
                 "hw_power_brake": 0x80}
        while not self.stop:
            try:
                self.samples.append(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM))
                self.power.append(nv.nvmlDeviceGetPowerUsage(self.h) / 1000.0)
                r = nv.nvmlDeviceGetCurrentClocksEventReasons(self.h) if hasattr(
                    nv, "nvmlDeviceGetCurrentClocksEventReasons") else nv.nvmlDeviceGetCurrentClocksThrottleReasons(self.h)
                for n, bit in names.items():
                    if r & bit:
                        self.reasons.add(n)
            except Exception:
                pass
            time.sleep(self.period)

    def __enter__(self):
        if self.nv:
            self.t.start()
        return self

    def __exit__(self, *a):
        self.stop = True
        if self.nv:
            self.t.join(timeout=1)

    def summary(self):
        s = sorted(self.samples)
        return {"sm_mhz": s[len(s) // 2] if s else None, "sm_mhz_min": s[0] if s else None,
                "sm_max_mhz": self.max_mhz, "samples": len(s), "power_w_max": max(self.power) if self.power else None,
                "reasons": sorted(self.reasons)}


def algorithmic(wl, T, e_act):
    H, I, k = wl["H"], wl["I"], wl["k"]
    Is = wl.get("shared", 0)
    flops = 6.0 * T * k * H * I + 6.0 * T * H * Is
    nH, nI = H // 128, I // 128
    wbytes = e_act * (3 * H * I + 12 * nH * nI) + (3 * H * Is + 12 * nH * (Is // 128) if Is else 0)
    abytes = 4 * T * H + 2 * wl["E"] * H + 8 * T * k
    return flops, wbytes + abytes


def _router_parts(wl, dev, seed):
    """Router weights, selection bias and logit bias of a synthetic layer (replicated on every rank)."""
    import torch
    E = wl["E"]
    g = torch.Generator(device=dev).manual_seed(seed + 12345)
    wr = (torch.randn(E, wl["H"], generator=g, device=dev) * 0.02).to(torch.bfloat16)
    bias = torch.randn(E, generator=g, device=dev) * 0.01 if wl["score"] == "sigmoid" else None
    logit_bias = None
    if wl.get("zipf"):
        # per-expert logit bias 3*log(p_e), p_e ~ rank_e^-1.2 with a seeded random assignment of ranks to experts
        ranks = (torch.randperm(E, generator=torch.Generator().manual_seed(seed * 31 + 5)) + 1).double()
        p = ranks ** -1.2
        logit_bias = (3.0 * torch.log(p / p.sum())).float().to(dev)
    return wr, bias, logit_bias


def _moe_config(wl):
    from torch_tpu_b200.layer import MoEConfig
    return MoEConfig(wl["H"], wl["I"], wl["E"], wl["k"], wl["score"], wl.get("groups", 1), wl.get("topk_groups", 1), True,
                     wl.get("scale", 1.0), wl.get("shared", 0))


def build_layer(wl, T_max, dev, seed, first_expert=0, n_local=None, fused_combine=False):
    import torch_tpu_b200  # noqa: F401
    from torch_tpu_b200 import weights as W
    from torch_tpu_b200.layer import FusedMoE
    n_local = wl["E"] if n_local is None else n_local
    w = W.random_experts(n_local, wl["H"], wl["I"], dev, seed=seed * 1000 + first_expert)
    wr, bias, logit_bias = _router_parts(wl, dev, seed)
    shared = W.random_experts(1, wl["H"], wl["shared"], dev, seed=seed + 777) if wl.get("shared") else None
    return FusedMoE(_moe_config(wl), wr, *w, bias=bias, shared=shared, logit_bias=logit_bias, max_tokens=T_max,
                    fused_combine=fused_combine)


def build_ep_layer(wl, T, dev, rank, world, seed=0, transport="p2p"):
    """The rank's shard of a synthetic expert-parallel layer.  Expert weights are seeded per (seed, first local
    expert), the replicated router/bias/shared expert by ``seed`` alone.  ``transport``: "nccl"
    (all_to_all_single) or "p2p" (peer-memory stores)."""
    import torch_tpu_b200  # noqa: F401
    from torch_tpu_b200 import weights as W
    from torch_tpu_b200.layer import FusedMoE
    E = wl["E"]
    El = E // world
    w = W.random_experts(El, wl["H"], wl["I"], dev, seed=seed * 1000 + rank * El)
    wr, bias, logit_bias = _router_parts(wl, dev, seed)
    shared = W.random_experts(1, wl["H"], wl["shared"], dev, seed=seed + 777) if wl.get("shared") else None
    layer = FusedMoE(_moe_config(wl), wr, *w, bias=bias, shared=shared, logit_bias=logit_bias, max_tokens=T,
                     alloc_workspace=False)
    if transport == "p2p":
        from torch_tpu_b200.ep_p2p import P2PFusedMoE
        ep = P2PFusedMoE(layer, E, max_tokens=T)
        ep.shared_ctas = int(os.environ.get("B200MOE_EP_SHARED_CTAS", ep.shared_ctas))  # A/B switch, see ep_p2p.py
        return ep
    from torch_tpu_b200.ep import EPFusedMoE
    return EPFusedMoE(layer, E)


def make_x(T, H, dev, seed, zipf_bias=None):
    import torch
    g = torch.Generator().manual_seed(seed)
    return torch.randn(T, H, generator=g).to(torch.bfloat16)


def time_steps(fn, steps, warmup, barrier=None, finish=None):
    """ms per step of one timed region: ``warmup`` untimed calls, then exactly ``steps`` calls between two CUDA
    events on the launching stream, a barrier + synchronize on both sides."""
    import torch
    for _ in range(warmup):
        fn()
    torch.cuda.synchronize()
    if barrier:
        barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    for _ in range(steps):
        fn()
    if finish:
        finish()   # e.g. make the timed stream wait for copies running on side streams
    e1.record()
    torch.cuda.synchronize()
    if barrier:
        barrier()
    return e0.elapsed_time(e1) / steps


def time_repeated(fn, steps, warmup, repeats, barrier=None, finish=None):
    """``repeats`` timed regions of ``steps`` steps each (warm-up before the first only); list of ms per step."""
    out = [time_steps(fn, steps, warmup, barrier, finish)]
    for _ in range(repeats - 1):
        out.append(time_steps(fn, steps, 0, barrier, finish))
    return out


def median(v):
    s = sorted(v)
    return s[len(s) // 2]


def launches_per_step(wl, T, world=1, ep="nccl"):
    import torch
    P = T * wl["k"]
    # router and selection: one kernel for few experts while its blocks of four tokens fit the SMs at once
    route = 1 if wl["E"] <= 16 and 16 < T <= 4 * torch.cuda.get_device_properties(0).multi_processor_count else 2
    sort = lambda pairs: 1 if pairs <= 8192 else 3
    if world > 1 and ep == "p2p":
        # router, route, permute | counts exchange, plan, dispatch, barrier | scales, tiles, 2 GEMMs, barrier | combine
        n = route + sort(P) + 4 + 5 + 1
        if wl.get("shared"):
            n += sort(T) + 1 + 2
        return n
    if world > 1:
        # router, route, permute, pack | unpack ids, permute (received rows), unpack rows, tiles, 2 GEMMs | invert, combine
        n = route + sort(P) + 1 + 1 + 3 + 1 + 1 + 2 + 2
        if wl.get("shared"):
            n += sort(T) + 1 + 2                          # permute (identity ids, tiles with it), quant, 2 GEMMs
        return n
    # router, route, permute (tiles with it), quant, 2 GEMMs, combine
    n = route + sort(P) + 1 + 2 + 1
    if wl.get("shared"):
        n += 1 + 2                                        # quant (lists with it), 2 GEMMs
    return n


# ---- CPU side: the oracle as checker (parity) and as baseline ---------------------------------------------------
def oracle_route(wl, logits, bias, logit_bias):
    from oracle import moe_oracle as O
    if wl["score"] == "softmax":
        if logit_bias is not None:
            logits = logits + logit_bias
        return O.route_softmax_topk(logits, wl["k"])
    return O.route_sigmoid_grouped(logits, bias, wl["groups"], wl["topk_groups"], wl["k"], wl["scale"])


def parity_check(wl, x_dev, y_dev, ids_dev, w_dev, local_w, shared, world=1, rank=0, n_tokens=None):
    """A sample of the step's tokens recomputed by the CPU oracle (W8A8 contract) from the experts' weights: the
    sampled tokens are rank 0's first ``n_tokens``; under expert parallelism the owners of the experts those tokens
    activate broadcast them (NCCL, outside any timed region).  Returns the record on rank 0, None elsewhere."""
    import torch
    from oracle import moe_oracle as O
    E = wl["E"]
    n = n_tokens or (64 if E <= 16 else 8)
    n = min(n, x_dev.shape[0])
    dev = x_dev.device
    El = E // world
    ids_s = ids_dev[:n].clone()
    if world > 1:
        import torch.distributed as dist
        dist.broadcast(ids_s, src=0)
    used = torch.unique(ids_s.long().clamp(0, E - 1)).cpu()
    gathered = []                                            # per owner: (expert ids, 6 tensors)
    for r in range(world):
        mine = used[(used >= r * El) & (used < (r + 1) * El)]
        if mine.numel() == 0:
            continue
        if rank == r:
            parts = [t[(mine - r * El).to(dev)].contiguous() for t in local_w]
        else:
            parts = [torch.empty((mine.numel(),) + tuple(t.shape[1:]), dtype=t.dtype, device=dev) for t in local_w]
        if world > 1:
            import torch.distributed as dist
            for t in parts:
                dist.broadcast(t.view(torch.uint8) if t.dtype == torch.float8_e4m3fn else t, src=r)
        if rank == 0:
            gathered.append((mine, [t.cpu() for t in parts]))
        del parts
    if rank != 0:
        return None
    order = torch.cat([g[0] for g in gathered])
    wts = [torch.cat([g[1][i] for g in gathered]) for i in range(6)]
    remap = torch.full((E,), 0, dtype=torch.long)
    remap[order] = torch.arange(order.numel())
    ids_c, w_c = ids_s.cpu(), w_dev[:n].float().cpu()
    sh = tuple(t[0].cpu() for t in shared) if shared is not None else None
    want = O.moe_layer_w8a8(x_dev[:n].cpu(), remap[ids_c.long()].to(torch.int32), tuple(wts), shared=sh, topk_w=w_c)
    m = O.parity_metrics(y_dev[:n].cpu(), want)
    return {"tokens": int(n), "max_rel": m["max_rel"], "cosine": m["cosine"],
            "ok": bool(m["max_rel"] <= 2e-2 and m["cosine"] >= 0.9995), "tolerance": "max_rel <= 2e-2, cosine >= 0.9995"}


def routing_exact(wl, layer, T):
    """ids of the whole batch against the oracle on the device's own logits (rows with a decidable top-k boundary)."""
    import torch
    from oracle import moe_oracle as O
    logits = layer.logits[:T].cpu()
    lb = layer.logit_bias.cpu() if layer.logit_bias is not None else None
    bias = layer.bias.cpu() if layer.bias is not None else None
    wid, _ = oracle_route(wl, logits, bias, lb)
    if wl["score"] == "softmax":
        ok = O.tie_free_rows(torch.softmax(logits + lb if lb is not None else logits, -1), wl["k"])
    else:
        ok = O.tie_free_rows(torch.sigmoid(logits) + bias, wl["k"], wl["groups"], wl["topk_groups"])
    return bool(torch.equal(layer.ids[:T].cpu()[ok], wid[ok])), float(ok.float().mean())


def cpu_step(wl, x, wr, bias, logit_bias, weights, shared, arith):
    """One whole step on the host: router matmul -> routing -> experts -> combine (+ shared expert)."""
    import torch
    from oracle import moe_oracle as O
    logits = x.float() @ wr.float().t()
    ids, w = oracle_route(wl, logits, bias, logit_bias)
    out = (O.experts_w8a8 if arith == "w8a8" else O.experts_w8a16)(x, ids, *weights)
    y = O.combine(out, w)
    if shared is not None:
        sh = [t[0] for t in shared]
        if arith == "w8a8":
            y = y + O.expert_mlp_w8a8(x.float(), *sh).to(torch.bfloat16)
        else:
            y = y + O.expert_mlp_w8a16(x, *sh)
    return y


def cpu_baseline_sample(wl, layer, sample_tokens):
    """The oracle (W8A8 contract) on the host cores over ``sample_tokens`` tokens of the same workload, the whole
    step inside the clock; only the experts the sample activates are copied from the device (outside the clock)."""
    import torch
    torch.set_num_threads(os.cpu_count())
    x = make_x(sample_tokens, wl["H"], "cpu", seed=4242)
    wr = layer.router_w.cpu()
    bias = layer.bias.cpu() if layer.bias is not None else None
    lb = layer.logit_bias.cpu() if layer.logit_bias is not None else None
    ids, _ = oracle_route(wl, x.float() @ wr.float().t(), bias, lb)
    used = torch.unique(ids.long())
    # sparse host copy: rows of the activated experts only (the step never touches the others)
    weights = []
    for t in layer.w:
        host = torch.empty((wl["E"],) + tuple(t.shape[1:]), dtype=t.dtype)
        host[used] = t[used.to(t.device)].cpu()
        weights.append(host)
    shared = tuple(t.cpu() for t in layer.shared) if layer.shared is not None else None
    t0 = time.perf_counter()
    cpu_step(wl, x, wr, bias, lb, weights, shared, "w8a8")
    secs = time.perf_counter() - t0
    return sample_tokens / secs, secs, int(used.numel())


def run_reference(args, wl):
    """`--impl reference`: the reference's CPU arithmetic (W8A16, bf16 roundings: a port of
    python/regression/test_llm/test_moe.py:10-98 with the dequantisation hoisted per expert, plus the router chain of
    test_torch_ops.py:439-455 and the bmm combine of test_bmm.py:118-134) on the host cores, at the SAME token count
    as the b200 arm, the whole step inside the clock.  Weights are generated on the CPU; nothing of the product
    package is imported.  A step takes seconds, so the number of timed steps is bounded by a time budget."""
    import torch
    from oracle import moe_oracle as O
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    torch.set_num_threads(os.cpu_count())
    T = wl["tokens"][0] if args.tokens is None else args.tokens
    E, H, I = wl["E"], wl["H"], wl["I"]
    t_gen = time.perf_counter()
    weights = O.make_expert_weights(E, H, I, seed=0)
    shared = O.make_expert_weights(1, H, wl["shared"], seed=777) if wl.get("shared") else None
    _, wr, _ = O.make_inputs(1, H, E, seed=0)
    g = torch.Generator().manual_seed(12345)
    bias = torch.randn(E, generator=g) * 0.01 if wl["score"] == "sigmoid" else None
    lb = O.zipf_bias(E, seed=0) if wl.get("zipf") else None
    xs = [make_x(T, H, "cpu", seed=100 + i) for i in range(2)]
    t_gen = time.perf_counter() - t_gen
    budget = args.cpu_budget_s
    times, warm = [], 0
    t_start = time.perf_counter()
    for i in range(args.warmup + args.steps):
        t0 = time.perf_counter()
        cpu_step(wl, xs[i % 2], wr, bias, lb, weights, shared, "w8a16")
        dt = time.perf_counter() - t0
        if i < min(args.warmup, 1) and dt < budget / 3:
            warm += 1                                  # one warm-up step when the budget allows it
        else:
            times.append(dt)
        if len(times) >= args.steps or (time.perf_counter() - t_start) > budget:
            break
    ms = 1000 * sum(times) / len(times)
    val = T / (ms / 1000)
    world = int(os.environ.get("WORLD_SIZE", "1"))
    line = {"impl": "reference", "metric": METRIC, "value": val, "unit": "tokens/s",
            "n_gpus": args.gpus, "steps": len(times), "warmup": warm, "ms_per_step": ms,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "bf16 activations x e4m3 weights dequantised to bf16 (cpu)",
            "data": "synthetic", "config": config_of(args.workload, wl, T, world, args.ep),
            "cpu_baseline": {"value": val, "unit": "tokens/s", "cores": os.cpu_count(), "kind": "port",
                             "sample": f"whole {T}-token steps (router + routing + experts + combine in the clock; "
                                       f"{len(times)} timed step(s) within a {budget:.0f} s budget; weights generated "
                                       f"on the host in {t_gen:.0f} s outside the clock)"},
            "e2e": {"value": val, "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


# ---- sub-records ------------------------------------------------------------------------------------------------
def roofline_frac(wl, T, e_act, ms, peaks):
    fl, nb = algorithmic(wl, T, e_act)
    fp8_peak = 2 * peaks["bf16"]
    t_tc, t_hbm = fl / (fp8_peak * 1e12), nb / (peaks["hbm"] * 1e9)
    if t_tc >= t_hbm:
        return "tensor", fl / (ms / 1000) / 1e12 / fp8_peak
    return "hbm", nb / (ms / 1000) / 1e9 / peaks["hbm"]


def single_gpu_config_record(name, T, dev, args, peaks):
    """Headline numbers of one of the other benchmark shapes on this GPU (device-resident input, CUDA events)."""
    import torch
    wl = WORKLOADS[name]
    layer = build_layer(wl, T, dev, seed=0)
    xs = [make_x(T, wl["H"], dev, seed=200 + i).to(dev) for i in range(4)]
    it = [0]
    use_graph = T <= 1024

    def step():
        (layer.forward_graph if use_graph else layer.forward)(xs[it[0] % 4])
        it[0] += 1
    ms_all = time_repeated(step, args.steps, 3, 3)
    ms = median(ms_all)
    y = layer.forward(xs[0])
    torch.cuda.synchronize()
    ids = layer.ids[:T]
    e_act = int(torch.unique(ids).numel())
    bound, frac = roofline_frac(wl, T, e_act, ms, peaks)
    ids_ok, _ = routing_exact(wl, layer, T)
    par = parity_check(wl, xs[0], y, ids, layer.topk_w[:T], layer.w, layer.shared)
    par["ids_exact"] = ids_ok
    rec = {"workload": f"{name}: {wl['desc']}, {T} tokens", "ms_per_step": ms, "ms_min": min(ms_all),
           "tokens_per_s": T / (ms / 1000), "cuda_graph": use_graph, "bound": bound, "frac": frac,
           "activated_experts": e_act, "device_status": int(layer.status.item()), "parity": par}
    del layer, xs
    torch.cuda.empty_cache()
    return rec


def ep_config_record(name, T, dev, rank, world, args):
    """One expert-parallel configuration (peer-memory exchange): step time (max over ranks) and per-phase times."""
    import torch
    import torch.distributed as dist
    wl = WORKLOADS[name]
    barrier = lambda: (dist.barrier(), torch.cuda.synchronize())  # noqa: E731
    ep = build_ep_layer(wl, T, dev, rank, world, seed=0, transport="p2p")
    xs = [make_x(T, wl["H"], dev, seed=500 + rank * 10 + i).to(dev) for i in range(4)]
    it = [0]

    def step():
        ep.forward(xs[it[0] % 4])
        it[0] += 1
    ms_all = time_repeated(step, max(5, args.steps // 2), 3, 3, barrier)
    phases = {}
    for _ in range(4):                                   # per-phase times of a few more steps
        ep.phase_events = []
        step()
        torch.cuda.synchronize()
        ev = ep.phase_events
        for (_, e0), (n1, e1) in zip(ev[:-1], ev[1:]):
            phases[n1] = phases.get(n1, 0.0) + e0.elapsed_time(e1) / 4
    ep.phase_events = None
    y = ep.forward(xs[0])
    torch.cuda.synchronize()
    layer = ep.layer
    status = int(ep.status.item()) | int(layer.status.item())
    par = parity_check(wl, xs[0], y, layer.ids[:T], layer.topk_w[:T], layer.w, layer.shared, world, rank)
    names = sorted(phases)
    t = torch.tensor([median(ms_all), min(ms_all), float(status)] + [phases[n] for n in names], device=dev,
                     dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms = float(t[0])
    rec = None
    if rank == 0:
        fl, _ = algorithmic(wl, T, wl["E"])
        rec = {"workload": f"{name}: {wl['desc']}, {T} tokens/GPU, experts sharded over {world} GPUs "
                           "(peer-memory exchange)",
               "ms_per_step": ms, "ms_min": float(t[1]), "tokens_per_s": T * world / (ms / 1000),
               "tflops_per_gpu": fl / (ms / 1000) / 1e12, "device_status": int(t[2]),
               "phase_ms_max_over_ranks": {n: float(v) for n, v in zip(names, t[3:])}, "parity": par}
    ep.close()
    del ep, xs
    torch.cuda.empty_cache()
    return rec


def bind_to_gpu_numa_node(index):
    """Run this process (and place its pinned host buffers, by first touch) on the NUMA node the GPU hangs off."""
    try:
        import pynvml
        pynvml.nvmlInit()
        bdf = pynvml.nvmlDeviceGetPciInfo(pynvml.nvmlDeviceGetHandleByIndex(index)).busId
        bdf = (bdf.decode() if isinstance(bdf, bytes) else bdf).lower()
        if len(bdf.split(":")[0]) == 8:
            bdf = bdf[4:]
        node = int(open(f"/sys/bus/pci/devices/{bdf}/numa_node").read())
        if node < 0:
            return None
        cpus = set()
        for part in open(f"/sys/devices/system/node/node{node}/cpulist").read().strip().split(","):
            a, _, b = part.partition("-")
            cpus.update(range(int(a), int(b or a) + 1))
        cpus &= os.sched_getaffinity(0)
        if cpus:
            os.sched_setaffinity(0, cpus)
        return node
    except Exception:
        return None


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--repeats", type=int, default=10, help="timed regions of --steps steps each; the median is reported")
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--workload", default="mixtral", choices=list(WORKLOADS))
    ap.add_argument("--tokens", type=int, default=None, help="tokens per GPU (default: the workload's headline size)")
    ap.add_argument("--sample-tokens", type=int, default=256, help="tokens of the CPU sample in the b200 arm")
    ap.add_argument("--cpu-budget-s", type=float, default=150.0, help="time budget of the reference arm's steps")
    ap.add_argument("--ep", default="p2p", choices=["p2p", "nccl"],
                    help="exchange of the expert-parallel runs (N > 1): peer-memory stores or NCCL all-to-all")
    ap.add_argument("--fused-combine", action="store_true",
                    help="form the weighted combine inside the down GEMM's epilogue (fp32 reductions)")
    ap.add_argument("--no-sweep", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-configs", action="store_true", help="skip the records of the other benchmark shapes")
    ap.add_argument("--no-parity", action="store_true")
    args = ap.parse_args()
    wl = WORKLOADS[args.workload]
    args.warmup = max(args.warmup, 3) if args.impl == "b200" else args.warmup
    if args.impl == "reference":
        return run_reference(args, wl)

    # Libraries (NCCL prints its version banner) write to stdout; the contract is ONE JSON line there.  Everything
    # but that line goes to stderr: fd 1 is pointed at fd 2 and the line is written to the saved descriptor.
    sys.stdout.flush()
    real_stdout = os.dup(1)
    os.dup2(2, 1)

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    numa = bind_to_gpu_numa_node(local) if world > 1 else None   # before any pinned allocation
    import torch
    import torch_tpu_b200  # noqa: F401
    from torch_tpu_b200 import lib as L
    from torch_tpu_b200 import ops

    torch.cuda.set_device(local)
    dev = f"cuda:{local}"
    barrier = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=torch.device(dev))
        barrier = lambda: (dist.barrier(), torch.cuda.synchronize())  # noqa: E731
    peaks = load_peaks()
    T = wl["tokens"][0] if args.tokens is None else args.tokens
    T_max = max([T] + ([] if args.tokens else wl["tokens"]))

    if world > 1:
        try:
            layer = build_ep_layer(wl, T, dev, rank, world, seed=0, transport=args.ep)
        except RuntimeError as exc:
            # peer memory cannot be mapped on this machine (the set-up fails on every rank together): run the
            # all-to-all exchange instead and say so in the line
            if args.ep != "p2p" or "peer memory" not in str(exc):
                raise
            sys.stderr.write(f"bench: {exc}; using the NCCL all-to-all exchange\n")
            args.ep = "nccl"
            layer = build_ep_layer(wl, T, dev, rank, world, seed=0, transport="nccl")
        base_layer = layer.layer
    else:
        layer = build_layer(wl, T_max, dev, seed=0, fused_combine=args.fused_combine)
        base_layer = layer

    xs = [make_x(T, wl["H"], dev, seed=100 + rank * 10 + i).to(dev) for i in range(4)]
    it = [0]

    # ---- the two GEMMs alone, first: ten short regions each while the GPU is still in its burst power state ---------
    # (the peak they are held against was measured as the best of ten short runs; the long loops below pull a 1 kW
    # part into its power cap within a few hundred milliseconds, and every later number is a sustained-state number)
    g1_all = g2_all = None
    if world == 1:
        def only(stage):
            def f():
                ops.experts(layer.out[:T], xs[0], *layer.w, layer.ids[:T], layer.topk_w[:T], shared=layer.shared,
                            workspace=layer.workspace, stages=stage, fused_combine=args.fused_combine)
            return f
        layer.forward(xs[0])
        g1_all = time_repeated(only(L.STAGE_GATE_UP), args.steps, 3, 10)
        g2_all = time_repeated(only(L.STAGE_DOWN), args.steps, 3, 10)

    # ---- device-resident throughput ---------------------------------------------------------------------------

    def step():
        layer.forward(xs[it[0] % 4])
        it[0] += 1

    with ClockSampler(local) as cs:
        ms_all = time_repeated(step, args.steps, args.warmup, args.repeats, barrier)
    clocks = cs.summary()
    ms = median(ms_all)
    status = int(base_layer.status.item())
    if world > 1 and args.ep == "p2p":
        status |= int(layer.status.item())

    # ---- end to end with host buffers ---------------------------------------------------------------------------
    xh = [x.cpu().pin_memory() for x in xs]
    oh = torch.empty(T, wl["H"], dtype=torch.bfloat16).pin_memory()

    def step_e2e():
        layer.forward_host(xh[it[0] % 4], oh)
        it[0] += 1

    e2e_all = time_repeated(step_e2e, args.steps, args.warmup, max(3, args.repeats // 2), barrier, finish=layer.host_join)
    ms_e2e = median(e2e_all)

    # the copies alone (same buffers, same streams, no layer): the ceiling the host link puts on the e2e figure
    hp = getattr(layer, "_hp")

    def step_copy_only():
        i = it[0] & 1
        it[0] += 1
        with torch.cuda.stream(hp["h2d"]):
            hp["x"][i][:T].copy_(xh[i], non_blocking=True)
        with torch.cuda.stream(hp["d2h"]):
            oh.copy_(hp["y"][i][:T], non_blocking=True)

    def join_copies():
        cur = torch.cuda.current_stream()
        cur.wait_stream(hp["h2d"])
        cur.wait_stream(hp["d2h"])
    ms_copy = median(time_repeated(step_copy_only, args.steps, 3, 3, barrier, finish=join_copies))

    if world > 1:
        import torch.distributed as dist
        t = torch.tensor([ms, ms_e2e, ms_copy, min(ms_all), float(status)], device=dev, dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms, ms_e2e, ms_copy, ms_min, status = float(t[0]), float(t[1]), float(t[2]), float(t[3]), int(t[4])
    else:
        ms_min = min(ms_all)

    line = {"metric": METRIC, "value": T * world / (ms / 1000), "unit": "tokens/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "fp8_e4m3 (fp32 accumulate)",
            "data": "synthetic", "config": config_of(args.workload, wl, T, world, args.ep),
            "repeats": args.repeats, "repeat_ms": [round(v, 5) for v in ms_all], "ms_min": ms_min,
            "ms_x_median_sm_mhz": (ms * clocks["sm_mhz"]) if clocks.get("sm_mhz") else None,
            "combine": "fused into the down GEMM's epilogue (fp32 reductions, order not fixed)" if args.fused_combine
            and world == 1 else "separate kernel over per-slot rows (deterministic)",
            "e2e": {"value": T * world / (ms_e2e / 1000), "unit": "tokens/s", "h2d_bytes_per_step": T * wl["H"] * 2,
                    "d2h_bytes_per_step": T * wl["H"] * 2, "ms_per_step": ms_e2e,
                    "copy_only_ms_per_step": ms_copy, "numa_node": numa},
            "gpu_launches": launches_per_step(wl, T, world, args.ep) * args.steps * args.repeats, "clocks": clocks,
            "device_status": status}

    # ---- parity of one more step, outside any timed region ----------------------------------------------------------
    failed = status != 0
    if not args.no_parity:
        x_last = xs[0]
        y = layer.forward(x_last)
        torch.cuda.synchronize()
        par = parity_check(wl, x_last, y, base_layer.ids[:T], base_layer.topk_w[:T], base_layer.w, base_layer.shared,
                           world, rank)
        if rank == 0:
            ids_ok, decidable = routing_exact(wl, base_layer, T)
            par["ids_exact"], par["decidable_rows"] = ids_ok, decidable
            line["parity"] = par
            failed = failed or not par["ok"] or not ids_ok

    if world == 1:
        # ---- roofline of the dominant kernel: gate/up GEMM alone on the filled workspace ---------------------------
        ids = layer.ids[:T]
        e_act = int(torch.unique(ids).numel())
        ms_g1, ms_g2 = median(g1_all), median(g2_all)
        flops, nbytes = algorithmic(wl, T, e_act)
        Is = wl.get("shared", 0)
        f_g1 = 4.0 * T * wl["k"] * wl["H"] * wl["I"] + 4.0 * T * wl["H"] * Is
        b_g1 = e_act * 2 * wl["H"] * wl["I"] + 2 * wl["H"] * Is + T * wl["k"] * (wl["H"] + wl["I"])
        fp8_peak = 2 * peaks["bf16"]
        t_tc, t_hbm = f_g1 / (fp8_peak * 1e12), b_g1 / (peaks["hbm"] * 1e9)
        best_g1 = min(g1_all)
        if t_tc >= t_hbm:
            roof = {"bound": "tensor", "achieved": f_g1 / (best_g1 / 1000) / 1e12, "peak": fp8_peak, "unit": "TFLOP/s"}
            roof["achieved_median"] = f_g1 / (ms_g1 / 1000) / 1e12
            roof["frac_median_vs_sustained_peak"] = roof["achieved_median"] / (2 * peaks["bf16_sus"])
        else:
            roof = {"bound": "hbm", "achieved": b_g1 / (best_g1 / 1000) / 1e9, "peak": peaks["hbm"], "unit": "GB/s"}
            roof["achieved_median"] = b_g1 / (ms_g1 / 1000) / 1e9
        roof["frac"] = roof["achieved"] / roof["peak"]
        roof["frac_median"] = roof["achieved_median"] / roof["peak"]
        roof["protocol"] = ("kernel alone, 10 regions of %d launches, CUDA events; achieved/frac = best region (how the "
                            "burst peak itself was taken: best of 10), *_median = median region" % args.steps)
        roof["traffic"], roof["traffic_note"] = ncu_traffic(args.workload, T)
        roof["traffic_unit"] = "bytes per launch (ncu dram read + write)"
        roof["algorithmic_bytes"] = b_g1
        roof["kernel"] = "moe_gemm_tc_kernel<0> (gate/up GEMM + SiLU*up + requantise)"
        roof["ms_per_launch"] = best_g1
        roof["ms_per_launch_median"] = ms_g1
        roof["region_ms"] = [round(v, 5) for v in g1_all]
        roof["peak_source"] = (f"{peaks['src']}: FP8 dense taken as 2 x the bf16 cuBLAS burst figure (the file holds "
                               "no FP8 number)" if roof["bound"] == "tensor" else f"{peaks['src']} copy bandwidth")
        roof["down_gemm_ms"] = min(g2_all)
        roof["down_gemm_ms_median"] = ms_g2
        roof["down_gemm_frac"] = 2.0 * T * wl["k"] * wl["H"] * wl["I"] / (min(g2_all) / 1000) / 1e12 / fp8_peak
        line["roofline"] = roof
        line["layer"] = {"flops_per_step": flops, "bytes_per_step": nbytes,
                         "tflops": flops / (ms / 1000) / 1e12, "gbs": nbytes / (ms / 1000) / 1e9,
                         "frac_of_fp8_peak": flops / (ms / 1000) / 1e12 / fp8_peak, "activated_experts": e_act}

        # ---- the other token counts of the workload ---------------------------------------------------------------
        if not args.no_sweep and args.tokens is None:
            sweep = []
            for Ts in wl["tokens"][1:]:
                xx = [make_x(Ts, wl["H"], dev, seed=300 + i).to(dev) for i in range(4)]
                j = [0]

                use_graph = Ts <= 1024   # launch-bound sizes: one graph launch instead of a dozen small ones

                def st():
                    (layer.forward_graph if use_graph else layer.forward)(xx[j[0] % 4])
                    j[0] += 1
                m_all = time_repeated(st, max(args.steps, 30), 5, 3)
                m = median(m_all)
                ea = int(torch.unique(layer.ids[:Ts]).numel())
                bound, frac = roofline_frac(wl, Ts, ea, m, peaks)
                sweep.append({"tokens": Ts, "cuda_graph": use_graph, "ms_per_step": m, "ms_min": min(m_all),
                              "tokens_per_s": Ts / (m / 1000), "bound": bound, "activated_experts": ea, "frac": frac})
            line["sweep"] = sweep

        # ---- CPU baseline (bounded sample; the weights of its experts come from the device) ---------------------------
        if not args.no_cpu:
            tps, secs, n_act = cpu_baseline_sample(wl, layer, args.sample_tokens)
            line["cpu_baseline"] = {"value": tps, "unit": "tokens/s", "cores": os.cpu_count(), "kind": "port",
                                    "sample": f"one {args.sample_tokens}-token step of the same layer on the host "
                                              f"(router, routing, {n_act} activated experts dequantised once each, "
                                              f"combine: {secs:.1f} s); a batch this small pays the dequantisation of "
                                              f"every expert for few tokens - the same-size CPU figure is the "
                                              f"--impl reference arm"}

        # ---- the other benchmark shapes -------------------------------------------------------------------------------
        if not args.no_configs and args.tokens is None and args.workload == "mixtral":
            del layer, base_layer, ids
            torch.cuda.empty_cache()
            layer = base_layer = None
            line["configs"] = [single_gpu_config_record(n, t, dev, args, peaks)
                               for n, t in (("small", 16), ("deepseek", 2048), ("qwen", 8192))]
            failed = failed or any(not c["parity"]["ok"] or not c["parity"]["ids_exact"] or c["device_status"]
                                   for c in line["configs"])
    elif not args.no_configs and args.workload == "mixtral" and args.tokens is None and args.ep == "p2p":
        # ---- expert-parallel records of the DeepSeek-V3 shape (4096 tokens/GPU) and, on 8 GPUs, the Qwen3 shape -------
        layer.close()
        del layer, base_layer
        torch.cuda.empty_cache()
        layer = None
        recs = [ep_config_record("deepseek", 4096, dev, rank, world, args)]
        if world == 8:
            recs.append(ep_config_record("qwen", 1024, dev, rank, world, args))
        if rank == 0:
            line["ep_configs"] = recs
            failed = failed or any(r["device_status"] or not r["parity"]["ok"] for r in recs)

    if rank == 0:
        sys.stdout.flush()
        os.write(real_stdout, (json.dumps(line) + "\n").encode())
    if world > 1:
        import torch.distributed as dist
        if layer is not None and hasattr(layer, "close"):
            layer.close()
        dist.destroy_process_group()
    if failed and rank == 0:
        sys.stderr.write("bench: device status word set or parity check failed (see the line)\n")
        sys.exit(3)


if __name__ == "__main__":
    main()
