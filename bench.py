#!/usr/bin/env python
"""Benchmark of the fused-MoE hot path: grouped_topk -> align -> expert GEMMs -> combine.

Workload at N=1: the DeepSeek-V3-shape FP8 block-quant layer (E=256, top-8 of 8
groups/4 kept, H=7168, I=2048) at M=8192 tokens, synthetic seeded inputs.
One step = one pass of the whole path over one batch.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference] [--tokens M]

Prints ONE JSON line (rank 0).  `value` is tokens/s with inputs resident in HBM;
`e2e` is the same metric through the public API with pinned HOST buffers (H2D of
activations and router logits, D2H of the layer output inside the timed region);
`roofline` describes the dominant kernel (GEMM1), timed with CUDA events inside
the timed steps; `cpu_baseline` is the CPU oracle on a bounded sample.
"""

from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import time

import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

DSV3 = dict(E=256, topk=8, n_group=8, topk_group=4, H=7168, I=2048, rsf=2.5)
L2_BYTES = 126 * 1024 * 1024


def load_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as fh:
            p = json.load(fh)
        return dict(hbm_gbs=float(p["hbm_gbs"]), bf16_tflops=float(p["bf16_tflops"]),
                    bf16_tflops_sustained=float(p.get("bf16_tflops_sustained", p["bf16_tflops"])),
                    source="measured")
    return dict(hbm_gbs=6650.0, bf16_tflops=1590.0, bf16_tflops_sustained=1400.0, source="fallback")


class ClockSampler:
    """nvidia-smi clock/throttle sampling during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits", "-lms", "20",
                 "-i", str(self.gpu)], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.15)
        self.proc.terminate()
        try:
            out, _ = self.proc.communicate(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
            out, _ = self.proc.communicate()
        rows, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in out.strip().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                rows.append((float(f[1]), float(f[3])))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        # "under load" = samples drawing at least 60 % of the highest power seen: the sampler also
        # runs a little before and after the timed region, where the clock is back at its maximum
        pmax = max((p for _, p in rows), default=0.0)
        load = sorted(c for c, p in rows if p >= 0.6 * pmax) or sorted(c for c, _ in rows)
        return {"sm_mhz": load[len(load) // 2] if load else None, "sm_max_mhz": max(mx) if mx else None,
                "samples": len(rows), "samples_under_load": len(load), "power_w_max": pmax,
                "reasons": sorted(reasons)}


def bind_to_gpu_cpus(gpu_index: int):
    """Pins THIS process to the CPUs NVML reports as local to its GPU (a process setting, not
    a GPU one), so that the pinned host buffers allocated afterwards land on that GPU's NUMA
    node: with several ranks per box, buffers on the far socket halve the host-copy rate.
    Returns the CPU count it bound to, or None when NVML or the call is unavailable."""
    try:
        import pynvml

        pynvml.nvmlInit()
        h = pynvml.nvmlDeviceGetHandleByIndex(gpu_index)
        words = (os.cpu_count() + 63) // 64
        mask = pynvml.nvmlDeviceGetCpuAffinity(h, words)
        cpus = {64 * i + b for i, w in enumerate(mask) for b in range(64) if (w >> b) & 1}
        cpus &= os.sched_getaffinity(0)
        if cpus:
            os.sched_setaffinity(0, cpus)
            return len(cpus)
    except Exception:
        pass
    return None


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def cpu_oracle_run(M_sample, seed_shift=0, E_used=None, threads=None):
    """Times the CPU oracle (torch-native restatement of the reference's golden
    path) on `M_sample` tokens of the DSV3 FP8 workload.  Returns tokens/s."""
    from oracle import moe_oracle as O

    threads = threads or os.cpu_count() or 1
    torch.set_num_threads(threads)
    c = DSV3
    E = c["E"]
    g = torch.Generator().manual_seed(1234 + seed_shift)
    x = torch.randn(M_sample, c["H"], generator=g).to(torch.bfloat16)
    logits = torch.randn(M_sample, E, generator=g)
    bias = torch.randn(E, generator=g) * 0.1
    tw, ti = O.grouped_topk_oracle(logits, c["n_group"], c["topk_group"], c["topk"], True, c["rsf"], bias, 1)
    used = torch.unique(ti).tolist()
    # Only the experts the sample touches are materialised, as a compact table
    # (ids remapped); four distinct N(0,0.02) block-quantised experts are
    # generated and repeated, which changes neither the arithmetic nor the time.
    n_used = len(used)
    remap = torch.full((E,), -1, dtype=torch.int64)
    remap[torch.tensor(used)] = torch.arange(n_used)
    b1, bs1 = O.quantize_weight_fp8_block(torch.randn(4, 2 * c["I"], c["H"], generator=g) * 0.02)
    b2, bs2 = O.quantize_weight_fp8_block(torch.randn(4, c["H"], c["I"], generator=g) * 0.02)
    sel = torch.arange(n_used) % 4
    w1, s1, w2, s2 = b1[sel], bs1[sel], b2[sel], bs2[sel]

    def step():
        tw_, ti_ = O.grouped_topk_oracle(logits, c["n_group"], c["topk_group"], c["topk"], True, c["rsf"], bias, 1)
        O.moe_align_block_size_oracle(ti_, 128, E)
        return O.fused_moe_fp8_block_oracle(x, w1, w2, s1, s2, tw_, remap[ti_.long()].to(torch.int32))

    return step, threads, len(used)


def fit_reference_tokens(want, steps, warmup, budget_s, seed_shift=0):
    """Largest power-of-two fraction of `want` tokens whose `steps + warmup` CPU passes fit
    `budget_s` seconds, judged from one timed pass.  Returns (tokens, step, threads,
    distinct experts, seconds of that first pass)."""
    M_s = want
    while True:
        step, threads, n_used = cpu_oracle_run(M_s, seed_shift)
        t0 = time.perf_counter()
        step()
        first = time.perf_counter() - t0
        if first * (steps + warmup) <= budget_s or M_s <= 16:
            return M_s, step, threads, n_used, first
        M_s //= 2


def run_reference(args):
    """--impl reference: the reference's torch-native path (CPU oracle port) on host cores."""
    rank, world, _ = dist_env()
    if rank != 0:
        return
    M_s, step, threads, n_used, _ = fit_reference_tokens(args.ref_tokens, args.steps, args.warmup,
                                                         args.ref_budget_s)
    for _ in range(max(0, args.warmup - 1)):  # the sizing pass above was the first warm-up pass
        step()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        step()
    dt = (time.perf_counter() - t0) / args.steps
    val = M_s / dt
    sample = (f"{M_s} tokens per step of the DSV3 FP8 layer ({n_used} distinct experts; the GPU arm runs "
              f"{args.tokens} tokens per step: the CPU sample is the largest that keeps {args.steps}+{args.warmup} "
              f"passes inside {args.ref_budget_s:.0f} s), CPU oracle restating the reference's torch goldens")
    line = {
        "impl": "reference", "metric": "fused_moe_layer_tokens_per_s", "value": val, "unit": "tokens/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "fp8_e4m3", "data": "synthetic",
        "config": {"workload": "deepseek_v3_fp8_block_moe_layer", "tokens": M_s, **DSV3},
        "cpu_baseline": {"value": val, "unit": "tokens/s", "cores": threads, "kind": "port", "sample": sample},
        "e2e": {"value": val, "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "tflops": 6.0 * M_s * DSV3["topk"] * DSV3["H"] * DSV3["I"] / dt / 1e12,
    }
    print(json.dumps(line), flush=True)


def measure_fp8_peak(dev, n=8192, reps=10):
    """Dense e4m3 x e4m3 -> bf16 library GEMM (torch._scaled_mm, per-tensor scales) of n^3,
    best of `reps`, CUDA events: the denominator of the FP8 roofline.  Runs once, outside
    every timed region.  Returns TFLOP/s or None when the library call is unavailable."""
    try:
        a = torch.randn((n, n), device=dev, dtype=torch.bfloat16).to(torch.float8_e4m3fn)
        b = torch.randn((n, n), device=dev, dtype=torch.bfloat16).to(torch.float8_e4m3fn).t()
        one = torch.ones((), device=dev, dtype=torch.float32)
        for _ in range(3):
            torch._scaled_mm(a, b, scale_a=one, scale_b=one, out_dtype=torch.bfloat16)
        best = None
        for _ in range(reps):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            torch._scaled_mm(a, b, scale_a=one, scale_b=one, out_dtype=torch.bfloat16)
            e1.record()
            torch.cuda.synchronize()
            ms = e0.elapsed_time(e1)
            best = ms if best is None or ms < best else best
        return 2.0 * n ** 3 / (best * 1e-3) / 1e12
    except Exception:
        return None


def run_sweep(args):
    """--sweep: every (configuration, M) point of the benchmark plan on one GPU.
    Prints one JSON line per point: ms (median, L2 flushed), TFLOP/s, algorithmic
    GB/s, the binding roofline and the achieved fraction of it."""
    import flaggems_vllm_b200 as fg
    from flaggems_vllm_b200 import testing as T

    torch.cuda.set_device(0)
    dev = torch.device("cuda", 0)
    peaks = load_peaks()
    flush = torch.empty(2 * L2_BYTES, dtype=torch.uint8, device=dev)

    def timeit(fn, iters):
        for _ in range(3):
            fn()
        ts = []
        for _ in range(iters):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            fn()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        ts.sort()
        return ts[len(ts) // 2]

    def graph_ms(fn, iters=20):
        """Device time of one step replayed from a CUDA graph (no launch gaps, L2 warm)."""
        fn()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            fn()
        g.replay()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(iters):
            g.replay()
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b) / iters

    def report(name, M, ms, flops, nbytes, peak_tf, extra=None):
        t_c, t_m = flops / (peak_tf * 1e12), nbytes / (peaks["hbm_gbs"] * 1e9)
        bound = "tensor" if t_c > t_m else "hbm"
        line = {"sweep": name, "M": M, "ms": ms, "tokens_per_s": M / (ms * 1e-3), "tflops": flops / (ms * 1e-3) / 1e12,
                "gbs": nbytes / (ms * 1e-3) / 1e9, "bound": bound, "floor_ms": max(t_c, t_m) * 1e3,
                "frac_of_roofline": max(t_c, t_m) * 1e3 / ms, "peaks": peaks["source"]}
        if extra:
            line.update(extra)
        print(json.dumps(line), flush=True)

    which = args.sweep.split(",")
    keep_m = {int(v) for v in args.sweep_m.split(",")} if args.sweep_m else None

    def sizes(all_m):
        return tuple(m for m in all_m if keep_m is None or m in keep_m)

    iters = lambda default: args.sweep_iters or default
    if "dsv3" in which:
        c = DSV3
        E, H, I, k = c["E"], c["H"], c["I"], c["topk"]
        w1, s1 = T.make_fp8_block_weights(E, 2 * I, H, dev, seed=100)
        w2, s2 = T.make_fp8_block_weights(E, H, I, dev, seed=200)
        for M in sizes((1, 32, 128, 1024, 8192)):
            x = T.make_activations(M, H, dev)
            logits, bias = T.make_router_inputs(M, E, dev, bias_std=args.router_bias_std)

            def step():
                tw, ti = fg.grouped_topk(logits, c["n_group"], c["topk_group"], k, True, c["rsf"], bias, 1)
                return fg.fused_experts_impl(x, w1, w2, tw, ti, use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2,
                                             block_shape=[128, 128])

            _, ti = fg.grouped_topk(logits, c["n_group"], c["topk_group"], k, True, c["rsf"], bias, 1)
            e_act = int(torch.unique(ti).numel())
            nbytes = e_act * (3 * H * I + (2 * I // 128) * (H // 128) * 4 + (H // 128) * (I // 128) * 4) \
                + M * H * 2 * 2 + M * E * 4 + k * 8 * M
            extra = {"distinct_experts": e_act}
            if M <= 1024 and not args.no_graph:
                extra["cuda_graph_replay_ms"] = graph_ms(step)
            report("dsv3_fp8", M, timeit(step, iters(10)), 6.0 * M * k * H * I, nbytes, 2 * peaks["bf16_tflops"], extra)
        del w1, w2, s1, s2
    if "mixtral" in which:
        E, H, I, k = 8, 4096, 14336, 2
        w1 = T.make_half_weights(E, 2 * I, H, dev, seed=1, chunk=1)
        w2 = T.make_half_weights(E, H, I, dev, seed=2, chunk=1)
        for M in sizes((1, 16, 64, 256, 1024, 4096, 16384)):
            x = T.make_activations(M, H, dev)
            logits, _ = T.make_router_inputs(M, E, dev)
            zero = torch.zeros(E, device=dev)

            def step():
                tw, ti = fg.grouped_topk(torch.softmax(logits, -1), 1, 1, k, True, 1.0, zero, 0)
                return fg.fused_experts_impl(x, w1, w2, tw.to(torch.bfloat16), ti)

            _, ti = fg.grouped_topk(torch.softmax(logits, -1), 1, 1, k, True, 1.0, zero, 0)
            e_act = int(torch.unique(ti).numel())
            nbytes = e_act * 3 * H * I * 2 + M * H * 2 * 2 + M * E * 4 + k * 8 * M
            extra = {"distinct_experts": e_act}
            if M <= 1024 and not args.no_graph:
                extra["cuda_graph_replay_ms"] = graph_ms(step)
            report("mixtral_bf16", M, timeit(step, iters(6)), 6.0 * M * k * H * I, nbytes, peaks["bf16_tflops"], extra)
        del w1, w2
    if "qwen3" in which:
        E, H, I, k = 128, 2048, 768, 8
        w1, s1 = T.make_int8_channel_weights(E, 2 * I, H, dev, seed=1)
        w2, s2 = T.make_int8_channel_weights(E, H, I, dev, seed=2)
        for M in sizes((1, 64, 512, 4096)):
            x = T.make_activations(M, H, dev)
            logits, _ = T.make_router_inputs(M, E, dev)
            zero = torch.zeros(E, device=dev)

            def step():
                tw, ti = fg.grouped_topk(torch.softmax(logits, -1), 1, 1, k, True, 1.0, zero, 0)
                return fg.fused_experts_impl(x, w1, w2, tw.to(torch.bfloat16), ti, use_int8_w8a16=True,
                                             per_channel_quant=True, w1_scale=s1, w2_scale=s2)

            _, ti = fg.grouped_topk(torch.softmax(logits, -1), 1, 1, k, True, 1.0, zero, 0)
            e_act = int(torch.unique(ti).numel())
            nbytes = e_act * (3 * H * I + 3 * I * 4 + H * 4) + M * H * 2 * 2 + M * E * 4 + k * 8 * M
            extra = {"distinct_experts": e_act}
            if M <= 1024 and not args.no_graph:
                extra["cuda_graph_replay_ms"] = graph_ms(step)
            report("qwen3_w8a16", M, timeit(step, iters(6)), 6.0 * M * k * H * I, nbytes, peaks["bf16_tflops"], extra)
    if "align" in which:
        for M in (1, 128, 2048, 8192):
            for skewed in (False, True):
                for bs in (64, 128):
                    ids = T.make_align_ids(M, 8, 256, dev, skewed=skewed)
                    ms = timeit(lambda: fg.moe_align_block_size(ids, bs, 256), 20)
                    nbytes = 4 * ids.numel() + 4 * (ids.numel() + 256 * (bs - 1)) + 4 * ((ids.numel() + 256 * (bs - 1)) // bs) + 4
                    print(json.dumps({"sweep": "align", "M": M, "skewed": skewed, "block_size": bs, "ms": ms,
                                      "ids_per_s": ids.numel() / (ms * 1e-3), "gbs": nbytes / (ms * 1e-3) / 1e9}),
                          flush=True)
    if "routing" in which:
        for M in (1, 32, 128, 1024, 8192, 16384):
            logits, bias = T.make_router_inputs(M, 256, dev)
            ms = timeit(lambda: fg.grouped_topk(logits, 8, 4, 8, True, 2.5, bias, 1), 20)
            print(json.dumps({"sweep": "grouped_topk_dsv3", "M": M, "ms": ms, "tokens_per_s": M / (ms * 1e-3)}),
                  flush=True)
        wr = torch.randn((256, 7168), device=dev).to(torch.bfloat16)
        for M in (1, 8, 32, 128, 256):
            xr = torch.randn((M, 7168), device=dev).to(torch.bfloat16)
            ms = timeit(lambda: fg.router_gemm(xr, wr), 20)
            nbytes = (256 + M) * 7168 * 2 + M * 256 * 4
            print(json.dumps({"sweep": "router_gemm_dsv3", "M": M, "ms": ms, "gbs": nbytes / (ms * 1e-3) / 1e9,
                              "tokens_per_s": M / (ms * 1e-3)}), flush=True)


def ep_parity_check(dist, dev, rank, world, layer, x, logits, bias, c, sample_tokens):
    """Expert-parallel correctness, run before the timed region at N > 1.

    (a) Three small layers (FP8 M=96, half precision M=64, FP8 M=1): every rank holds the full
        seeded weights, runs the expert-parallel step on its own tokens and compares with the
        single-GPU layer of the same tokens.
    (b) `sample_tokens` tokens per rank of the full-size step against the CPU oracle; only the
        experts those tokens use are broadcast from their owners.
    Returns {"max_rel_l2", "min_cos", "ok", ...}; limits are the layer tolerance (relative L2
    <= 1e-2, cosine >= 0.9999).  The per-rank partial sums are rounded to bf16 before the final
    sum, one rounding more than the single-GPU layer."""
    import flaggems_vllm_b200 as fg
    from flaggems_vllm_b200 import _lib, ep
    from flaggems_vllm_b200 import testing as T
    from oracle import moe_oracle as O

    worst, mincos, status = 0.0, 1.0, 0
    cases = []
    for mode, (M, E, H, I, k) in (("fp8", (96, 32, 512, 256, 8)), ("half", (64, 16, 256, 256, 4)),
                                  ("fp8", (1, 32, 512, 256, 8))):
        xs = T.make_activations(M, H, dev, seed=50 + rank)
        lg, bs = T.make_router_inputs(M, E, dev, seed=60 + rank)
        El = E // world
        sl = slice(rank * El, (rank + 1) * El)
        if mode == "fp8":
            w1, s1 = T.make_fp8_block_weights(E, 2 * I, H, dev, seed=1, std=H ** -0.5)
            w2, s2 = T.make_fp8_block_weights(E, H, I, dev, seed=2, std=I ** -0.5)
            tw, ti = fg.grouped_topk(lg, 8, 4, k, True, 2.5, torch.zeros_like(bs), 1)
            full = fg.fused_experts_impl(xs, w1, w2, tw, ti, use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2,
                                         block_shape=[128, 128])
            small = ep.ExpertParallelMoE(w1[sl].contiguous(), w2[sl].contiguous(), s1[sl].contiguous(),
                                         s2[sl].contiguous(), E, mode=_lib.MODE_FP8_BLOCK)
        else:
            w1 = T.make_half_weights(E, 2 * I, H, dev, seed=1, std=H ** -0.5)
            w2 = T.make_half_weights(E, H, I, dev, seed=2, std=I ** -0.5)
            tw, ti = fg.grouped_topk(torch.softmax(lg, -1), 1, 1, k, True, 1.0, torch.zeros_like(bs), 0)
            full = fg.fused_experts_impl(xs, w1, w2, tw, ti)
            small = ep.ExpertParallelMoE(w1[sl].contiguous(), w2[sl].contiguous(), None, None, E, mode=_lib.MODE_HALF)
        got = small.forward(xs, tw, ti)
        torch.cuda.synchronize()
        rl2, cs = O.rel_l2(got.float().cpu(), full.float().cpu()), O.cosine(got.float().cpu(), full.float().cpu())
        worst, mincos = max(worst, rl2), min(mincos, cs)
        cases.append(rl2)
    status |= fg.read_status(dev)

    # ---- (b) sampled tokens of the full-size step against the CPU oracle
    E, k, M = c["E"], c["topk"], x.shape[0]
    El = E // world
    tw, ti = fg.grouped_topk(logits, c["n_group"], c["topk_group"], k, True, c["rsf"], bias, 1)
    out = layer.forward(x, tw, ti)
    torch.cuda.synchronize()
    status |= fg.read_status(dev)
    n_s = min(sample_tokens, M)
    idx = torch.linspace(0, M - 1, n_s, device=dev).long()
    ids_s = ti[idx]
    need = torch.zeros(E, dtype=torch.int32, device=dev)
    need[ids_s.reshape(-1).long()] = 1
    union = need.clone()
    dist.all_reduce(union, op=dist.ReduceOp.MAX)
    mine = need.cpu().bool()
    tabs = {"w1": [], "s1": [], "w2": [], "s2": []}
    remap = torch.full((E,), -1, dtype=torch.int64)
    for e in torch.nonzero(union.cpu()).reshape(-1).tolist():
        owner, el = divmod(e, El)
        parts = {}
        for name, t in (("w1", layer.w1), ("s1", layer.s1), ("w2", layer.w2), ("s2", layer.s2)):
            buf = t[el].clone() if rank == owner else torch.empty_like(t[0])
            flat = buf.view(torch.uint8) if buf.dtype == torch.float8_e4m3fn else buf
            dist.broadcast(flat, owner)
            parts[name] = buf
        if mine[e]:
            remap[e] = len(tabs["w1"])
            for name in tabs:
                tabs[name].append(parts[name].cpu())
    torch.set_num_threads(max(1, (os.cpu_count() or 1) // world))
    w1t, s1t, w2t, s2t = (torch.stack(tabs[n]) for n in ("w1", "s1", "w2", "s2"))
    ref = O.fused_moe_fp8_block_oracle(x[idx].cpu(), w1t, w2t, s1t, s2t, tw[idx].cpu(),
                                       remap[ids_s.cpu().long()].to(torch.int32))
    got = out[idx].float().cpu()
    rl2, cs = O.rel_l2(got, ref), O.cosine(got, ref)
    worst_t = torch.tensor([max(worst, rl2), -min(mincos, cs), float(status)], dtype=torch.float64, device=dev)
    dist.all_reduce(worst_t, op=dist.ReduceOp.MAX)
    w, mc, stt = float(worst_t[0]), -float(worst_t[1]), int(worst_t[2])
    return {"max_rel_l2": w, "min_cos": mc, "ok": bool(w <= 1e-2 and mc >= 0.9999 and stt == 0),
            "kernel_status": stt, "rank0_small_cases_rel_l2": cases, "rank0_full_size_sample_rel_l2": rl2,
            "full_size_sample_tokens_per_rank": n_s,
            "what": "max over ranks: 3 small layers vs the single-GPU layer, and sampled tokens of the "
                    "full-size step vs the CPU oracle (limits 1e-2 / 0.9999; the per-rank partial sums are "
                    "rounded to bf16 once more than on one GPU)"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--tokens", type=int, default=8192, help="tokens per GPU per step")
    ap.add_argument("--ref-tokens", type=int, default=256,
                    help="tokens per step of the CPU reference arm (halved until the run fits --ref-budget-s)")
    ap.add_argument("--ref-budget-s", type=float, default=240.0, help="wall-clock budget of the CPU reference arm")
    ap.add_argument("--cpu-baseline-tokens", type=int, default=256)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--ep-chunks", type=int, default=1,
                    help="token chunks per expert-parallel step (each on its own stream and communicator)")
    ap.add_argument("--ep-overlap", type=int, default=0,
                    help="1: expert-parallel combine in two column halves, the first half's all-to-all beside the "
                         "second half's GEMM 2")
    ap.add_argument("--ep-free-sms", type=int, default=16, help="SMs the second GEMM 2 leaves to the all-to-all")
    ap.add_argument("--ep-check-tokens", type=int, default=-1,
                    help="tokens per rank of the full-size expert-parallel step checked against the CPU oracle "
                         "(0: skip; default 16 at 2 GPUs, 8 at 4, 4 at 8: every rank runs the oracle on its share "
                         "of the host cores, and each token brings about 8 experts to widen)")
    ap.add_argument("--router-bias-std", type=float, default=0.02,
                    help="spread of the synthetic score-correction bias; the scores are i.i.d., so a small "
                         "spread gives the balanced expert load a trained bias produces")
    ap.add_argument("--experts", type=int, default=DSV3["E"],
                    help="expert count (smaller values give the small case used for ncu captures)")
    ap.add_argument("--sweep-m", default="", help="comma list: keep only these token counts of a --sweep")
    ap.add_argument("--sweep-iters", type=int, default=0, help="timed iterations per --sweep point (0: default)")
    ap.add_argument("--no-graph", action="store_true", help="--sweep: skip the CUDA-graph replay timing of small M")
    ap.add_argument("--sweep", default="", help="comma list of dsv3,mixtral,qwen3,align,routing: print one line per point")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3) if args.impl == "b200" else args.warmup
    if args.sweep:
        run_sweep(args)
        return
    if args.impl == "reference":
        run_reference(args)
        return

    import flaggems_vllm_b200 as fg
    from flaggems_vllm_b200 import fused_moe
    from flaggems_vllm_b200 import testing as T

    rank, world, local = dist_env()
    if world > 1:
        from flaggems_vllm_b200 import ep  # expert-parallel wrapper
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    else:
        ep = None
        dist = None
        torch.cuda.set_device(0)
    dev = torch.device("cuda", torch.cuda.current_device())
    c = dict(DSV3, E=args.experts)
    M, E, H, I, k = args.tokens, c["E"], c["H"], c["I"], c["topk"]
    E_local = E // world
    peaks = load_peaks()

    # ---- resident inputs
    w1, s1 = T.make_fp8_block_weights(E_local, 2 * I, H, dev, seed=100 + rank)
    w2, s2 = T.make_fp8_block_weights(E_local, H, I, dev, seed=200 + rank)
    x = T.make_activations(M, H, dev, seed=300 + rank)
    logits, bias = T.make_router_inputs(M, E, dev, seed=400 + rank, bias_std=args.router_bias_std)
    if world > 1:
        dist.broadcast(bias, 0)
    flush = torch.empty(2 * L2_BYTES, dtype=torch.uint8, device=dev)
    layer = ep.ExpertParallelMoE(w1, w2, s1, s2, E, dist.group.WORLD, chunks=args.ep_chunks,
                                 overlap_combine=bool(args.ep_overlap), free_sms=args.ep_free_sms) if world > 1 else None
    ep_parity = None
    if args.ep_check_tokens < 0:
        args.ep_check_tokens = max(4, 32 // max(world, 2))
    if world > 1 and args.ep_check_tokens > 0:
        ep_parity = ep_parity_check(dist, dev, rank, world, layer, x, logits, bias, c, args.ep_check_tokens)
    fp8_peak = measure_fp8_peak(dev) if world == 1 else None

    def device_step():
        tw, ti = fg.grouped_topk(logits, c["n_group"], c["topk_group"], k, True, c["rsf"], bias, 1)
        if layer is not None:
            return layer.forward(x, tw, ti)
        return fg.fused_experts_impl(x, w1, w2, tw, ti, use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2,
                                     block_shape=[128, 128])

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    stage_ms = {}
    stage_events = []

    def hook(name):
        ev = torch.cuda.Event(enable_timing=True)
        ev.record(torch.cuda.current_stream())
        stage_events.append((name, ev))

    def timed(fn, steps, record_stages=False):
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
        barrier()
        for i in range(steps):
            flush.zero_()  # L2 flush between iterations (inputs of small M would otherwise stay in L2)
            if record_stages:
                fused_moe.STAGE_HOOK = hook
                hook("begin")
            evs[i][0].record()
            fn()
            evs[i][1].record()
            fused_moe.STAGE_HOOK = None
        barrier()
        total = sum(a.elapsed_time(b) for a, b in evs)
        t = torch.tensor([total], dtype=torch.float64, device=dev)
        if dist is not None:
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item()) / steps

    # the clock sampler starts before the warm-up (nvidia-smi needs a moment to produce its first
    # line, more so with eight GPUs in the box); only its samples under load are used
    sampler = ClockSampler(local)
    sampler.start()
    from flaggems_vllm_b200 import _lib as _native

    for _ in range(args.warmup):
        device_step()
    launches0 = _native.LAUNCHES
    ms = timed(device_step, args.steps, record_stages=(world == 1))
    launches = _native.LAUNCHES - launches0
    clocks = sampler.stop()
    if world == 1:
        prev = None
        for name, ev in stage_events:
            if name != "begin" and prev is not None:
                stage_ms.setdefault(name, []).append(prev.elapsed_time(ev))
            prev = ev
    status = fg.read_status(dev)

    # ---- expert parallel: where the step's time goes and what the all-to-alls achieve.  A few extra
    # steps with an event after every stage (outside the timed region above); bytes are the rows that
    # leave this GPU, the time of a collective includes waiting for the slowest peer to reach it.
    ep_stages = None
    if world > 1 and args.ep_chunks == 1:
        stage_events.clear()
        timed(device_step, 5, record_stages=True)
        per = {}
        prev = None
        for name, ev in stage_events:
            if name != "begin" and prev is not None:
                per.setdefault(name, []).append(prev.elapsed_time(ev))
            prev = ev
        med = {n: sorted(v)[len(v) // 2] for n, v in per.items()}
        nb = layer.last_bytes
        t = torch.tensor([med.get("ep_dispatch", 0.0), med.get("ep_combine", 0.0), float(nb["dispatch"]),
                          float(nb["combine"])], dtype=torch.float64, device=dev)
        tmax, tmin = t.clone(), t.clone()
        dist.all_reduce(tmax, op=dist.ReduceOp.MAX)
        dist.all_reduce(tmin, op=dist.ReduceOp.MIN)
        dist.all_reduce(t, op=dist.ReduceOp.SUM)
        mean = (t / world).tolist()

        def gbs(nbytes, ms_):
            return nbytes / (ms_ * 1e-3) / 1e9 if ms_ > 0 else None

        ep_stages = {
            "stage_ms_rank0": med,
            "a2a": {"dispatch_ms_max": float(tmax[0]), "dispatch_ms_min": float(tmin[0]),
                    "combine_ms_max": float(tmax[1]), "combine_ms_min": float(tmin[1]),
                    "dispatch_bytes_out_per_gpu": mean[2], "combine_bytes_out_per_gpu": mean[3],
                    "dispatch_gbs_per_gpu": gbs(mean[2], float(tmax[0])), "combine_gbs_per_gpu": gbs(mean[3], float(tmax[1])),
                    "dispatch_gbs_last_arriver": gbs(mean[2], float(tmin[0])),
                    "combine_gbs_last_arriver": gbs(mean[3], float(tmin[1])),
                    "nvlink_gbs_per_direction": {"nominal": 900.0, "measured_peer_copy": 770.0},
                    "note": "bytes leaving one GPU, one direction, / time inside the collective: `max` is the rank "
                            "that waited longest for its peers (load skew included), `min` the rank that arrived "
                            "last and saw the transfer alone"}}

    # ---- end to end with host buffers through the public API
    # Every step copies its activations and router logits from pinned host memory, runs the
    # public ops, and copies the layer output back to pinned host memory.  Two figures:
    #   serial    - copy in, compute, copy out on one stream (latency of an isolated step)
    #   pipelined - the same three phases on three streams with double-buffered device
    #               inputs, so step i+1's H2D and step i-1's D2H overlap step i's kernels
    #               (how a serving loop would drive it); reported as `e2e`.
    numa = bind_to_gpu_cpus(local) if world > 1 else None
    hx = torch.empty((M, H), dtype=torch.bfloat16).pin_memory()
    hl = torch.empty((M, E), dtype=torch.float32).pin_memory()
    hx.copy_(x.cpu())
    hl.copy_(logits.cpu())
    hout = [torch.empty((M, H), dtype=torch.bfloat16).pin_memory() for _ in range(2)]
    dx = [torch.empty_like(x) for _ in range(2)]
    dl = [torch.empty_like(logits) for _ in range(2)]

    def layer_call(xi, li):
        tw, ti = fg.grouped_topk(li, c["n_group"], c["topk_group"], k, True, c["rsf"], bias, 1)
        if layer is not None:
            return layer.forward(xi, tw, ti)
        return fg.fused_experts_impl(xi, w1, w2, tw, ti, use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2,
                                     block_shape=[128, 128])

    def e2e_serial_step():
        dx[0].copy_(hx, non_blocking=True)
        dl[0].copy_(hl, non_blocking=True)
        hout[0].copy_(layer_call(dx[0], dl[0]), non_blocking=True)

    for _ in range(3):
        e2e_serial_step()
    e2e_serial_ms = timed(e2e_serial_step, max(3, args.steps // 2))

    s_in, s_out = torch.cuda.Stream(), torch.cuda.Stream()
    s_comp = torch.cuda.current_stream()

    def e2e_pipelined(steps):
        """Returns total milliseconds for `steps` pipelined steps (device clock)."""
        in_ready = [torch.cuda.Event() for _ in range(2)]
        comp_done = [torch.cuda.Event() for _ in range(2)]
        out_done = [torch.cuda.Event() for _ in range(2)]
        keep = [None, None]
        barrier()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record(s_comp)
        s_in.wait_event(t0)
        s_out.wait_event(t0)
        for i in range(steps):
            b = i % 2
            with torch.cuda.stream(s_in):
                if i >= 2:
                    s_in.wait_event(comp_done[b])      # step i-2 has finished reading these inputs
                dx[b].copy_(hx, non_blocking=True)
                dl[b].copy_(hl, non_blocking=True)
                in_ready[b].record(s_in)
            s_comp.wait_event(in_ready[b])
            out = layer_call(dx[b], dl[b])
            comp_done[b].record(s_comp)
            with torch.cuda.stream(s_out):
                s_out.wait_event(comp_done[b])
                if i >= 2:
                    s_out.wait_event(out_done[b])
                out.record_stream(s_out)
                hout[b].copy_(out, non_blocking=True)
                out_done[b].record(s_out)
            keep[b] = out
        s_comp.wait_stream(s_out)
        s_comp.wait_stream(s_in)
        t1.record(s_comp)
        barrier()
        tt = torch.tensor([t0.elapsed_time(t1)], dtype=torch.float64, device=dev)
        if dist is not None:
            dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        return float(tt.item())

    e2e_pipelined(3)
    e2e_steps = max(4, args.steps)
    e2e_ms = e2e_pipelined(e2e_steps) / e2e_steps

    # What the host link alone allows: the same H2D and D2H copies of one step, both directions at
    # once, on every rank at the same time and with no kernels running (the ceiling of `e2e`).
    def copies_only(reps=5):
        barrier()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record(s_comp)
        s_in.wait_event(t0)
        s_out.wait_event(t0)
        for _ in range(reps):
            with torch.cuda.stream(s_in):
                dx[0].copy_(hx, non_blocking=True)
                dl[0].copy_(hl, non_blocking=True)
            with torch.cuda.stream(s_out):
                hout[0].copy_(dx[1], non_blocking=True)
        s_comp.wait_stream(s_in)
        s_comp.wait_stream(s_out)
        t1.record(s_comp)
        barrier()
        tt = torch.tensor([t0.elapsed_time(t1) / reps], dtype=torch.float64, device=dev)
        if dist is not None:
            dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        return float(tt.item())

    copies_only(2)
    copy_ms = copies_only()

    total_tokens = M * world
    flops = 6.0 * total_tokens * k * H * I
    value = total_tokens / (ms * 1e-3)
    line = {
        "metric": "fused_moe_layer_tokens_per_s", "value": value, "unit": "tokens/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "fp8_e4m3", "data": "synthetic",
        "config": {"workload": "deepseek_v3_fp8_block_moe_layer", "tokens_per_gpu": M, "global_tokens": total_tokens,
                   **c, "experts_per_gpu": E_local, "router_bias_std": args.router_bias_std, "parallelism": f"ep{world}" if world > 1 else "single", "ep_chunks": args.ep_chunks if world > 1 else None, "ep_overlap_combine": bool(args.ep_overlap) if world > 1 else None,
                   "l2": "flushed between iterations (252 MB memset); weights 11.3 GB >> L2"},
        "tflops": flops / (ms * 1e-3) / 1e12,
        "e2e": {"value": total_tokens / (e2e_ms * 1e-3), "unit": "tokens/s", "ms_per_step": e2e_ms,
                "h2d_bytes_per_step": hx.numel() * 2 + hl.numel() * 4, "d2h_bytes_per_step": hout[0].numel() * 2,
                "mode": "three streams, double-buffered: H2D / kernels / D2H of neighbouring steps overlap",
                "serial_ms_per_step": e2e_serial_ms, "serial_value": total_tokens / (e2e_serial_ms * 1e-3),
                "host_copies_only_ms_per_step": copy_ms,
                "host_copies_only_gbs_per_rank": (hx.numel() * 2 + hl.numel() * 4 + hout[0].numel() * 2) / (copy_ms * 1e-3) / 1e9,
                "host_copies_note": "one step's H2D and D2H copies alone, both directions at once on all ranks, no "
                                    "kernels: the ceiling the host link puts on e2e",
                "cpus_bound": numa},
        # kernel-launching calls into libmoe_sm100.so counted inside the timed region on this rank
        "gpu_launches": launches,
        "clocks": clocks, "kernel_status": status,
    }
    if world == 1:
        med = {n: sorted(v)[len(v) // 2] for n, v in stage_ms.items()}
        line["stage_ms"] = med
        # dominant kernel: GEMM1 (2*M*k*2I*H flop per launch); FP8 peak is not in
        # MEASURED_PEAKS.json, so 2x the measured bf16 burst figure is used
        g1 = sum(stage_ms["gemm1"]) / len(stage_ms["gemm1"])
        f1 = 2.0 * M * k * (2 * I) * H
        peak2x = 2.0 * peaks["bf16_tflops"]
        peak = fp8_peak if fp8_peak else peak2x
        # DRAM traffic of one GEMM1 launch: ncu (dram__bytes_read+write, one pass) on this workload, 8192
        # tokens and 256 experts, gave 8.66 + 0.17 GB for 7.713 GB of algorithmic bytes (weights of the experts in
        # use + e4m3 activations + scales + the e4m3 intermediate), a ratio of 1.145 (the sorted rows are
        # read eight times as often as the tokens); 32 experts and 1024 tokens give 1.10.
        _, ti0 = fg.grouped_topk(logits, c["n_group"], c["topk_group"], k, True, c["rsf"], bias, 1)
        e_act = int(torch.unique(ti0).numel())
        alg1 = e_act * (2 * I * H + (2 * I // 128) * (H // 128) * 4) + M * H + M * (H // 128) * 4 + M * k * I
        ach = f1 / (g1 * 1e-3) / 1e12
        line["roofline"] = {"kernel": "tc_gemm_kernel<fp8,gemm1>", "bound": "tensor", "achieved": ach,
                            "peak": peak, "unit": "TFLOP/s", "frac": ach / peak,
                            "peak_fp8_measured": fp8_peak, "frac_vs_2x_bf16": ach / peak2x,
                            "frac_of_sustained": ach / (2.0 * peaks["bf16_tflops_sustained"]),
                            "traffic": 1.145 * alg1, "traffic_source": "ncu DRAM bytes of this launch over its algorithmic bytes (x1.145)",
                            "algorithmic_bytes": alg1,
                            "peak_source": ("torch._scaled_mm e4m3 8192^3, best of 10, CUDA events, measured in this run"
                                            if fp8_peak else f"2 x bf16_tflops of {peaks['source']} peaks"),
                            "ms_per_launch": g1, "experts_in_use": e_act,
                            "layer_tflops": flops / (ms * 1e-3) / 1e12, "layer_frac": flops / (ms * 1e-3) / 1e12 / peak}
        wbytes = E * 3 * H * I + (E * (2 * I // 128) * (H // 128) + E * (H // 128) * (I // 128)) * 4
        B = wbytes + M * H * 2 * 2 + M * E * 4 + k * 8 * M
        line["layer_hbm"] = {"algorithmic_bytes": B, "achieved_gbs": B / (ms * 1e-3) / 1e9,
                             "peak_gbs": peaks["hbm_gbs"], "frac": B / (ms * 1e-3) / 1e9 / peaks["hbm_gbs"]}
    if ep_parity is not None:
        line["ep_parity"] = ep_parity
    if ep_stages is not None:
        line["ep_stages"] = ep_stages
    if rank == 0 and world == 1 and not args.no_cpu_baseline and E == DSV3["E"]:
        # same sample size as the reference arm; one sizing/warm-up pass, one timed pass
        Ms, step, threads, n_used, _ = fit_reference_tokens(args.cpu_baseline_tokens, 1, 1, 60.0)
        t0 = time.perf_counter()
        step()
        dt = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": Ms / dt, "unit": "tokens/s", "cores": threads, "kind": "port",
                                "ms_per_step": dt * 1e3,
                                "sample": f"{Ms} tokens of the same layer ({n_used} distinct experts; the GPU step is {M} "
                                          "tokens), one timed pass after one warm-up, CPU oracle (torch-native "
                                          "restatement of the reference goldens)"}
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist is not None:
        dist.destroy_process_group()
    if status != 0:
        print(f"kernel status word = {status} (a kernel reported a failure)", file=sys.stderr)
        sys.exit(3)
    if ep_parity is not None and not ep_parity["ok"]:
        print(f"expert-parallel parity check failed: {ep_parity}", file=sys.stderr)
        sys.exit(4)


if __name__ == "__main__":
    main()
