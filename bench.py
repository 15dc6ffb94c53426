#!/usr/bin/env python
"""Benchmark of the attention-forward hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--no-sweep]
    python -m torch.distributed.run --nnodes=1 --nproc-per-node N ... bench.py --gpus N ...

One "step" = one causal attention forward over one batch of the headline workload: the attention
problem of one GPT-2 XL layer at prefill, B=32 sequences PER GPU, H=25, N=1024, d=64, bf16
(weak scaling: every GPU gets its own batch; (batch, head) problems are independent, so there is no
collective on the data path -- NCCL is only used for the timing barrier and the max over ranks).
Inputs are synthetic (seeded N(0,1)); 420 MB per GPU, larger than the 126 MB L2.

Rank 0 prints ONE JSON line.  `value` is aggregate causal-adjusted TFLOP/s (2*B*H*N^2*d per
forward) with inputs resident in HBM; `e2e` is the same metric through the public
`custom_flash_attn.forward` call with host buffers (pinned host -> device copies of q, k, v and the
device -> host copy of O inside the timed region); `roofline` compares the kernel with the
measured bf16 tensor peak; `cpu_baseline` times the CPU oracle (a port of the reference's
standard-PyTorch attention) on a bounded sample on this box's host cores; `extra.sweep` holds the
other attention configurations (sharded over ranks by (batch, head)).

`--impl reference` runs the reference project's own implementation of the path instead -- its
CUDA kernel, compiled unmodified from the reference sources by oracle/build_ref.py and checked
against the CPU oracle on a small shape before it is timed -- on the same workload, metric and
unit, one replica per rank, and prints the same line with "impl": "reference"; its `cpu_baseline`
is the CPU port of the reference's standard-PyTorch attention on a bounded sample.  Where that
library is absent (it is built only where the reference sources are), the CPU port is what is timed.

The timed region of the headline is K steps repeated back to back until it spans at least 200 ms
(`timed_launches` of them; `ms_per_step` is the mean over all), so that the maximum over ranks is not
decided by a few microseconds of launch jitter; `roofline.sustained` is the same launch kept going
for two seconds with the clocks sampled through it.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

from tfg_flashattention_b200 import workloads  # noqa: E402

METRIC = "causal_attention_fwd_tflops"
UNIT = "TFLOP/s"
# DRAM bytes per launch of fa_fwd_kernel on the headline workload (dram__bytes_read.sum +
# dram__bytes_write.sum).  Captured with ncu at B=12 (118.03 + 19.01 MB per launch) and scaled by
# 32/12 to the benchmark's B=32: every (batch, head) is independent, so traffic grows in proportion.
NCU_TRAFFIC_BYTES_PER_LAUNCH = 137.04e6 * 32 / 12
NCU_TRAFFIC_NOTE = ("ncu capture at B=12 scaled by 32/12; reads equal Q+K+V exactly, writes are a lower bound "
                    "(part of O is still in L2 when the small capture's kernel ends)")
E2E_CHUNKS = 8                # batch slices the host-buffer call pipelines through PCIe
E2E_CHUNKS_MULTI = 4          # fewer, larger copies when several ranks share the host's memory system
CPU_SAMPLE_BATCH = 4          # batch entries (x25 heads) the CPU legs compute per repetition


def load_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            p = json.load(f)
        return {"bf16_tflops": float(p["bf16_tflops"]), "bf16_tflops_sustained": float(p.get("bf16_tflops_sustained", 0)),
                "hbm_gbs": float(p["hbm_gbs"]), "source": "measured"}
    except Exception:
        return {"bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0, "hbm_gbs": 6650.0, "source": "fallback"}


class ClockSampler:
    """Samples SM clock and throttle reasons of one GPU with nvidia-smi while a region runs."""
    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: str):
        self.index = index
        self.proc = None
        self.lines = []
        self.thread = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None
            return
        self.thread = threading.Thread(target=self._pump, daemon=True)
        self.thread.start()

    def _pump(self):
        for line in self.proc.stdout:
            self.lines.append((time.time(), line.strip()))

    def stop(self, t0=None, t1=None):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.15)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            pass
        rows = [l for (t, l) in self.lines if (t0 is None or t >= t0 - 0.05) and (t1 is None or t <= t1 + 0.15)]
        if not rows:
            rows = [l for (_, l) in self.lines]
        sm, smax, reasons, power = [], [], set(), []
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for r in rows:
            f = [x.strip() for x in r.split(",")]
            if len(f) < 8:
                continue
            try:
                sm.append(float(f[0])); smax.append(float(f[1])); power.append(float(f[2]))
            except ValueError:
                continue
            for name, val in zip(names, f[4:8]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "power_w_max": max(power) if power else None,
                "samples": len(sm), "reasons": sorted(reasons)}


def dist_setup(n_gpus):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    elif n_gpus > 1:
        raise SystemExit("--gpus N > 1 must be launched with torch.distributed.run (one rank per GPU)")
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()
    torch.cuda.synchronize()


def max_over_ranks(x: float, world: int) -> float:
    if world == 1:
        return x
    import torch.distributed as dist
    t = torch.tensor([x], device="cuda", dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def device_inputs(w, rank, heads=None):
    """bf16 device tensors of workload w (seed offset by rank for per-GPU batches)."""
    g = torch.Generator(device="cuda").manual_seed(w.seed + 1000 * rank)
    shape = (w.B, w.H, w.N, w.d) if heads is None else (heads, 1, w.N, w.d)
    q, k, v = (torch.randn(shape, device="cuda", generator=g, dtype=torch.float32).bfloat16() for _ in range(3))
    if w.stress_k_rows:
        idx = torch.randperm(w.N, device="cuda", generator=g)[: max(1, w.N // 100)]
        k[:, :, idx, :] *= 4.0
    return q, k, v


def n_input_sets(q):
    """How many copies of (q, k, v, o) to rotate through so that consecutive launches cannot be
    served from the 126 MB L2: enough for 400 MB in total, at most 8."""
    one_set = 4 * q.numel() * 2
    return max(1, min(8, -(-400_000_000 // one_set)))


def gather_over_ranks(x: float, world: int):
    if world == 1:
        return [x]
    import torch.distributed as dist
    t = torch.tensor([x], device="cuda", dtype=torch.float64)
    out = [torch.zeros_like(t) for _ in range(world)]
    dist.all_gather(out, t)
    return [float(o.item()) for o in out]


def time_kernel(cfa, q, k, v, causal, steps, warmup, world, min_window_ms=0.0, detail=None):
    """ms per step, max over ranks; CUDA events on the launching (current torch) stream.  Small
    problems rotate through several copies of their inputs (n_input_sets).  With min_window_ms the
    block of `steps` launches is repeated back to back (same event pair) until the timed region is
    at least that long; `detail`, a dict, receives the launch count and the per-rank figures."""
    sets = [(q, k, v, torch.empty_like(q))]
    for _ in range(n_input_sets(q) - 1):
        sets.append((q.clone(), k.clone(), v.clone(), torch.empty_like(q)))
    n = len(sets)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for i in range(max(warmup, n)):
        qq, kk, vv, oo = sets[i % n]
        cfa.forward(qq, kk, vv, causal=causal, out=oo)
    torch.cuda.synchronize()
    repeats = 1
    if min_window_ms > 0:
        e0.record()                      # a second, already warm block sizes the timed region
        for i in range(n):
            qq, kk, vv, oo = sets[i % n]
            cfa.forward(qq, kk, vv, causal=causal, out=oo)
        e1.record()
        torch.cuda.synchronize()
        est = max_over_ranks(e0.elapsed_time(e1) / n, world)                   # same count on every rank
        repeats = max(1, int(-(-min_window_ms // max(est * steps, 1e-6))))
    launches = steps * repeats
    barrier(world)
    e0.record()
    for i in range(launches):
        qq, kk, vv, oo = sets[i % n]
        cfa.forward(qq, kk, vv, causal=causal, out=oo)
    e1.record()
    barrier(world)
    ms = e0.elapsed_time(e1) / launches
    if detail is not None:
        detail["timed_launches"] = launches
        detail["ms_per_step_by_rank"] = [round(x, 5) for x in gather_over_ranks(ms, world)]
    return max_over_ranks(ms, world)


def time_sustained(cfa, q, k, v, seconds, sampler_id):
    """The headline launch back to back for `seconds`, clocks sampled through it (this rank only):
    what the kernel holds once power and temperature have settled, next to the burst figure."""
    sets = [(q, k, v, torch.empty_like(q))]
    sampler = ClockSampler(sampler_id)
    sampler.start()
    time.sleep(0.3)
    torch.cuda.synchronize()
    t0 = time.time()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    launches = 0
    e0.record()
    while time.time() - t0 < seconds:
        for _ in range(200):
            cfa.forward(q, k, v, causal=True, out=sets[0][3])
        launches += 200
    e1.record()
    torch.cuda.synchronize()
    t1 = time.time()
    clocks = sampler.stop(t0, t1)
    return e0.elapsed_time(e1) / launches, launches, clocks


def bind_near_gpu(local):
    """Run this rank (and so allocate its pinned host buffers, first touch) on the cores nearest
    its GPU, as `nvidia-smi topo -m` reports them.  Returns the CPU set used, or None."""
    try:
        out = subprocess.run(["nvidia-smi", "topo", "-m"], capture_output=True, text=True, timeout=20).stdout
        for line in out.splitlines():
            f = line.split()
            if f and f[0] == f"GPU{local}":
                for tok in f[1:]:
                    if tok[0].isdigit() and ("-" in tok or "," in tok):
                        cpus = set()
                        for part in tok.split(","):
                            lo, _, hi = part.partition("-")
                            cpus.update(range(int(lo), int(hi or lo) + 1))
                        os.sched_setaffinity(0, cpus)
                        return tok
    except Exception:
        pass
    return None


def time_e2e(cfa, w, rank, steps, warmup, world, detail=None):
    """ms per step through the public host-buffer call (custom_flash_attn.forward_host): pinned
    q, k, v -> device, forward, O -> pinned host, all inside the timed region; the call cuts the
    batch into slices so that uploads, kernels and downloads overlap."""
    qd, kd, vd = device_inputs(w, rank)
    hq, hk, hv = (t.cpu().pin_memory() for t in (qd, kd, vd))
    ho = torch.empty_like(hq).pin_memory()
    del qd, kd, vd

    def step():
        # the public host-buffer call: chunked upload / kernel / download pipeline
        cfa.forward_host(hq, hk, hv, out=ho, chunks=E2E_CHUNKS if world == 1 else E2E_CHUNKS_MULTI)

    for _ in range(max(1, warmup)):
        step()
    barrier(world)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        step()
    e1.record()
    barrier(world)
    mine = e0.elapsed_time(e1) / steps
    ms = max_over_ranks(mine, world)
    nbytes = hq.numel() * 2
    if detail is not None:
        detail["ms_per_step_by_rank"] = [round(x, 3) for x in gather_over_ranks(mine, world)]
        detail["host_link_gbs_by_rank"] = [round(4 * nbytes / (x * 1e-3) / 1e9, 1)
                                           for x in gather_over_ranks(mine, world)]
    return ms, 3 * nbytes, nbytes


def time_add_layernorm(rows, cols, steps, warmup):
    """s = a + resid (written in place over resid), y = LayerNorm(s): 4 * rows * cols * 2 algorithmic
    bytes per launch.  Buffer sets are rotated so that no launch finds its inputs in L2."""
    from tfg_flashattention_b200.block_ops import add_layernorm
    g = torch.Generator(device="cuda").manual_seed(13)
    one_set = 3 * rows * cols * 2
    n_sets = max(2, min(8, int(400e6 // one_set) + 1))
    sets = [(torch.randn(rows, cols, device="cuda", generator=g).bfloat16(),
             torch.randn(rows, cols, device="cuda", generator=g).bfloat16(),
             torch.empty(rows, cols, device="cuda", dtype=torch.bfloat16)) for _ in range(n_sets)]
    scale = torch.ones(cols, device="cuda", dtype=torch.bfloat16)
    shift = torch.zeros(cols, device="cuda", dtype=torch.bfloat16)
    def step(i):
        a, x, y = sets[i % n_sets]
        add_layernorm(a, x, scale, shift, 1e-5, sum_out=x, norm_out=y)
    for i in range(warmup):
        step(i)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for i in range(steps):
        step(i)
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / steps
    return {"rows": rows, "cols": cols, "us_per_launch": round(ms * 1e3, 2),
            "gbs": round(4.0 * rows * cols * 2 / (ms * 1e-3) / 1e9, 1), "buffer_sets_rotated": n_sets,
            "kernel": "fa::fa_add_layernorm_kernel"}


def time_linear_small(M, N, K, steps, warmup):
    """y = x W^T + b for M rows, one pass over W (N * K * 2 algorithmic bytes per launch).  Enough
    different weight matrices are rotated that no launch finds its weights in L2."""
    from tfg_flashattention_b200.block_ops import linear_small
    g = torch.Generator(device="cuda").manual_seed(17)
    n_sets = max(2, min(32, -(-300_000_000 // (N * K * 2))))
    ws = [(torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16() for _ in range(n_sets)]
    b = torch.randn(N, device="cuda", generator=g).bfloat16()
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    y = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    for i in range(max(warmup, 3)):
        linear_small(x, ws[i % n_sets], b, out=y)
    torch.cuda.synchronize()
    # the kernel lives inside CUDA graphs in generation (a launch from Python costs more than the
    # kernel runs): record `steps` launches as one graph and time its replay
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for i in range(steps):
            linear_small(x, ws[i % n_sets], b, out=y)
    graph.replay()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    graph.replay()
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / steps
    return {"M": M, "N": N, "K": K, "us_per_launch": round(ms * 1e3, 2),
            "gbs": round(N * K * 2 / (ms * 1e-3) / 1e9, 1), "weight_sets_rotated": n_sets,
            "timing": "one CUDA-graph replay of all launches", "kernel": "fa::fa_linear_small_kernel"}


def cpu_attention_sample(w, reps, threads):
    """Time the CPU oracle on CPU_SAMPLE_BATCH batch entries of workload w.  Returns TFLOP/s."""
    from oracle.attention_oracle import manual_attention
    torch.set_num_threads(threads)
    bs = min(CPU_SAMPLE_BATCH, w.B)
    g = torch.Generator().manual_seed(w.seed)
    q, k, v = (torch.randn(bs, w.H, w.N, w.d, generator=g) for _ in range(3))
    flops = 2.0 * bs * w.H * w.N * w.N * w.d
    manual_attention(q[:1], k[:1], v[:1], causal=True)           # warm the thread pool
    times = []
    for _ in range(reps):
        t0 = time.perf_counter()
        manual_attention(q, k, v, causal=True)
        times.append(time.perf_counter() - t0)
    return flops / statistics.median(times) / 1e12, bs, times


def bench_config(w):
    """The workload description both arms print."""
    return {"workload": "gpt2-xl-layer-attention (config 4 attention shape)",
            "B_per_gpu": w.B, "H": w.H, "N": w.N, "d": w.d, "causal": True,
            "flops_convention": "causal-adjusted 2*B*H*N^2*d",
            "l2_policy": "inputs (420 MB per GPU) larger than L2 (126 MB)",
            "sharding": "independent (batch, head) problems per GPU, no collective"}


def time_rotating(fn, q, k, v, steps, warmup):
    """ms per call of fn(q, k, v, out) on this rank, rotating input copies like time_kernel."""
    sets = [(q, k, v, torch.empty_like(q))]
    for _ in range(n_input_sets(q) - 1):
        sets.append((q.clone(), k.clone(), v.clone(), torch.empty_like(q)))
    n = len(sets)
    for i in range(max(warmup, n)):
        fn(*sets[i % n])
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for i in range(steps):
        fn(*sets[i % n])
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / steps


def reference_kernel_checked():
    """The reference project's CUDA kernel (oracle/_ref), or None with a reason.  Before anything
    is timed it is run once on a small ragged shape and compared with the CPU oracle."""
    from oracle import ref_kernel
    if not ref_kernel.available():
        return None, "oracle/_ref/libref_v1.so absent (built by oracle/build_ref.py where the reference sources are)"
    if not torch.cuda.is_available():
        return None, "no CUDA device"
    from oracle.attention_oracle import manual_attention
    g = torch.Generator().manual_seed(5)
    q, k, v = (torch.randn(2, 3, 200, 64, generator=g).bfloat16() for _ in range(3))
    o = ref_kernel.forward(q.cuda(), k.cuda(), v.cuda()).float().cpu()
    ref = manual_attention(q.float(), k.float(), v.float(), causal=True)
    err = (o - ref).abs().max().item()
    if not err <= 2e-2:
        return None, f"reference kernel disagrees with the oracle on the check shape (max-abs {err:.3e})"
    return ref_kernel, None


def run_comparators(cfa, peaks):
    """Other implementations of the same problem, timed on this rank in the same run (timing only):
    torch's scaled_dot_product_attention -- what every reference test compares with
    (test/py/test_cuda_implementation.py:49-52, 83, 112) -- with its default, flash and cuDNN
    back ends, and the reference project's own CUDA kernel (always causal)."""
    import torch.nn.functional as F
    from torch.nn.attention import SDPBackend, sdpa_kernel
    ref_kernel, why = reference_kernel_checked()
    rows = []
    shapes = [("headline B=32 H=25 N=1024", workloads.config4_attention()), ("config 1", workloads.config1()),
              ("config 3 N=4096", workloads.config3(4096, True)), ("config 3 N=4096", workloads.config3(4096, False))]
    for label, w in shapes:
        q, k, v = device_inputs(w, 0)
        steps = 20 if w.N <= 1024 else 8
        row = {"workload": label, "B": w.B, "H": w.H, "N": w.N, "causal": w.causal}
        def tf(ms):
            return round(w.flops() / (ms * 1e-3) / 1e12, 1)
        ms = time_rotating(lambda a, b, c, o: cfa.forward(a, b, c, causal=w.causal, out=o), q, k, v, steps, 3)
        row["this_library"] = {"ms": round(ms, 4), "tflops": tf(ms)}
        for name, backend in (("sdpa_default", None), ("sdpa_flash", SDPBackend.FLASH_ATTENTION),
                              ("sdpa_cudnn", SDPBackend.CUDNN_ATTENTION)):
            try:
                fn = lambda a, b, c, o: F.scaled_dot_product_attention(a, b, c, is_causal=w.causal)
                if backend is None:
                    ms = time_rotating(fn, q, k, v, steps, 3)
                else:
                    with sdpa_kernel(backend):
                        ms = time_rotating(fn, q, k, v, steps, 3)
                row[name] = {"ms": round(ms, 4), "tflops": tf(ms)}
            except Exception as e:   # a back end that refuses the shape
                row[name] = {"unavailable": str(e).splitlines()[0][:120]}
        if not w.causal:
            row["reference_v1_kernel"] = {"unavailable": "the reference kernel is always causal"}
        elif ref_kernel is None:
            row["reference_v1_kernel"] = {"unavailable": why}
        else:
            ms = time_rotating(lambda a, b, c, o: ref_kernel.forward(a, b, c, out=o), q, k, v, 3, 1)
            row["reference_v1_kernel"] = {"ms": round(ms, 3), "tflops": tf(ms)}
        for name in ("sdpa_default", "sdpa_flash", "sdpa_cudnn", "reference_v1_kernel"):
            if "ms" in row[name]:
                row[name]["this_library_speedup"] = round(row[name]["ms"] / row["this_library"]["ms"], 2)
        rows.append(row)
        del q, k, v
        torch.cuda.empty_cache()
    return rows


def run_reference(args, w):
    """The reference arm.  The reference's implementation of this path is its CUDA kernel
    (src/cpp/v1.cu + headers/v1_implementation.hpp): it is what is timed, one replica per rank on
    the same workload, `value` with inputs resident in HBM and `e2e` through host buffers (pinned
    host -> device copies of q, k, v, kernel, device -> host copy of O inside the timed region,
    which is what a caller of the reference binding with host data has to do).  `cpu_baseline` is
    the CPU port of the reference's standard-PyTorch attention on a bounded sample (rank 0).
    Where the reference kernel is not available the CPU port is what is timed, on rank 0 alone."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    ref_kernel, why = reference_kernel_checked() if torch.cuda.is_available() else (None, "no CUDA device")
    threads = os.cpu_count() or 1
    if ref_kernel is None:
        if rank != 0:
            return
        tf, bs, times = cpu_attention_sample(w, reps=max(1, args.steps), threads=threads)
        sample = f"{bs} of {w.B} batch entries ({bs * w.H} of {w.B * w.H} heads) per step, fp32, torch CPU"
        dt = statistics.median(times)
        line = {
            "impl": "reference", "metric": METRIC, "value": tf, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "config": bench_config(w),
            "note": f"reference CUDA kernel unavailable ({why}): CPU port timed on rank 0 only, value does not scale with --gpus",
            "cpu_baseline": {"value": tf, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample},
            "e2e": {"value": tf, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "gpu_launches": 0,
        }
        print(json.dumps(line), flush=True)
        return

    world, rank, local = dist_setup(args.gpus)
    torch.cuda.set_device(local)
    # the reference launcher launches on the current device's legacy default stream (v1.cu:33-34;
    # its query of device 0's properties, :7-8, only feeds dead code): one replica per rank
    q, k, v = device_inputs(w, rank)
    o = torch.empty_like(q)
    # at least three untimed launches: the first ones of this 50 ms kernel run at the clocks of an
    # idle GPU and were seen to take half again as long
    steps, warmup = max(1, args.steps), max(3, args.warmup)
    for _ in range(warmup):
        ref_kernel.forward(q, k, v, out=o)
    barrier(world)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        ref_kernel.forward(q, k, v, out=o)
    e1.record()
    barrier(world)
    ms = max_over_ranks(e0.elapsed_time(e1) / steps, world)
    value = world * w.flops() / (ms * 1e-3) / 1e12
    # end to end with host buffers
    hq, hk, hv = (t.cpu().pin_memory() for t in (q, k, v))
    ho = torch.empty_like(hq).pin_memory()
    def e2e_step():
        dq, dk, dv = (t.to("cuda", non_blocking=True) for t in (hq, hk, hv))
        ho.copy_(ref_kernel.forward(dq, dk, dv), non_blocking=True)
    e2e_step()
    barrier(world)
    n_e2e = max(2, min(steps, 5))
    e0.record()
    for _ in range(n_e2e):
        e2e_step()
    e1.record()
    barrier(world)
    e2e_ms = max_over_ranks(e0.elapsed_time(e1) / n_e2e, world)
    nbytes = hq.numel() * 2
    cpu = None
    if rank == 0:
        tf, bs, times = cpu_attention_sample(w, reps=3, threads=threads)
        cpu = {"value": tf, "unit": UNIT, "cores": threads, "kind": "port",
               "sample": f"{bs} of {w.B} batch entries ({bs * w.H} of {w.B * w.H} heads), median of "
                         f"{len(times)} repetitions, fp32 torch CPU (the reference's standard-PyTorch branch)"}
        line = {
            "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": steps, "warmup": warmup, "ms_per_step": ms, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
            "config": bench_config(w),
            "note": "the reference project's own CUDA kernel (flash_attention_forward_kernel<32,32,2,64,bf16>, "
                    "fp32 FMA, no tensor cores), compiled unmodified for sm_100a, one replica per rank",
            "reference_kind": "reference CUDA kernel (oracle/_ref/libref_v1.so)",
            "cpu_baseline": cpu,
            "e2e": {"value": world * w.flops() / (e2e_ms * 1e-3) / 1e12, "unit": UNIT, "ms_per_step": e2e_ms,
                    "h2d_bytes_per_step": 3 * nbytes, "d2h_bytes_per_step": nbytes},
            "gpu_launches": steps,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-sweep", action="store_true", help="skip the extra configurations")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--no-sustained", action="store_true",
                    help="skip the two-second sustained leg and the 200 ms minimum window (runs under a profiler)")
    ap.add_argument("--decode-case", default=None, metavar="B,H,kv_len",
                    help="time only this decode step (small runs for profilers); prints a short line")
    ap.add_argument("--ln-case", default=None, metavar="rows,cols",
                    help="time only the residual add + LayerNorm kernel on this shape (for profiling)")
    ap.add_argument("--linear-case", default=None, metavar="M,N,K",
                    help="time only the few-rows Linear kernel on this shape (for profiling)")
    ap.add_argument("--case", default=None, metavar="B,H,N,causal",
                    help="time only this attention problem (small runs for profilers); prints a short line")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3) if args.impl == "ours" else args.warmup

    w = workloads.config4_attention()
    if args.impl == "reference":
        run_reference(args, w)
        return

    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device: the attention kernel has no CPU fallback")
    world, rank, local = dist_setup(args.gpus)
    torch.cuda.set_device(local)
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    peaks = load_peaks()

    if args.decode_case:
        db, dh, dn = (int(x) for x in args.decode_case.split(","))
        g = torch.Generator(device="cuda").manual_seed(11)
        dq = torch.randn(db, dh, 64, device="cuda", generator=g).bfloat16()
        n_sets = max(1, min(8, int(400e6 // (2 * db * dh * dn * 128)) + 1))
        caches = [(torch.randn(db, dh, dn, 64, device="cuda", generator=g).bfloat16(),
                   torch.randn(db, dh, dn, 64, device="cuda", generator=g).bfloat16()) for _ in range(n_sets)]
        do = torch.empty_like(dq)
        for i in range(args.warmup):
            cfa.decode(dq, *caches[i % n_sets], dn, out=do)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for i in range(args.steps):
            cfa.decode(dq, *caches[i % n_sets], dn, out=do)
        e1.record()
        torch.cuda.synchronize()
        dms = e0.elapsed_time(e1) / args.steps
        print(json.dumps({"decode_case": args.decode_case, "us_per_step": dms * 1e3,
                          "gbs": 2.0 * db * dh * dn * 128 / (dms * 1e-3) / 1e9,
                          "status": cfa.last_status()}), flush=True)
        return

    if args.ln_case:
        lr, lc = (int(x) for x in args.ln_case.split(","))
        print(json.dumps({"ln_case": args.ln_case, **time_add_layernorm(lr, lc, args.steps, args.warmup)}), flush=True)
        return

    if args.linear_case:
        lm, ln_, lk = (int(x) for x in args.linear_case.split(","))
        print(json.dumps({"linear_case": args.linear_case, **time_linear_small(lm, ln_, lk, args.steps, args.warmup)}), flush=True)
        return

    if args.case:
        cb, ch, cn, cc = (int(x) for x in args.case.split(","))
        cw = workloads.AttnWorkload("case", cb, ch, cn, seed=5, causal=bool(cc))
        cq, ck, cv = device_inputs(cw, rank)
        cms = time_kernel(cfa, cq, ck, cv, cw.causal, args.steps, args.warmup, world)
        if rank == 0:
            print(json.dumps({"case": args.case, "ms_per_step": cms, "tflops": cw.flops() / cms / 1e9,
                              "status": cfa.last_status()}), flush=True)
        return

    # ---------------------------------------------------------------- headline: kernel, HBM-resident
    q, k, v = device_inputs(w, rank)
    try:
        gpu_id = "GPU-" + str(torch.cuda.get_device_properties(torch.cuda.current_device()).uuid)
    except Exception:
        gpu_id = str(torch.cuda.current_device())
    # first the K steps alone, from an idle GPU: the burst figure (a few milliseconds at the full
    # clock); then the timed region proper, long enough for the power limit to be felt
    burst_ms = time_kernel(cfa, q, k, v, True, args.steps, args.warmup, world)
    burst = {"tflops_per_gpu": round(w.flops() / (burst_ms * 1e-3) / 1e12, 1), "ms_per_step": round(burst_ms, 5),
             "launches": args.steps, "frac_of_burst_peak": round(w.flops() / (burst_ms * 1e-3) / 1e12 / peaks["bf16_tflops"], 4)}
    sampler = ClockSampler(gpu_id)
    sampler.start()
    time.sleep(0.3)
    t0 = time.time()
    headline = {}
    ms = time_kernel(cfa, q, k, v, True, args.steps, args.warmup, world,
                     min_window_ms=0.0 if args.no_sustained else 200.0, detail=headline)
    t1 = time.time()
    clocks = sampler.stop(t0, t1)
    status = cfa.last_status()
    if status != 0:
        raise SystemExit(f"kernel watchdog reported {status:#x}")
    flops = w.flops()
    value = world * flops / (ms * 1e-3) / 1e12
    per_gpu = value / world
    del q, k, v

    # ---------------------------------------------------------------- end to end with host buffers
    cpu_set = bind_near_gpu(local) if world > 1 else None
    e2e_detail = {"cpu_affinity": cpu_set, "chunks": E2E_CHUNKS if world == 1 else E2E_CHUNKS_MULTI}
    e2e_ms, h2d, d2h = time_e2e(cfa, w, rank, max(3, min(args.steps, 10)), 2, world, detail=e2e_detail)
    e2e_value = world * flops / (e2e_ms * 1e-3) / 1e12

    # ---------------------------------------------------------------- the other attention configs
    sweep = []
    if not args.no_sweep:
        cases = [workloads.config1()]
        cases += [workloads.config3(n, c) for n in (512, 1024, 2048, 4096) for c in (True, False)]
        cases += [workloads.config5(n) for n in (8192, 16384, 32768)]
        for cw in cases:
            sl = workloads.shard_heads(cw.B * cw.H, world, rank)
            heads = sl.stop - sl.start
            steps = 20 if cw.N <= 4096 else (8 if cw.N <= 8192 else 4)
            if heads > 0:
                cq, ck, cv = device_inputs(cw, rank, heads=heads)
                n_sets = n_input_sets(cq)
                cms = time_kernel(cfa, cq, ck, cv, cw.causal, steps, 3, world)
                del cq, ck, cv
            else:
                n_sets = 0
                barrier(world); barrier(world)
                cms = max_over_ranks(0.0, world)
            tf = cw.flops() / (cms * 1e-3) / 1e12
            sweep.append({"workload": cw.name, "B": cw.B, "H": cw.H, "N": cw.N, "causal": cw.causal,
                          "ms": round(cms, 4), "tflops": round(tf, 1),
                          "frac_of_peak_per_gpu": round(tf / world / peaks["bf16_tflops"], 4),
                          "input_sets_rotated": n_sets})
        if cfa.last_status() != 0:
            raise SystemExit("kernel watchdog fired during the sweep")

    # ---------------------------------------------------------------- GPT-2 prefill (the callers)
    prefill = []
    if not args.no_sweep:
        from tfg_flashattention_b200 import gpt2
        for name, batch, seed, steps in (("gpt2-small", 8, 1, 7), ("gpt2-xl", 32, 3, 5)):
            cfg = gpt2.gpt2_config(name, impl_type="cuda")
            model = gpt2.init_random(gpt2.GPTModel(cfg, dtype=torch.bfloat16), seed=seed).cuda().eval()
            model.prepare_for_inference()     # fused QKV GEMM, vocabulary padded to a multiple of 64
            ids = torch.randint(0, cfg["vocab_size"], (batch, 1024),
                                generator=torch.Generator().manual_seed(seed + rank)).cuda()
            def timed_forwards(fwd):
                # one event pair per forward; the median is robust against a first-use stall
                # (cuBLAS kernel loading, allocator growth) landing inside the timed steps
                for _ in range(3):
                    fwd(ids)
                barrier(world)
                evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
                       for _ in range(steps)]
                for e0, e1 in evs:
                    e0.record()
                    fwd(ids)
                    e1.record()
                barrier(world)
                times = [e0.elapsed_time(e1) for e0, e1 in evs]
                return (max_over_ranks(statistics.median(times), world),
                        max_over_ranks(sum(times) / len(times), world))
            with torch.no_grad():
                eager_ms, _ = timed_forwards(model)
                # the same forward recorded once as a CUDA graph and replayed: every step still
                # copies the token ids in and runs all kernels, only the host launch gaps go
                graphed = model.capture_prefill(batch, 1024)
                pms, pms_mean = timed_forwards(graphed)
                logits = graphed(ids)
            tok_s = world * batch * 1024 / (pms * 1e-3)
            prefill.append({"model": name, "batch_per_gpu": batch, "seq_len": 1024, "dtype": "bf16",
                            "weights": f"random N(0,0.02) seed {seed}", "ms_per_forward": round(pms, 3), "ms_per_forward_mean": round(pms_mean, 3), "timing": f"median of {steps} forwards, CUDA events; one CUDA-graph replay per forward",
                            "ms_per_forward_eager": round(eager_ms, 3),
                            "tokens_per_s": round(tok_s, 1),
                            "model_tflops_per_gpu": round(tok_s / world * gpt2.prefill_flops_per_token(cfg, 1024) / 1e12, 1),
                            "attention": "fa::fa_fwd_kernel on strided [B,N,H,d] views, every layer",
                            "block_ops": "fa::fa_add_layernorm_kernel (residual add + LayerNorm), GELU in the cuBLASLt GEMM epilogue, fused QKV GEMM",
                            "logits": "all positions"})
            del graphed
            del model, ids, logits
            torch.cuda.empty_cache()
        if cfa.last_status() != 0:
            raise SystemExit("kernel watchdog fired during the prefill runs")

    # ---------------------------------------------------------------- decode step (KV-cache attention)
    decode = []
    if not args.no_sweep:
        for (db, dh, dn) in ((32, 25, 1024), (1, 25, 1024), (8, 25, 8192)):
            g = torch.Generator(device="cuda").manual_seed(11 + rank)
            dq = torch.randn(db, dh, 64, device="cuda", generator=g).bfloat16()
            # several cache sets rotated between launches so that K/V come from HBM, not from L2
            n_sets = max(1, min(8, int(400e6 // (2 * db * dh * dn * 128)) + 1))
            caches = [(torch.randn(db, dh, dn, 64, device="cuda", generator=g).bfloat16(),
                       torch.randn(db, dh, dn, 64, device="cuda", generator=g).bfloat16())
                      for _ in range(n_sets)]
            do = torch.empty_like(dq)
            for i in range(5):
                cfa.decode(dq, *caches[i % n_sets], dn, out=do)
            barrier(world)
            steps = 40
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for i in range(steps):
                cfa.decode(dq, *caches[i % n_sets], dn, out=do)
            e1.record()
            barrier(world)
            dms = max_over_ranks(e0.elapsed_time(e1) / steps, world)
            nbytes = 2.0 * db * dh * dn * 128                      # K and V read once
            decode.append({"B_per_gpu": db, "H": dh, "kv_len": dn, "us_per_step": round(dms * 1e3, 2),
                           "gbs_per_gpu": round(nbytes / (dms * 1e-3) / 1e9, 1),
                           "frac_of_hbm_peak": round(nbytes / (dms * 1e-3) / 1e9 / peaks["hbm_gbs"], 3),
                           "cache_sets_rotated": n_sets,
                           "kernels": "fa::fa_decode_kernel"})
            del caches, dq, do
            torch.cuda.empty_cache()
        if cfa.last_status() != 0:
            raise SystemExit("kernel watchdog fired during the decode runs")

    # ---------------------------------------------------------------- residual add + LayerNorm kernel
    add_ln = []
    if not args.no_sweep:
        for rows, cols in ((32 * 1024, 1600), (8 * 1024, 768)):      # GPT-2 XL B=32 and small B=8 prefill
            r = time_add_layernorm(rows, cols, 40, 5)
            r["frac_of_hbm_peak"] = round(r["gbs"] / peaks["hbm_gbs"], 3)
            add_ln.append(r)

    # ---------------------------------------------------------------- Linear for one row (generation)
    lin = []
    if not args.no_sweep:
        for M, N, K in ((1, 4800, 1600), (1, 1600, 6400), (1, 50257, 1600)):   # GPT-2 XL: QKV, MLP-proj, head
            r = time_linear_small(M, N, K, 100, 10)
            r["frac_of_hbm_peak"] = round(r["gbs"] / peaks["hbm_gbs"], 3)
            lin.append(r)

    # ---------------------------------------------------------------- the reference's own benchmark
    # "time for 20 tokens" (model_inference.py:444-465): B=1, a ~70-token prompt, 20 new tokens,
    # here with random-init weights and random token ids; with the K/V cache and the one-launch step,
    # and with the reference's recompute loop through the prefill kernel.
    gen = []
    if not args.no_sweep and rank == 0:
        from tfg_flashattention_b200 import gpt2
        for name, seed, gb, gp in (("gpt2-small", 1, 1, 72), ("gpt2-xl", 3, 1, 72), ("gpt2-xl", 3, 8, 900)):
            cfg = gpt2.gpt2_config(name, impl_type="cuda")
            model = gpt2.init_random(gpt2.GPTModel(cfg, dtype=torch.bfloat16), seed=seed).cuda().eval()
            model.prepare_for_inference()
            prompt = torch.randint(0, cfg["vocab_size"], (gb, gp), generator=torch.Generator().manual_seed(123)).cuda()
            row = {"model": name, "prompt_tokens": gp, "new_tokens": 20, "batch": gb, "dtype": "bf16",
                   "note": "a step is one kernel launch (fa_b200_gpt_step), the prompt runs eagerly; "
                           "kv_cache_graph_ms: with a GenerationSession kept across calls, kv_cache_ms: default arguments"}
            session = gpt2.GenerationSession(model, gb, 1024)      # caches + recorded decode step, reused
            for label, kw in (("kv_cache_graph_ms", {"session": session}), ("kv_cache_ms", {}),
                              ("recompute_ms", {"use_cache": False})):
                gpt2.generate(model, prompt, 20, 1024, temperature=0.0, **kw)
                torch.cuda.synchronize()
                times = []
                for _ in range(3):
                    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                    e0.record()
                    gpt2.generate(model, prompt, 20, 1024, temperature=0.0, **kw)
                    e1.record()
                    torch.cuda.synchronize()
                    times.append(e0.elapsed_time(e1))
                row[label] = round(statistics.median(times), 2)
            del session
            gen.append(row)
            del model
            torch.cuda.empty_cache()
    if world > 1:
        barrier(world)

    # ---------------------------------------------------------------- a small problem: host cost vs kernel
    small = None
    comparators = None
    if not args.no_sweep and rank == 0 and world == 1:
        cw = workloads.config1()
        cq, ck, cv = device_inputs(cw, rank)
        co = torch.empty_like(cq)
        for _ in range(5):
            cfa.forward(cq, ck, cv, out=co)
        torch.cuda.synchronize()
        # host time of one call: launches into an idle stream, nothing to wait for
        t_host = []
        for _ in range(200):
            torch.cuda.synchronize()
            h0 = time.perf_counter()
            cfa.forward(cq, ck, cv, out=co)
            t_host.append(time.perf_counter() - h0)
        # kernel alone: the launches recorded once as a CUDA graph and replayed
        n_rec = 50
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(n_rec):
                cfa.forward(cq, ck, cv, out=co)
        graph.replay()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        graph.replay()
        e1.record()
        torch.cuda.synchronize()
        g_us = e0.elapsed_time(e1) / n_rec * 1e3
        e_ms = time_rotating(lambda a, b, c, o: cfa.forward(a, b, c, out=o), cq, ck, cv, 200, 5)
        small = {"workload": "config 1 (B=4 H=12 N=1024 causal)",
                 "host_us_per_call_median": round(statistics.median(t_host) * 1e6, 2),
                 "eager_us_per_launch": round(e_ms * 1e3, 2),
                 "eager_tflops": round(cw.flops() / (e_ms * 1e-3) / 1e12, 1),
                 "graph_replay_us_per_launch": round(g_us, 2),
                 "graph_replay_tflops": round(cw.flops() / (g_us * 1e-6) / 1e12, 1),
                 "note": "graph replay: same buffers every launch (25 MB, L2-resident); eager: rotating copies"}
        del graph, cq, ck, cv, co
        comparators = run_comparators(cfa, peaks)
        if cfa.last_status() != 0:
            raise SystemExit("kernel watchdog fired during the comparator runs")

    # ---------------------------------------------------------------- sustained leg (last GPU leg)
    # the headline launch kept going for two seconds: what it holds at settled clocks and power.
    # It comes after every other leg, because it leaves the GPU at its power limit for a while.
    q, k, v = device_inputs(w, rank)
    sus_ms, sus_launches, sus_clocks = time_sustained(cfa, q, k, v, 0.02 if args.no_sustained else 2.0, gpu_id)
    sus_tf = flops / (sus_ms * 1e-3) / 1e12
    sustained = {"tflops": round(sus_tf, 1), "ms_per_launch": round(sus_ms, 5), "launches": sus_launches,
                 "seconds": round(sus_ms * sus_launches * 1e-3, 2),
                 "sm_mhz_median": sus_clocks.get("sm_mhz"), "power_w_max": sus_clocks.get("power_w_max"),
                 "reasons": sus_clocks.get("reasons"),
                 "frac_of_sustained_peak": round(sus_tf / peaks["bf16_tflops_sustained"], 4) if peaks["bf16_tflops_sustained"] else None,
                 "frac_of_burst_peak": round(sus_tf / peaks["bf16_tflops"], 4),
                 "ms_times_sm_mhz": round(sus_ms * (sus_clocks.get("sm_mhz") or 0), 2),
                 "burst_ms_times_sm_mhz": round(ms * (clocks.get("sm_mhz") or 0), 2)}
    del q, k, v

    # ---------------------------------------------------------------- CPU baseline (rank 0, N=1 only)
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        threads = os.cpu_count() or 1
        tf, bs, times = cpu_attention_sample(w, reps=5, threads=threads)
        cpu = {"value": tf, "unit": UNIT, "cores": threads, "kind": "port",
               "sample": f"{bs} of {w.B} batch entries ({bs * w.H} of {w.B * w.H} heads), "
                         f"median of {len(times)} repetitions, fp32 torch CPU"}

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
            "config": bench_config(w),
            "tflops_per_gpu": per_gpu,
            "frac_of_bf16_peak": per_gpu / peaks["bf16_tflops"],
            "frac_of_bf16_peak_sustained": (per_gpu / peaks["bf16_tflops_sustained"]) if peaks["bf16_tflops_sustained"] else None,
            "frac_of_bf16_nominal_2250": per_gpu / 2250.0,
            "roofline": {"bound": "tensor", "achieved": per_gpu, "peak": peaks["bf16_tflops"],
                         "unit": "TFLOP/s", "frac": per_gpu / peaks["bf16_tflops"],
                         "traffic": NCU_TRAFFIC_BYTES_PER_LAUNCH, "traffic_note": NCU_TRAFFIC_NOTE,
                         "peak_source": f"of {peaks['source']}",
                         "algorithmic_bytes": w.bytes(), "kernel": "fa::fa_fwd_kernel<2, true, false, false> (dynamic schedule, causal)",
                         "burst": burst, "sustained": sustained},
            "e2e": dict({"value": e2e_value, "unit": UNIT, "ms_per_step": e2e_ms,
                         "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h}, **e2e_detail),
            "timed_launches": headline.get("timed_launches"),
            "gpu_launches": headline.get("timed_launches"),
            "clocks": clocks,
            "cpu_baseline": cpu,
            "extra": {"ms_per_step_by_rank": headline.get("ms_per_step_by_rank"), "comparators": comparators,
                      "small_problem": small, "sweep": sweep, "gpt2_prefill": prefill, "decode_step": decode, "add_layernorm": add_ln, "linear_small": lin,
                      "generate_20_tokens": gen},
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
