#!/usr/bin/env python
"""Benchmark of the quantized-matmul path.

    python bench.py --gpus N --steps K --warmup W [--impl reference]

N = 1  workload "w8a8_prefill_8b": one step = the four W8A8 prefill GEMMs of an 8B-class decoder
       layer at M = 8192 tokens (K x N = 4096x6144, 4096x28672, 4096x4096, 14336x4096), each
       preceded by the per-token dynamic quantization of its bf16 activations; bf16 outputs.
N > 1  workload "w8a8_row_parallel_allreduce": M = 4096, K = 28672 sharded evenly over the ranks,
       N = 8192; one step = dynamic quantization of the rank's activation shard + matmul +
       allreduce of the bf16 partials (strong scaling: the total work is fixed).

`value` counts GEMM operations only (2*M*N*K) over the device time of whole steps with inputs
resident in HBM; `e2e` is the same metric through the torch operators with pinned host buffers,
host<->device copies inside the timed region.  `roofline` describes the dominant kernel (the
tcgen05 CTA-pair GEMM; its four launches are timed with CUDA events around CUDA-graph replays, so
the host's launch cost is not in the figure), `cpu_baseline` the CPU restatement of the path timed
on this host's cores; `extras` holds the other configurations at one GPU (dynamic quant, W8A8
decode, W4A16 decode) as GB/s of algorithmic bytes against the measured copy bandwidth.
With `--impl reference` the CPU path itself is the thing measured.

    python bench.py --case quant_matmul --M 8192 --K 4096 --N 6144 [--algo 1] [--iters 3] [--buffers 2] [--graph]
    python bench.py --case dynamic_quant --M 8192 --K 14336
    python bench.py --case w4a16 | w4a16_prepacked --M 16 --K 8192 --N 28672
    python bench.py --case rms_norm_quant --M 8192 --K 4096

`--case` runs ONE kernel of the library a few times on synthetic data and prints its CUDA-event time per
launch: the target of `ncu` captures (the summaries under profiles/ quote these commands); it prints no
bench line.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import sys
import threading
import time
from pathlib import Path

import torch

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

PREFILL_M = 8192
PREFILL_GEMMS = [("qkv", 4096, 6144), ("gate_up", 4096, 28672), ("o_proj", 4096, 4096), ("down", 14336, 4096)]
ROWPAR = dict(M=4096, K=28672, N=8192)
# dram__bytes_read.sum + dram__bytes_write.sum of one launch of w8a8_pair_kernel per prefill shape (K, N), from ncu
PAIR_DRAM_BYTES = {(4096, 6144): 65926656 + 69236736, (4096, 28672): 203958272 + 439107328,
                   (4096, 4096): 53308928 + 34690816, (14336, 4096): 510722048 + 59542528}
CPU_ROW_BLOCK = 2048  # token rows per call of the CPU path
NOMINAL_INT8_TOPS = 4500.0  # NVIDIA's B200 dense int8 figure (9 POPS with 2:4 sparsity / 2)
NOMINAL_HBM_GBS = 8000.0


def prefill_config():
    """`config` of the N = 1 line; both arms print the same dict."""
    resident = sum(PREFILL_M * K * 2 + K * N + PREFILL_M * N * 2 for _, K, N in PREFILL_GEMMS)
    return {"workload": "w8a8_prefill_8b", "M": PREFILL_M, "gemms_KxN": [[K, N] for _, K, N in PREFILL_GEMMS],
            "step": "per GEMM: dynamic quant of bf16 activations + W8A8 matmul with fused dequant to bf16",
            "l2": f"inputs larger than L2: {resident / 1e6:.0f} MB touched per step"}


def rowpar_config(world):
    """`config` of the N > 1 lines; both arms print the same dict."""
    M, K, N = ROWPAR["M"], ROWPAR["K"], ROWPAR["N"]
    kr = K // world
    return {"workload": "w8a8_row_parallel_allreduce", "M": M, "K": K, "N": N, "k_per_rank": kr,
            "step": "dynamic quant of the rank's shard + W8A8 matmul + allreduce of bf16 partials",
            "l2": f"inputs larger than L2: {(M * kr * 2 + kr * N + M * N * 2) / 1e6:.0f} MB per rank"}


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return dict(hbm_gbs=d["hbm_gbs"], bf16=d["bf16_tflops"], bf16_sustained=d["bf16_tflops_sustained"],
                    source="measured")
    return dict(hbm_gbs=6650.0, bf16=1590.0, bf16_sustained=1400.0, source="fallback")


# ----------------------------------------------------------------------------------------------
# clocks sampler (reads only)
# ----------------------------------------------------------------------------------------------
class ClockSampler:
    REASONS = {0x1: "gpu_idle", 0x2: "applications_clocks_setting", 0x4: "sw_power_cap", 0x8: "hw_slowdown",
               0x10: "sync_boost", 0x20: "sw_thermal_slowdown", 0x40: "hw_thermal_slowdown",
               0x80: "hw_power_brake_slowdown", 0x100: "display_clock_setting"}

    def __init__(self, index: int):
        self.samples, self.reasons, self.max_mhz = [], set(), None
        self._stop = threading.Event()
        self._thread = None
        try:
            import pynvml

            pynvml.nvmlInit()
            self._nv = pynvml
            self._h = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self._h, pynvml.NVML_CLOCK_SM)
        except Exception:
            self._nv = None

    def _run(self):
        nv = self._nv
        while not self._stop.is_set():
            try:
                self.samples.append(nv.nvmlDeviceGetClockInfo(self._h, nv.NVML_CLOCK_SM))
                mask = nv.nvmlDeviceGetCurrentClocksEventReasons(self._h)
                for bit, name in self.REASONS.items():
                    if mask & bit and name != "gpu_idle":
                        self.reasons.add(name)
            except Exception:
                pass
            time.sleep(0.01)

    def __enter__(self):
        if self._nv is not None:
            self._thread = threading.Thread(target=self._run, daemon=True)
            self._thread.start()
        return self

    def __exit__(self, *exc):
        self._stop.set()
        if self._thread is not None:
            self._thread.join()

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": self.max_mhz, "reasons": ["unavailable"]}
        return {"sm_mhz": statistics.median(self.samples), "sm_max_mhz": self.max_mhz,
                "reasons": sorted(self.reasons)}


# ----------------------------------------------------------------------------------------------
# distributed plumbing
# ----------------------------------------------------------------------------------------------
def dist_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("LOCAL_RANK", 0)), int(os.environ.get("WORLD_SIZE", 1))


def max_over_ranks(ms: float, world: int, dev) -> float:
    if world == 1:
        return ms
    import torch.distributed as dist

    t = torch.tensor([ms], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(world: int):
    if world > 1:
        import torch.distributed as dist

        dist.barrier()
    torch.cuda.synchronize()


def timed_region(step_fn, steps: int, world: int, dev) -> float:
    """barrier+sync, `steps` steps between two CUDA events on the launching stream, sync; max over ranks (ms)."""
    barrier(world)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        step_fn()
    e1.record()
    torch.cuda.synchronize()
    barrier(world)
    return max_over_ranks(e0.elapsed_time(e1), world, dev)


# ----------------------------------------------------------------------------------------------
# reference arm / CPU baseline: the CPU restatement on the host cores
# ----------------------------------------------------------------------------------------------
def cpu_prefill_sample(rows: int, seed: int = 0):
    """The 4-GEMM prefill step on `rows` of the 8192 tokens, reference-style CPU path."""
    from oracle import qmm_oracle as O

    g = torch.Generator().manual_seed(seed)
    work = []
    ops = 0
    for _, K, N in PREFILL_GEMMS:
        x = torch.randn((rows, K), generator=g).to(torch.bfloat16)
        w = torch.randint(-127, 128, (K, N), generator=g, dtype=torch.int8).float()
        scale = torch.empty(N).uniform_(1e-3, 1e-2, generator=g)
        work.append((x, w, scale))
        ops += 2 * rows * K * N

    def step():
        for x, w, scale in work:
            for r0 in range(0, rows, CPU_ROW_BLOCK):  # row blocks bound the host memory of the fp32 intermediates
                O.cpu_path_w8a8(x[r0:r0 + CPU_ROW_BLOCK], w, scale, None)

    return step, ops


def cpu_rowpar_sample(rows: int, seed: int = 0):
    from oracle import qmm_oracle as O

    g = torch.Generator().manual_seed(seed)
    K, N = ROWPAR["K"], ROWPAR["N"]
    x = torch.randn((rows, K), generator=g).to(torch.bfloat16)
    w = torch.randint(-127, 128, (K, N), generator=g, dtype=torch.int8).float()
    scale = torch.empty(N).uniform_(1e-3, 1e-2, generator=g)

    def step():
        for r0 in range(0, rows, CPU_ROW_BLOCK):
            O.cpu_path_w8a8(x[r0:r0 + CPU_ROW_BLOCK], w, scale, None)

    return step, 2 * rows * K * N


def run_reference(args):
    """The CPU restatement of the path on the host cores, on the SAME configuration as the GPU arm: all
    8192 (4096) token rows per step.  A step is 3.6 TOP (1.9 TOP) of fp32 BLAS, a few seconds on a server CPU;
    QMM_REF_ROWS=<n> shrinks the row count for a quick look (the line then says so in `config.sample`)."""
    rank, _, world = dist_env()
    if rank != 0:
        return
    torch.set_num_threads(os.cpu_count() or 1)
    if args.gpus == 1:
        full_rows, config = PREFILL_M, prefill_config()
        rows = int(os.environ.get("QMM_REF_ROWS", full_rows))
        step, ops = cpu_prefill_sample(rows)
    else:
        full_rows, config = ROWPAR["M"], rowpar_config(args.gpus)
        rows = int(os.environ.get("QMM_REF_ROWS", full_rows))
        step, ops = cpu_rowpar_sample(rows)
    sample = (f"all {full_rows} token rows of the step" if rows == full_rows
              else f"{rows} of {full_rows} token rows (QMM_REF_ROWS)")
    if rows != full_rows:
        config = dict(config, sample=sample)
    if args.gpus > 1:
        sample += "; full K=28672 on one host (no sharding: one CPU)"
    for _ in range(max(args.warmup, 1)):
        step()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        step()
    dt = time.perf_counter() - t0
    tops = ops * args.steps / dt / 1e12
    line = {
        "impl": "reference", "metric": "W8A8 GEMM TOPS", "value": tops, "unit": "TOPS", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt / args.steps * 1e3, "higher_is_better": True,
        "scaling": "strong", "vs_baseline": None, "dtype": "int8", "data": "synthetic",
        "config": config,
        "cpu_baseline": {"value": tops, "unit": "TOPS", "cores": torch.get_num_threads(), "kind": "port",
                         "sample": sample},
        "e2e": {"value": tops, "unit": "TOPS", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "note": "reference = CPU restatement of the path (oracle port, torch fp32 BLAS in exact K chunks); the "
                "reference snapshot has no implementation of these operators and cannot be built here",
    }
    print(json.dumps(line), flush=True)


# ----------------------------------------------------------------------------------------------
# our arm
# ----------------------------------------------------------------------------------------------
def time_kernel(fn, iters: int) -> float:
    """Average device time of one call (ms), CUDA events on the launching stream."""
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    for _ in range(iters):
        fn()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / iters


def time_kernel_graph(fn, launches: int = 6, replays: int = 5) -> float:
    """Average device time of one call (ms) with the host taken out: `launches` calls are captured into a
    CUDA graph on a side stream (after a warm-up there) and the graph is replayed.  For kernels of a few
    tens of microseconds the Python + tensor-map + launch cost of a call exceeds the kernel itself, and
    back-to-back eager launches would time the host.  Falls back to eager timing if capture fails."""
    try:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(3):
                fn()
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for _ in range(launches):
                fn()
        graph.replay()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(replays):
            graph.replay()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / (replays * launches)
    except Exception:
        torch.cuda.synchronize()
        return time_kernel(fn, launches * replays)


def run_prefill(args, pkg, dev):
    capi = pkg.capi
    ops_mod = pkg.load_ops()
    peaks = measured_peaks()
    M = PREFILL_M
    g = torch.Generator(device=dev).manual_seed(2024)
    layers = []
    for name, K, N in PREFILL_GEMMS:
        x = torch.randn((M, K), generator=g, device=dev, dtype=torch.float32).to(torch.bfloat16)
        w = torch.randint(-127, 128, (K, N), generator=g, device=dev, dtype=torch.int8)
        scale = torch.empty(N, device=dev).uniform_(1e-3, 1e-2, generator=g)
        out = torch.empty((M, N), device=dev, dtype=torch.bfloat16)
        layers.append(dict(name=name, K=K, N=N, x=x, w=w, scale=scale, out=out))
    total_ops = sum(2 * M * L["K"] * L["N"] for L in layers)

    def step():
        for L in layers:
            q, s = capi.dynamic_quant(L["x"])
            capi.quant_matmul(q, L["w"], L["scale"], pertoken_scale=s, output_dtype=torch.bfloat16, out=L["out"])

    for _ in range(max(args.warmup, 3)):
        step()
    with ClockSampler(dev.index) as clocks:
        ms = timed_region(step, args.steps, 1, dev)
    value = total_ops * args.steps / (ms * 1e-3) / 1e12

    # ---- roofline of the dominant kernel: the tile GEMM alone, event-timed per shape
    gemm_ms = 0.0
    per_shape = {}
    gemm_clocks = ClockSampler(dev.index)
    gemm_clocks.__enter__()
    for L in layers:
        q, s = capi.dynamic_quant(L["x"])
        fn = lambda L=L, q=q, s=s: capi.quant_matmul(q, L["w"], L["scale"], pertoken_scale=s,  # noqa: E731
                                                      output_dtype=torch.bfloat16, out=L["out"])
        for _ in range(3):
            fn()
        # replayed from a CUDA graph: an eager launch through ctypes costs more host time than the
        # shorter GEMMs run, and the events would then time the host
        t = time_kernel_graph(fn)
        gemm_ms += t
        per_shape[L["name"]] = {"ms": t, "tops": 2 * M * L["K"] * L["N"] / (t * 1e-3) / 1e12}
    gemm_clocks.__exit__()
    achieved = total_ops / (gemm_ms * 1e-3) / 1e12
    # Denominator: the int8 tensor pipe's own issue-rate ceiling, measured here in operations per clock and SM
    # (operands resident in shared memory, one CTA per SM) and taken at the SM clock sampled while the GEMMs
    # above were timed - the microbenchmark itself draws enough power to leave the burst clock within a
    # millisecond, so its own TOPS figure belongs to another clock and is printed beside it.
    pipe = capi.int8_mma_peak(1024)
    gclk = gemm_clocks.summary()
    n_sm = torch.cuda.get_device_properties(dev).multi_processor_count
    gemm_mhz = gclk["sm_mhz"] or clocks.summary()["sm_mhz"] or pipe["sm_mhz"]
    peak_at_clock = pipe["ops_per_clk_per_sm"] * n_sm * gemm_mhz * 1e6 / 1e12
    roofline = {"bound": "tensor", "kernel": "w8a8_pair_kernel", "achieved": achieved, "peak": peak_at_clock,
                "unit": "TFLOP/s", "frac": achieved / peak_at_clock, "traffic": sum(PAIR_DRAM_BYTES.values()),
                "traffic_note": "dram read+write bytes of one ncu-captured launch per shape, summed over the four "
                                "launches of a step (profiles/w8a8_pair_kernel_prefill_8b.md)",
                "algorithmic_bytes": sum(M * L["K"] + L["K"] * L["N"] + 2 * M * L["N"] for L in layers),
                "peak_note": "measured in this run: tcgen05.mma.kind::i8 128x256x32 issued back to back from shared "
                             f"memory on every SM gives {pipe['ops_per_clk_per_sm']:.0f} int8 ops per clock and SM; "
                             f"x {n_sm} SMs x {gemm_mhz:.0f} MHz (median SM clock while the GEMMs were timed); "
                             "MEASURED_PEAKS.json holds no int8 figure",
                "int8_pipe": pipe, "gemm_clocks": gclk, "frac_of_nominal_4500": achieved / NOMINAL_INT8_TOPS,
                "frac_of_2x_measured_bf16_burst": achieved / (2.0 * peaks["bf16"]), "per_shape": per_shape}

    # ---- the same four GEMMs in a loop of several seconds: what the board sustains under its power cap
    def gemms_only():
        for L in layers:
            capi.quant_matmul(L["q"], L["w"], L["scale"], pertoken_scale=L["s"], output_dtype=torch.bfloat16,
                              out=L["out"])

    for L in layers:
        L["q"], L["s"] = capi.dynamic_quant(L["x"])
    sustained = None
    if args.quick:
        roofline["sustained"] = None
        print(json.dumps({"metric": "W8A8 GEMM TOPS", "value": value, "unit": "TOPS", "n_gpus": 1, "steps": args.steps,
                          "warmup": max(args.warmup, 3), "ms_per_step": ms / args.steps, "config": prefill_config(),
                          "clocks": clocks.summary(), "gpu_launches": 8 * args.steps, "roofline": roofline,
                          "quick": True}), flush=True)
        return
    try:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            gemms_only()
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for _ in range(8):
                gemms_only()
        graph.replay()
        torch.cuda.synchronize()
        replays = max(8, int(3.2 / (8 * gemm_ms * 1e-3)))
        with ClockSampler(dev.index) as sclk:
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(replays):
                graph.replay()
            e1.record()
            torch.cuda.synchronize()
        sus_s = e0.elapsed_time(e1) * 1e-3
        sus_tops = total_ops * 8 * replays / sus_s / 1e12
        with ClockSampler(dev.index) as pclk:
            pipe_sus = capi.int8_mma_peak(int(3.0 * 1.2e9 / (128 * 64)))  # about three seconds at 1.2 GHz
        sc = sclk.summary()
        sustained = {"seconds": sus_s, "tops": sus_tops, "clocks": sc,
                     "ms_per_step_x_sm_mhz": (sus_s * 1e3 / (8 * replays)) * (sc["sm_mhz"] or 0),
                     "burst_ms_per_step_x_sm_mhz": gemm_ms * (clocks.summary()["sm_mhz"] or 0),
                     "int8_pipe_sustained": dict(pipe_sus, clocks=pclk.summary()),
                     "frac_of_pipe_at_same_clock": (sus_tops / (pipe_sus["ops_per_clk_per_sm"] * n_sm * sc["sm_mhz"] * 1e-6)
                                                    if sc["sm_mhz"] else None),
                     "frac_of_sustained_pipe_run": sus_tops / pipe_sus["tops"] if pipe_sus["tops"] else None,
                     "frac_of_nominal_4500": sus_tops / NOMINAL_INT8_TOPS,
                     "note": "CUDA-graph replays of the four GEMMs alone for >= 3 s; sw_power_cap pulls the SM clock "
                             "down, time x clock shows how much of the slowdown the clock explains"}
    except Exception as e:  # the sustained record must not take the headline line down
        sustained = {"error": repr(e)}
    roofline["sustained"] = sustained

    # ---- end to end through the torch operators, host buffers pinned
    host_x = [torch.empty((M, L["K"]), dtype=torch.bfloat16).pin_memory() for L in layers]
    host_y = [torch.empty((M, L["N"]), dtype=torch.bfloat16).pin_memory() for L in layers]
    for hx, L in zip(host_x, layers):
        hx.copy_(L["x"])
    h2d = sum(hx.numel() * 2 for hx in host_x)
    d2h = sum(hy.numel() * 2 for hy in host_y)
    copy_in, copy_out = torch.cuda.Stream(), torch.cuda.Stream()
    main = torch.cuda.current_stream()
    dx = [torch.empty_like(L["x"]) for L in layers]

    def e2e_step():
        evs = []
        with torch.cuda.stream(copy_in):
            for hx, d in zip(host_x, dx):
                d.copy_(hx, non_blocking=True)
                ev = torch.cuda.Event()
                ev.record(copy_in)
                evs.append(ev)
        for i, L in enumerate(layers):
            main.wait_event(evs[i])
            q, s = ops_mod.npu_dynamic_quant(dx[i])
            y = ops_mod.npu_quant_matmul(q, L["w"], L["scale"], pertoken_scale=s, output_dtype=torch.bfloat16)
            done = torch.cuda.Event()
            done.record(main)
            copy_out.wait_event(done)
            with torch.cuda.stream(copy_out):
                host_y[i].copy_(y, non_blocking=True)
                y.record_stream(copy_out)
        main.wait_stream(copy_out)
        main.wait_stream(copy_in)

    e2e_steps = max(2, min(args.steps, 10))
    for _ in range(2):
        e2e_step()
    e2e_ms = timed_region(e2e_step, e2e_steps, 1, dev)
    e2e_value = total_ops * e2e_steps / (e2e_ms * 1e-3) / 1e12

    extras = secondary_workloads(capi, dev, peaks)
    cpu = cpu_baseline()
    line = {
        "metric": "W8A8 GEMM TOPS", "value": value, "unit": "TOPS", "n_gpus": 1, "steps": args.steps,
        "warmup": max(args.warmup, 3), "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "strong",
        "vs_baseline": None, "dtype": "int8", "data": "synthetic",
        "config": prefill_config(),
        "clocks": clocks.summary(),
        "e2e": {"value": e2e_value, "unit": "TOPS", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                "steps": e2e_steps, "ms_per_step": e2e_ms / e2e_steps,
                "path": "torch.ops.npu.npu_dynamic_quant + npu_quant_matmul, pinned host buffers, weights resident"},
        "gpu_launches": 8 * args.steps,
        "roofline": roofline, "cpu_baseline": cpu, "extras": extras,
    }
    print(json.dumps(line), flush=True)


def secondary_workloads(capi, dev, peaks):
    """Other configurations at 1 GPU: HBM-bound kernels in GB/s of algorithmic bytes (weights rotate over
    buffers larger than L2 in total, so they are never L2-resident)."""
    out = {}
    hbm = peaks["hbm_gbs"]
    try:
        # dynamic quant: 2*M*K read + M*K written + 4*M
        for (M, K) in [(8192, 4096), (8192, 14336)]:
            xs = [torch.randn((M, K), device=dev, dtype=torch.bfloat16) for _ in range(3)]
            i = [0]

            def f():
                i[0] += 1
                capi.dynamic_quant(xs[i[0] % 3])

            for _ in range(3):
                f()
            t = time_kernel_graph(f)
            gbs = (3 * M * K + 4 * M) / (t * 1e-3) / 1e9
            out[f"dynamic_quant_{M}x{K}"] = {"us": t * 1e3, "GB/s": gbs, "frac_of_measured_hbm": gbs / hbm,
                                             "frac_of_8TB/s": gbs / NOMINAL_HBM_GBS}
            del xs
        # W8A8 decode
        for (K, N) in [(8192, 28672), (28672, 8192)]:
            ws = [torch.randint(-127, 128, (K, N), dtype=torch.int8, device=dev) for _ in range(3)]
            scale = torch.empty(N, device=dev).uniform_(1e-3, 1e-2)
            for M in (1, 8, 32, 128):
                a = torch.randint(-127, 128, (M, K), dtype=torch.int8, device=dev)
                pt = torch.empty(M, device=dev).uniform_(1e-2, 5e-2)
                y = torch.empty((M, N), dtype=torch.bfloat16, device=dev)
                i = [0]

                def f():
                    i[0] += 1
                    capi.quant_matmul(a, ws[i[0] % 3], scale, pertoken_scale=pt, output_dtype=torch.bfloat16, out=y)

                for _ in range(3):
                    f()
                t = time_kernel_graph(f)
                nbytes = K * N + M * K + 2 * M * N + 4 * N + 4 * M
                gbs = nbytes / (t * 1e-3) / 1e9
                out[f"w8a8_decode_M{M}_K{K}_N{N}"] = {"us": t * 1e3, "GB/s": gbs, "frac_of_measured_hbm": gbs / hbm,
                                                      "frac_of_8TB/s": gbs / NOMINAL_HBM_GBS}
                if N == 28672 and M in (1, 128):
                    # the allocation-free entry point on the same problem: same kernel + one memset of its
                    # built-in scratch per call
                    st = torch.cuda.current_stream

                    def g():
                        i[0] += 1
                        wq = ws[i[0] % 3]
                        capi.check(capi.lib().qmm_quant_matmul_decode_noalloc(
                            a.data_ptr(), K, wq.data_ptr(), N, 1, scale.data_ptr(), N, pt.data_ptr(), None,
                            capi.DTYPE_NONE, y.data_ptr(), capi.DTYPE_BF16, N, M, N, K, st().cuda_stream),
                            "qmm_quant_matmul_decode_noalloc")

                    for _ in range(3):
                        g()
                    tn = time_kernel_graph(g)
                    out[f"w8a8_decode_noalloc_M{M}_K{K}_N{N}"] = {"us": tn * 1e3, "GB/s": nbytes / (tn * 1e-3) / 1e9,
                                                                  "extra_us_vs_caller_scratch": (tn - t) * 1e3}
            del ws
        # W4A16 decode
        K, N, group = 8192, 28672, 128
        packs = [torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), device=dev, dtype=torch.int64).to(torch.int32)
                 for _ in range(3)]
        sc = torch.empty((K // group, N), device=dev).uniform_(5e-3, 2e-2).to(torch.bfloat16)
        of = torch.empty((K // group, N), device=dev).uniform_(-1, 1).to(torch.bfloat16)
        for M in (1, 16, 64):
            x = torch.randn((M, K), device=dev, dtype=torch.bfloat16)
            i = [0]

            def f():
                i[0] += 1
                capi.weight_quant_batchmatmul(x, packs[i[0] % 3], sc, of, group_size=group)

            t = time_kernel_graph(f)
            nbytes = K * N // 2 + 2 * 2 * (K // group) * N + 2 * M * K + 2 * M * N
            gbs = nbytes / (t * 1e-3) / 1e9
            out[f"w4a16_decode_M{M}_K{K}_N{N}"] = {"us": t * 1e3, "GB/s": gbs, "frac_of_measured_hbm": gbs / hbm,
                                                   "frac_of_8TB/s": gbs / NOMINAL_HBM_GBS,
                                                   "layout": "stock int32 [K, N/8]"}
        # the same problem over prepacked weights (one-time layout pass, not timed: weights are static)
        bufs = [capi.w4a16_prepack(p, sc, of, group_size=group) for p in packs]
        del packs
        for M in (1, 16, 64):
            x = torch.randn((M, K), device=dev, dtype=torch.bfloat16)
            i = [0]

            def f():
                i[0] += 1
                capi.weight_quant_batchmatmul_prepacked(x, bufs[i[0] % 3], N)

            t = time_kernel_graph(f)
            nbytes = K * N // 2 + 2 * 2 * (K // group) * N + 2 * M * K + 2 * M * N
            gbs = nbytes / (t * 1e-3) / 1e9
            out[f"w4a16_prepacked_decode_M{M}_K{K}_N{N}"] = {"us": t * 1e3, "GB/s": gbs,
                                                             "frac_of_measured_hbm": gbs / hbm,
                                                             "frac_of_8TB/s": gbs / NOMINAL_HBM_GBS,
                                                             "layout": "prepacked k-major stream"}
        del bufs
        # rms_norm fused with dynamic quant: 2*M*K read + M*K written + 8*M (scale, rstd)
        for (M, K) in [(8192, 4096)]:
            xs = [torch.randn((M, K), device=dev, dtype=torch.bfloat16) for _ in range(3)]
            gamma = torch.rand(K, device=dev).to(torch.bfloat16)
            i = [0]

            def f():
                i[0] += 1
                capi.rms_norm_dynamic_quant(xs[i[0] % 3], gamma, 1e-6)

            for _ in range(3):
                f()
            t = time_kernel_graph(f)
            gbs = (3 * M * K + 8 * M + 2 * K) / (t * 1e-3) / 1e9
            out[f"rms_norm_dynamic_quant_{M}x{K}"] = {"us": t * 1e3, "GB/s": gbs, "frac_of_measured_hbm": gbs / hbm,
                                                      "frac_of_8TB/s": gbs / NOMINAL_HBM_GBS}
            del xs
    except Exception as e:  # secondary numbers must not take the headline line down
        out["error"] = repr(e)
    return out


def cpu_baseline():
    """The CPU restatement of the prefill step on a bounded sample, all host threads."""
    torch.set_num_threads(os.cpu_count() or 1)
    rows = 256
    step, ops = cpu_prefill_sample(rows)
    step()
    t0 = time.perf_counter()
    n = 0
    while True:
        step()
        n += 1
        dt = time.perf_counter() - t0
        if dt >= 10.0 or n >= 50:
            break
    return {"value": ops * n / dt / 1e12, "unit": "TOPS", "cores": torch.get_num_threads(), "kind": "port",
            "sample": f"{rows} of 8192 token rows through all four GEMMs, {n} repetitions in {dt:.1f} s"}


def rowpar_parity(step, q, s, w, scale, hcom, rank, world, dev, M, N, nrows=64):
    """One more step outside the timed region, checked: rank 0 gathers every rank's quantized activations and
    scales for `nrows` sampled token rows and its weight shard, evaluates the CPU oracle of the operator on
    those rows at the full size of the configuration, and compares; every rank's whole output is compared
    with rank 0's bit for bit.  (The oracle call is the checker, not part of anything timed.)"""
    import torch.distributed as dist

    out = step()
    torch.cuda.synchronize()
    rows = torch.linspace(0, M - 1, nrows, device=dev).long().unique()
    q_rows = [torch.empty((rows.numel(), q.shape[1]), dtype=torch.int8, device=dev) for _ in range(world)]
    s_rows = [torch.empty((rows.numel(),), dtype=torch.float32, device=dev) for _ in range(world)]
    w_all = [torch.empty_like(w) for _ in range(world)] if rank == 0 else None
    dist.all_gather(q_rows, q[rows].contiguous())
    dist.all_gather(s_rows, s[rows].contiguous())
    dist.gather(w, w_all, dst=0)
    ref = out.clone()
    dist.broadcast(ref, src=0)
    same = torch.tensor([1 if torch.equal(ref.view(torch.int16), out.view(torch.int16)) else 0], device=dev)
    dist.all_reduce(same, op=dist.ReduceOp.MIN)
    result = None
    if rank == 0:
        from oracle import qmm_oracle as O
        import numpy as np

        total, rounded = O.mm_all_reduce([t.cpu() for t in q_rows], [t.cpu() for t in w_all], scale.cpu(),
                                         [t.cpu() for t in s_rows], output_dtype=torch.bfloat16)
        got = out[rows].float().cpu().numpy()
        mag = np.zeros_like(total)
        for r in range(world):
            mag += np.abs(O.quant_matmul(q_rows[r].cpu(), w_all[r].cpu(), scale.cpu(), pertoken_scale=s_rows[r].cpu(),
                                         output_dtype=torch.bfloat16).float().numpy())
        err = np.abs(got - total)
        bound = 1e-2 * np.abs(total) + 1e-2 * mag
        result = {"rows": int(rows.numel()), "cols": int(N), "K_total": int(q.shape[1] * world),
                  "max_err_over_bound": float(np.max(err / np.maximum(bound, 1e-30))),
                  "within_rtol_1e-2": bool(np.all(err <= bound)),
                  "bit_exact_vs_oracle": bool(torch.equal(out[rows].cpu().view(torch.int16), rounded.view(torch.int16))),
                  "all_ranks_identical": bool(same.item() == 1),
                  "note": "oracle = per-rank fp32-epilogue results rounded to bf16, summed in fp32 in rank order, "
                          "rounded once; the peer-memory kernel adds in the same order (bit-exact), NCCL need not"}
    return result


def run_rowpar(args, pkg, dev, rank, world):
    import torch.distributed as dist

    sys.path.insert(0, str(ROOT / "ascend-python_b200"))
    import torch_npu
    from ascend_python_b200.sharding import k_shard_bounds

    capi = pkg.capi
    M, K, N = ROWPAR["M"], ROWPAR["K"], ROWPAR["N"]
    b = k_shard_bounds(K, world)
    Kr = b[rank + 1] - b[rank]
    g = torch.Generator(device=dev).manual_seed(100 + rank)
    x = torch.randn((M, Kr), generator=g, device=dev, dtype=torch.float32).to(torch.bfloat16)
    w = torch.randint(-127, 128, (Kr, N), generator=g, device=dev, dtype=torch.int8)
    scale = torch.empty(N, device=dev).uniform_(1e-3, 1e-2, generator=torch.Generator(device=dev).manual_seed(7))
    hcom = torch_npu.get_comm_name()
    total_ops = 2 * M * N * K

    def step():
        q, s = torch_npu.npu_dynamic_quant(x)
        return torch_npu.npu_mm_all_reduce_base(q, w, hcom, reduce_op="sum", dequant_scale=scale, pertoken_scale=s)

    for _ in range(max(args.warmup, 3)):
        step()
    with ClockSampler(dev.index) as clocks:
        ms = timed_region(step, args.steps, world, dev)
    value = total_ops * args.steps / (ms * 1e-3) / 1e12

    # matmul alone and allreduce alone (for the overlap figure), max over ranks
    q, s = torch_npu.npu_dynamic_quant(x)
    y = torch.empty((M, N), device=dev, dtype=torch.bfloat16)
    gemm = lambda: capi.quant_matmul(q, w, scale, pertoken_scale=s, output_dtype=torch.bfloat16, out=y)  # noqa: E731
    for _ in range(3):
        gemm()
    gemm_ms = max_over_ranks(time_kernel(gemm, 10), world, dev)
    ar = lambda: dist.all_reduce(y)  # noqa: E731
    for _ in range(3):
        ar()
    barrier(world)
    ar_ms = max_over_ranks(time_kernel(ar, 10), world, dev)

    parity = rowpar_parity(step, q, s, w, scale, hcom, rank, world, dev, M, N)
    stats_timed = capi.comm_stats(hcom)

    host_x = torch.empty((M, Kr), dtype=torch.bfloat16).pin_memory()
    host_x.copy_(x)
    host_y = torch.empty((M, N), dtype=torch.bfloat16).pin_memory()
    dx = torch.empty_like(x)

    def e2e_step():
        dx.copy_(host_x, non_blocking=True)
        q, s = torch_npu.npu_dynamic_quant(dx)
        out = torch_npu.npu_mm_all_reduce_base(q, w, hcom, reduce_op="sum", dequant_scale=scale, pertoken_scale=s)
        host_y.copy_(out, non_blocking=True)

    e2e_steps = max(2, min(args.steps, 10))
    for _ in range(2):
        e2e_step()
    e2e_ms = timed_region(e2e_step, e2e_steps, world, dev)
    peaks = measured_peaks()
    # the same measured ceiling as the 1-GPU line: ops per clock and SM of the int8 tensor pipe x SMs x the SM clock
    # sampled during the timed region
    pipe = capi.int8_mma_peak(1024) if rank == 0 else None
    if rank == 0:
        step_ms = ms / args.steps
        achieved = (total_ops / world) / (gemm_ms * 1e-3) / 1e12
        n_sm = torch.cuda.get_device_properties(dev).multi_processor_count
        mhz = clocks.summary()["sm_mhz"] or pipe["sm_mhz"]
        int8_peak = pipe["ops_per_clk_per_sm"] * n_sm * mhz * 1e6 / 1e12
        line = {
            "metric": "W8A8 GEMM TOPS", "value": value, "unit": "TOPS", "n_gpus": world, "steps": args.steps,
            "warmup": max(args.warmup, 3), "ms_per_step": step_ms, "higher_is_better": True, "scaling": "strong",
            "vs_baseline": None, "dtype": "int8", "data": "synthetic",
            "config": rowpar_config(world),
            "allreduce_path": dict(stats_timed, note="calls of npu_mm_all_reduce_base on rank 0 up to the end of the "
                                   "timed region and the parity step, counted by the library per path taken: its own "
                                   "kernels over peer memory (of which: output tiles pushed to their owners by the "
                                   "matmul's epilogue; of which: reduce + gather done by the matmul kernel's own "
                                   "communication warps, no second kernel) or NCCL"),
            "parity": parity,
            "clocks": clocks.summary(),
            "e2e": {"value": total_ops * e2e_steps / (e2e_ms * 1e-3) / 1e12, "unit": "TOPS",
                    "h2d_bytes_per_step": host_x.numel() * 2, "d2h_bytes_per_step": host_y.numel() * 2,
                    "steps": e2e_steps, "ms_per_step": e2e_ms / e2e_steps},
            "gpu_launches": args.steps * (2 if stats_timed["peer_fused_calls"] >= args.steps else 3),
            "roofline": {"bound": "tensor", "kernel": "w8a8_pair_kernel", "achieved": achieved, "peak": int8_peak,
                         "unit": "TFLOP/s", "frac": achieved / int8_peak, "traffic": None,
                         "peak_note": f"per GPU, matmul alone: {pipe['ops_per_clk_per_sm']:.0f} int8 ops per clock and SM "
                                      f"(measured in this run) x {n_sm} SMs x {mhz:.0f} MHz (median SM clock of the "
                                      "timed region)",
                         "frac_of_2x_measured_bf16_sustained": achieved / (2.0 * peaks["bf16_sustained"])},
            "overlap": {"gemm_ms": gemm_ms, "nccl_allreduce_ms": ar_ms, "step_ms": step_ms,
                        "allreduce_busbw_GB/s": 2 * (world - 1) / world * M * N * 2 / (ar_ms * 1e-3) / 1e9,
                        "roofline_ms": max(gemm_ms, ar_ms)},
            "cpu_baseline": None,
        }
        print(json.dumps(line), flush=True)
    barrier(world)
    torch_npu.destroy_comm(hcom)


def run_case(args):
    """One kernel, a few launches (see the module docstring): what the ncu captures profile."""
    from __graft_entry__ import load_package

    capi = load_package().capi
    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    M, K, N = args.M, args.K, args.N
    nb = max(args.buffers, 1)
    if args.case == "quant_matmul":
        a = torch.randint(-127, 128, (M, K), dtype=torch.int8, device=dev)
        ws = [torch.randint(-127, 128, (K, N), dtype=torch.int8, device=dev) for _ in range(nb)]
        scale = torch.empty(N, device=dev).uniform_(1e-3, 1e-2)
        pt = torch.empty(M, device=dev).uniform_(1e-2, 5e-2)
        out = torch.empty((M, N), dtype=torch.bfloat16, device=dev)
        fn = lambda i: capi.quant_matmul(a, ws[i % nb], scale, pertoken_scale=pt,  # noqa: E731
                                         output_dtype=torch.bfloat16, algo=args.algo, out=out)
    elif args.case == "dynamic_quant":
        xs = [torch.randn((M, K), device=dev, dtype=torch.bfloat16) for _ in range(nb)]
        fn = lambda i: capi.dynamic_quant(xs[i % nb])  # noqa: E731
    elif args.case == "dense_matmul":
        # the bf16 matmul of npu_mm_reduce_scatter_base / npu_all_gather_base_mm, through a one-rank communicator
        import ctypes

        uid = ctypes.create_string_buffer(capi.UNIQUE_ID_BYTES)
        capi.check(capi.lib().qmm_comm_unique_id(uid), "qmm_comm_unique_id")
        capi.check(capi.lib().qmm_comm_init_rank(b"bench_solo", uid, 1, 0), "qmm_comm_init_rank")
        a = torch.randn((M, K), device=dev, dtype=torch.bfloat16)
        ws = [torch.randn((K, N), device=dev, dtype=torch.bfloat16) for _ in range(nb)]
        out = torch.empty((M, N), dtype=torch.bfloat16, device=dev)
        st = torch.cuda.current_stream

        def fn(i):
            capi.check(capi.lib().qmm_mm_reduce_scatter(a.data_ptr(), capi.DTYPE_BF16, K, ws[i % nb].data_ptr(), N, 1, None,
                                                        out.data_ptr(), N, M, N, K, b"bench_solo", b"sum", 0, None, 0,
                                                        st().cuda_stream), "qmm_mm_reduce_scatter")
    elif args.case == "rms_norm_quant":
        xs = [torch.randn((M, K), device=dev, dtype=torch.bfloat16) for _ in range(nb)]
        gamma = torch.randn(K, device=dev, dtype=torch.bfloat16)
        fn = lambda i: capi.rms_norm_dynamic_quant(xs[i % nb], gamma, 1e-6)  # noqa: E731
    elif args.case == "rms_norm":
        xs = [torch.randn((M, K), device=dev, dtype=torch.bfloat16) for _ in range(nb)]
        gamma = torch.randn(K, device=dev, dtype=torch.bfloat16)
        fn = lambda i: capi.rms_norm(xs[i % nb], gamma, 1e-6)  # noqa: E731
    elif args.case == "quant_matmul_int8":
        # the requantized int8 output (in the matmul kernels' epilogue)
        a = torch.randint(-127, 128, (M, K), dtype=torch.int8, device=dev)
        ws = [torch.randint(-127, 128, (K, N), dtype=torch.int8, device=dev) for _ in range(nb)]
        scale = torch.empty(N, device=dev).uniform_(1e-5, 1e-4)
        offset = torch.empty(N, device=dev).uniform_(-4, 4)
        pt = torch.empty(M, device=dev).uniform_(0.5, 2.0)
        fn = lambda i: capi.quant_matmul_int8(a, ws[i % nb], scale, offset=offset, pertoken_scale=pt)  # noqa: E731
    else:
        x = torch.randn((M, K), device=dev, dtype=torch.bfloat16)
        packs = [torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), device=dev, dtype=torch.int64).to(torch.int32)
                 for _ in range(nb)]
        sc = torch.empty((K // 128, N), device=dev).uniform_(5e-3, 2e-2).to(torch.bfloat16)
        of = torch.empty((K // 128, N), device=dev).uniform_(-1, 1).to(torch.bfloat16)
        if args.case == "w4a16_prepacked":
            bufs = [capi.w4a16_prepack(p, sc, of, group_size=128) for p in packs]
            del packs
            fn = lambda i: capi.weight_quant_batchmatmul_prepacked(x, bufs[i % nb], N)  # noqa: E731
        else:
            fn = lambda i: capi.weight_quant_batchmatmul(x, packs[i % nb], sc, of, group_size=128)  # noqa: E731
    fn(0)
    torch.cuda.synchronize()
    eager_us = time_kernel(lambda c=[0]: (c.__setitem__(0, c[0] + 1), fn(c[0]))[1], args.iters) * 1e3
    assert capi.device_status() == 0
    graph_us = float("nan")
    if args.graph:
        graph_us = time_kernel_graph(lambda c=[0]: (c.__setitem__(0, c[0] + 1), fn(c[0]))[1], launches=args.iters) * 1e3
        assert capi.device_status() == 0
    print(f"{args.case} M={M} K={K} N={N}: {eager_us:.1f} us per eager launch, {graph_us:.1f} us per launch in a graph")


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--case", default=None, choices=["quant_matmul", "dynamic_quant", "w4a16", "w4a16_prepacked",
                                                     "rms_norm_quant", "dense_matmul", "rms_norm", "quant_matmul_int8"],
                    help="run one kernel a few times (profiling target) instead of the benchmark")
    ap.add_argument("--M", type=int, default=8192)
    ap.add_argument("--K", type=int, default=4096)
    ap.add_argument("--N", type=int, default=6144)
    ap.add_argument("--algo", type=int, default=0)
    ap.add_argument("--iters", type=int, default=3)
    ap.add_argument("--buffers", type=int, default=1, help="--case: rotate over this many weight/input buffers")
    ap.add_argument("--graph", action="store_true", help="--case: also time the launches replayed from a CUDA graph")
    ap.add_argument("--quick", action="store_true",
                    help="N = 1: headline step and roofline only (no sustained loop, extras, end-to-end or CPU legs); "
                         "what the launch list under profiles/ was captured on")
    args = ap.parse_args()
    if args.case is not None:
        run_case(args)
        return

    if args.gpus > 1 and "WORLD_SIZE" not in os.environ:
        # launched by hand without torchrun: start one rank per GPU ourselves
        os.execvp(sys.executable, [sys.executable, "-m", "torch.distributed.run", "--nnodes=1",
                                   f"--nproc-per-node={args.gpus}", "--master-addr", "127.0.0.1", "--master-port",
                                   str(29400 + os.getpid() % 500), str(Path(__file__).resolve()), *sys.argv[1:]])

    if args.impl == "reference":
        run_reference(args)
        return

    from __graft_entry__ import load_package

    rank, local_rank, world = dist_env()
    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device: there is no CPU fallback for the product path")
    dev = torch.device("cuda", local_rank)
    torch.cuda.set_device(dev)
    pkg = load_package()
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl", rank=rank, world_size=world, device_id=dev)
        try:
            run_rowpar(args, pkg, dev, rank, world)
        finally:
            dist.destroy_process_group()
    else:
        run_prefill(args, pkg, dev)


if __name__ == "__main__":
    main()
