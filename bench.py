#!/usr/bin/env python3
"""Benchmark of the MTP speculative decode step on the Llama-3-8B-shaped INT4 g128 configuration
(32 layers, hidden 4096, 32 q / 8 kv heads, head 128, FFN 14336, vocab 128256, bf16 embeddings / lm_head,
one MTP layer; paged bf16 KV with 16-token pages; prompt 512, k = 3, batch 1).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl b200|reference]

A "step" is one speculative cycle of the stream: k draft steps, one (k+1)-lane verify, on-device acceptance
and the draft catch-up.  `value` = accepted (emitted) tokens per second over exactly K steps, device-timed with
CUDA events on the engine's stream (state resident in HBM); `e2e` = the same metric through the public engine
API for a whole 256-token event, host wall clock around the `run_until_idle` call that decodes it, every step's
host->device uploads and device->host read-back inside the timed region.  `parity` = the first cycles of a short
event (16-token prompt) compared token by token and cycle by cycle with the CPU oracle (oracle/parity.py) - the
oracle cycles of that comparison are also the `cpu_baseline` sample.  Weights are synthetic N(0, 0.02) (seeded), written as a compiled package on local
disk by the native package writer and mounted through the C ABI.  Each step streams ~4.7 GB of weights, far
larger than the 126 MB L2, so no L2 flush is needed between steps.
"""

from __future__ import annotations

import argparse
import json
import os
import shutil
import statistics
import subprocess
import sys
import tempfile
import threading
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

PROMPT_TOKENS = 512
EVENT_TOKENS = 256
DRAFTS = 3
METRIC = "accepted tokens/s (8B INT4, MTP k=3)"
UNIT = "tokens/s"
STACK_TRAFFIC_RATIO = 1.037  # DRAM bytes over algorithmic bytes of a four-layer verify launch (ncu; summary under profiles/)
NOMINAL_HBM_GBS = 8000.0


def measured_peaks():
    path = ROOT / "MEASURED_PEAKS.json"
    if path.exists():
        data = json.loads(path.read_text())
        return float(data["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def package_dir(spec_name: str) -> Path:
    base = Path(os.environ.get("NERVE_B200_BENCH_DIR", tempfile.gettempdir())) / "nerve_b200_bench"
    return base / spec_name


def bench_spec():
    from llmoop_b200.synth import LLAMA3_8B_INT4, ModelSpec

    return ModelSpec(name="llama3_8b_int4_mtp", seed=0, **LLAMA3_8B_INT4)


def ensure_package(spec, device: str):
    """Writes the synthetic 8B package once per box (about 6 GB on local disk)."""
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import iter_checkpoint_torch

    directory = package_dir(spec.name)
    if (directory / "vulkan_resident_package.json").exists():
        return directory
    staging = directory.with_name(directory.name + f".tmp{os.getpid()}")
    shutil.rmtree(staging, ignore_errors=True)
    write_package(spec, staging, tensors=iter_checkpoint_torch(spec, device), hash_tensors=False)
    try:
        staging.rename(directory)
    except OSError:
        shutil.rmtree(staging, ignore_errors=True)  # another rank won the race
    return directory


def prompt_tokens(vocab: int, seed: int = 0):
    import numpy as np

    return [int(t) for t in np.random.default_rng(seed).integers(0, vocab, size=PROMPT_TOKENS)]


class ClockSampler:
    """Samples SM clocks and throttle reasons while the timed region runs: through NVML every 10 ms (read-only
    queries), or with nvidia-smi every 100 ms where the NVML binding is missing."""

    QUERY = ("clocks.sm,clocks.max.sm,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
    REASON_BITS = (("sw_power_cap", 0x4), ("hw_slowdown", 0x8), ("sw_thermal_slowdown", 0x20), ("hw_thermal_slowdown", 0x40))

    def __init__(self, index: int):
        self.index = index
        self.process = None
        self.thread = None
        self.lines = []
        self.stop = threading.Event()

    def _nvml_loop(self, nvml, handle):
        maximum = nvml.nvmlDeviceGetMaxClockInfo(handle, nvml.NVML_CLOCK_SM)
        while not self.stop.is_set():
            try:
                clock = nvml.nvmlDeviceGetClockInfo(handle, nvml.NVML_CLOCK_SM)
                reasons = nvml.nvmlDeviceGetCurrentClocksEventReasons(handle) if hasattr(nvml, "nvmlDeviceGetCurrentClocksEventReasons") \
                    else nvml.nvmlDeviceGetCurrentClocksThrottleReasons(handle)
            except Exception:
                break
            flags = ["Active" if reasons & bit else "Not Active" for _, bit in self.REASON_BITS]
            # the column order of the nvidia-smi query: hw_slowdown, hw_thermal_slowdown, sw_thermal_slowdown, sw_power_cap
            self.lines.append(f"{clock}, {maximum}, {hex(reasons)}, {flags[1]}, {flags[3]}, {flags[2]}, {flags[0]}")
            self.stop.wait(0.01)

    def __enter__(self):
        try:
            import pynvml

            pynvml.nvmlInit()
            handle = pynvml.nvmlDeviceGetHandleByIndex(self.index)
            self.thread = threading.Thread(target=self._nvml_loop, args=(pynvml, handle), daemon=True)
            self.thread.start()
            return self
        except Exception:
            self.thread = None
        try:
            self.process = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except OSError:
            self.process = None
        return self

    def _read(self):
        for line in self.process.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *_):
        self.stop.set()
        if self.process is not None:
            self.process.terminate()
            try:
                self.process.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.process.kill()
        elif self.thread is not None:
            self.thread.join(timeout=2)

    def summary(self):
        clocks, maxima, reasons = [], [], set()
        for line in self.lines:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 7:
                continue
            try:
                clocks.append(float(parts[0]))
                maxima.append(float(parts[1]))
            except ValueError:
                continue
            for name, value in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"), parts[3:7]):
                if value.lower().startswith("active"):
                    reasons.add(name)
        if not clocks:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(clocks), "sm_max_mhz": max(maxima), "reasons": sorted(reasons), "samples": len(clocks)}


def run_event(engine, stream_id, prompt, max_tokens, teacher=None):
    """One whole input event through the public API: the prompt and the first cycle in one call, the rest of the
    event in a second one whose host wall clock is the end-to-end decode time.  Returns (tokens, report of the
    second call, tokens it produced / its wall seconds)."""
    engine.reset_stream_transient_state(stream_id)
    engine.set_teacher_tokens(stream_id, teacher or [])
    engine.enqueue_input_event(stream_id, prompt, max_tokens)
    first, first_report = engine.run(1)
    run_event.prefill_ms = first_report.prefill_ns * 1e-6  # host clock around the prompt's chunk(s), synchronised at the sampled token
    start = time.perf_counter()
    outputs, report = engine.run_until_idle()
    wall = time.perf_counter() - start
    tokens = [token for _, token, _, _ in first] + [token for _, token, _, _ in outputs]
    return tokens, report, len(outputs) / wall


def prefill_line(spec, milliseconds):
    """The 512-token prompt as one chunk: INT4 GEMMs on the tcgen05 tensor cores (target layers and the MTP layer's
    warm-up), tiled attention, one sampled token; flops = 2 x tokens x dense-layer weights."""
    path = ROOT / "MEASURED_PEAKS.json"
    sustained = float(json.loads(path.read_text()).get("bf16_tflops_sustained", 1400.0)) if path.exists() else 1400.0
    q_width, kv_width = spec.q_heads * spec.head_dim, spec.kv_heads * spec.head_dim
    per_layer = spec.hidden * (q_width + 2 * kv_width) + q_width * spec.hidden + 3 * spec.hidden * spec.ffn
    flops = 2.0 * PROMPT_TOKENS * per_layer * (spec.layers + 1)
    tflops = flops / (milliseconds * 1e-3) / 1e12 if milliseconds > 0 else 0.0
    return {"tokens": PROMPT_TOKENS, "ms": milliseconds, "tokens_per_s": PROMPT_TOKENS / (milliseconds * 1e-3) if milliseconds > 0 else 0.0,
            "tflops": tflops, "frac_of_measured_sustained_bf16": tflops / sustained, "peak_tflops": sustained}


def timed_cycles(engine, stream_id, prompt, budget_tokens, warmup, steps, teacher, barrier):
    """Prefill + `warmup` untimed cycles, then exactly `steps` cycles timed on the device."""
    import torch

    engine.reset_stream_transient_state(stream_id)
    engine.set_teacher_tokens(stream_id, teacher or [])
    engine.enqueue_input_event(stream_id, prompt, budget_tokens)
    engine.run(max(1, warmup))
    torch.cuda.synchronize()
    barrier()
    start = time.perf_counter()
    _, report = engine.run(steps)
    torch.cuda.synchronize()
    wall = time.perf_counter() - start
    barrier()
    if report.cycle_count != steps:
        raise RuntimeError(f"timed region ran {report.cycle_count} cycles instead of {steps}")
    engine.interrupt_stream(stream_id)
    return report, wall


SAMPLE_PROMPT_TOKENS = 16


def short_event(engine, stream_id, prompt, tokens):
    """The event the CPU leg replays: a 16-token prompt and `tokens` greedy tokens with k = 3 on the mounted package;
    returns (tokens, cycle log)."""
    engine.reset_stream_transient_state(stream_id)
    engine.set_teacher_tokens(stream_id, [])
    engine.set_cycle_logging(True)
    engine.enqueue_input_event(stream_id, prompt[:SAMPLE_PROMPT_TOKENS], tokens)
    outputs, _ = engine.run_until_idle()
    cycles = [{key: (list(value) if isinstance(value, list) else int(value)) for key, value in cycle.items()} for cycle in engine.cycle_log()]
    engine.set_cycle_logging(False)
    return [token for _, token, _, _ in outputs], cycles


def cpu_cycle_sample(directory, seconds_budget=150.0, max_cycles=None, cuda_run=None):
    """The CPU oracle (a port of the reference's shader arithmetic; the reference's Vulkan path cannot run on
    this box) on all host threads: speculative cycles at a 16-token context.  KV bytes are under 2 % of a cycle
    at the benchmark's context, so the short context does not change the rate materially.  With `cuda_run`
    (tokens, cycle log of the same event on the GPU) the oracle follows that run and the parity report comes back
    with the sample."""
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream
    from oracle.parity import follow_generation, summary

    # torchrun exports OMP_NUM_THREADS=1 to its workers; the sample is meant to use every host thread
    try:
        import ctypes

        ctypes.CDLL("libgomp.so.1").omp_set_num_threads(os.cpu_count() or 1)
    except OSError:
        pass
    package = OraclePackage(directory)
    oracle = Oracle(package)
    stream = OracleStream(package, 64)
    prompt = prompt_tokens(package.vocab)[:SAMPLE_PROMPT_TOKENS]
    durations, emitted, parity = [], 0, None
    if cuda_run is not None:
        tokens, cycles = cuda_run
        report = follow_generation(oracle, stream, prompt, tokens, cycles, DRAFTS, prefill_chunk=SAMPLE_PROMPT_TOKENS, max_cycles=max_cycles,
                                   cycle_seconds=durations, seconds_budget=seconds_budget)
        emitted = report["tokens_compared"] - 1
        parity = summary(report)
        parity["event"] = f"prompt {SAMPLE_PROMPT_TOKENS} + {len(tokens)} greedy tokens, k = {DRAFTS}, CUDA run followed by the CPU oracle"
        parity["divergence_list"] = report["divergences"][:8]
        parity["note"] = ("32 layers of random weights amplify one bf16 rounding of the hidden state to a few 1e-2 of a logit (logits reach +-6): the "
                          "oracle, the kernel-per-operator path and the persistent kernel differ mutually by that much "
                          "(tests/test_gpu_config2_parity.py), so near-ties up to that size may fall either way; accepted_equal says the "
                          "per-cycle bookkeeping followed the oracle through every one of them; control_kernel_per_operator_path is the "
                          "same replay of the path whose operators match the oracle to the last bf16 bit in at least 97 % of their "
                          "outputs one by one; which of the two parts from the oracle, and how often, varies with the build")
    else:
        token, _ = oracle.prefill(stream, prompt, sample_last=True)
        begin = time.perf_counter()
        while True:
            start = time.perf_counter()
            cycle = oracle.speculative_cycle(stream, token, DRAFTS)
            durations.append(time.perf_counter() - start)
            emitted += len(cycle["emitted"])
            token = cycle["emitted"][-1]
            if max_cycles is not None and len(durations) >= max_cycles:
                break
            if time.perf_counter() - begin > seconds_budget or stream.next_tick > 48:
                break
    total = sum(durations)
    return {"cycles": len(durations), "tokens": emitted, "seconds": total, "tokens_per_s": emitted / total,
            "ms_per_cycle": 1e3 * total / len(durations), "parity": parity}


def main():
    parser = argparse.ArgumentParser()
    parser.add_argument("--gpus", type=int, default=1)
    parser.add_argument("--steps", type=int, default=200)
    parser.add_argument("--warmup", type=int, default=8)
    parser.add_argument("--impl", default="b200", choices=["b200", "reference"])
    parser.add_argument("--skip-cpu-baseline", action="store_true")
    args = parser.parse_args()

    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    warmup = max(3, args.warmup)
    steps = max(1, args.steps)
    cores = os.cpu_count() or 1
    # Several GPUs: one stream, the weights sharded tensor-parallel over the ranks (strong scaling; every rank runs
    # the same calls and meets the others in the exchange).  NERVE_B200_BENCH_REPLICAS=1 instead runs one
    # independent stream per GPU on replicated weights (weak scaling, no collective on the data path).
    tensor_parallel = world > 1 and os.environ.get("NERVE_B200_BENCH_REPLICAS", "0") != "1"
    config = {
        "workload": "configs[1]: Llama-3-8B-shaped INT4 g128 + MTP k=3, prompt 512, batch 1, natural acceptance",
        "prompt_tokens": PROMPT_TOKENS, "draft_tokens": DRAFTS, "kv_page_tokens": 16,
        "l2": "each step streams ~4.7 GB of weights (inputs larger than the 126 MB L2); no flush",
        "weights": "synthetic N(0,0.02), seeded; INT4 symmetric g128 + bf16 scales; bf16 embeddings/lm_head",
    }

    if args.impl == "reference":
        # The reference's own implementation of this path is Vulkan-only (unavailable on this box); its CPU
        # restatement is timed instead.  Rank 0 alone works.
        if rank != 0:
            return
        import torch

        spec = bench_spec()
        directory = ensure_package(spec, "cuda" if torch.cuda.is_available() else "cpu")
        sample = cpu_cycle_sample(directory, seconds_budget=150.0, max_cycles=steps + warmup)
        config = {**config, "workload": "configs[1]: Llama-3-8B-shaped INT4 g128 + MTP k=3, batch 1, natural acceptance - a bounded CPU sample: "
                                        f"speculative cycles at a {SAMPLE_PROMPT_TOKENS}-token context (the 512-token prefill is not repeated on the host cores)",
                  "prompt_tokens": SAMPLE_PROMPT_TOKENS}
        line = {
            "impl": "reference", "metric": METRIC, "value": sample["tokens_per_s"], "unit": UNIT, "n_gpus": args.gpus,
            "steps": sample["cycles"], "steps_requested": steps, "warmup": 0, "ms_per_step": sample["ms_per_cycle"],
            "higher_is_better": True, "scaling": "strong" if tensor_parallel else "weak", "vs_baseline": None, "dtype": "int4 weights, bf16 activations, f32 accumulate",
            "data": "synthetic", "config": config,
            "cpu_baseline": {"value": sample["tokens_per_s"], "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": f"{sample['cycles']} speculative cycles (k=3) at a 16-token context, OpenMP over output rows"},
            "e2e": {"value": sample["tokens_per_s"], "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        }
        print(json.dumps(line))
        return

    import torch
    import torch.distributed as dist

    import llmoop_b200 as nb

    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device: the CUDA path has no CPU fallback")
    torch.cuda.set_device(local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local_rank))

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    spec = bench_spec()
    if rank == 0:
        directory = ensure_package(spec, f"cuda:{local_rank}")
    barrier()
    directory = package_dir(spec.name)
    peer_exchange = tensor_parallel and os.environ.get("NERVE_B200_TP_EXCHANGE", "1") != "0"
    prompt = prompt_tokens(spec.vocab, seed=0 if tensor_parallel else rank)

    # natural-mode budget: one token per cycle when no draft is accepted, up to k+1 when all are
    budget = (warmup + steps) * (DRAFTS + 1) + 8
    capacity = PROMPT_TOKENS + max(budget, EVENT_TOKENS + 8) + 64  # the context ring never wraps in this workload
    package = nb.Package(directory, device=local_rank, capacity_tokens=capacity, page_tokens=16, max_streams=1,
                         max_lanes=PROMPT_TOKENS, verify_level=0, tp_rank=rank if tensor_parallel else 0,
                         tp_size=world if tensor_parallel else 1)
    info = package.info
    engine = nb.Engine(package)
    if tensor_parallel:
        unique_id = torch.zeros(128, dtype=torch.uint8, device="cuda")
        if rank == 0:
            unique_id.copy_(torch.frombuffer(bytearray(nb.tensor_parallel_unique_id()), dtype=torch.uint8))
        dist.broadcast(unique_id, src=0)
        engine.init_tensor_parallel(rank, world, bytes(unique_id.cpu().numpy().tobytes()))
        if peer_exchange:  # the persistent kernel's exchange over peer memory: handles travel through the process group
            mine = torch.frombuffer(bytearray(engine.tp_exchange_handle()), dtype=torch.uint8).cuda()
            handles = [torch.zeros(64, dtype=torch.uint8, device="cuda") for _ in range(world)]
            dist.all_gather(handles, mine)
            connected = torch.ones(1, dtype=torch.int32, device="cuda")
            try:
                engine.tp_connect([bytes(handle.cpu().numpy().tobytes()) for handle in handles])
            except nb.NerveError as error:  # e.g. no peer access between two of the GPUs
                print(f"rank {rank}: peer exchange not available ({error}); NCCL path", file=sys.stderr)
                connected.zero_()
            dist.all_reduce(connected, op=dist.ReduceOp.MIN)
            if int(connected.item()) == 0:  # all ranks or none: the others would wait for this one inside the kernel
                engine.set_decode_stack(False)
                peer_exchange = False
    if os.environ.get("NERVE_B200_DECODE_STACK", "1") == "0":  # the kernel-per-operator path, for comparisons
        engine.set_decode_stack(False)
    engine.set_prefill_chunk(PROMPT_TOKENS)
    engine.add_stream(0, seed=0, speculative_draft_tokens=DRAFTS)

    # ---- e2e: whole events through the public API (natural, then teacher-forced with the same tokens)
    natural_tokens, natural_report, _ = run_event(engine, 0, prompt, EVENT_TOKENS)
    natural_tokens, natural_report, natural_rate = run_event(engine, 0, prompt, EVENT_TOKENS)
    forced_tokens, forced_report, forced_rate = run_event(engine, 0, prompt, EVENT_TOKENS, teacher=natural_tokens)
    if forced_tokens != natural_tokens:
        raise RuntimeError("teacher-forced run diverged from the natural greedy run")
    # the short event the CPU oracle replays afterwards (rank 0): tokens and per-cycle acceptance of this very mount
    sample_run = short_event(engine, 0, prompt, 40)
    # the control of that replay (one GPU): the same event on the kernel-per-operator path, whose operators agree with
    # the oracle to the last bf16 bit in at least 97 % of their outputs - what the model's own chaos does to a token sequence
    control_run = None
    if world == 1 and info["target_decode_stack"] and os.environ.get("NERVE_B200_DECODE_STACK", "1") != "0":
        engine.set_decode_stack(False)
        control_run = short_event(engine, 0, prompt, 40)
        engine.set_decode_stack(True)

    # ---- value: exactly K cycles, device-timed, clocks sampled meanwhile
    teacher_long = None
    with ClockSampler(local_rank) as sampler:
        natural_timed, natural_timed_wall = timed_cycles(engine, 0, prompt, budget, warmup, steps, None, barrier)
    clocks = sampler.summary()
    # teacher tokens for the long forced run: the natural continuation of the same budget
    long_tokens, _, _ = run_event(engine, 0, prompt, budget)
    forced_timed, _ = timed_cycles(engine, 0, prompt, budget, warmup, min(steps, (budget - 8) // (DRAFTS + 1) - warmup), long_tokens, barrier)

    # ---- roofline of the dominant kernel: per-launch CUDA events around the INT4 linears of a few cycles
    engine.set_profiling(True)
    profiled, _ = timed_cycles(engine, 0, prompt, budget, warmup, min(steps, 16), None, barrier)
    engine.set_profiling(False)

    stack_kernel = bool(info["target_decode_stack"]) and os.environ.get("NERVE_B200_DECODE_STACK", "1") != "0" and (not tensor_parallel or peer_exchange)

    def reduce_max(value):
        if world == 1:
            return value
        tensor = torch.tensor([value], dtype=torch.float64, device="cuda")
        dist.all_reduce(tensor, op=dist.ReduceOp.MAX)
        return float(tensor.item())

    def reduce_sum(value):
        if world == 1 or tensor_parallel:  # tensor-parallel ranks all carry the one stream: nothing to add up
            return value
        tensor = torch.tensor([value], dtype=torch.float64, device="cuda")
        dist.all_reduce(tensor, op=dist.ReduceOp.SUM)
        return float(tensor.item())

    seconds = reduce_max(natural_timed.device_ms * 1e-3)
    tokens = reduce_sum(float(natural_timed.generated_tokens))
    forced_seconds = reduce_max(forced_timed.device_ms * 1e-3)
    forced_total = reduce_sum(float(forced_timed.generated_tokens))
    e2e_natural = reduce_sum(natural_rate)
    e2e_forced = reduce_sum(forced_rate)

    peak, peak_kind = measured_peaks()
    verify_ms = natural_timed.verify_ms_sum / max(1, natural_timed.verify_steps)
    verify_bytes = natural_timed.verify_bytes / max(1, natural_timed.verify_steps)
    verify_gbs = verify_bytes / (verify_ms * 1e-3) / 1e9
    int4_gbs = profiled.int4_bytes / (profiled.int4_ms * 1e-3) / 1e9 if profiled.int4_ms > 0 else 0.0
    line = {
        "metric": METRIC, "value": tokens / seconds, "unit": UNIT, "n_gpus": world, "steps": steps, "warmup": warmup,
        "ms_per_step": 1e3 * seconds / steps, "higher_is_better": True, "scaling": "strong" if tensor_parallel else "weak", "vs_baseline": None,
        "dtype": "int4 weights, bf16 activations, f32 accumulate", "data": "synthetic",
        "config": {**config, "parallelism": ((f"tp{world}: dense layers sharded by rows / columns, partial sums exchanged over peer memory inside the persistent kernel"
                                               if peer_exchange else f"tp{world}: dense layers sharded by rows / columns, 2 NCCL all-reduces per layer") if tensor_parallel
                                              else "replicated streams (one per GPU)") if world > 1 else "single GPU",
                   "capacity_tokens": capacity},
        "modes": {
            "natural": {"tokens_per_s": tokens / seconds, "acceptance": natural_timed.accepted_draft_token_count /
                        max(1, natural_timed.proposed_draft_token_count), "e2e_tokens_per_s": e2e_natural},
            "teacher_forced": {"tokens_per_s": forced_total / forced_seconds,
                               "acceptance": forced_timed.accepted_draft_token_count / max(1, forced_timed.proposed_draft_token_count),
                               "e2e_tokens_per_s": e2e_forced, "steps": forced_timed.cycle_count},
        },
        "verify_step": {"ms": verify_ms, "algorithmic_bytes": verify_bytes, "gbs": verify_gbs,
                        "frac_of_nominal_8tbs": verify_gbs / NOMINAL_HBM_GBS, "frac_of_measured_copy": verify_gbs / peak},
        # The dominant kernel is the persistent decode stack kernel (all layers of a stack in one launch; its
        # algorithmic bytes are the tile-major INT4 weights + scales + norm weights of the stack), or - with it
        # switched off - the per-matrix INT4 kernel.  traffic: DRAM bytes per launch = algorithmic bytes x the
        # ratio ncu measured on a four-layer launch of the same width (dram__bytes_read.sum + dram__bytes_write.sum
        # over algorithmic bytes; traffic grows in proportion to the layers); no capture of the per-matrix kernel
        # is kept, so its traffic is null.
        "roofline": {"kernel": "decode_stack_kernel" if stack_kernel else "linear_int4_mma_kernel", "bound": "hbm", "achieved": int4_gbs, "peak": peak, "peak_kind": peak_kind,
                     "unit": "GB/s", "frac": int4_gbs / peak,
                     "traffic": STACK_TRAFFIC_RATIO * profiled.int4_bytes / max(1, profiled.int4_launches) if stack_kernel else None,
                     "launches_timed": profiled.int4_launches,
                     "bytes_per_launch": profiled.int4_bytes / max(1, profiled.int4_launches)},
        "e2e": {"value": e2e_natural, "unit": UNIT,
                "h2d_bytes_per_step": natural_report.h2d_bytes / max(1, natural_report.cycle_count),
                "d2h_bytes_per_step": natural_report.d2h_bytes / max(1, natural_report.cycle_count),
                "event": f"prompt {PROMPT_TOKENS} + {EVENT_TOKENS} tokens via enqueue_input_event / run / run_until_idle; host wall clock around the "
                         "run_until_idle call that decodes everything after the first cycle"},
        "prefill": prefill_line(spec, run_event.prefill_ms),
        "gpu_launches": natural_timed.kernel_launches,
        "clocks": clocks,
        "package": {"verify_step_weight_bytes": info["verify_step_weight_bytes"], "draft_step_weight_bytes": info["draft_step_weight_bytes"],
                    "kv_bytes_per_token": info["kv_bytes_per_token"]},
    }
    if rank == 0 and not args.skip_cpu_baseline:
        # the CPU oracle follows the short event this mount just ran: parity of tokens and per-cycle acceptance, and -
        # on one GPU - the cpu_baseline sample (several GPUs: a shorter replay, enough to check the sharded run)
        if world == 1:
            engine.close()
            package.unmount()
        sample = cpu_cycle_sample(directory, seconds_budget=25.0 if world == 1 else 12.0, cuda_run=sample_run)
        line["parity"] = sample["parity"]
        if control_run is not None:
            control = cpu_cycle_sample(directory, seconds_budget=12.0, cuda_run=control_run)["parity"]
            line["parity"]["control_kernel_per_operator_path"] = {key: control[key] for key in (
                "tokens_compared", "cycles_compared", "tokens_equal", "accepted_equal", "divergences", "violations", "largest_gap_at_a_divergence")}
        if world == 1:
            line["cpu_baseline"] = {
                "value": sample["tokens_per_s"], "unit": UNIT, "cores": cores, "kind": "port",
                "sample": f"{sample['cycles']} speculative cycles (k=3) of the same package at a {SAMPLE_PROMPT_TOKENS}-token context "
                          f"({sample['ms_per_cycle']:.0f} ms per cycle), OpenMP over output rows"}
    if world > 1:
        barrier()  # the other ranks wait for rank 0's replay before the group is torn down
    if rank == 0:
        print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
