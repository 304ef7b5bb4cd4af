"""Benchmark of the Gemma4 decode step.  python bench.py --gpus N --steps K --warmup W

One "step" = one decode step (one new token for every sequence of the batch) through all layers,
the tied LM head and the fused arg-max. Prints ONE JSON line (rank 0).

  value      decode tokens/s with everything resident in HBM: the captured step graph is replayed
             K times, each step's arg-max fed back on the device (oxg4_decode_greedy), timed with
             CUDA events on the library's stream.
  e2e        the same metric through the public per-token call (decode_topk): every step copies
             the token ids host->device, replays the graph, copies (id, score) device->host and
             synchronises, exactly what the reference's generate loop does per token.
  roofline   dominant kernel (gate/up projection): algorithmic bytes / mean device time of that
             kernel, measured with CUDA events around each launch in eager profiling steps run
             right after the timed region; `step_*` keys give the whole-step figure.
  cpu_baseline / --impl reference: the CPU oracle (a port of the reference's arithmetic; the
             reference has no CPU forward pass of its own) on this box's host cores.
  tp         (default workload only) the ~12B workload tensor-parallel over all N ranks, N = 1 included:
             tokens/s, step time, per-kind kernel times and the time spent in the per-layer all-reduces,
             so that a 1/2/4/8-GPU series of this command also measures the path's real exchange step
             (the default ~4B workload itself runs one replica per GPU: no data-path collective).

Weights are seeded random N(0, 0.02) (generated with torch on the GPU when one is present, then
handed to the library through its host-pointer upload call); prompts are seeded uniform ids.
Inputs streamed per step (weights + KV) are far larger than the 126 MB L2, so no L2 flush is needed.
"""
import argparse
import importlib
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "decode_tokens_per_s"
UNIT = "tok/s"
DEFAULT_WORKLOAD = "c3"          # ~4B-class, batch 1: the configuration the 70%-of-HBM target is quoted on
# gate/up launch: dram read + write bytes per launch from the ncu captures summarised in profiles/ (the tcgen05 kernel on the
# ~12B widths, single GPU; the one-row kernel has not been captured in its present form)
NCU_TRAFFIC_BYTES = {"c4": 246000000}
TP_RECORD_PROMPT = 8192          # prompt length of the tensor-parallel (~12B) record that accompanies the default run


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def algorithmic_bytes(cfg, batch, contexts, wb=2, kvb=2):
    """weights + KV bytes one decode step must read (activations and KV writes excluded)."""
    H, D = cfg["hidden_size"], cfg["head_dim"]
    Nq, Nkv, I, V = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["intermediate_size"], cfg["vocab_size"]
    per_layer = (H * (Nq + 2 * Nkv) * D + Nq * D * H + 3 * H * I) * wb
    total = cfg["num_hidden_layers"] * per_layer + V * H * wb
    kv = 0
    for t in cfg["layer_types"]:
        for ctx in contexts:
            vis = min(ctx, cfg["sliding_window"]) if t == "sliding_attention" else ctx
            kv += 2 * vis * Nkv * D * kvb
    return total + kv, {"weights": total, "kv": kv, "gateup_launch": 2 * I * H * wb}


def torch_weights(cfg, device):
    """Seeded N(0, 0.02) BF16 weights generated on `device`, yielded as (name, uint16 array)."""
    import torch
    syn = importlib.import_module("oxide-beta_b200").synthetic
    gen = torch.Generator(device=device).manual_seed(0)
    for name, shape, kind in syn.weight_names(cfg):
        if kind == "matrix":
            t = torch.empty(shape, dtype=torch.float32, device=device).normal_(0.0, 0.02, generator=gen)
        else:
            t = torch.ones(shape, dtype=torch.float32, device=device)
        yield name, t.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)


class ClockSampler:
    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits",
                                          "-lms", "100", "-i", str(self.gpu)], stdout=self.file,
                                         stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self):
        out = {"sm_mhz": None, "sm_max_mhz": None, "reasons": []}
        if self.proc is None:
            return out
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.file.flush()
        self.file.seek(0)
        sm, mx, reasons = [], [], set()
        for line in self.file.read().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for name, v in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"), f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(name)
        os.unlink(self.file.name)
        if sm:
            out = {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                   "samples": len(sm)}
        return out


def cpu_oracle_run(cfg, weights_iter, prompt, steps, warmup):
    """Times the CPU oracle: ingests `prompt`, then `warmup` + `steps` greedy decode steps."""
    from oracle import oracle as orc
    orc.set_num_threads(os.cpu_count() or 1)      # torchrun exports OMP_NUM_THREADS=1
    m = orc.OracleModel(cfg, orc.REF_BF16, kv_bf16=True)
    for name, a in weights_iter:
        m.set_weight(name, a)
    cache = m.new_cache(len(prompt) + steps + warmup + 1)
    for t in prompt[:-1]:
        cache.prefill_token(int(t))
    tok = int(prompt[-1])
    for _ in range(warmup):
        tok = int(cache.decode_topk(tok, 1, 1.0, False)[0][0])
    t0 = time.perf_counter()
    for _ in range(steps):
        tok = int(cache.decode_topk(tok, 1, 1.0, False)[0][0])
    dt = time.perf_counter() - t0
    return steps / dt, dt, orc.num_threads()


def run_workload(pkg, dist, rank, local_rank, world, name, tp, prompt_len, steps, warmup, layers=None, vocab=None,
                 keep_host=False, e2e=True, sampler=None, cache_fill="prefill"):
    """Loads workload `name` (tensor-parallel over `tp` ranks, or one replica per rank), ingests the
    prompts, then times `steps` decode steps after `warmup`. Returns the measurements of this rank
    (times already reduced to the maximum over ranks)."""
    import torch
    syn = pkg.synthetic
    w = syn.workload(name)
    cfg, B = w["cfg"], w["batch"]
    if layers or vocab:
        cfg = syn.scaled_down(cfg, layers=layers, vocab=vocab)
    if prompt_len is None:
        prompt_len = w["prompt"] if isinstance(w["prompt"], int) else None
    t_load = time.perf_counter()
    state = pkg.Gemma4CudaState(pkg.Gemma4TextConfig(cfg), local_rank, pkg.BF16, tp_rank=rank if tp > 1 else 0,
                                tp_size=tp)
    host_weights = []
    for wname, a in torch_weights(cfg, f"cuda:{local_rank}"):
        state.upload(wname, a)
        if keep_host:
            host_weights.append((wname, a))
    state.finalize()
    if tp > 1:
        ids = [pkg.Gemma4CudaState.tp_unique_id() if rank == 0 else None]
        dist.broadcast_object_list(ids, src=0)
        state.tp_init(ids[0])
    torch.cuda.empty_cache()
    load_s = time.perf_counter() - t_load

    if prompt_len is None:           # ragged workload: per-sequence prompt lengths from seed 2
        lens = syn.ragged_lengths(B, w["prompt"][0], w["prompt"][1], seed=2).tolist()
    else:
        lens = [prompt_len] * B
    total_steps = warmup + steps
    max_seq = [n + 2 * total_steps + 16 for n in lens]
    table = state.new_cache_table(max_seq, batch=B, kv_dtype=pkg.BF16)
    tp_exchange = "nccl"
    if tp > 1 and 8 <= B <= 64 and not os.environ.get("OXG4_TP_NCCL"):
        # the sums after O and down travel through peer memory (plain stores into the other ranks' gather buffers)
        # instead of NCCL all-reduces: measured faster (~12B workload, 4 GPUs: 7.60 vs 8.10 ms per step)
        handles = [None] * world
        dist.all_gather_object(handles, table.tp_export())
        table.tp_connect(handles)
        tp_exchange = "peer-memory"
    t_pre = time.perf_counter()
    if cache_fill == "synthetic":
        # the K/V pools receive a pseudo-random pattern instead of the prompts' K/V: same bytes per step, no prefill
        table.fill_synthetic(lens)
        first = (np.arange(B, dtype=np.uint32) * 7919 + 11) % cfg["vocab_size"]
    else:
        prompts = [syn.prompt_ids(cfg["vocab_size"], n, seed=1 + b) for b, n in enumerate(lens)]
        logits = state.prefill_prompt(np.concatenate(prompts), table, lens=lens)
        first = np.atleast_2d(logits).argmax(-1).astype(np.uint32)
    prefill_s = time.perf_counter() - t_pre

    # device-resident loop: warm-up, then the timed K steps bracketed by barrier + synchronize
    ids, _ = state.decode_greedy(first, table, warmup)
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    if sampler:
        sampler.start()                    # SM clocks and throttle reasons DURING the timed region
    launches1 = state.kernel_launches()
    ids, ms_step = state.decode_greedy(ids[-1], table, steps)
    torch.cuda.synchronize()
    launches_timed = state.kernel_launches() - launches1
    if dist:
        dist.barrier()
    tok = ids[-1].copy()
    e2e_s, e2e_steps, inter_token_ms = float("nan"), 0, [float("nan")]
    if e2e:
        # end to end: the per-token public call with host buffers (H2D token ids, D2H (id, score), one sync)
        for _ in range(3):
            r = state.decode_topk(tok, table, 1, 1.0, True)
            tok = np.array([r[0][0]], dtype=np.uint32) if B == 1 else r[0][:, 0].copy()
        e2e_steps = min(steps, total_steps - 3)
        t0 = time.perf_counter()
        stamps = [t0]
        for _ in range(e2e_steps):
            r = state.decode_topk(tok, table, 1, 1.0, True)
            tok = np.array([r[0][0]], dtype=np.uint32) if B == 1 else r[0][:, 0].copy()
            stamps.append(time.perf_counter())
        e2e_s = stamps[-1] - t0
        inter_token_ms = sorted(1000.0 * (b_ - a_) for a_, b_ in zip(stamps[:-1], stamps[1:]))
    clocks = sampler.stop() if sampler else None
    if dist:
        t = torch.tensor([ms_step, e2e_s if e2e else 0.0], device="cuda", dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms_step, e2e_s = float(t[0]), float(t[1]) if e2e else e2e_s

    # per-kernel timing: eager steps with CUDA events around every launch and collective
    contexts = [table.position(b) for b in range(B)]
    prof, prof_step = {}, {}
    n_prof = 5
    for _ in range(n_prof):
        for k, v in state.profile_step(tok, table).items():
            prof[k] = prof.get(k, 0.0) + v / n_prof
        for k, v in state.profile_step(tok, table, totals=True).items():
            prof_step[k] = prof_step.get(k, 0.0) + v / n_prof
    step_bytes, parts = algorithmic_bytes(cfg, B, contexts)
    parts["gateup_launch"] //= tp          # a rank streams its shard of the projection
    if dist:
        dist.barrier()                     # no rank frees its cache table while a peer may still read it
    del table
    state.close()
    torch.cuda.empty_cache()
    return dict(cfg=cfg, B=B, lens=lens, tp=tp, tp_exchange=tp_exchange, ms_step=ms_step, e2e_s=e2e_s,
                e2e_steps=e2e_steps, inter_token_ms=inter_token_ms, contexts=contexts, prof=prof, prof_step=prof_step,
                step_bytes=step_bytes, parts=parts, load_s=load_s, prefill_s=prefill_s,
                launches_timed=int(launches_timed), host_weights=host_weights, steps=steps, warmup=warmup,
                clocks=clocks)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=256)
    ap.add_argument("--warmup", type=int, default=16)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default=DEFAULT_WORKLOAD)
    ap.add_argument("--prompt", type=int, default=None, help="override the prompt length")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-tp-record", action="store_true",
                    help="skip the tensor-parallel ~12B measurement that accompanies the default workload")
    ap.add_argument("--tp-prompt", type=int, default=TP_RECORD_PROMPT, help="prompt length of the tensor-parallel record")
    ap.add_argument("--cache-fill", default="prefill", choices=["prefill", "synthetic"],
                    help="synthetic: K/V pools filled with a pseudo-random pattern at the prompt lengths instead of "
                         "ingesting the prompts (decode timing at long contexts without the prefill time)")
    ap.add_argument("--layers", type=int, default=None, help="profiling aid: keep only the first LAYERS layers")
    ap.add_argument("--vocab", type=int, default=None, help="profiling aid: shrink the vocabulary")
    ap.add_argument("--design", default=None, choices=["pabovik", "nozurax"],
                    help="instead of the workload: prefill and decode throughput and per-kernel times of this design at a few "
                         "sizes, beside models of equal width, depth and feed-forward: Gemma 4, for nozurax also Pabovik (bench_layered.py)")
    args = ap.parse_args()
    if args.design:
        import bench_layered
        bench_layered.main(args.design)
        return
    warmup = max(args.warmup, 3)

    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    pkg = importlib.import_module("oxide-beta_b200")
    syn = pkg.synthetic

    import torch
    has_gpu = torch.cuda.is_available()

    # ------------------------------------------------------------------ reference arm (CPU oracle)
    if args.impl == "reference":
        if rank != 0:
            return
        # torchrun exports OMP_NUM_THREADS=1 to every rank; the CPU reference uses all host cores
        os.environ["OMP_NUM_THREADS"] = str(os.cpu_count() or 1)
        w = syn.workload(args.workload)
        cfg = w["cfg"]
        if args.layers or args.vocab:
            cfg = syn.scaled_down(cfg, layers=args.layers, vocab=args.vocab)
        # a bounded sample of the workload: the step count asked for, after a short prompt (ingesting the
        # full prompt token by token on the CPU would take minutes and is outside the timed region anyway)
        sample_prompt = 32
        steps = args.steps
        weights = torch_weights(cfg, "cuda:0" if has_gpu else "cpu")
        prompt = syn.prompt_ids(cfg["vocab_size"], sample_prompt, seed=1)
        tps, dt, cores = cpu_oracle_run(cfg, weights, prompt, steps, warmup)
        sample = (f"{steps} greedy decode steps at batch 1 after a {sample_prompt}-token prompt "
                  f"(full {args.workload} weights, BF16 recipe, OpenMP over {cores} threads)")
        print(json.dumps({
            "impl": "reference", "metric": METRIC, "value": tps, "unit": UNIT, "n_gpus": args.gpus, "steps": steps,
            "warmup": warmup, "ms_per_step": 1000.0 * dt / steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
            "config": {"workload": args.workload, "batch": 1, "prompt": sample_prompt,
                       "note": "CPU port of the reference arithmetic; the reference has no CPU forward pass"},
            "cpu_baseline": {"value": tps, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample},
            "e2e": {"value": tps, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}))
        return

    # ------------------------------------------------------------------ our arm
    if not has_gpu:
        raise SystemExit("bench.py needs a CUDA device: the library has no CPU path")
    torch.cuda.set_device(local_rank)
    dist = None
    # The one JSON line is the only thing this program writes to its standard output: libraries that print
    # there (NCCL announces its version on stdout) are sent to stderr for the length of the run.
    sys.stdout.flush()
    json_fd = os.dup(1)
    os.dup2(2, 1)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=torch.device("cuda", local_rank))

    # the 12B / 27B workloads are tensor-parallel across the ranks; the smaller ones run one replica per GPU
    tp = world if (world > 1 and args.workload in ("c4", "c5")) else 1
    keep_host = (rank == 0 and world == 1 and not args.no_cpu_baseline and args.workload in ("c1", "c2", "c3"))
    r = run_workload(pkg, dist, rank, local_rank, world, args.workload, tp, args.prompt, args.steps, warmup,
                     args.layers, args.vocab, keep_host=keep_host, sampler=ClockSampler(local_rank),
                     cache_fill=args.cache_fill)
    clocks = r["clocks"]
    cfg, B, lens, ms_step = r["cfg"], r["B"], r["lens"], r["ms_step"]
    replicas = world // tp
    value = replicas * B * 1000.0 / ms_step
    e2e_value = replicas * B * r["e2e_steps"] / r["e2e_s"]
    peak, peak_kind = peaks()
    gu_ms = r["prof"].get("gateup", float("nan"))
    achieved = r["parts"]["gateup_launch"] / (gu_ms * 1e-3) / 1e9
    # as the library picks it for BF16 weights (one sequence with projections of more than 1 MB per SM, which take gemv_kernel, is no workload)
    gu_kernel = ("gemv_mma_kernel<PRO_NORM, EPI_GATEUP>" if B < (8 if tp > 1 else 2) else
                 "tc_gemm_kernel (tcgen05, gate and up maps)" if B <= 256 else
                 "gemv_rows_kernel<PRO_NORM, EPI_GATEUP>")
    roofline = {"bound": "hbm", "kernel": gu_kernel + " (gate/up projection)",
                "achieved": achieved, "peak": peak, "peak_kind": f"of {peak_kind}", "unit": "GB/s",
                "frac": achieved / peak, "traffic": NCU_TRAFFIC_BYTES.get(args.workload) if tp == 1 else None,
                "bytes_per_launch": r["parts"]["gateup_launch"], "ms_per_launch": gu_ms,
                "step_bytes": r["step_bytes"], "step_achieved": r["step_bytes"] / (ms_step * 1e-3) / 1e9,
                "step_frac": r["step_bytes"] / (ms_step * 1e-3) / 1e9 / (peak * tp),
                "kernel_ms": {k: round(v, 5) for k, v in r["prof"].items()}}

    # the tensor-parallel record: the ~12B workload split over all N ranks (N = 1 included), so that the
    # 1/2/4/8-GPU series of the default workload also carries a strong-scaling curve with a real exchange
    tp_record = None
    if args.workload == DEFAULT_WORKLOAD and not args.no_tp_record and not (args.layers or args.vocab):
        t_steps, t_warm = min(args.steps, 64), min(warmup, 8)
        t = run_workload(pkg, dist, rank, local_rank, world, "c4", world, args.tp_prompt, t_steps, t_warm, e2e=False)
        ar = t["prof_step"].get("allreduce", 0.0) + t["prof_step"].get("allgather", 0.0)
        tp_record = {
            "workload": "c4", "tp": world, "batch": t["B"], "prompt": args.tp_prompt, "steps": t_steps, "warmup": t_warm,
            "context_at_timing": t["contexts"][0], "value": t["B"] * 1000.0 / t["ms_step"], "unit": UNIT,
            "ms_per_step": t["ms_step"], "scaling": "strong", "exchange": t["tp_exchange"] if world > 1 else "none",
            "step_bytes": t["step_bytes"], "step_frac": t["step_bytes"] / (t["ms_step"] * 1e-3) / 1e9 / (peak * world),
            "kernel_ms": {k: round(v, 5) for k, v in t["prof"].items()},
            "kernel_ms_per_step": {k: round(v, 4) for k, v in t["prof_step"].items()},
            "collectives_ms_per_step": round(ar, 4),
            "note": "eager event timing per launch (no overlap between launches); ms_per_step is the graph replay",
            "load_s": round(t["load_s"], 2), "prefill_s": round(t["prefill_s"], 2)}

    if rank != 0:
        dist.destroy_process_group()
        return
    out = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps, "warmup": warmup,
        "ms_per_step": ms_step, "higher_is_better": True, "scaling": "strong" if tp > 1 else "weak", "vs_baseline": None, "dtype": "bf16",
        "data": "synthetic",
        "config": {"workload": args.workload + (f" (reduced: layers={args.layers} vocab={args.vocab})"
                                                 if (args.layers or args.vocab) else ""),
                   "batch": B, "prompt": lens[0] if len(set(lens)) == 1 else "ragged",
                   "context_at_timing": r["contexts"][0] if len(set(lens)) == 1 else
                   {"min": min(r["contexts"]), "mean": round(sum(r["contexts"]) / B), "max": max(r["contexts"])},
                   "cache_fill": ("prompts ingested by the chunked prefill" if args.cache_fill == "prefill" else
                                  "synthetic: K/V pools filled with a pseudo-random pattern at the prompt lengths, no prefill"),
                   "kv_dtype": "bf16", "page_tokens": 256,
                   "parallelism": "single GPU" if world == 1 else (f"tp{tp} (sums after O and down: {r['tp_exchange']})"
                                                                   if tp > 1 else f"{world} independent replicas"),
                   "l2": "per-step inputs (weights + KV) exceed the 126 MB L2; no flush",
                   "load_s": round(r["load_s"], 2), "prefill_s": round(r["prefill_s"], 2)},
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": 4 * B + 28, "d2h_bytes_per_step": 8 * B,
                "steps": r["e2e_steps"], "p50_inter_token_ms": r["inter_token_ms"][len(r["inter_token_ms"]) // 2],
                "p95_inter_token_ms": r["inter_token_ms"][int(len(r["inter_token_ms"]) * 0.95)]},
        "gpu_launches": r["launches_timed"],
        "clocks": clocks,
        "roofline": roofline,
    }
    if tp_record is not None:
        out["tp"] = tp_record
    if keep_host:
        sample_prompt, cpu_steps = 32, 8
        tps, dt, cores = cpu_oracle_run(cfg, r["host_weights"], syn.prompt_ids(cfg["vocab_size"], sample_prompt, seed=1),
                                        cpu_steps, 2)
        out["cpu_baseline"] = {"value": tps, "unit": UNIT, "cores": cores, "kind": "port",
                               "sample": f"{cpu_steps} greedy decode steps at batch 1 after a {sample_prompt}-token "
                                         f"prompt, full {args.workload} weights, BF16 recipe"}
    sys.stdout.flush()
    os.write(json_fd, (json.dumps(out) + "\n").encode())
    if dist:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
