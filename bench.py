"""Benchmark of the SageAttention3 hot path (pre-pass + FP4 attention) on B200.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--workload NAME] [--impl reference]

One step = one pass of the hot path (smoothing, NVFP4 quantization, attention) over one batch of seeded
synthetic input.  Default workload: B=4, H=32, Nq=Nk=32768, D=128, bf16, non-causal -- the configuration the
reference's headline "attention TOPS at hd128, N=32k" is quoted on.  TOPS = 4*B*H*Nq*Nk*D / time
(halved for causal), the reference's formula (bench/bench_baseline.py:31 in the reference project).

With N > 1 (launched by torch.distributed.run, one rank per GPU) every rank runs the whole workload on its
own (batch, head) shard with no data-path collective (weak scaling); the reported value is the units all
ranks processed divided by the slowest rank's device time.  The same line carries, under "ulysses", the
strong-scaling arm of the two long-sequence video workloads (tokens sharded over the ranks, all-to-all before and
after attention; at N = 1 the plain call on the same workload), and under "parity" a check of the timed output: one
whole query tile of one head against the CPU oracle.

`--impl reference` times the reference's math on the host cores instead: the torch-fp32 CPU restatement of
the reference pipeline (the reference's own kernels only execute on sm_120 hardware), on a bounded sample
of the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import pathlib
import statistics
import subprocess
import sys
import threading
import time

ROOT = pathlib.Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

WORKLOADS = {
    # name: B, Hq, Hkv, Nq, Nk, D, causal, layout, input kwargs
    "c2_hd128_32k": dict(B=4, Hq=32, Hkv=32, Nq=32768, Nk=32768, D=128, causal=False, layout="HND",
                         inp=dict(k_offset_std=3.0)),
    "c2_hd64_32k": dict(B=4, Hq=64, Hkv=64, Nq=32768, Nk=32768, D=64, causal=False, layout="HND",
                        inp=dict(k_offset_std=3.0)),
    "c3_cogvideox": dict(B=2, Hq=48, Hkv=48, Nq=17776, Nk=17776, D=64, causal=False, layout="HND",
                         inp=dict(k_outlier_channels=4)),
    "c4_hunyuan": dict(B=1, Hq=24, Hkv=24, Nq=119056, Nk=119056, D=128, causal=False, layout="HND",
                       inp=dict(k_offset_std=2.0)),
    "c5_llama_gqa": dict(B=8, Hq=32, Hkv=8, Nq=8192, Nk=8192, D=128, causal=True, layout="NHD",
                         inp=dict(rope_base=500000.0)),
    "ncu_small": dict(B=1, Hq=16, Hkv=16, Nq=16384, Nk=16384, D=128, causal=False, layout="HND",
                      inp=dict(k_offset_std=3.0)),
    "ncu_small_hd64": dict(B=1, Hq=32, Hkv=32, Nq=16384, Nk=16384, D=64, causal=False, layout="HND",
                           inp=dict(k_offset_std=3.0)),
    "ncu_small_causal": dict(B=1, Hq=32, Hkv=8, Nq=8192, Nk=8192, D=128, causal=True, layout="NHD",
                             inp=dict(rope_base=500000.0)),
    "c1_small": dict(B=1, Hq=2, Hkv=2, Nq=1024, Nk=1024, D=128, causal=False, layout="HND",
                     inp=dict(k_offset_std=3.0)),
}
NOMINAL_FP4_TFLOPS = 9000.0     # dense NVFP4, B200 datasheet
FALLBACK_HBM_GBS, FALLBACK_BF16_TFLOPS = 6650.0, 1590.0


def flops_of(w) -> float:
    f = 4.0 * w["B"] * w["Hq"] * w["Nq"] * w["Nk"] * w["D"]
    return f / 2 if w["causal"] else f


def prepass_bytes_of(w) -> float:
    """Algorithmic bytes of the pre-pass: every input element read once (2 B), its code (1/2 B) and scale
    (1/16 B) written once, plus delta_s and the means in 16 bit."""
    nqp, nkp = -(-w["Nq"] // 128) * 128, -(-w["Nk"] // 128) * 128
    nq_el = w["B"] * w["Hq"] * w["Nq"] * w["D"]
    nk_el = w["B"] * w["Hkv"] * w["Nk"] * w["D"]
    b = (nq_el + 2 * nk_el) * (2 + 0.5 + 1 / 16)
    b += 2.0 * w["B"] * w["Hq"] * (nqp // 128) * nkp
    b += 2.0 * (w["B"] * w["Hkv"] * w["D"] + w["B"] * w["Hq"] * (nqp // 128) * w["D"])
    return b


def launches_per_step(w, base: int) -> int:
    """Kernels of one call: `base` (stage, K and attention; one more for q.km, which the stand-alone pre-pass and the LSE need) and
    one for the K mean beyond 16 384 keys."""
    return base + (1 if w["Nk"] > 16384 else 0)


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return dict(hbm_gbs=d["hbm_gbs"], bf16=d["bf16_tflops"], bf16_sustained=d.get("bf16_tflops_sustained", d["bf16_tflops"]),
                    source="measured")
    return dict(hbm_gbs=FALLBACK_HBM_GBS, bf16=FALLBACK_BF16_TFLOPS, bf16_sustained=1400.0, source="fallback")


class ClockSampler:
    """Samples SM clocks and throttle reasons with nvidia-smi while the timed region runs."""
    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index, self.proc, self.lines = index, None, []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=lambda: self.lines.extend(self.proc.stdout), daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return dict(sm_mhz=None, sm_max_mhz=None, reasons=["nvidia-smi unavailable"])
        self.proc.terminate()
        self.t.join(timeout=5)
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 7:
                continue
            try:
                sm.append(float(f[0])); mx.append(float(f[1]))
            except ValueError:
                continue
            for n, v in zip(names, f[3:7]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        busy = [x for x in sm if x > 0]
        return dict(sm_mhz=statistics.median(busy) if busy else None, sm_max_mhz=max(mx) if mx else None,
                    reasons=sorted(reasons), samples=len(sm))


# --------------------------------------------------------------------------------------------------
def cpu_reference_sample(w, n: int | None = None, heads: int | None = None):
    """One bounded sample of the workload on the host cores with the CPU oracle: `heads` query heads (default: the
    query heads of one kv head) of one batch entry at sequence length `n` (default min(N, 4096)), same dtype, head
    dim, mask and input distributions.  Returns (flops, seconds, description)."""
    import torch
    from oracle import sage3_oracle as O
    n = min(w["Nq"], 4096) if n is None else n
    group = w["Hq"] // w["Hkv"]
    hq = group if heads is None else heads
    hkv = max(1, hq // group)
    q, k, v = O.make_inputs(1, hq, hkv, n, n, w["D"], seed=4242, **w["inp"])
    t0 = time.perf_counter()
    O.sageattn3_oracle(q, k, v, is_causal=w["causal"])
    dt = time.perf_counter() - t0
    f = 4.0 * hq * n * n * w["D"] / (2 if w["causal"] else 1)
    return f, dt, f"{hq} query head(s) of one batch entry at Nq=Nk={n}, D={w['D']}, same distributions"


def cpu_baseline_report(w, cores: int, budget_s: float = 14.0):
    """The CPU oracle timed on the host cores: the small configuration at its full size, then one head of the
    benchmark workload at N = 4096 and N = 8192; the full-length figure is an extrapolation (time grows with N^2
    at fixed width) and is labelled as one."""
    import torch
    torch.set_num_threads(cores)
    c1 = WORKLOADS["c1_small"]
    out, t_start = {}, time.perf_counter()
    f, dt, _ = cpu_reference_sample(c1, n=c1["Nq"], heads=c1["Hq"])          # warm-up (thread pool, allocator)
    f, dt, d1 = cpu_reference_sample(c1, n=c1["Nq"], heads=c1["Hq"])
    out["c1_small_full_size"] = dict(tops=f / dt / 1e12, seconds=dt, sample=d1)
    best = None
    for n in (4096, 8192):
        if n > w["Nq"] or time.perf_counter() - t_start > budget_s:
            break
        f, dt, dn = cpu_reference_sample(w, n=n)
        out[f"N{n}"] = dict(tops=f / dt / 1e12, seconds=dt, sample=dn)
        best = (f / dt / 1e12, n, dt, dn)
    if best is None:
        f, dt, dn = cpu_reference_sample(w)
        best = (f / dt / 1e12, min(w["Nq"], 4096), dt, dn)
    tops, n, dt, dn = best
    group = w["Hq"] // w["Hkv"]
    full_s = dt * (w["Nq"] / n) ** 2 * (w["B"] * w["Hq"] / group)
    return dict(value=tops, unit="TOPS", cores=cores, kind="port", sample=dn, measured=out,
                extrapolated_seconds_for_the_whole_workload=full_s,
                extrapolation="EXTRAPOLATED, not measured: time of the largest measured sample x (N / n)^2 x (batch x heads)")


def parity_of_timed_output(w, qh, kh, vh, oh, tile: int | None = None):
    """One whole 128-row query tile of the output the timed steps produced, against the CPU oracle run on the same
    inputs.  qh / oh: [1, group, N, D] host tensors (the query heads of kv head 0 of batch 0), kh / vh: [1, 1, N, D].
    The oracle quantizes the whole head, then evaluates the sampled rows against all keys."""
    from oracle import sage3_oracle as O
    nt = (w["Nq"] + 127) // 128
    tile = nt // 3 if tile is None else tile
    rows = slice(tile * 128, min(w["Nq"], (tile + 1) * 128))
    pp = O.prepass(qh, kh, vh)
    ref = O.attention_from_prepass(pp, is_causal=w["causal"], q_rows=slice(tile * 128, (tile + 1) * 128))
    got = oh[:, :, rows]
    return dict(cos=O.cosine(got, ref), rel_l1=O.rel_l1(got, ref), rows=f"batch 0, kv head 0, query rows {rows.start}..{rows.stop - 1}",
                gate="cos >= 0.999 and rel_l1 <= 0.01 against the CPU oracle")


def run_reference(args, w):
    """`--impl reference`: the reference's math on the host cores (rank 0 only)."""
    if int(os.environ.get("RANK", "0")) != 0:
        return
    import torch
    cores = os.cpu_count() or 1
    torch.set_num_threads(cores)
    for _ in range(max(args.warmup, 0)):
        cpu_reference_sample(w)
    tot_f, tot_t, desc = 0.0, 0.0, ""
    for _ in range(args.steps):
        f, dt, desc = cpu_reference_sample(w)
        tot_f += f
        tot_t += dt
    tops = tot_f / tot_t / 1e12
    line = dict(impl="reference", metric="attention TOPS (4*B*H*Nq*Nk*D/t) of the smooth+NVFP4-quantize+attend path", value=tops,
                unit="TOPS", n_gpus=args.gpus, steps=args.steps, warmup=args.warmup, ms_per_step=1e3 * tot_t / args.steps,
                higher_is_better=True, scaling="weak", vs_baseline=None, dtype="fp4 (e2m1 x ue4m3), fp32 accumulate", data="synthetic",
                config=dict(workload=args.workload, **{k_: w[k_] for k_ in ("B", "Hq", "Hkv", "Nq", "Nk", "D", "causal", "layout")}),
                cpu_baseline=dict(value=tops, unit="TOPS", cores=cores, kind="port", sample=desc + " per step"),
                e2e=dict(value=tops, unit="TOPS", h2d_bytes_per_step=0, d2h_bytes_per_step=0), gpu_launches=0)
    print(json.dumps(line))


def make_inputs_on_device(w, dev, seed, Nq=None, Nk=None):
    """Seeded synthetic input of a workload, generated on the device (the full tensors are several GB)."""
    import torch
    g = torch.Generator(device=dev).manual_seed(seed)
    B, Hq, Hkv, D = (w[k_] for k_ in ("B", "Hq", "Hkv", "D"))
    Nq, Nk = (w["Nq"] if Nq is None else Nq), (w["Nk"] if Nk is None else Nk)
    shp_q = (B, Hq, Nq, D) if w["layout"] == "HND" else (B, Nq, Hq, D)
    shp_k = (B, Hkv, Nk, D) if w["layout"] == "HND" else (B, Nk, Hkv, D)
    q = torch.empty(shp_q, dtype=torch.bfloat16, device=dev).normal_(generator=g)
    k = torch.empty(shp_k, dtype=torch.bfloat16, device=dev).normal_(generator=g)
    v = torch.empty(shp_k, dtype=torch.bfloat16, device=dev).normal_(generator=g)
    off_std = w["inp"].get("k_offset_std", 0.0)
    if off_std:
        off_shape = (B, Hkv, 1, D) if w["layout"] == "HND" else (B, 1, Hkv, D)
        k += (off_std * torch.randn(off_shape, device=dev, generator=g)).to(torch.bfloat16)
    if w["inp"].get("k_outlier_channels"):
        idx = torch.randperm(D, device=dev, generator=g)[: w["inp"]["k_outlier_channels"]]
        k[..., idx] *= 2
    # (RoPE of the Llama-shaped workload changes values, not shapes or timing; the parity tests cover it.)
    return q, k, v


def time_sequence_parallel(name, steps, warmup, rank, world, dev, ring=False, overlap_groups=1, peer=False):
    """Strong-scaling arm on workload `name`: every rank holds the token shard [rank N/P, (rank + 1) N/P) of all heads;
    one step = exchange, pre-pass, attention, exchange (at one GPU: the plain call).  The exchange is NCCL all-to-alls
    (`ulysses_attention`) or, with `peer`, direct loads and stores in the other ranks' buffers (`PeerUlysses`).
    Device time, max over ranks."""
    import torch
    import torch.distributed as dist
    from sageattention_b200 import sageattn3
    from sageattention_b200.ulysses import PeerUlysses, ring_attention, ulysses_attention
    w = WORKLOADS[name]
    if w["Nq"] % world or w["Hq"] % world or w["Hkv"] % world or w["causal"]:
        return dict(skipped=f"token / head counts of {name} are not divisible by {world} GPUs")
    q, k, v = make_inputs_on_device(w, dev, 7000 + rank, w["Nq"] // world, w["Nk"] // world)
    stream = torch.cuda.current_stream()
    prof = []

    pu = None
    if peer and world > 1:
        # the shards live in the buffers every rank has mapped, as when a caller's projections write there directly
        # (`PeerUlysses.stage()`); both alternating buffer sets are filled once, outside the timed region
        pu = PeerUlysses(w["B"], w["Hq"], w["Hkv"], w["Nq"] // world, w["D"], torch.bfloat16, device=dev)
        for views in pu._views:
            for dst, src in zip(views[:3], (q, k, v)):
                dst.copy_(src)

    def step(profile=None):
        if world == 1:
            return sageattn3(q, k, v, tensor_layout=w["layout"])
        if pu is not None:
            return pu(*pu.stage())
        if ring:
            return ring_attention(q, k, v, tensor_layout=w["layout"])
        return ulysses_attention(q, k, v, tensor_layout=w["layout"], overlap_groups=overlap_groups, profile=profile)

    for _ in range(max(warmup, 3)):
        step()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    a, b_ = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record(stream)
    for _ in range(steps):
        step()
    b_.record(stream)
    torch.cuda.synchronize()
    ms = a.elapsed_time(b_) / steps
    split = None
    if world > 1 and not ring and pu is None:
        step(prof)                                   # one more step with phase marks, outside the timed region
        torch.cuda.synchronize()
        ev = dict(prof)
        if all(n_ in ev for n_ in ("start", "exchanged_in", "attended", "exchanged_out")):
            split = [ev["start"].elapsed_time(ev["exchanged_in"]), ev["exchanged_in"].elapsed_time(ev["attended"]),
                     ev["attended"].elapsed_time(ev["exchanged_out"])]
        t = torch.tensor([ms] + (split or [0.0, 0.0, 0.0]), device=dev, dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms, split = t[0].item(), (t[1:].tolist() if split else None)
    elif world > 1:
        t = torch.tensor([ms], device=dev, dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = t.item()
    if pu is not None:
        pu.close()
    del q, k, v
    torch.cuda.empty_cache()
    res = dict(tops=flops_of(w) / (ms * 1e-3) / 1e12, ms_per_step=ms, steps=steps, scaling="strong",
               tokens_per_rank=w["Nq"] // world, heads_per_rank=w["Hq"] // world,
               sharding=("one GPU: plain call" if world == 1 else
                         "ulysses sequence parallel, peer to peer: shards read and written in place over NVLink, two barriers" if pu is not None else
                         "ring attention (NCCL send/recv of K/V shards, LSE merge)" if ring else
                         "ulysses sequence parallel: NCCL all-to-all before and after attention"))
    if split:
        res.update(exchange_in_ms=split[0], attn_ms=split[1], exchange_out_ms=split[2], a2a_ms=split[0] + split[2])
        res["all_to_all_bytes_per_rank_per_step"] = 4 * (world - 1) / world * (w["B"] * w["Hq"] * (w["Nq"] // world) * w["D"]) * 2
    return res


def run_ulysses(args, w, rank, world, local, dev):
    """`--ulysses`: the strong-scaling arm alone, as its own JSON line."""
    import torch.distributed as dist
    sampler = ClockSampler(local)
    if rank == 0:
        sampler.start()
    res = time_sequence_parallel(args.workload, args.steps, args.warmup, rank, world, dev, ring=args.ring,
                                 overlap_groups=max(1, args.overlap_groups), peer=args.peer)
    clocks = sampler.stop() if rank == 0 else None
    if rank == 0:
        if "skipped" in res:
            raise SystemExit(res["skipped"])
        groups = max(1, args.overlap_groups)
        print(json.dumps(dict(
            metric="attention TOPS (4*B*H*Nq*Nk*D/t) of the smooth+NVFP4-quantize+attend path", value=res["tops"], unit="TOPS",
            n_gpus=world, steps=args.steps, warmup=max(args.warmup, 3), ms_per_step=res["ms_per_step"], higher_is_better=True,
            scaling="strong", vs_baseline=None, dtype="fp4 (e2m1 x ue4m3), fp32 accumulate", data="synthetic",
            config=dict(workload=args.workload, l2="inputs larger than L2", head_slices_in_flight=groups,
                        **{k_: v_ for k_, v_ in res.items() if k_ not in ("tops", "ms_per_step", "steps", "scaling")}),
            clocks=clocks, gpu_launches=((launches_per_step(w, 4) + 1) * world if args.ring else launches_per_step(w, 3) * groups + 4) * args.steps)))
    if world > 1:
        dist.destroy_process_group()


# --------------------------------------------------------------------------------------------------
def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--workload", default="c2_hd128_32k", choices=sorted(WORKLOADS))
    ap.add_argument("--impl", default="sage3_b200", choices=["sage3_b200", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=4)
    ap.add_argument("--no-cpu-baseline", action="store_true", help="skip the CPU oracle legs (cpu_baseline and the parity check)")
    ap.add_argument("--no-ulysses", action="store_true", help="skip the sequence-parallel arm of the default line")
    ap.add_argument("--ulysses", action="store_true",
                    help="strong scaling: the workload's tokens are sharded over the ranks (all-to-all before and after attention)")
    ap.add_argument("--ring", action="store_true", help="with --ulysses: ring attention instead of the all-to-all exchange")
    ap.add_argument("--peer", action="store_true", help="with --ulysses: peer-to-peer exchange (PeerUlysses) instead of NCCL all-to-alls")
    ap.add_argument("--overlap-groups", type=int, default=0,
                    help="with --ulysses: head slices whose all-to-all overlaps the kernels of the others (0 = one slice, no overlap)")
    args = ap.parse_args()
    w = WORKLOADS[args.workload]
    if args.impl == "reference":
        run_reference(args, w)
        return

    import torch
    import torch.distributed as dist
    from sageattention_b200 import Sage3Problem, sageattn3_offload

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world != args.gpus:
        raise SystemExit(f"--gpus {args.gpus} but WORLD_SIZE={world}: launch with torch.distributed.run --nproc-per-node {args.gpus}")
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        # NCCL prints its version banner to stdout while the communicator is created; stdout is for the one
        # JSON line, so file descriptor 1 points at stderr until the first collective has completed
        sys.stdout.flush()
        saved_stdout = os.dup(1)
        os.dup2(2, 1)
        try:
            dist.init_process_group("nccl", device_id=dev)
            dist.barrier()
            torch.cuda.synchronize()
        finally:
            os.dup2(saved_stdout, 1)
            os.close(saved_stdout)

    B, Hq, Hkv, Nq, Nk, D = (w[k_] for k_ in ("B", "Hq", "Hkv", "Nq", "Nk", "D"))
    if args.ulysses:
        run_ulysses(args, w, rank, world, local, dev)
        return
    q, k, v = make_inputs_on_device(w, dev, 2000 + rank)
    flops = flops_of(w)
    stream = torch.cuda.current_stream()
    prob = Sage3Problem(q, k, v, tensor_layout=w["layout"], is_causal=w["causal"])

    def step(ev=None):
        if ev is not None:
            ev[0].record(stream)
        prob.prepass()
        if ev is not None:
            ev[1].record(stream)
        prob.attention()
        if ev is not None:
            ev[2].record(stream)

    for _ in range(max(args.warmup, 3)):
        step()
    torch.cuda.synchronize()
    prob.check_status()

    sampler = ClockSampler(local)
    if rank == 0:
        sampler.start()
        time.sleep(0.3)
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    evs = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(args.steps)]
    t_begin, t_end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t_begin.record(stream)
    for i in range(args.steps):
        step(evs[i])
    t_end.record(stream)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    clocks = sampler.stop() if rank == 0 else None
    total_ms = t_begin.elapsed_time(t_end)
    pre_ms = sum(e[0].elapsed_time(e[1]) for e in evs) / args.steps
    att_ms = sum(e[1].elapsed_time(e[2]) for e in evs) / args.steps
    prob.check_status()
    if world > 1:
        t = torch.tensor([total_ms, pre_ms, att_ms], device=dev, dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms, pre_ms, att_ms = t.tolist()

    # the output of the last timed step, for the parity check below (one head's worth of rows goes to the host)
    parity_in = None
    if rank == 0 and not args.no_cpu_baseline:
        hnd = (lambda t_: t_) if w["layout"] == "HND" else (lambda t_: t_.transpose(1, 2))
        group = Hq // Hkv
        parity_in = tuple(hnd(t_)[:1, :n_].contiguous().cpu() for t_, n_ in ((q, group), (k, 1), (v, 1), (prob.out, group)))

    # end to end through the public call: pinned host tensors in, host tensor out, copies inside the timed region
    e2e = None
    if args.e2e_steps > 0:
        qh, kh, vh = (t_.cpu().pin_memory() for t_ in (q, k, v))
        oh = torch.empty(q.shape, dtype=q.dtype).pin_memory()
        del prob
        torch.cuda.synchronize()

        def e2e_step():
            # the public call for host-resident operands: copies in, pre-pass, attention and copy out, pipelined
            # over (batch, kv-head) chunks; it returns when the result is in host memory
            sageattn3_offload(qh, kh, vh, out=oh, tensor_layout=w["layout"], is_causal=w["causal"], device=dev)

        for _ in range(3):          # warm-up: allocator, pinned pages, clocks
            e2e_step()
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        a, b_ = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(args.e2e_steps):
            e2e_step()
        b_.record(stream)
        torch.cuda.synchronize()
        e2e_ms = a.elapsed_time(b_) / args.e2e_steps
        if world > 1:
            t = torch.tensor([e2e_ms], device=dev, dtype=torch.float64)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            e2e_ms = t.item()
        nbytes = lambda t_: t_.numel() * t_.element_size()
        e2e = dict(value=world * flops / (e2e_ms * 1e-3) / 1e12, unit="TOPS", ms_per_step=e2e_ms,
                   h2d_bytes_per_step=world * (nbytes(qh) + nbytes(kh) + nbytes(vh)), d2h_bytes_per_step=world * nbytes(oh))     # whole job
        del qh, kh, vh, oh
        from sageattention_b200 import sageattn3_offload_release
        sageattn3_offload_release()
    else:
        del prob
    del q, k, v
    torch.cuda.empty_cache()

    # strong-scaling arm (sequence parallel) on the two long-sequence video workloads, every rank takes part
    ulysses = None
    if args.workload == "c2_hd128_32k" and not args.no_ulysses:
        ulysses = {}
        for name, n_steps in (("c4_hunyuan", 5), ("c3_cogvideox", 10)):
            res = time_sequence_parallel(name, n_steps, 3, rank, world, dev)
            if world > 1 and "skipped" not in res:
                # both transports; the headline of the arm is the faster one, the other is kept beside it
                res_p = time_sequence_parallel(name, n_steps, 3, rank, world, dev, peer=True)
                best, other = (res_p, res) if res_p["tops"] >= res["tops"] else (res, res_p)
                res = dict(best, other_transport=other)
            ulysses[name] = res

    if rank != 0:
        if world > 1:
            dist.destroy_process_group()
        return

    peaks = measured_peaks()
    ms_per_step = total_ms / args.steps
    att_tops = flops / (att_ms * 1e-3) / 1e12
    fp4_peak = 4.0 * peaks["bf16_sustained"]          # dense FP4 is 4x dense bf16 on this part
    # DRAM traffic of one attention launch: a constant taken from one stored ncu capture of the small profiling case
    # (16 heads x 16384 tokens, D = 128: 160.6 MB = dram__bytes_read.sum + dram__bytes_write.sum), scaled by B*H*N; the
    # kernel reads each head's operands once from DRAM and writes its output once, so its traffic grows in that proportion.
    traffic, traffic_src = None, None
    if D == 128 and not w["causal"]:
        traffic = 160.6e6 * (B * Hq * Nq) / (16 * 16384.0)
        traffic_src = "constant from a stored ncu capture of a smaller case (not measured in this run), scaled in proportion to B*H*N"
    line = dict(
        metric="attention TOPS (4*B*H*Nq*Nk*D/t) of the smooth+NVFP4-quantize+attend path", value=world * flops / (ms_per_step * 1e-3) / 1e12,
        unit="TOPS", n_gpus=world, steps=args.steps, warmup=max(args.warmup, 3), ms_per_step=ms_per_step, higher_is_better=True,
        scaling="weak", vs_baseline=None, dtype="fp4 (e2m1 x ue4m3), fp32 accumulate", data="synthetic",
        config=dict(workload=args.workload, B=B, Hq=Hq, Hkv=Hkv, Nq=Nq, Nk=Nk, D=D, causal=w["causal"], layout=w["layout"],
                    in_dtype="bf16", l2="inputs larger than L2 (3.2 GB of q/k/v per step)" if flops > 1e12 else "small case, L2 resident",
                    sharding="independent (batch, head) shards per rank, no collective"),
        attn_kernel=dict(ms=att_ms, tops=att_tops), prepass=dict(ms=pre_ms, gbs=prepass_bytes_of(w) / (pre_ms * 1e-3) / 1e9,
                                                                 frac_of_hbm_peak=prepass_bytes_of(w) / (pre_ms * 1e-3) / 1e9 / peaks["hbm_gbs"],
                                                                 algorithmic_bytes=prepass_bytes_of(w)),
        roofline=dict(bound="tensor", kernel="attn_fwd_kernel", achieved=att_tops, peak=fp4_peak, unit="TFLOP/s", frac=att_tops / fp4_peak,
                      traffic=traffic, traffic_source=traffic_src, peak_source=f"4 x bf16_tflops_sustained of MEASURED_PEAKS.json ({peaks['source']})",
                      frac_of_nominal_fp4=att_tops / NOMINAL_FP4_TFLOPS),
        clocks=clocks, e2e=e2e, gpu_launches=launches_per_step(w, 4) * args.steps, ulysses=ulysses,
    )
    if not args.no_cpu_baseline:
        line["parity"] = parity_of_timed_output(w, *parity_in)
        line["cpu_baseline"] = cpu_baseline_report(w, os.cpu_count() or 1)
    print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
