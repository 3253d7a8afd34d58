#!/usr/bin/env python
"""Benchmark of the FP8 GEMM path: the DeepSeek-V3 Linear shape sweep.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

One step = one pass of fp8_gemm over every (shape, M) pair of the sweep, M-major so that
540 MB of other weights stream between two uses of any weight (inputs larger than L2).
`value`  : aggregate fp8_gemm TFLOP/s with FP8 activations, weights and scales resident in HBM.
`e2e`    : the same sweep through the drop-in module (`kernel.act_quant` + `kernel.fp8_gemm`) with the
           bf16 activations in pinned host memory and the bf16 results read back to the host, every step.
`roofline`: the tcgen05 token-major kernel (launches with M >= 256), flops / CUDA-event time of its launches
           (each M column of the sweep is one CUDA graph, bracketed by events).
`cpu_baseline` / `--impl reference`: the CPU restatement of the reference's kernel.py (oracle/) on the
           host cores, on a bounded sample of the sweep (the M = 64 column).

N > 1: every rank holds the TP=N shard of each Linear (column-parallel N/ws, row-parallel K/ws followed
by an NCCL all_reduce of the partial output, as model.py:262-264 does); total work is fixed (strong scaling).
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

ROOT = os.path.dirname(os.path.abspath(__file__))
for _p in (ROOT, os.path.join(ROOT, "deepseek-v3_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

MS = [1, 8, 32, 64, 256, 1024, 4096, 16384]
# name, K (in), N (out), parallel kind under tensor parallelism (model.py:208-267)
BASE_SHAPES = [
    ("wq_a", 7168, 1536, "replicated"),
    ("wq_b", 1536, 24576, "column"),
    ("wkv_a", 7168, 576, "replicated"),
    ("wkv_b", 512, 32768, "column"),
    ("wo", 16384, 7168, "row"),
    ("dense_w13", 7168, 18432, "column"),
    ("dense_w2", 18432, 7168, "row"),
    ("expert_w13", 7168, 2048, "expert"),       # routed experts are never TP-sliced: a rank owns whole experts
    ("expert_w2", 2048, 7168, "expert"),
]
SHARED = [("shared_w13", 7168, 2048, "column"), ("shared_w2", 2048, 7168, "row")]


def shard(shape, tp):
    name, K, N, kind = shape
    if kind == "column":
        return (f"{name}/tp{tp}", K, N // tp, kind)
    if kind == "row":
        return (f"{name}/tp{tp}", K // tp, N, kind)
    return shape


def sweep_rows(world: int, rank: int = 0):
    """Rows of the sweep this rank executes: (name, K, N, kind, needs_all_reduce, counted).

    The global problem set is the same for every world size (the 9 full Linear shapes
    and 7 shapes that are already the TP=8 per-rank slice).  With more than one rank it is spread the way the
    reference's tensor parallelism spreads it (model.py:208-267, 636-666):
      * column-parallel: every rank N/ws rows of W; row-parallel: every rank K/ws columns of W, partial
        outputs summed with all_reduce;
      * replicated Linears (wq_a, wkv_a) run on every rank, as they do in the model; their flops are
        counted once;
      * whole-expert GEMMs and the ready-made TP=8 slices are single-rank problems: each is owned by one
        rank (round-robin), the way different ranks own different experts.
    `counted` says whether this rank's execution adds to the job's flop count."""
    slices = [shard(s, 8) for s in BASE_SHAPES + SHARED if s[3] in ("column", "row")]
    slices = [(n.replace("/tp8", "@tp8-slice"), k, o, kind) for n, k, o, kind in slices]
    if world == 1:
        rows = [(n, k, o, kind, False, True) for n, k, o, kind in BASE_SHAPES]
        rows += [(n, k, o, kind, False, True) for n, k, o, kind in slices]
        return rows
    rows = []
    owner = 0
    # row-parallel Linears first: their all_reduce is issued on a communication stream and overlaps the GEMMs after them
    for s in sorted(BASE_SHAPES, key=lambda r: 0 if r[3] == "row" else 1):
        n, k, o, kind = s
        if kind in ("column", "row"):
            n, k, o, kind = shard(s, world)
            rows.append((n, k, o, kind, kind == "row", True))
        elif kind == "replicated":
            rows.append((n, k, o, kind, False, rank == 0))
        else:  # expert
            if owner % world == rank:
                rows.append((n, k, o, kind, False, True))
            owner += 1
    for n, k, o, kind in slices:
        if owner % world == rank:
            rows.append((n, k, o, "slice", False, True))
        owner += 1
    return rows


def gemm_flops(M, N, K):
    return 2.0 * M * N * K


def gemm_bytes(M, N, K):
    kc = -(-K // 128)
    return M * K + N * K + 4 * M * kc + 4 * (-(-N // 128)) * kc + 2 * M * N


# ncu captures of one launch each (commands and figures in the named summaries): measured DRAM bytes,
# the (M, N, K) of the captured problem, the summary file.
NCU_TRAFFIC = {
    "token_major": (185.80e6 + 132.54e6, (4096, 18432, 7168), "profiles/fp8_gemm_tw_token_major_4096x18432x7168.md"),
    "weight_major": (117.67e6 + 4.22e6, (8, 7168, 16384), "profiles/fp8_gemm_tc_weight_major_8x7168x16384.md"),
}

def read_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return {"hbm_gbs": d["hbm_gbs"], "bf16_tflops": d["bf16_tflops"],
                "bf16_tflops_sustained": d.get("bf16_tflops_sustained", d["bf16_tflops"]), "source": "measured"}
    return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0, "source": "fallback"}


class ClockSampler:
    """Samples SM clock and throttle reasons of one GPU with nvidia-smi while a region runs."""
    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index, self.lines, self.proc = index, [], None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                          "-lms", "100", "-i", str(self.index)], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=lambda: self.lines.extend(self.proc.stdout), daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.t.join(timeout=5)
        sm, mx, pw, reasons = [], [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 7:
                continue
            try:
                sm.append(float(f[0])); mx.append(float(f[1])); pw.append(float(f[2]))
            except ValueError:
                continue
            for nm, v in zip(names, f[3:7]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        # "under load": the upper half of the samples by clock excludes idle gaps around the region
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "power_w_max": max(pw) if pw else None, "reasons": sorted(reasons), "samples": len(sm)}


# --------------------------------------------------------------------------------------
# reference arm / CPU baseline: the oracle port on the host cores
# --------------------------------------------------------------------------------------

def cpu_sample_inputs(rows, M, seed=0):
    import torch
    from oracle import oracle as O
    g = torch.Generator().manual_seed(seed)
    cases = []
    for name, K, N, *_ in rows:
        w = (torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16)
        wq, ws = O.weight_quant(w)
        x = torch.randn(M, K, generator=g).to(torch.bfloat16)
        cases.append((name, x, wq, ws))
    return cases


def cpu_pass(cases):
    """act_quant + fp8_gemm on the CPU oracle for every case; returns (seconds, gemm flops)."""
    from oracle import oracle as O
    t0 = time.perf_counter()
    fl = 0.0
    for _, x, wq, ws in cases:
        xq, xs = O.act_quant(x)
        O.fp8_gemm(xq, xs, wq, ws)
        fl += gemm_flops(x.size(0), wq.size(0), x.size(1))
    return time.perf_counter() - t0, fl


def bf16_linear_leg(rows, M, budget_s=8.0):
    """model.py:155-157 on the host: weight_dequant once, then F.linear in bf16 with all the threads torch has.
    Bounded: shapes are taken in order until the time budget is spent."""
    import torch
    import torch.nn.functional as F
    torch.set_num_threads(max(1, len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)))
    g = torch.Generator().manual_seed(1)
    t_total, fl, used = 0.0, 0.0, []
    for name, K, N, *_ in rows:
        if N * K > (40 << 20):
            continue                                           # keep the sample bounded: the three 117-132 MB weights are left out
        w = (torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16)
        x = torch.randn(M, K, generator=g).to(torch.bfloat16)
        F.linear(x, w)
        reps, t0 = 0, time.perf_counter()
        while reps < 3 or time.perf_counter() - t0 < 0.25:      # a quarter of a second per shape
            F.linear(x, w)
            reps += 1
        t_total += time.perf_counter() - t0
        fl += reps * gemm_flops(M, N, K)
        used.append(name)
        if t_total > budget_s:
            break
    return {"value": fl / t_total / 1e12 if t_total else None, "unit": "TFLOP/s", "threads": torch.get_num_threads(),
            "cpu_count": os.cpu_count(), "sample": f"bf16 F.linear (model.py:155-157) at M={M} on {len(used)} shapes of the sweep "
                                                   f"(weights up to 40 MB), repeated for 0.25 s each, {t_total:.2f} s"}


REFERENCE_SAMPLE_M = 64


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    from oracle import oracle as O
    # torch.distributed.run exports OMP_NUM_THREADS=1 to its ranks; the reference arm is meant to use
    # every host core this process may run on
    try:
        O.set_num_threads(len(os.sched_getaffinity(0)))
    except AttributeError:
        O.set_num_threads(os.cpu_count() or 1)
    rows = sweep_rows(1)
    M = REFERENCE_SAMPLE_M
    cases = cpu_sample_inputs(rows, M)
    for _ in range(args.warmup):
        cpu_pass(cases)
    t, fl = 0.0, 0.0
    for _ in range(args.steps):
        dt, f = cpu_pass(cases)
        t += dt
        fl += f
    val = fl / t / 1e12
    sample = f"M={M} column of the sweep ({len(rows)} shapes), act_quant+fp8_gemm per shape"
    cfg = workload_config(1)
    cfg["workload"] = (f"bounded sample of the sweep: the M={M} column only ({len(rows)} (K->N) rows), act_quant + fp8_gemm "
                       "per shape on the host; the GPU arm reports the same column as `same_sample_as_reference`")
    cfg["m_values"] = [M]
    line = {
        "impl": "reference", "metric": "fp8_gemm_tflops_v3_shape_sweep", "value": val, "unit": "TFLOP/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": t / args.steps * 1e3,
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "fp8_e4m3 x fp8_e4m3 -> fp32",
        "data": "synthetic", "config": cfg,
        "cpu_baseline": {"value": val, "unit": "TFLOP/s", "cores": O.num_threads(), "kind": "port", "sample": sample,
                         "bf16_linear": bf16_linear_leg(rows, M)},
        "e2e": {"value": val, "unit": "TFLOP/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
        "note": "reference = CPU restatement of inference/kernel.py (oracle/dsv3_oracle.c, OpenMP); the Python/Triton "
                "reference is not part of this repository",
    }
    print(json.dumps(line), flush=True)


def workload_config(world):
    rows = sweep_rows(1)
    return {
        "workload": "fp8_gemm sweep over DeepSeek-V3 Linear shapes (dim 7168), "
                    f"{len(rows)} (K->N) rows x M in {MS}; activations N(0,1) bf16 -> act_quant, weights N(0,0.02) "
                    "quantised per 128x128 block",
        "shapes": [f"{n}:{k}->{o}" for n, k, o, *_ in rows],
        "m_values": MS, "block_size": 128,
        "parallelism": "single GPU" if world == 1 else
                       f"tp{world}: the same problem set; column-parallel N/ws, row-parallel K/ws + NCCL all_reduce, "
                       "replicated Linears on every rank (counted once), expert and TP=8-slice problems owned round-robin; "
                       "all_reduce on a communication stream, GEMMs leave it --comm-sms SMs while one is in flight",
        "l2": "inputs larger than L2: the sweep runs M-major, so >500 MB of other weights stream between two "
              "uses of any weight (L2 is 126 MB)",
    }


# --------------------------------------------------------------------------------------
# GPU arm
# --------------------------------------------------------------------------------------

def run_ours(args):
    import torch
    import torch.distributed as dist
    import dsv3_b200
    import kernel

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world != args.gpus:
        raise SystemExit(f"--gpus {args.gpus} but WORLD_SIZE={world}: launch with torch.distributed.run")
    # stdout carries the one JSON line and nothing else: whatever libraries print while the run lasts (NCCL's
    # version banner, for one) is sent to stderr, and stdout is put back just before the line is printed
    sys.stdout.flush()
    saved_stdout = os.dup(1)
    os.dup2(2, 1)
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
    torch.set_default_dtype(torch.bfloat16)
    torch.manual_seed(1234 + rank)
    peaks = read_peaks()
    rows = sweep_rows(world, rank)

    # ---- synthetic, resident inputs -------------------------------------------------
    Mmax = max(MS)
    acts = {}       # K -> (x bf16, xq fp8, xs fp32), all [Mmax, ...]
    for K in sorted({r[1] for r in rows}):
        x = torch.randn(Mmax, K, device=dev, dtype=torch.bfloat16)
        xq, xs = kernel.act_quant(x)
        acts[K] = (x, xq, xs)
    weights = {}
    for name, K, N, *_ in rows:
        w = (torch.randn(N, K, device=dev, dtype=torch.float32) * 0.02).to(torch.bfloat16)
        weights[name] = dsv3_b200.weight_quant(w)
        del w
    plan = [(name, K, N, M, ar) for M in MS for (name, K, N, _, ar, _c) in rows]   # M-major
    my_flops = sum(gemm_flops(M, N, K) for M in MS for (_, K, N, _, _, counted) in rows if counted)
    total_flops = my_flops
    if world > 1:
        tt = torch.tensor([my_flops], device=dev, dtype=torch.float64)
        dist.all_reduce(tt)
        total_flops = tt.item()
    ref_flops = sum(gemm_flops(M, N, K) for M in MS for (_, K, N, *_r) in sweep_rows(1))
    assert abs(total_flops - ref_flops) <= 1e-9 * ref_flops, (total_flops, ref_flops)

    # high priority: when SMs come free, the collective's CTAs go ahead of the next GEMM's (already queued under
    # programmatic dependent launch)
    comm = torch.cuda.Stream(device=dev, priority=-1) if world > 1 else None
    sm_total = torch.cuda.get_device_properties(dev).multi_processor_count

    def column(M, collectives=True, with_act_quant=False):
        """fp8_gemm for every shape of the sweep at one M (one CUDA graph per column).  The all_reduce of a
        row-parallel Linear (model.py:263-264) is issued on a communication stream as soon as its GEMM is done and
        joins the main stream at the end of the column, so it runs under the GEMMs that follow."""
        cur = torch.cuda.current_stream()
        pending = []
        # While an all_reduce is (by estimate) in flight, the GEMMs leave it `--comm-sms` SMs: a persistent kernel on
        # every SM keeps the collective's CTAs waiting until it ends, and the GEMM launched after that finds SMs
        # taken and runs a straggling round.  t_gemm / t_comm_end: estimated device time since the column began.
        t_gemm, t_comm_end, limited = 0.0, 0.0, False
        for name, K, N, _, ar, _c in rows:
            x, xq, xs = acts[K]
            wq, ws = weights[name]
            want = collectives and args.comm_sms > 0 and t_gemm < t_comm_end
            if want != limited:
                dsv3_b200.set_num_sms(sm_total - args.comm_sms if want else 0)
                limited = want
            if with_act_quant:
                xq_m, xs_m = kernel.act_quant(x[:M])
                y = kernel.fp8_gemm(xq_m, xs_m, wq, ws)
            else:
                y = kernel.fp8_gemm(xq[:M], xs[:M], wq, ws)
            t_gemm += gemm_flops(M, N, K) / 1.8e15 + 3e-6
            if ar and collectives:
                ev = torch.cuda.Event()
                ev.record(cur)
                comm.wait_event(ev)
                with torch.cuda.stream(comm):
                    dist.all_reduce(y)
                y.record_stream(comm)
                pending.append(y)
                if M * N * 2 >= (4 << 20):
                    t_comm_end = max(t_gemm, t_comm_end) + 2.0 * (world - 1) / world * (M * N * 2) / 550e9 + 20e-6
        if limited:
            dsv3_b200.set_num_sms(0)
        if pending:
            ev = torch.cuda.Event()
            ev.record(comm)
            cur.wait_event(ev)

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    # The decode-sized launches last a few microseconds, less than the host needs to issue one, so
    # each M column is captured once into a CUDA graph and a step replays the eight graphs: the GPU
    # then runs the launches back to back.  Capture happens on the stream the warm-up ran on so the
    # split-K workspace of that stream already exists.
    side = torch.cuda.Stream(device=dev)
    graphs, graphs_nocomm, graphs_linear = {}, {}, {}
    with torch.cuda.stream(side):
        for _ in range(max(args.warmup, 3)):
            for M in MS:
                column(M)
        for M in MS:
            column(M, with_act_quant=True)
        dsv3_b200.check_device_status()

        def capture(**kw):
            out = {}
            for M in MS:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=side):
                    column(M, **kw)
                out[M] = g
            return out
        graphs = capture()
        graphs_linear = capture(with_act_quant=True)
        if world > 1:
            graphs_nocomm = capture(collectives=False)
        for M in MS:
            graphs[M].replay()
    barrier()

    def timed_pass(gs, steps):
        """Replays the eight column graphs `steps` times; returns (ms, per-step list of per-column event lists)."""
        evs = []
        barrier()
        with torch.cuda.stream(side):
            a = torch.cuda.Event(enable_timing=True); b = torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(steps):
                marks = [torch.cuda.Event(enable_timing=True) for _ in range(len(MS) + 1)]
                marks[0].record()
                for i, M in enumerate(MS):          # M-major: every weight is used once per column
                    gs[M].replay()
                    marks[i + 1].record()
                evs.append(marks)
            b.record()
        barrier()
        t = a.elapsed_time(b)
        if world > 1:
            tt = torch.tensor([t], device=dev, dtype=torch.float64)
            dist.all_reduce(tt, op=dist.ReduceOp.MAX)
            t = tt.item()
        return t, evs

    sampler = ClockSampler(local)
    if rank == 0:
        sampler.start()
    # ---- timed region 1: resident inputs ----------------------------------------------
    ms, col_events = timed_pass(graphs, args.steps)
    dsv3_b200.check_device_status()
    # the same sweep as the two-operator Linear of model.py:158-160 (act_quant + fp8_gemm), still device resident
    ms_linear, _ = timed_pass(graphs_linear, args.steps)
    # N > 1: the same GEMMs without the collectives, to tell compute from communication
    ms_nocomm, nocomm_events = (timed_pass(graphs_nocomm, args.steps) if world > 1 else (None, None))
    dsv3_b200.check_device_status()

    # ---- timed region 2: end to end through the drop-in module, host buffers ----------
    hx = {K: torch.empty(Mmax, K, dtype=torch.bfloat16, pin_memory=True).copy_(acts[K][0].cpu()) for K in acts}
    max_out = max(M * N for _, _, N, M, _ in plan)
    hy = torch.empty(max_out, dtype=torch.bfloat16, pin_memory=True)
    h2d = sum(M * K * 2 for _, K, _, M, _ in plan)
    d2h = sum(M * N * 2 for _, _, N, M, _ in plan)

    # Three streams, the way a host program would pipeline the public API: activations go up on one,
    # act_quant + fp8_gemm run on the second, results come down on the third (PCIe is full duplex), with
    # two device-side input buffers so that an upload can run ahead of the GEMM that consumes the other.
    s_in, s_out = torch.cuda.Stream(device=dev), torch.cuda.Stream(device=dev)
    Kmax = max(acts)
    xbuf = [torch.empty(Mmax * Kmax, device=dev, dtype=torch.bfloat16) for _ in range(2)]

    def e2e_step(items=None):
        done = [None, None]      # event: the GEMM that read xbuf[i] has finished
        for i, (name, K, N, M, ar) in enumerate(plan if items is None else items):
            wq, ws = weights[name]
            b = i & 1
            with torch.cuda.stream(s_in):
                if done[b] is not None:
                    s_in.wait_event(done[b])
                x = xbuf[b][: M * K].view(M, K)
                x.copy_(hx[K][:M], non_blocking=True)
                up = torch.cuda.Event()
                up.record(s_in)
            with torch.cuda.stream(side):
                side.wait_event(up)
                xq, xs = kernel.act_quant(x)
                y = kernel.fp8_gemm(xq, xs, wq, ws)
                if ar:
                    dist.all_reduce(y)
                done[b] = torch.cuda.Event()
                done[b].record(side)
            with torch.cuda.stream(s_out):
                s_out.wait_event(done[b])
                hy[: M * N].view(M, N).copy_(y, non_blocking=True)
                y.record_stream(s_out)
        side.wait_stream(s_out)
        side.wait_stream(s_in)

    with torch.cuda.stream(side):
        e2e_step()
    barrier()
    s0 = torch.cuda.Event(enable_timing=True); s1 = torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(side):
        s0.record()
        for _ in range(args.steps):
            e2e_step()
        s1.record()
    barrier()
    ms_e2e = s0.elapsed_time(s1)
    if world > 1:
        tt = torch.tensor([ms_e2e], device=dev, dtype=torch.float64)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        ms_e2e = tt.item()
    dsv3_b200.check_device_status()
    # the reference arm's sample (the M = 64 column), end to end, for a like-for-like ratio
    sample_items = [it for it in plan if it[3] == REFERENCE_SAMPLE_M]
    with torch.cuda.stream(side):
        e2e_step(sample_items)
    barrier()
    q0 = torch.cuda.Event(enable_timing=True); q1 = torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(side):
        q0.record()
        for _ in range(args.steps):
            e2e_step(sample_items)
        q1.record()
    barrier()
    ms_e2e_sample = q0.elapsed_time(q1)
    if world > 1:
        tt = torch.tensor([ms_e2e_sample], device=dev, dtype=torch.float64)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        ms_e2e_sample = tt.item()
    clocks = sampler.stop() if rank == 0 else None

    # ---- per-shape table at the M values the targets are stated for (single GPU): every problem alone, a CUDA
    # graph of launches over distinct copies of the weight (more than L2 in total)
    per_shape = None
    if world == 1 and not args.no_per_shape:
        per_shape = []
        fp8_pk = 2.0 * peaks["bf16_tflops"]
        for name, K, N, *_r in rows:
            wq0, ws0 = weights[name]
            R = max(2, min(32, -(-(256 << 20) // (N * K))))
            copies = [(wq0, ws0)] + [(wq0.clone(), ws0.clone()) for _ in range(R - 1)]
            for M in (1, 64, 4096, 16384):
                _, xq, xs = acts[K]
                with torch.cuda.stream(side):
                    for wq, ws in copies[:2]:
                        kernel.fp8_gemm(xq[:M], xs[:M], wq, ws)
                    g = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(g, stream=side):
                        for wq, ws in copies:
                            kernel.fp8_gemm(xq[:M], xs[:M], wq, ws)
                    g.replay()
                    a = torch.cuda.Event(enable_timing=True); b = torch.cuda.Event(enable_timing=True)
                    a.record()
                    g.replay(); g.replay()
                    b.record()
                torch.cuda.synchronize()
                us = a.elapsed_time(b) * 1e3 / (2 * R)
                t_c = gemm_flops(M, N, K) / (fp8_pk * 1e12) * 1e6
                t_m = gemm_bytes(M, N, K) / (peaks["hbm_gbs"] * 1e9) * 1e6
                bound = "tensor" if t_c > t_m else "hbm"
                target = 0.70 if M >= 4096 else 0.75
                entry = {"shape": name, "K": K, "N": N, "M": M, "us": round(us, 2), "bound": bound,
                         "tflops": round(gemm_flops(M, N, K) / us / 1e6, 1), "gbs": round(gemm_bytes(M, N, K) / us / 1e3),
                         "roofline_us": round(max(t_c, t_m), 2), "frac": round(max(t_c, t_m) / us, 3), "target": target}
                if M <= 64 and max(t_c, t_m) < 2.5:
                    # a launch costs about 2.5 us on this GPU whatever it does (the reference's own Triton launches measure
                    # 2.6 us on its smallest problem): a roofline time below that cannot be met by any single launch
                    entry["out_of_reach"] = "roofline time is below the cost of a launch"
                per_shape.append(entry)
                del g
            del copies
        dsv3_b200.check_device_status()

    # ---- per-kernel roofline from the per-column events of region 1 -------------------
    big_t = big_f = small_t = small_b = 0.0
    n_big = n_small = 0
    per_column = {}
    for marks in col_events:
        for i, M in enumerate(MS):
            dt = marks[i].elapsed_time(marks[i + 1]) * 1e-3
            fl = sum(gemm_flops(M, N, K) for _, K, N, *_r in rows)
            by = sum(gemm_bytes(M, N, K) for _, K, N, *_r in rows)
            acc = per_column.setdefault(M, [0.0, 0, fl, by])
            acc[0] += dt; acc[1] += 1
            if M >= 256:
                big_t += dt; big_f += fl; n_big += len(rows)
            elif M <= 64:
                small_t += dt; small_b += by; n_small += len(rows)
    # FP8 issues at twice the bf16 rate.  The burst figure is the denominator: the timed region lasts a fraction of a
    # second; the fraction of the sustained figure (a seconds-long cuBLAS loop under the power cap) is given beside it.
    fp8_peak = 2.0 * peaks["bf16_tflops"]
    fp8_sustained = 2.0 * peaks["bf16_tflops_sustained"]
    # DRAM traffic per launch: ncu's dram__bytes_read.sum + dram__bytes_write.sum of one captured launch
    # (bench.py --single, summaries under profiles/) divided by that problem's algorithmic bytes, applied
    # to the average algorithmic bytes of the launches timed here (traffic tracks the operand and result
    # sizes: each is moved once).
    big_b = sum(gemm_bytes(M, N, K) for M in MS if M >= 256 for _, K, N, *_r in rows) / max(1, n_big // max(1, len(col_events)))
    small_avg = sum(gemm_bytes(M, N, K) for M in MS if M <= 64 for _, K, N, *_r in rows) / max(1, n_small // max(1, len(col_events)))
    ratio_big = NCU_TRAFFIC["token_major"][0] / gemm_bytes(*NCU_TRAFFIC["token_major"][1])
    ratio_small = NCU_TRAFFIC["weight_major"][0] / gemm_bytes(*NCU_TRAFFIC["weight_major"][1])
    ach_big = big_f / big_t / 1e12 if big_t else None
    roofline = {
        "kernel": "token-major tcgen05 kernels (launches with M >= 256): fp8_gemm_tw_kernel (CTA pairs, 256x256 tiles), "
                  "fp8_gemm_tm_kernel (CTA pairs, 256x128 tiles, where 256-wide tiles fill the last round badly) "
                  "and fp8_gemm_tc_kernel<128,false> (split-K)",
        "bound": "tensor", "achieved": ach_big, "peak": fp8_peak, "unit": "TFLOP/s",
        "frac": ach_big / fp8_peak if big_t else None,
        "frac_of_sustained": ach_big / fp8_sustained if big_t else None,
        "traffic": ratio_big * big_b if n_big else None, "traffic_unit": "bytes per launch (average launch)",
        "traffic_source": f"{NCU_TRAFFIC['token_major'][2]}: measured / algorithmic bytes = {ratio_big:.2f}",
        "peak_source": f"2 x bf16_tflops (burst) of MEASURED_PEAKS.json ({peaks['source']}): the timed region is a fraction of a "
                       f"second; frac_of_sustained uses 2 x bf16_tflops_sustained = {fp8_sustained:.0f}",
        "launches": n_big, "avg_launch_us": big_t / n_big * 1e6 if n_big else None,
        "algorithmic": "2*M*N*K flops per launch",
        "includes_collectives": world > 1,
    }
    roofline_decode = {
        "kernel": "decode launches (M <= 64): fp8_gemm_tc_kernel<BN,true> (tcgen05, weight-major tiles, split-K) and "
                  "fp8_linear_small_kernel (M <= 8, small weights)",
        "bound": "hbm", "achieved": small_b / small_t / 1e9 if small_t else None, "peak": peaks["hbm_gbs"], "unit": "GB/s",
        "frac": (small_b / small_t / 1e9) / peaks["hbm_gbs"] if small_t else None,
        "traffic": ratio_small * small_avg if n_small else None, "traffic_unit": "bytes per launch (average launch)",
        "traffic_source": f"{NCU_TRAFFIC['weight_major'][2]}: measured / algorithmic bytes = {ratio_small:.2f}",
        "peak_source": f"hbm_gbs of MEASURED_PEAKS.json ({peaks['source']})",
        "launches": n_small, "algorithmic": "M*K + N*K + scales + 2*M*N bytes per launch",
        "includes_collectives": world > 1,
    }
    # N > 1: compute (the same graphs without collectives) against the full step, per column
    breakdown = None
    if world > 1:
        comp = {M: 0.0 for M in MS}
        for marks in nocomm_events:
            for i, M in enumerate(MS):
                comp[M] += marks[i].elapsed_time(marks[i + 1])
        full = {M: per_column[M][0] * 1e3 for M in MS}
        n = len(nocomm_events)
        breakdown = {
            "compute_ms_per_step": ms_nocomm / args.steps, "comm_exposed_ms_per_step": (ms - ms_nocomm) / args.steps,
            "per_column": {f"M={M}": {"compute_ms": comp[M] / n, "step_ms": full[M] / len(col_events),
                                      "comm_exposed_ms": full[M] / len(col_events) - comp[M] / n} for M in MS},
            "note": "rank 0's device times; compute = the same CUDA graphs captured without the all_reduce calls; the "
                    "all_reduce of a row-parallel Linear runs on a communication stream under the following GEMMs",
        }
        roofline["achieved_compute_only"] = (sum(gemm_flops(M, N, K) for M in MS if M >= 256 for _, K, N, *_r in rows) /
                                             (sum(comp[M] for M in MS if M >= 256) / n * 1e-3) / 1e12)
    detail = {f"M={k}": {"us_per_column": v[0] / v[1] * 1e6, "tflops": v[2] / (v[0] / v[1]) / 1e12,
                         "gbs": v[3] / (v[0] / v[1]) / 1e9, "launches": len(rows)} for k, v in per_column.items()}

    def shutdown():
        """Tear down in an order NCCL accepts: graphs that captured collectives go first.  A timer ends
        the process if the teardown itself blocks (the measurement is already printed by then)."""
        if world == 1:
            return
        killer = threading.Timer(45.0, lambda: os._exit(0))
        killer.daemon = True
        killer.start()
        graphs.clear()
        graphs_nocomm.clear()
        graphs_linear.clear()
        torch.cuda.synchronize()
        dist.barrier()
        dist.destroy_process_group()
        killer.cancel()

    if rank != 0:
        shutdown()
        return

    # ---- CPU baseline (rank 0, N=1 only): the oracle on a bounded sample ----------------
    cpu = None
    if world == 1 and not args.no_cpu_baseline:
        from oracle import oracle as O
        cases = cpu_sample_inputs(sweep_rows(1), 64)
        dt, fl = cpu_pass(cases)
        cpu = {"value": fl / dt / 1e12, "unit": "TFLOP/s", "cores": O.num_threads(), "kind": "port",
               "sample": f"M=64 column of the sweep ({len(cases)} shapes), act_quant+fp8_gemm per shape, one pass, {dt:.1f} s",
               "bf16_linear": bf16_linear_leg(sweep_rows(1), REFERENCE_SAMPLE_M)}

    agg = total_flops * args.steps / (ms * 1e-3) / 1e12
    agg_e2e = total_flops * args.steps / (ms_e2e * 1e-3) / 1e12
    line = {
        "metric": "fp8_gemm_tflops_v3_shape_sweep", "value": agg, "unit": "TFLOP/s", "n_gpus": world,
        "steps": args.steps, "warmup": max(args.warmup, 3), "ms_per_step": ms / args.steps,
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
        "dtype": "fp8_e4m3 x fp8_e4m3 -> fp32", "data": "synthetic", "config": workload_config(world),
        "roofline": roofline, "roofline_decode": roofline_decode, "cpu_baseline": cpu,
        "e2e": {"value": agg_e2e, "unit": "TFLOP/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                "ms_per_step": ms_e2e / args.steps,
                "path": "pinned host bf16 activations -> kernel.act_quant -> kernel.fp8_gemm -> bf16 result to pinned host; "
                        "weights resident on the device; upload, compute and download on three streams"},
        "gpu_launches": len(plan) * args.steps, "gpu_launches_e2e": 2 * len(plan) * args.steps,
        "clocks": clocks, "per_column": detail,
        # the two-operator Linear of model.py:158-160 (act_quant + fp8_gemm per problem), device resident
        "value_act_quant_plus_gemm": total_flops * args.steps / (ms_linear * 1e-3) / 1e12,
        # the sample the reference arm times (its config.workload): the M = 64 column
        "same_sample_as_reference": {
            "workload": f"M={REFERENCE_SAMPLE_M} column of the sweep",
            "value": per_column[REFERENCE_SAMPLE_M][2] / (per_column[REFERENCE_SAMPLE_M][0] / per_column[REFERENCE_SAMPLE_M][1]) / 1e12,
            "e2e": (sum(gemm_flops(M, N, K) for _, K, N, M, _ in sample_items) * args.steps / (ms_e2e_sample * 1e-3) / 1e12
                    if world == 1 else None),
            "unit": "TFLOP/s"},
        "comm_breakdown": breakdown, "per_shape": per_shape,
    }
    sys.stdout.flush()
    os.dup2(saved_stdout, 1)
    print(json.dumps(line), flush=True)
    os.dup2(2, 1)
    shutdown()


def run_single(args):
    """One (M, N, K) problem, `steps` launches of act_quant / fp8_gemm / weight_dequant: the small case
    the ncu captures under profiles/ are taken on.  Prints per-launch CUDA-event times."""
    import torch
    import dsv3_b200
    import kernel
    M, N, K = (int(v) for v in args.single.split(","))
    torch.cuda.set_device(0)
    torch.set_default_dtype(torch.bfloat16)
    torch.manual_seed(0)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    wq, ws = dsv3_b200.weight_quant((torch.randn(N, K, device="cuda") * 0.02).to(torch.bfloat16))
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    out = {"M": M, "N": N, "K": K}
    for name, fn in (("act_quant", lambda: kernel.act_quant(x)), ("fp8_gemm", None),
                     ("weight_dequant", lambda: kernel.weight_dequant(wq, ws))):
        if fn is None:
            xq, xs = kernel.act_quant(x)
            fn = lambda: kernel.fp8_gemm(xq, xs, wq, ws)
        ts = []
        for i in range(args.warmup + args.steps):
            flush.zero_()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record(); fn(); e1.record()
            torch.cuda.synchronize()
            if i >= args.warmup:
                ts.append(e0.elapsed_time(e1) * 1e3)
        out[name + "_us"] = sorted(ts)[len(ts) // 2]
    dsv3_b200.check_device_status()
    out["fp8_gemm_tflops"] = gemm_flops(M, N, K) / out["fp8_gemm_us"] / 1e6
    out["fp8_gemm_gbs"] = gemm_bytes(M, N, K) / out["fp8_gemm_us"] / 1e3
    print(json.dumps(out), flush=True)


def run_detail(args):
    """Per-(shape, M) table: every problem of the sweep timed alone.  A CUDA graph holds R launches
    over R distinct weight copies (R x weight bytes >= 256 MB, more than L2), so launches run back to
    back on weights that are not cache-resident.  Prints one JSON line per problem."""
    import torch
    import dsv3_b200
    import kernel
    torch.cuda.set_device(0)
    dev = torch.device("cuda", 0)
    torch.set_default_dtype(torch.bfloat16)
    torch.manual_seed(7)
    peaks = read_peaks()
    fp8_peak = 2.0 * peaks["bf16_tflops_sustained"]
    rows = sweep_rows(1)
    ms_list = [int(v) for v in args.detail_m.split(",")] if args.detail_m else MS
    side = torch.cuda.Stream(device=dev)
    out = []
    for name, K, N, *_ in rows:
        R = max(2, min(64, -(-(256 << 20) // (N * K))))
        w = (torch.randn(N, K, device=dev, dtype=torch.float32) * 0.02).to(torch.bfloat16)
        wq0, ws0 = dsv3_b200.weight_quant(w)
        del w
        copies = [(wq0.clone(), ws0.clone()) for _ in range(R)]
        for M in ms_list:
            x = torch.randn(M, K, device=dev, dtype=torch.bfloat16)
            xq, xs = kernel.act_quant(x)
            with torch.cuda.stream(side):
                for wq, ws in copies[:2]:
                    kernel.fp8_gemm(xq, xs, wq, ws)
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=side):
                    for wq, ws in copies:
                        kernel.fp8_gemm(xq, xs, wq, ws)
                g.replay()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                for _ in range(args.steps):
                    g.replay()
                e1.record()
            torch.cuda.synchronize()
            us = e0.elapsed_time(e1) * 1e3 / (args.steps * R)
            tf, gb = gemm_flops(M, N, K) / us / 1e6, gemm_bytes(M, N, K) / us / 1e3
            t_roof = max(gemm_flops(M, N, K) / (fp8_peak * 1e12), gemm_bytes(M, N, K) / (peaks["hbm_gbs"] * 1e9)) * 1e6
            r = {"shape": name, "K": K, "N": N, "M": M, "us": round(us, 2), "tflops": round(tf, 1), "gbs": round(gb, 0),
                 "roofline_us": round(t_roof, 2), "frac_of_roofline": round(t_roof / us, 3),
                 "bound": "tensor" if gemm_flops(M, N, K) / (fp8_peak * 1e12) > gemm_bytes(M, N, K) / (peaks["hbm_gbs"] * 1e9) else "hbm"}
            out.append(r)
            print(json.dumps(r), flush=True)
            del g
        del copies
    dsv3_b200.check_device_status()


def run_moe_layer(args):
    """One DeepSeekMoE layer at V3 dims (dim 7168, 256 routed experts of moe_inter 2048,
    sigmoid gate with bias, 8 groups / 4 kept, top-8, route_scale 2.5, one shared expert), T tokens.
    Routed experts are sharded E/ws per rank and the routed output is all_reduced (model.py:658-666, 691-692).
    Times the reference's expert loop (model.py:683-689, restated on the drop-in operators, with its host
    synchronisations) and the grouped path; prints one JSON line."""
    import torch
    import torch.distributed as dist
    import torch.nn.functional as F
    import dsv3_b200
    import kernel

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    # stdout carries the one JSON line and nothing else: whatever libraries print while the run lasts (NCCL's
    # version banner, for one) is sent to stderr, and stdout is put back just before the line is printed
    sys.stdout.flush()
    saved_stdout = os.dup(1)
    os.dup2(2, 1)
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
    torch.set_default_dtype(torch.bfloat16)
    dim, inter, E, topk, n_groups, topk_groups, route_scale = 7168, 2048, args.moe_experts, 8, 8, 4, 2.5
    T = args.moe_tokens
    n_local = E // world
    start = rank * n_local

    class Lin:
        scale_fmt = None

        def __init__(self, N, K, gen):
            w = (torch.randn(N, K, device=dev, dtype=torch.float32, generator=gen) * 0.02).to(torch.bfloat16)
            self.weight, sc = dsv3_b200.weight_quant(w)
            self.weight.scale = sc

        def __call__(self, x):
            xq, xs = kernel.act_quant(x)
            return kernel.fp8_gemm(xq, xs, self.weight, self.weight.scale)

    class Expert:
        def __init__(self, d, i, gen):
            self.w1, self.w2, self.w3 = Lin(i, d, gen), Lin(d, i, gen), Lin(i, d, gen)

        def __call__(self, x):
            return self.w2(F.silu(self.w1(x)) * self.w3(x))

    class Layer:
        pass

    gen = torch.Generator(device=dev).manual_seed(1000 + rank)
    shared_gen = torch.Generator(device=dev).manual_seed(77)
    moe = Layer()
    moe.dim, moe.n_routed_experts, moe.n_local_experts = dim, E, n_local
    moe.experts_start_idx, moe.experts_end_idx = start, start + n_local
    moe.experts = [Expert(dim, inter, gen) if start <= i < start + n_local else None for i in range(E)]
    shared = Expert(dim, inter // world, shared_gen)       # column/row-parallel slice of the shared expert
    gate_gen = torch.Generator(device=dev).manual_seed(5)
    gate_w = (torch.randn(E, dim, device=dev, dtype=torch.float32, generator=gate_gen) * 0.02).to(torch.bfloat16)
    gate_b = torch.randn(E, device=dev, dtype=torch.float32, generator=gate_gen) * 0.01

    def gate(x):                                            # Gate.forward, model.py:566-598 (sigmoid + bias + groups)
        scores = F.linear(x, gate_w).sigmoid()
        original = scores
        sc = (scores + gate_b).view(x.size(0), n_groups, -1)
        group_scores = sc.topk(2, dim=-1)[0].sum(dim=-1)
        idx = group_scores.topk(topk_groups, dim=-1)[1]
        mask = sc.new_ones(x.size(0), n_groups, dtype=torch.bool).scatter_(1, idx, False)
        sc = sc.masked_fill(mask.unsqueeze(-1), float("-inf")).flatten(1)
        indices = torch.topk(sc, topk, dim=-1)[1]
        weights = original.gather(1, indices)
        weights = weights / weights.sum(dim=-1, keepdim=True) * route_scale
        return weights.type_as(x), indices

    def shared_experts(x):
        z = shared(x)
        if world > 1:
            dist.all_reduce(z)
        return z

    moe.gate, moe.shared_experts = gate, shared_experts

    def loop_forward(x):                                    # MoE.forward, model.py:669-693
        weights, indices = moe.gate(x)
        y = torch.zeros_like(x)
        counts = torch.bincount(indices.flatten(), minlength=E).tolist()
        for i in range(start, start + n_local):
            if counts[i] == 0:
                continue
            idx, top = torch.where(indices == i)
            y[idx] += moe.experts[i](x[idx]) * weights[idx, top, None]
        z = moe.shared_experts(x)
        if world > 1:
            dist.all_reduce(y)
        return y + z

    def grouped_forward(x):
        return dsv3_b200.grouped_moe_forward(moe, x, world_size=world)

    xgen = torch.Generator(device=dev).manual_seed(9)
    x = torch.randn(T, dim, device=dev, dtype=torch.float32, generator=xgen).to(torch.bfloat16)

    def timeit(fn):
        for _ in range(max(2, args.warmup)):
            out = fn(x)
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.steps):
            out = fn(x)
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / args.steps
        if world > 1:
            tt = torch.tensor([ms], device=dev, dtype=torch.float64)
            dist.all_reduce(tt, op=dist.ReduceOp.MAX)
            ms = tt.item()
        return ms, out

    ms_loop, out_loop = timeit(loop_forward)
    ms_grp, out_grp = timeit(grouped_forward)
    dsv3_b200.check_device_status()
    err = (out_grp.float() - out_loop.float()).abs()
    rms = out_loop.float().pow(2).mean().sqrt()
    ok = bool((err <= 2e-2 * (out_loop.float().abs() + rms)).all())
    flops = 2.0 * 3 * dim * inter * (T * topk + T)           # routed pairs + shared expert
    if rank == 0:
        sys.stdout.flush()
        os.dup2(saved_stdout, 1)
        print(json.dumps({
            "metric": "moe_layer_tokens_per_s", "value": T / (ms_grp * 1e-3), "unit": "tokens/s", "n_gpus": world,
            "steps": args.steps, "warmup": max(2, args.warmup), "ms_per_step": ms_grp, "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None, "dtype": "fp8_e4m3 x fp8_e4m3 -> fp32", "data": "synthetic",
            "config": {"workload": f"DeepSeekMoE layer, dim {dim}, {E} routed experts (inter {inter}) "
                                   f"+ 1 shared, top-{topk}, T={T} tokens, experts sharded {n_local} per rank"},
            "grouped_ms": ms_grp, "expert_loop_ms": ms_loop, "speedup_vs_expert_loop": ms_loop / ms_grp,
            "grouped_tflops": flops / (ms_grp * 1e-3) / 1e12, "agrees_with_expert_loop": ok,
        }), flush=True)
    if world > 1:
        killer = threading.Timer(45.0, lambda: os._exit(0))
        killer.daemon = True
        killer.start()
        dist.barrier()
        dist.destroy_process_group()
        killer.cancel()


def run_decode_step(args):
    """One decode step of the 671B-shaped model at tensor parallelism = world.

    Per layer the Linear sequence of model.py at M = batch rows: MLA wq_a, wq_b, wkv_a, weight_dequant(wkv_b), wo
    (+ all_reduce) (model.py:461-496); layers 0-2 the dense MLP w1, w3, w2 (+ all_reduce) (model.py:500-532); layers
    3-60 the MoE layer: gate, routed experts of this rank (256 / world), shared expert (+ all_reduce), all_reduce
    (model.py:669-693).  Attention scores, RoPE, norms, embedding and the bf16 head are outside the path and not
    executed, so the figure is the time of the FP8 GEMM path of a step, not of the whole model.  Weights: random-init,
    block-quantised; a few distinct instances of each layer kind (each larger than L2) are visited in rotation, which
    keeps weights out of L2 between two uses without holding 85 GB per rank.
    Modes: `operators` = the reference's call structure on the drop-in operators (act_quant + fp8_gemm per Linear,
    Python expert loop with its host synchronisations); `seams` = linear seam (fused decode Linear), grouped MoE,
    weight_dequant cache, SwiGLU folded into the quantisation; `graph` = the seams step captured once in a CUDA graph and
    replayed."""
    import torch
    import torch.distributed as dist
    import torch.nn.functional as F
    import dsv3_b200
    import kernel
    from dsv3_b200 import linear_seam as L

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    sys.stdout.flush()
    saved_stdout = os.dup(1)
    os.dup2(2, 1)
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
    torch.set_default_dtype(torch.bfloat16)
    peaks = read_peaks()
    dim, q_lora, kv_lora, rope, heads, nope, vdim = 7168, 1536, 512, 64, 128, 128, 128
    inter, moe_inter, E, topk, n_groups, topk_groups, route_scale = 18432, 2048, 256, 8, 8, 4, 2.5
    n_layers, n_dense = 61, 3
    # shard shapes: the real world size, or (single process) the per-rank shapes of a larger tensor-parallel group
    tp = args.decode_tp_shapes if (world == 1 and args.decode_tp_shapes > 0) else world
    n_local = E // tp
    start = rank * n_local
    gen = torch.Generator(device=dev).manual_seed(4000 + rank)

    class Lin:
        scale_fmt = None

        def __init__(self, N, K):
            w = (torch.randn(N, K, device=dev, dtype=torch.float32, generator=gen) * 0.02).to(torch.bfloat16)
            self.weight, sc = dsv3_b200.weight_quant(w)
            self.weight.scale = sc
            self.bytes = N * K

    class Expert:
        def __init__(self, d, i):
            self.w1, self.w2, self.w3 = Lin(i, d), Lin(d, i), Lin(i, d)

    class Attn:
        def __init__(self):
            self.wq_a, self.wq_b = Lin(q_lora, dim), Lin(heads * (nope + rope) // tp, q_lora)
            self.wkv_a, self.wkv_b = Lin(kv_lora + rope, dim), Lin(heads * (nope + vdim) // tp, kv_lora)
            self.wo = Lin(dim, heads * vdim // tp)
            self.bytes = sum(l.bytes for l in (self.wq_a, self.wq_b, self.wkv_a, self.wkv_b, self.wo))

    class Dense:
        def __init__(self):
            self.w1, self.w3, self.w2 = Lin(inter // tp, dim), Lin(inter // tp, dim), Lin(dim, inter // tp)
            self.bytes = 3 * self.w1.bytes

    class MoE:
        def __init__(self):
            self.dim, self.n_routed_experts, self.n_local_experts, self.n_activated_experts = dim, E, n_local, topk
            self.experts_start_idx, self.experts_end_idx = start, start + n_local
            self.experts = [Expert(dim, moe_inter) if start <= i < start + n_local else None for i in range(E)]
            self.shared = Expert(dim, moe_inter // tp)
            g2 = torch.Generator(device=dev).manual_seed(77)          # the gate is replicated: same on every rank
            self.gate_w = (torch.randn(E, dim, device=dev, dtype=torch.float32, generator=g2) * 0.02).to(torch.bfloat16)
            self.gate_b = torch.randn(E, device=dev, dtype=torch.float32, generator=g2) * 0.01

        def gate(self, x):                                            # Gate.forward, model.py:566-598
            scores = F.linear(x, self.gate_w).sigmoid()
            original = scores
            sc = (scores + self.gate_b).view(x.size(0), n_groups, -1)
            group_scores = sc.topk(2, dim=-1)[0].sum(dim=-1)
            idx = group_scores.topk(topk_groups, dim=-1)[1]
            mask = sc.new_ones(x.size(0), n_groups, dtype=torch.bool).scatter_(1, idx, False)
            sc = sc.masked_fill(mask.unsqueeze(-1), float("-inf")).flatten(1)
            indices = torch.topk(sc, topk, dim=-1)[1]
            weights = original.gather(1, indices)
            weights = weights / weights.sum(dim=-1, keepdim=True) * route_scale
            return weights.type_as(x), indices

    n_inst = max(2, args.decode_instances)
    attn = [Attn() for _ in range(n_inst)]
    dense = [Dense() for _ in range(min(n_inst, n_dense))]
    moes = [MoE() for _ in range(n_inst)]
    torch.cuda.synchronize()

    # f3: the one-shot all-reduce over peer-mapped buffers for the decode-sized partial results (opt-in in the
    # library; measured here next to NCCL as a second graph of the same step)
    oneshot = {"ar": None, "on": False}
    if world > 1:
        try:
            oneshot["ar"] = dsv3_b200.P2PAllReduce(max_bytes=256 << 10)   # larger messages stay on NCCL
        except Exception as e:      # no peer access between the ranks' GPUs: NCCL only
            sys.stderr.write(f"one-shot all-reduce unavailable: {e}\n")

    def all_reduce(y):
        if world > 1:
            if oneshot["on"] and oneshot["ar"].fits(y):
                oneshot["ar"].all_reduce(y)
            else:
                dist.all_reduce(y)
        return y

    ops = {"k": kernel}       # the operator module the `operators` mode calls (the drop-in, or the reference's own)

    def lin_ops(x, l):                                               # model.py:158-160 on the drop-in operators
        xq, xs = ops["k"].act_quant(x)
        return ops["k"].fp8_gemm(xq, xs, l.weight, l.weight.scale)

    ref_kernel = None
    if args.reference_kernel_dir:
        # builder-run comparison only: the reference's own kernel.py (Triton), imported from a directory outside the repo
        import importlib.util
        spec = importlib.util.spec_from_file_location("_reference_kernel", os.path.join(args.reference_kernel_dir, "kernel.py"))
        ref_kernel = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(ref_kernel)

    def lin_seam(x, l):
        return L.linear(x, l.weight)

    def mlp(x, e, lin, reduce=True):
        if lin is lin_seam:                                          # the MLP seam: SwiGLU folded into the quantisation
            hq, hs = dsv3_b200.swiglu_quant(lin(x, e.w1), lin(x, e.w3))
            y = kernel.fp8_gemm(hq, hs, e.w2.weight, e.w2.weight.scale)
        else:
            y = lin(F.silu(lin(x, e.w1)) * lin(x, e.w3), e.w2)      # model.py:532, 633
        return all_reduce(y) if reduce else y

    def moe_loop(m, x):                                              # MoE.forward, model.py:669-693
        weights, indices = m.gate(x)
        y = torch.zeros_like(x)
        counts = torch.bincount(indices.flatten(), minlength=E).tolist()
        for i in range(start, start + n_local):
            if counts[i] == 0:
                continue
            idx, top = torch.where(indices == i)
            y[idx] += mlp(x[idx], m.experts[i], lin_ops, reduce=False) * weights[idx, top, None]
        z = mlp(x, m.shared, lin_ops)
        return all_reduce(y) + z

    def moe_grouped(m, x):
        m.shared_experts = lambda t: mlp(t, m.shared, lin_seam)
        return dsv3_b200.grouped_moe_forward(m, x, world_size=world)

    def step(x, a_in, seams):
        lin = lin_seam if seams else lin_ops
        out = None
        for layer in range(n_layers):
            if seams:
                L.reset_memo()      # every layer has its own input in the model: no reuse of a quantisation across layers
            a = attn[layer % len(attn)]
            q = lin(lin(x, a.wq_a), a.wq_b)                           # model.py:464 (q_norm is outside the path)
            kv = lin(x, a.wkv_a)                                      # model.py:468
            wkv_b = (kernel if seams else ops["k"]).weight_dequant(a.wkv_b.weight, a.wkv_b.weight.scale)     # model.py:481
            o = all_reduce(lin(a_in, a.wo))                           # model.py:496, 263-264
            if layer < n_dense:
                out = mlp(x, dense[layer % len(dense)], lin)
            else:
                m = moes[layer % len(moes)]
                out = moe_grouped(m, x) if seams else moe_loop(m, x)
        return out, q, kv, wkv_b, o

    side = torch.cuda.Stream(device=dev)
    results = {}
    for B in [int(v) for v in args.decode_batch.split(",")]:
        xg = torch.Generator(device=dev).manual_seed(9)               # the same tokens on every rank
        x = torch.randn(B, dim, device=dev, dtype=torch.float32, generator=xg).to(torch.bfloat16)
        a_in = torch.randn(B, heads * vdim // tp, device=dev, dtype=torch.float32, generator=xg).to(torch.bfloat16)
        # weight bytes a step touches on this rank: everything but the routed experts no token of the batch chose
        with torch.no_grad():
            touched = 0
            for layer in range(n_dense, n_layers):
                _, idx = moes[layer % len(moes)].gate(x)
                loc = idx[(idx >= start) & (idx < start + n_local)]
                touched += int(torch.unique(loc).numel()) * 3 * dim * moe_inter
        step_bytes = (n_layers * attn[0].bytes + n_dense * dense[0].bytes + (n_layers - n_dense) * 3 * dim * (moe_inter // tp) + touched)
        res = {}

        def timed(fn, reps):
            fn()
            if world > 1:
                dist.barrier()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(reps):
                fn()
            e1.record()
            torch.cuda.synchronize()
            t = e0.elapsed_time(e1) / reps
            if world > 1:
                tt = torch.tensor([t], device=dev, dtype=torch.float64)
                dist.all_reduce(tt, op=dist.ReduceOp.MAX)
                t = tt.item()
            return t

        with torch.cuda.stream(side), torch.no_grad():
            dsv3_b200.disable_weight_dequant_cache()
            if ref_kernel is not None:
                ops["k"] = ref_kernel
                step(x, a_in, False)                                  # Triton JIT + autotune
                res["reference_kernels_ms"] = timed(lambda: step(x, a_in, False), 1)
                ops["k"] = kernel
            if not args.decode_skip_operators:
                res["operators_ms"] = timed(lambda: step(x, a_in, False), 1)
            dsv3_b200.enable_weight_dequant_cache(4 << 30)
            L.reset_memo()
            res["seams_ms"] = timed(lambda: step(x, a_in, True), max(2, args.steps))
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                outs = step(x, a_in, True)
            res["graph_ms"] = timed(g.replay, max(3, args.steps))
            del g, outs
            if oneshot["ar"] is not None:
                oneshot["on"] = True
                step(x, a_in, True)
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=side):
                    outs = step(x, a_in, True)
                res["graph_oneshot_allreduce_ms"] = timed(g.replay, max(3, args.steps))
                del g, outs
                oneshot["on"] = False
        dsv3_b200.check_device_status()
        best = min(res["graph_ms"], res.get("graph_oneshot_allreduce_ms", res["graph_ms"]))
        res.update(batch=B, tokens_per_s=B / (best * 1e-3), step_weight_bytes=step_bytes,
                   hbm_gbs=step_bytes / (best * 1e-3) / 1e9, frac_of_hbm=step_bytes / (best * 1e-3) / 1e9 / peaks["hbm_gbs"])
        results[f"B={B}"] = res
    dsv3_b200.disable_weight_dequant_cache()
    if rank == 0:
        sys.stdout.flush()
        os.dup2(saved_stdout, 1)
        first = results[next(iter(results))]
        print(json.dumps({
            "metric": "decode_tokens_per_s_671B_shapes_gemm_path", "value": first["tokens_per_s"], "unit": "tokens/s",
            "n_gpus": world, "steps": max(3, args.steps), "warmup": 1, "ms_per_step": first["graph_ms"], "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None, "dtype": "fp8_e4m3 x fp8_e4m3 -> fp32", "data": "synthetic",
            "config": {"workload": f"GEMM path of 61 layers of DeepSeek-V3 671B Linear shapes at TP={tp}"
                                   + (" (one rank's shards on one GPU, no collectives)" if tp != world else "") + ", "
                                   f"one decode step (M = batch rows), {n_inst} distinct instances per layer kind visited in rotation; "
                                   "attention scores, RoPE, norms, embedding and head are not executed",
                       "batches": args.decode_batch},
            "per_batch": results,
        }), flush=True)
        os.dup2(2, 1)
    if world > 1:
        killer = threading.Timer(45.0, lambda: os._exit(0))
        killer.daemon = True
        killer.start()
        torch.cuda.synchronize()
        if oneshot["ar"] is not None:
            oneshot["ar"].close()
        dist.barrier()
        dist.destroy_process_group()
        killer.cancel()



def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--comm-sms", type=int, default=32,
                    help="N > 1: SMs the GEMMs leave to an all_reduce that is in flight (0: none)")
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-per-shape", action="store_true", help="skip the per-shape table of the default run")
    ap.add_argument("--single", default=None, metavar="M,N,K",
                    help="run one problem instead of the sweep (the case ncu captures are taken on)")
    ap.add_argument("--detail", action="store_true", help="per-(shape, M) table instead of the aggregate sweep")
    ap.add_argument("--detail-m", default=None, metavar="M1,M2,...", help="restrict --detail to these M values")
    ap.add_argument("--moe-layer", action="store_true", help="one MoE layer, expert loop vs grouped")
    ap.add_argument("--moe-tokens", type=int, default=2048)
    ap.add_argument("--moe-experts", type=int, default=256)
    ap.add_argument("--decode-step", action="store_true", help="one 671B-shaped decode step")
    ap.add_argument("--decode-batch", default="1,16,64")
    ap.add_argument("--decode-instances", type=int, default=2, help="distinct weight instances per layer kind")
    ap.add_argument("--decode-tp-shapes", type=int, default=0,
                    help="single process only: use one rank's shard shapes of a TP group of this size (no collectives)")
    ap.add_argument("--decode-skip-operators", action="store_true", help="skip the slow reference-structure mode")
    ap.add_argument("--reference-kernel-dir", default=None,
                    help="--decode-step only: directory holding the reference's kernel.py; adds the reference-structure mode on "
                         "the reference's own Triton kernels (a comparison for whoever has the reference at hand; never needed)")
    args = ap.parse_args()
    if args.decode_step:
        run_decode_step(args)
    elif args.moe_layer:
        run_moe_layer(args)
    elif args.single:
        run_single(args)
    elif args.detail:
        run_detail(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
