"""Headline benchmark: FA2 forward + backward, bf16, B16 H16 S2048 D128 causal, on N B200s.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

One step = one forward and one backward pass (delta preprocess, dQ/dK/dV kernel, dQ convert) over
one batch of seeded synthetic inputs. With N > 1 (launched through torch.distributed.run) every rank
runs the same workload on its own inputs (independent (batch, head) units, no collective on the data
path), so the job is weak-scaled: value = FLOPs of all ranks / max-over-ranks device time.
Rank 0 prints one JSON line.

`--impl reference` times the reference path that can run here: the crate's test-harness naive
attention (fp32, CPU) restated in oracle/attention_oracle.py, on a bounded sample of the same
workload, with all host threads.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))
sys.path.insert(0, str(ROOT / "kernels-community-rs_b200"))

import torch  # noqa: E402

B, H, S, D = 16, 16, 2048, 128
CAUSAL = True
FWD_FLOPS = 4.0 * B * H * S * S * D * 0.5
BWD_FLOPS = 2.5 * FWD_FLOPS
METRIC = "FA2 fwd/bwd TFLOP/s bf16 B16 H16 S2048 D128 causal; % of B200 dense peak"
WORKLOAD = "FA2 forward+backward, causal, B=16, H_q=H_kv=16, S=2048, D=128, bf16"
# Long-context leg (strong scaling): one seeded tensor, heads split over the ranks.
LC_S, LC_H = 16384, 32
LC_FWD_FLOPS = 4.0 * LC_H * LC_S * LC_S * D * 0.5
LC_BWD_FLOPS = 2.5 * LC_FWD_FLOPS


def measured_peaks():
    f = ROOT / "MEASURED_PEAKS.json"
    if f.exists():
        d = json.loads(f.read_text())
        return d.get("bf16_tflops", 1590.0), d.get("bf16_tflops_sustained"), "measured"
    return 1590.0, 1400.0, "fallback"


class ClockSampler:
    """Samples SM clock and throttle reasons through NVML (read-only) while the timed region runs."""

    def __init__(self, index):
        self.index, self.samples, self._stop = index, [], threading.Event()
        self._t = threading.Thread(target=self._run, daemon=True)
        self.max_mhz = None

    def _run(self):
        try:
            import pynvml as nv

            nv.nvmlInit()
            visible = os.environ.get("CUDA_VISIBLE_DEVICES")
            phys = self.index
            if visible:
                ids = [x for x in visible.split(",") if x.strip()]
                if self.index < len(ids) and ids[self.index].strip().isdigit():
                    phys = int(ids[self.index])
            h = nv.nvmlDeviceGetHandleByIndex(phys)
            self.max_mhz = nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM)
            while not self._stop.is_set():
                mhz = nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)
                reasons = nv.nvmlDeviceGetCurrentClocksEventReasons(h) if hasattr(
                    nv, "nvmlDeviceGetCurrentClocksEventReasons") else nv.nvmlDeviceGetCurrentClocksThrottleReasons(h)
                self.samples.append((mhz, reasons))
                self._stop.wait(0.002)
        except Exception as e:  # clocks are reported as unknown rather than failing the bench
            self.error = f"{type(e).__name__}: {e}"

    def __enter__(self):
        self._t.start()
        return self

    def __exit__(self, *exc):
        self._stop.set()
        self._t.join(timeout=6)

    def summary(self):
        bits = {"hw_slowdown": 0x8, "sw_power_cap": 0x4, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40,
                "hw_power_brake_slowdown": 0x80}
        sm = sorted(m for m, _ in self.samples)
        seen = 0
        for _, r in self.samples:
            seen |= int(r)
        out = {"sm_mhz": sm[len(sm) // 2] if sm else None, "sm_max_mhz": self.max_mhz,
               "reasons": sorted(n for n, b in bits.items() if seen & b), "samples": len(self.samples)}
        if hasattr(self, "error"):
            out["error"] = self.error
        return out


def make_inputs(seed, pin=False):
    g = torch.Generator().manual_seed(seed)
    ts = [torch.randn(B, S, H, D, generator=g).to(torch.bfloat16) for _ in range(4)]  # q, k, v, dO
    return [t.pin_memory() for t in ts] if pin else ts


def cpu_reference_sample(pairs, threads):
    """fp32 naive attention forward + explicit backward on `pairs` (batch, head) units; seconds."""
    from oracle.attention_oracle import attention_backward, attention_forward

    torch.set_num_threads(threads)
    g = torch.Generator().manual_seed(1)
    q, k, v, do = [torch.randn(1, S, pairs, D, generator=g).to(torch.bfloat16) for _ in range(4)]
    t0 = time.perf_counter()
    out, lse = attention_forward(q, k, v, causal=CAUSAL)
    attention_backward(q, k, v, do, causal=CAUSAL, out=out, lse=lse)
    return time.perf_counter() - t0


def run_reference(args, rank):
    if rank != 0:
        return
    threads = os.cpu_count() or 1
    pairs = 8
    cpu_reference_sample(1, threads)  # warm-up (also pages torch in)
    for _ in range(max(args.warmup - 1, 0)):
        cpu_reference_sample(pairs, threads)
    times = [cpu_reference_sample(pairs, threads) for _ in range(args.steps)]
    t = sum(times) / len(times)
    flops = (FWD_FLOPS + BWD_FLOPS) * pairs / (B * H)
    value = flops / t / 1e12
    sample = f"{pairs} of the {B * H} (batch, head) units per step, forward + backward, fp32 on the host CPU"
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "TFLOP/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": t * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": WORKLOAD, "sample": sample},
        "cpu_baseline": {"value": value, "unit": "TFLOP/s", "cores": threads, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": "TFLOP/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


def run_long_context(ops, dev, rank, world, timed, steps):
    """B=1, H=32, S=16384, D=128, bf16, causal, seed 4: rank r of N runs heads shard_heads(32, 32, N, r) as
    strided views of the one seeded tensor (fixed total work: strong scaling, no collective in the timed
    region). Afterwards, once, the shards of O, LSE, dQ, dK, dV are all-gathered (NCCL) and rank 0 compares
    them with its own unsharded run."""
    import torch.distributed as dist
    from flash_attn2_b200.sharding import gather_shards, shard_heads

    if LC_H % world:
        return {"skipped": f"{LC_H} heads do not split over {world} ranks"}
    g = torch.Generator().manual_seed(4)
    full = [torch.randn(1, LC_S, LC_H, D, generator=g).to(torch.bfloat16).to(dev) for _ in range(4)]
    hq, hkv = shard_heads(LC_H, LC_H, world, rank)
    q, k, v, do = [t[:, :, hq] for t in full]
    acc = torch.empty(LC_S * (hq.stop - hq.start) * D, dtype=torch.float32, device=dev)
    state = {}

    def fwd():
        state["o"], state["lse"] = ops.fwd(q, k, v, causal=True, split=False)  # the bits of the unsharded run

    def bwd():
        delta = ops.bwd_preprocess(do, state["o"])
        state["g"] = ops.bwd(q, k, v, do, state["lse"], delta, causal=True, dq_accum=acc)

    for _ in range(3):
        fwd()
        bwd()
    ms_f = timed(fwd, steps)
    ms_b = timed(bwd, steps)
    res = {"workload": f"FA2 forward+backward, causal, B=1, H_q=H_kv={LC_H}, S={LC_S}, D={D}, bf16, seed 4",
           "scaling": "strong", "sharding": f"{LC_H // world} heads per GPU, strided views of the full tensors",
           "fwd_ms": ms_f, "bwd_ms": ms_b, "fwd_tflops": LC_FWD_FLOPS / ms_f / 1e9, "bwd_tflops": LC_BWD_FLOPS / ms_b / 1e9,
           "tflops": (LC_FWD_FLOPS + LC_BWD_FLOPS) / (ms_f + ms_b) / 1e9}
    # verification, outside every timed region
    dq, dk, dv = state["g"]
    shards = {"out": (state["o"], 2), "lse": (state["lse"], 1), "dq": (dq, 2), "dk": (dk, 2), "dv": (dv, 2)}
    if world > 1:
        gathered = {n: gather_shards(t, dim) for n, (t, dim) in shards.items()}
    else:
        gathered = {n: t for n, (t, _) in shards.items()}
    if rank == 0:
        o, lse = ops.fwd(*full[:3], causal=True, split=False)
        delta = ops.bwd_preprocess(full[3], o)
        ref = dict(zip(("dq", "dk", "dv"), ops.bwd(*full, lse, delta, causal=True)), out=o, lse=lse)
        verify = {}
        for n, t in gathered.items():
            if torch.equal(t, ref[n]):
                verify[n] = "bit-identical"
            else:
                verify[n] = "max abs diff %.3e" % (t.float() - ref[n].float()).abs().max().item()
        res["gathered_vs_unsharded"] = verify
        res["gather"] = "NCCL all_gather of the head shards" if world > 1 else "single rank"
    if world > 1:
        dist.barrier()
    return res


def run_ours(args, rank, world):
    import torch.distributed as dist
    from flash_attn2_b200 import cabi_ops as ops
    import flash_attn2_b200 as plugin

    local = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)

    host = make_inputs(1 + rank, pin=True)
    q, k, v, do = [t.to(dev, non_blocking=True) for t in host]
    acc = torch.empty(B * S * H * D, dtype=torch.float32, device=dev)
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731
    k0, k1 = ev(), ev()
    k0.record(), k1.record()  # materialise the handles
    torch.cuda.synchronize()

    launches = {"n": 0}  # kernels of this library enqueued: forward 1, delta preprocess 1, backward 2 (dQ/dK/dV + dQ convert)

    def fwd_only():
        launches["n"] += 1
        return ops.fwd(q, k, v, causal=CAUSAL)

    def bwd_only(o, lse, events=None):
        launches["n"] += 3
        delta = ops.bwd_preprocess(do, o)
        return ops.bwd(q, k, v, do, lse, delta, causal=CAUSAL, dq_accum=acc, kernel_events=events)

    def step():
        o, lse = fwd_only()
        return bwd_only(o, lse)

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    def timed(fn, n):
        barrier()
        e0, e1 = ev(), ev()
        e0.record()
        for _ in range(n):
            fn()
        e1.record()
        barrier()
        ms = e0.elapsed_time(e1)
        if world > 1:
            t = torch.tensor([ms], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms / n

    for _ in range(args.warmup):
        step()
    # The clock record covers the timed region of `value` only: the legs below pause between kernels, and an
    # idle GPU's clock says nothing about the run.
    with ClockSampler(local) as clocks:
        launches["n"] = 0
        ms_step = timed(step, args.steps)
        launches_timed = launches["n"]
    # Per-kernel figures for the roofline and the per-pass targets. Every leg starts from the same state: a
    # pause, then its own warm-up. Without it the legs measured last come out 5-9 % slower than the same
    # loop run first (the GPU's power management after 50-100 ms of back-to-back kernels), so the order of
    # the legs, not the kernels, would set the figures.
    def settle(fn):
        barrier()
        time.sleep(0.3)
        for _ in range(max(3, args.warmup)):
            fn()

    settle(fwd_only)
    ms_fwd = timed(fwd_only, args.steps)
    o, lse = fwd_only()
    settle(lambda: bwd_only(o, lse))
    ms_bwd = timed(lambda: bwd_only(o, lse), args.steps)
    settle(lambda: bwd_only(o, lse))
    kt = []
    for _ in range(args.steps):
        bwd_only(o, lse, events=(k0, k1))
        torch.cuda.synchronize()
        kt.append(k0.elapsed_time(k1))
    ms_bwd_kernel = sum(kt) / len(kt)
    status = ops.device_status()
    if status != 0:
        raise RuntimeError(f"kernel pipeline reported a stalled wait (status {status})")

    # Sustained leg: the same step back to back for at least a second, so that the GPU settles at the clock
    # its power limit allows; reported beside the burst figure with its own clock record.
    sustained = None
    if not args.kernels_only:
        n_sus = max(args.steps, int(1100.0 / ms_step) + 1)
        with ClockSampler(local) as sus_clocks:
            ms_sus = timed(step, n_sus)
        sustained = {"steps": n_sus, "ms_per_step": ms_sus, "clocks": sus_clocks.summary()}

    long_context = None
    if not args.kernels_only and args.batch == 16:
        long_context = run_long_context(ops, dev, rank, world, timed, max(3, args.steps // 2))

    # End to end through the operator (plugin) API with host buffers: H2D of q, k, v, dO, the
    # tvm-ffi forward + backward, D2H of O, LSE, dQ, dK, dV.
    outs_host = [torch.empty_like(host[0]).pin_memory() for _ in range(4)]
    lse_host = torch.empty(B, H, S, dtype=torch.float32).pin_memory()
    h2d = sum(t.numel() * t.element_size() for t in host)
    d2h = sum(t.numel() * t.element_size() for t in outs_host) + lse_host.numel() * 4

    # Three streams, two buffer slots: the H2D copy of step i + 1 and the D2H copy of step i - 1 run under
    # the kernels of step i (PCIe is full duplex). Every step still moves its own inputs and outputs inside
    # the timed region.
    s_in, s_c, s_out = torch.cuda.Stream(dev), torch.cuda.Stream(dev), torch.cuda.Stream(dev)
    dev_in = [[torch.empty_like(t, device=dev) for t in host] for _ in range(2)]
    in_ready = [torch.cuda.Event() for _ in range(2)]
    in_free = [torch.cuda.Event() for _ in range(2)]
    c_done = [torch.cuda.Event() for _ in range(2)]
    out_done = [torch.cuda.Event() for _ in range(2)]
    hold = [None, None]

    def e2e_pipeline(n):
        for i in range(n):
            sl = i & 1
            if hold[sl] is not None:
                out_done[sl].synchronize()  # the outputs of step i - 2 have left the device
            with torch.cuda.stream(s_in):
                if i >= 2:
                    s_in.wait_event(in_free[sl])
                for dst, src in zip(dev_in[sl], host):
                    dst.copy_(src, non_blocking=True)
                in_ready[sl].record(s_in)
            with torch.cuda.stream(s_c):
                s_c.wait_event(in_ready[sl])
                qd, kd, vd, dod = dev_in[sl]
                out, lse_d, _, _ = plugin.fwd(qd, kd, vd, is_causal=CAUSAL)
                dq, dk, dv, _ = plugin.bwd(dod, qd, kd, vd, out, lse_d, is_causal=CAUSAL)
                in_free[sl].record(s_c)
                c_done[sl].record(s_c)
            with torch.cuda.stream(s_out):
                s_out.wait_event(c_done[sl])
                for dst, src in zip(outs_host, (out, dq, dk, dv)):
                    src.record_stream(s_out)
                    dst.copy_(src, non_blocking=True)
                lse_d.record_stream(s_out)
                lse_host.copy_(lse_d, non_blocking=True)
                out_done[sl].record(s_out)
            hold[sl] = (out, lse_d, dq, dk, dv)

    def timed_pipeline(n):
        barrier()
        e0, e1 = ev(), ev()
        cur = torch.cuda.current_stream(dev)
        e0.record(cur)
        for st in (s_in, s_c, s_out):
            st.wait_event(e0)
        e2e_pipeline(n)
        for st in (s_in, s_c, s_out):
            done = torch.cuda.Event()
            done.record(st)
            cur.wait_event(done)
        e1.record(cur)
        barrier()
        ms = e0.elapsed_time(e1)
        if world > 1:
            t = torch.tensor([ms], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms / n

    ms_e2e = None
    if not args.kernels_only:
        e2e_steps = max(4, min(args.steps, 8))
        timed_pipeline(2)
        hold[0] = hold[1] = None
        ms_e2e = timed_pipeline(e2e_steps)

    if rank == 0:
        peak, peak_sustained, peak_kind = measured_peaks()
        total = (FWD_FLOPS + BWD_FLOPS) * world
        tf = lambda fl, ms: fl / ms / 1e9  # noqa: E731
        traffic = None
        tfile = ROOT / "profiles" / "ncu_traffic.json"
        if tfile.exists() and (B, D) == (16, 128):
            traffic = json.loads(tfile.read_text()).get("bwd_kernel_dram_bytes_per_launch")
        cpu = None
        if world == 1 and not args.kernels_only:
            threads = os.cpu_count() or 1
            pairs = 16
            cpu_reference_sample(1, threads)
            t = cpu_reference_sample(pairs, threads)
            cpu = {"value": (FWD_FLOPS + BWD_FLOPS) * pairs / (B * H) / t / 1e12, "unit": "TFLOP/s", "cores": threads,
                   "kind": "port",
                   "sample": f"{pairs} of the {B * H} (batch, head) units, forward + backward, fp32 on the host CPU"}
        achieved = tf(BWD_FLOPS, ms_bwd_kernel)
        line = {
            "metric": METRIC if (B, D) == (16, 128) else METRIC.replace("B16", f"B{B}").replace("D128", f"D{D}") + " (not the headline configuration)",
            "value": tf(total, ms_step), "unit": "TFLOP/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
            "config": {"workload": WORKLOAD if (B, D) == (16, 128) else WORKLOAD.replace("B=16", f"B={B}").replace("D=128", f"D={D}") + " (not the headline configuration)",
                       "global_batch": B * world, "sharding": "independent batches per GPU",
                       "l2": "inputs and outputs (1.1 GB per step at B=16) exceed the 126 MB L2",
                       "value_path": "C ABI (fa2_fwd, fa2_bwd_preprocess, fa2_bwd) with a preallocated dQ accumulator, inputs resident in HBM",
                       "e2e_path": "tvm-ffi operators (fwd_lse, bwd_preprocess, bwd_all) with pinned host buffers"},
            "detail": {
                "fwd_tflops": tf(FWD_FLOPS * world, ms_fwd), "bwd_tflops": tf(BWD_FLOPS * world, ms_bwd),
                "fwd_ms": ms_fwd, "bwd_ms": ms_bwd, "bwd_kernel_ms": ms_bwd_kernel,
                "fwd_frac_of_peak": tf(FWD_FLOPS, ms_fwd) / peak, "bwd_frac_of_peak": tf(BWD_FLOPS, ms_bwd) / peak,
                "peak_tflops": peak, "peak_sustained_tflops": peak_sustained, "peak_kind": peak_kind,
                "sustained": None if sustained is None else dict(
                    sustained, tflops=tf(total, sustained["ms_per_step"]),
                    frac_of_sustained_peak=None if not peak_sustained else tf(total / world, sustained["ms_per_step"]) / peak_sustained),
                "long_context": long_context,
            },
            "roofline": {"kernel": "bwd_kernel<128, bf16>" if D <= 128 else "bwd_wide_pair_kernel<bf16>" if D in (192, 256) else "bwd_wide_kernel<bf16>", "bound": "tensor", "achieved": achieved, "peak": peak,
                         "unit": "TFLOP/s", "frac": achieved / peak, "traffic": traffic, "peak_kind": peak_kind},
            "roofline_fwd": {"kernel": "fwd_kernel<128, bf16>" if D <= 128 else "fwd_wide_kernel<bf16>", "bound": "tensor", "achieved": tf(FWD_FLOPS, ms_fwd),
                             "peak": peak, "unit": "TFLOP/s", "frac": tf(FWD_FLOPS, ms_fwd) / peak},
            "cpu_baseline": cpu,
            "e2e": None if ms_e2e is None else {"value": tf(total, ms_e2e), "unit": "TFLOP/s",
                                                 "h2d_bytes_per_step": h2d * world, "d2h_bytes_per_step": d2h * world,
                                                 "ms_per_step": ms_e2e},
            "gpu_launches": launches_timed,
            "clocks": clocks.summary(),
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--batch", type=int, default=16,
                    help="batch size; 16 is the benchmark, smaller values only size ncu captures")
    ap.add_argument("--kernels-only", action="store_true",
                    help="skip the end-to-end and CPU-baseline legs (for ncu captures)")
    ap.add_argument("--head-dim", type=int, default=128,
                    help="head dim; 128 is the benchmark, others (with --kernels-only) size ncu captures of the other kernels")
    args = ap.parse_args()
    if args.head_dim != 128 and not args.kernels_only:
        ap.error("--head-dim other than 128 goes with --kernels-only")
    args.warmup = max(args.warmup, 3) if args.impl == "ours" else args.warmup
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    global B, D, FWD_FLOPS, BWD_FLOPS
    if args.batch != B or args.head_dim != D:
        B, D = args.batch, args.head_dim
        FWD_FLOPS = 4.0 * B * H * S * S * D * 0.5
        BWD_FLOPS = 2.5 * FWD_FLOPS
    if args.impl == "reference":
        run_reference(args, rank)
    else:
        run_ours(args, rank, world)


if __name__ == "__main__":
    main()
