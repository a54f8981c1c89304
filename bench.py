"""Benchmark: BLS12-446 G1 MSM points/s on B200 (one JSON line on rank 0).

Workload (the plain single-GPU configuration): one G1 MSM of n = 2^20
points per GPU, scalars uniform in [0, r) with 1% zeros and 1% ones, bases
P_i = t_i * G with 2% duplicated, 5 x u64 limbs per scalar, seeded synthetic
data (no dataset).  With N GPUs each rank runs the same shape on its own
shard (weak scaling); the shards' partial sums are exchanged with one
all_gather and added on the device, as a sharded MSM does.

Keys beyond the driver contract:
  roofline      the additions of entries (affine rounds, accumulation): their fixed op count
                (798 IMAD per Fp product) against the measured mad.lo peak of
                this GPU (bound "imad": the path is exact integer arithmetic;
                neither tensor cores nor HBM bound it)
  msm_roofline  the whole MSM against the same peak, with the fixed op count
  value         timed steps run round-robin over PIPELINE_STREAMS streams
                (consecutive MSMs overlap); ms_per_step_serial is one stream,
                and the phase times and roofline come from that serial pass
  cpu_baseline  the reference's own host code (oracle/_ref) on the host cores
  extra         Fp 2^26, Fp2 2^24 and G2 2^18 measurements, phase breakdown,
                the batched (512 MSMs) and served workloads

--impl reference times the reference's CPU implementation of the path
(oracle/_ref, all host threads) on a bounded sample of the same workload.
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

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

LOG2N = 20
G2_LOG2N = 18
# the timed plain-MSM steps run round-robin over this many streams: one MSM's
# latency-bound tail (upper reduction levels, window combine) then
# overlaps the next MSM's accumulation (G1 2^20: 10.8 -> 10.1 ms per MSM)
PIPELINE_STREAMS = 3
# CPU baseline sample: the first 2^16 points (about 1 s per pass on 16 host
# cores); the repo arm reports the median of CPU_RUNS passes
CPU_SAMPLE = 1 << 16
CPU_RUNS = 5
FP_MICRO = 1 << 26
FP2_MICRO = 1 << 24
METRIC = "MSM points/s (G1 2^20, G2 2^18) batched vs plain on 1 B200, bit-exact; p99 ms"


# fixed-base window tables (window widths) for the resident-table workloads
PRECOMPUTE_BATCH = (8, 10, 12, 14, 16)
PRECOMPUTE_SERVE = {1: (11, 14, 17, 20), 2: (11, 13, 16)}

def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-extra", action="store_true", help="skip the Fp / G2 / CPU side measurements")
    ap.add_argument("--msm-only", metavar="G,LOG2N", default=None,
                    help="profiling workload: plain MSMs of group G (1 or 2) over 2^LOG2N synthetic points, "
                         "--warmup untimed and --steps timed calls, one JSON line with time and phases")
    return ap.parse_args()


def host_threads() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


# ---------------------------------------------------------------------------
# clocks sampled during the timed region
# ---------------------------------------------------------------------------
class ClockSampler:
    """SM clock, its maximum and the active clock-event reasons, read (never
    set) every 10 ms during the timed region through NVML, with nvidia-smi as
    the fallback.  Entering waits for the first sample, so even a region of a
    few tens of milliseconds is covered."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    # NVML clock-event reason bits
    REASONS = {"sw_power_cap": 0x4, "hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40}

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.proc = None
        self.lines = []
        self.samples = []   # (sm MHz, max MHz, reason bits)
        self.stop = threading.Event()
        self.nvml = None

    def _handle(self):
        import pynvml
        pynvml.nvmlInit()
        try:
            import torch
            pr = torch.cuda.get_device_properties(self.gpu)
            bus = f"{pr.pci_domain_id:08x}:{pr.pci_bus_id:02x}:{pr.pci_device_id:02x}.0"
            return pynvml, pynvml.nvmlDeviceGetHandleByPciBusId(bus)
        except Exception:
            return pynvml, pynvml.nvmlDeviceGetHandleByIndex(self.gpu)

    def _poll(self):
        nv, h = self.nvml
        get_reasons = getattr(nv, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
            nv.nvmlDeviceGetCurrentClocksThrottleReasons
        while True:
            try:
                self.samples.append((nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM),
                                     nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM), int(get_reasons(h))))
            except Exception:
                return
            if self.stop.wait(0.01):
                return

    def __enter__(self):
        try:
            self.nvml = self._handle()
            self.t = threading.Thread(target=self._poll, daemon=True)
            self.t.start()
            t0 = time.perf_counter()
            while not self.samples and time.perf_counter() - t0 < 1.0:
                time.sleep(0.002)
            return self
        except Exception:
            self.nvml = None
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except (OSError, FileNotFoundError):
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.nvml is not None:
            self.stop.set()
            self.t.join(timeout=2)
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], None, set()
        for clk, mclk, bits in self.samples:
            sm.append(float(clk))
            mx = float(mclk)
            for nm, b in self.REASONS.items():
                if bits & b:
                    reasons.add(nm)
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(sm),
                "source": "nvml" if self.samples else "nvidia-smi"}


# ---------------------------------------------------------------------------
# Additions of G1 2^20 entries (four k_affine_round<Fp> launches and
# k_accumulate<Fp>): DRAM bytes of the four rounds and their pipe utilisation,
# from the ncu capture summarised in profiles/k_affine_round.md
ADD_TRAFFIC_NCU = 13.95e9
ADD_PIPES_NCU = {"fmaheavy_imad": 0.725, "alu": 0.237, "issue": 0.347}

# CPU baseline: reference host code (or the oracle port) on a bounded sample
# ---------------------------------------------------------------------------
def cpu_baseline_run(points, scalars, threads):
    import oracle
    t0 = time.perf_counter()
    res = oracle.ref_msm_pippenger(points, scalars, group=1, threads=threads)
    kind = "reference"
    if res is None:
        oracle.msm_pippenger(points, scalars, group=1, threads=threads)
        kind = "port"
    dt = time.perf_counter() - t0
    return len(points) / dt, kind, dt


def cpu_sample_inputs(n):
    """First n points of the benchmark workload, computed on the CPU."""
    from concurrent.futures import ThreadPoolExecutor

    import oracle
    from gpu_msm_b200 import workload as wl
    sc = wl.make_scalars(1 << LOG2N, seed=42)[:n]
    logs = wl.make_base_logs(1 << LOG2N, seed=4242)[:n]
    g = oracle.g1_generator()
    ts = wl.limbs_to_ints(logs)
    with ThreadPoolExecutor(max_workers=host_threads()) as ex:
        pts = list(ex.map(lambda t: oracle.scalar_mul(g, t), ts))
    return np.concatenate(pts), sc


def run_reference(args, rank, world):
    """--impl reference: rank 0 times the reference CPU path; others exit."""
    if rank != 0:
        return
    threads = host_threads()
    pts, sc = cpu_sample_inputs(CPU_SAMPLE)
    # warm-up passes over the whole sample (the first pass of a process runs
    # about a quarter slower: thread start-up, page faults)
    for _ in range(max(1, args.warmup)):
        cpu_baseline_run(pts, sc, threads)
    times, kind = [], "reference"
    for _ in range(args.steps):
        _, kind, dt = cpu_baseline_run(pts, sc, threads)
        times.append(dt)
    t = statistics.mean(times)
    value = CPU_SAMPLE / t
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "points/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": t * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u64 limbs (exact integer)", "data": "synthetic",
        "config": {"workload": f"G1 MSM, 2^{LOG2N}-point workload, timed on its first {CPU_SAMPLE} points",
                   "scalar_limbs": 5, "parallelism": "host threads"},
        "cpu_baseline": {"value": value, "unit": "points/s", "cores": threads, "kind": kind,
                         "sample": f"first {CPU_SAMPLE} points of the G1 2^{LOG2N} workload per step; "
                                   "4-bit windows, projective buckets, combine_buckets_cpu_projective_g1"},
        "e2e": {"value": value, "unit": "points/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------
# our arm
# ---------------------------------------------------------------------------
def run_msm_only(args):
    """Plain single-GPU MSMs of one group and size (the workload the ncu
    summaries of profiles/ are captured on for sizes other than the bench's)."""
    import torch

    import gpu_msm_b200 as gm
    from gpu_msm_b200 import workload as wl
    group, log2n = (int(x) for x in args.msm_only.split(","))
    if group not in (1, 2) or not 1 <= log2n <= 24:
        raise SystemExit("--msm-only G,LOG2N with G in {1, 2} and 1 <= LOG2N <= 24")
    n = 1 << log2n
    dev = torch.device("cuda", 0)
    logs = wl.make_base_logs(n, seed=4343)
    pts = gm.generator_mul_batch(torch.from_numpy(logs.view(np.int64)).to(dev), group=group)
    sc = torch.from_numpy(wl.make_scalars(n, seed=43).view(np.int64)).to(dev)
    out = torch.empty(gm.G1P_WORDS if group == 1 else gm.G2P_WORDS, dtype=torch.int64, device=dev)
    for _ in range(args.warmup):
        gm.msm_device(pts, sc, group=group, out=out)
    torch.cuda.synchronize()
    gm.profile_enable(True)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.steps):
        gm.msm_device(pts, sc, group=group, out=out)
    e1.record()
    torch.cuda.synchronize()
    acc = {}
    for k, v in gm.profile_collect():
        if k != "start":
            acc.setdefault(k, []).append(v)
    gm.profile_enable(False)
    ms = e0.elapsed_time(e1) / args.steps
    print(json.dumps({"workload": f"plain G{group} MSM, n=2^{log2n}", "ms_per_msm": ms, "points_per_s": n / (ms / 1e3),
                      "phases_ms": {k: statistics.mean(v) for k, v in acc.items()}}), flush=True)


def run_ours(args, rank, world, local_rank):
    import torch
    import torch.distributed as dist

    import gpu_msm_b200 as gm
    from gpu_msm_b200 import workload as wl

    dev = torch.device("cuda", local_rank)
    torch.cuda.set_device(dev)
    n = 1 << LOG2N

    # inputs of this rank's shard, resident in HBM before timing
    sc = wl.make_scalars(n, seed=42 + 1000 * rank)
    logs = wl.make_base_logs(n, seed=4242 + 1000 * rank)
    sc_d = torch.from_numpy(sc.view(np.int64)).to(dev)
    pts_d = gm.generator_mul_batch(torch.from_numpy(logs.view(np.int64)).to(dev), group=1)
    torch.cuda.synchronize()
    c = gm.default_window(1, n, 5)
    entries = int(wl.signed_digit_counts(sc, c).sum())

    # one result (and gather) buffer per stream, so that MSMs in flight on
    # different streams never share one
    outs = [torch.empty(gm.G1P_WORDS, dtype=torch.int64, device=dev) for _ in range(PIPELINE_STREAMS)]
    gathered = [torch.empty(world * gm.G1P_WORDS, dtype=torch.int64, device=dev) if world > 1 else None
                for _ in range(PIPELINE_STREAMS)]

    def step(k, stream):
        with torch.cuda.stream(stream):
            gm.msm_device(pts_d, sc_d, group=1, out=outs[k], stream=stream)
            if world > 1:
                dist.all_gather_into_tensor(gathered[k], outs[k])
                gm.sum_projective(gathered[k].view(world, gm.G1P_WORDS), group=1, out=outs[k], stream=stream)

    main = torch.cuda.current_stream()
    side = [torch.cuda.Stream() for _ in range(PIPELINE_STREAMS)]

    def run_steps(steps, pipelined):
        """Device time per step (ms): one stream, or steps round-robin over
        PIPELINE_STREAMS streams (one step's latency-bound tail -- upper
        reduction levels, window combine -- overlaps the next step's
        accumulation)."""
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev0.record(main)
        if pipelined:
            for s in side:
                s.wait_stream(main)
            for i in range(steps):
                step(i % PIPELINE_STREAMS, side[i % PIPELINE_STREAMS])
            for s in side:
                main.wait_stream(s)
        else:
            for _ in range(steps):
                step(0, main)
        ev1.record(main)
        torch.cuda.synchronize()
        return ev0.elapsed_time(ev1) / steps

    def max_over_ranks(ms):
        t = torch.tensor([ms], dtype=torch.float64, device=dev)
        if world > 1:
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    for _ in range(args.warmup):
        step(0, main)
    torch.cuda.synchronize()

    # serial pass (one stream, phase events on): the per-phase times and the
    # dominant kernel's duration for the roofline, free of other MSMs' kernels
    gm.profile_enable(True)
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    ms = run_steps(args.steps, pipelined=False)
    phases = gm.profile_collect()
    gm.profile_enable(False)
    serial_ms_max = max_over_ranks(ms)
    serial_aff = gm.canonical_affine(gm.to_numpy_proj(outs[0], 1), 1)

    # timed region: the same steps, pipelined over PIPELINE_STREAMS streams
    # (untimed first until every stream's MSM has its workspace: a pass can
    # find one fewer than it would use, since an allocation that waits lets an
    # earlier MSM's workspace come free)
    for _ in range(PIPELINE_STREAMS):
        run_steps(max(args.warmup, PIPELINE_STREAMS), pipelined=True)
    gm.launch_count_reset()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    with ClockSampler(local_rank) as clk:
        ms_pipe = run_steps(args.steps, pipelined=True)
    if world > 1:
        dist.barrier()
    launches = gm.launch_count_reset()
    ms_max = max_over_ranks(ms_pipe)
    value = world * n / (ms_max / 1e3)
    # every pipelined step's result equals the serial one (compared in affine
    # form: projective coordinates depend on the order of additions in a bucket)
    pipelined_ok = all(np.array_equal(gm.canonical_affine(gm.to_numpy_proj(o, 1), 1), serial_aff) for o in outs)

    # per-phase averages and the dominant kernel
    acc = {}
    for name, v in phases:
        if name == "start":
            continue
        acc.setdefault(name, []).append(v)
    phase_ms = {k: statistics.mean(v) for k, v in acc.items()}

    # end to end through the host-buffer API: every rank takes part (at N > 1
    # the steps' partial sums are gathered and combined inside the timed region)
    e2e = measure_e2e(args, gm, sc, pts_d, world=world, dev=dev)

    if rank != 0:
        return

    # multiply-add ceilings of this GPU (project microbenchmark): mad.lo alone
    # (the roofline peak) and the lo/hi mix of an integer Montgomery product
    sink = torch.empty(148 * 8 * 256 * 4, dtype=torch.int32, device=dev)
    iters = 4096
    peaks = {}
    for mode in (0, 1):
        gm.imad_probe(64, sink, mode=mode)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = 0.0
        for _ in range(3):
            e0.record()
            cnt = gm.imad_probe(iters, sink, mode=mode)
            e1.record()
            torch.cuda.synchronize()
            best = max(best, cnt / (e0.elapsed_time(e1) / 1e3))
        peaks[mode] = best
    # roofline denominator: the IMAD issue peak (mad.lo only), against which
    # the fixed op count (798 IMAD per Fp product) is quoted.  The lo/hi mix
    # of an integer Montgomery product runs well below it (the hi halves take
    # extra pipe time).
    imad_peak = peaks[1]

    # additions of entries: affine rounds and the accumulation of what they
    # leave.  Every entry is counted as one affine addition (6 products with
    # its share of the inversion); those that the accumulation adds in XYZZ
    # form take 10, so the rate is a lower bound.
    acc_ms = phase_ms.get("affine", 0.0) + phase_ms.get("accumulate", float("nan"))
    acc_imad = 798.0 * 6 * entries
    achieved = acc_imad / (acc_ms / 1e3)
    msm_ops = wl.msm_roofline_imad(n, 1)

    line = {
        "metric": METRIC, "value": value, "unit": "points/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_max, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "u32 limbs (exact integer)", "data": "synthetic",
        "config": {"workload": f"plain single G1 MSM, n=2^{LOG2N} per GPU, scalars < r (5 x u64), "
                               "1% zeros, 1% ones, bases t_i*G with 2% duplicates",
                   "window_bits": c, "entries": entries, "parallelism": f"points sharded x{world}",
                   "streams": f"{PIPELINE_STREAMS} (consecutive steps round-robin; each step a full MSM)",
                   "l2": "inputs 168 MB > 126 MB L2 (no flush)"},
        "ms_per_step_serial": serial_ms_max,
        "pipelined_results_equal": bool(pipelined_ok),
        "roofline": {"bound": "imad", "kernel": "k_affine_round<Fp> + k_accumulate<Fp>", "achieved": achieved / 1e12,
                     "peak": imad_peak / 1e12, "unit": "TIMAD/s", "frac": achieved / imad_peak,
                     # dram__bytes_read + dram__bytes_write of one MSM's affine rounds,
                     # from the ncu capture summarised in profiles/k_affine_round.md
                     "traffic": ADD_TRAFFIC_NCU,
                     "traffic_unit": "bytes per MSM (ncu, affine rounds)",
                     "work": f"798 IMAD-equivalents x 6 Fp mults x {entries} entries per MSM",
                     "peak_source": "measured: gm_imad_probe mode 1 (independent mad.lo chains over all SMs)",
                     "peak_lo_hi_mix": peaks[0] / 1e12,
                     "products_on": "IMAD pipe (CIOS, mad.lo.cc/madc.hi.cc)",
                     "pipes_busy_ncu": ADD_PIPES_NCU},
        "msm_roofline": {"ops_imad": msm_ops, "achieved": msm_ops / (ms_max / 1e3) / 1e12,
                         "frac": msm_ops / (ms_max / 1e3) / imad_peak, "unit": "TIMAD/s",
                         "frac_serial": msm_ops / (serial_ms_max / 1e3) / imad_peak},
        "phases_ms": phase_ms,
        "gpu_launches": int(launches),
    }
    line["clocks"] = clk.summary()

    line["e2e"] = e2e
    if world == 1:
        if not args.no_extra:
            line["extra"] = measure_extra(gm, wl, dev, imad_peak)
            pts_h = gm.to_numpy_points(pts_d[:CPU_SAMPLE], 1)
            cpu_baseline_run(pts_h, sc[:CPU_SAMPLE], host_threads())   # warm-up pass
            runs = [cpu_baseline_run(pts_h, sc[:CPU_SAMPLE], host_threads()) for _ in range(CPU_RUNS)]
            vals = sorted(r[0] for r in runs)
            kind = runs[0][1]
            line["cpu_baseline"] = {
                "value": statistics.median(vals), "unit": "points/s", "cores": host_threads(), "kind": kind,
                "runs": vals,
                "sample": f"first {CPU_SAMPLE} points of this workload, median of {CPU_RUNS} passes after a warm-up pass "
                          f"({sum(r[2] for r in runs):.1f} s in all), reference-structured "
                          "Pippenger: 4-bit windows, projective buckets, combine per window"}
    print(json.dumps(line), flush=True)


def measure_e2e(args, gm, sc, pts_d, world=1, dev=None):
    """End to end through the public host-buffer API, pinned host buffers:
    every step copies its points and scalars to the device, runs the MSM and
    reads its result back to the host.

    value: gm_g1_msm_host_async round-robin on PIPELINE_STREAMS streams, so
    that one step's copies overlap the previous steps' compute (each step's
    copies and result read are still inside the timed region).  sync_value: the blocking
    g1_msm_limbs_wrapper, one MSM at a time (one GPU only).  With N ranks each
    rank runs the steps on its own shard; the steps' partial sums are then
    gathered once and added on the device, inside the timed region, and the
    time is the maximum over ranks."""
    import torch
    n = len(sc)
    pts_pin = torch.empty((n, gm.G1_WORDS), dtype=torch.int64, pin_memory=True)
    pts_pin.copy_(pts_d.cpu())
    sc_pin = torch.empty((n, 5), dtype=torch.int64, pin_memory=True)
    sc_pin.copy_(torch.from_numpy(sc.view(np.int64)))
    pts_np = pts_pin.numpy().view(np.uint64).view(gm.G1).reshape(-1)
    sc_np = sc_pin.numpy().view(np.uint64)
    # at least 24 steps: filling and draining the three-stream pipeline (the
    # first step's copies, the last step's tail, ~7 ms in all) then weigh
    # under 2 % of the per-step time (measured: 10 steps 16.64 ms, 24 steps
    # 15.95 ms, against 15.68 ms for device-resident inputs)
    steps = max(24, args.steps)

    for _ in range(2):
        ref = gm.msm(pts_np, sc_np, group=1, montgomery=True)
    sync_dt = None
    if world == 1:
        t0 = time.perf_counter()
        for _ in range(steps):
            gm.msm(pts_np, sc_np, group=1, montgomery=True)
        sync_dt = (time.perf_counter() - t0) / steps

    ns = PIPELINE_STREAMS
    streams = [torch.cuda.Stream() for _ in range(ns)]
    res_pin = torch.zeros((steps + ns, gm.G1P_WORDS), dtype=torch.int64, pin_memory=True)
    res_np = res_pin.numpy().view(np.uint64).view(gm.G1P).reshape(-1)
    err_pin = torch.ones(steps + ns, dtype=torch.int32, pin_memory=True)
    err_np = err_pin.numpy().view(np.uint32)
    for i in range(ns):
        gm.msm_host_async(pts_np, sc_np, res_np[i:i + 1], stream=streams[i], err=err_np[i:i + 1])
    for st in streams:
        st.synchronize()
    if world > 1:
        import torch.distributed as dist
        dist.barrier()
    t0 = time.perf_counter()
    for i in range(ns, steps + ns):
        gm.msm_host_async(pts_np, sc_np, res_np[i:i + 1], stream=streams[i % ns], err=err_np[i:i + 1])
    for st in streams:
        st.synchronize()
    if world > 1:
        # every step's full MSM: its partial sums from all ranks, gathered
        # once and added on the device, then read back
        parts = torch.from_numpy(res_np[ns:].view(np.uint64).view(np.int64).reshape(-1).copy()).to(dev)
        gathered = torch.empty(world * parts.numel(), dtype=torch.int64, device=dev)
        dist.all_gather_into_tensor(gathered, parts)
        g = gathered.view(world, steps, gm.G1P_WORDS)
        full = torch.empty((steps, gm.G1P_WORDS), dtype=torch.int64, device=dev)
        for k in range(steps):
            gm.sum_projective(g[:, k, :].contiguous(), group=1, out=full[k])
        full_h = full.cpu()
    dt = time.perf_counter() - t0
    if world > 1:
        t = torch.tensor([dt], dtype=torch.float64, device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        dt = float(t.item())
    dt /= steps
    want = gm.canonical_affine(ref.reshape(1), 1)
    ok = bool(err_np.max() == 0) and all(
        np.array_equal(gm.canonical_affine(res_np[i:i + 1], 1), want) for i in range(steps + ns))
    out = {"value": world * n / dt, "unit": "points/s", "h2d_bytes_per_step": n * (120 + 40),
           "d2h_bytes_per_step": 168 + 4, "ms_per_step": dt * 1e3,
           "api": f"gm_g1_msm_host_async on {ns} streams (host buffers, pinned)", "results_equal": ok}
    if world > 1:
        fh = full_h.numpy().view(np.uint64).view(gm.G1P).reshape(-1)
        first = gm.canonical_affine(fh[:1], 1)
        out["api"] += (f"; each rank its own shard, the {steps} steps' partial sums gathered once and added "
                       "on the device inside the timed region, max over ranks")
        out["results_equal"] = ok and all(np.array_equal(gm.canonical_affine(fh[k:k + 1], 1), first)
                                          for k in range(steps))
        out["h2d_bytes_per_step"] = world * n * (120 + 40)
        out["d2h_bytes_per_step"] = world * (168 + 4) + 168
    else:
        out.update({"sync_value": n / sync_dt, "sync_ms_per_step": sync_dt * 1e3,
                    "sync_api": "g1_msm_limbs_wrapper (host buffers, pinned)"})
    return out


def measure_fp2_micro(gm, wl, dev, imad_peak, reps=5, check_n=1 << 14):
    """Fp2 microbench: 2^24 independent fp2_mont_mul pairs (3-product
    Karatsuba, i^2 = -1), Montgomery form, element-wise over device arrays --
    the work of the reference's fp2_mul_array_host without its per-call copies.
    2,394 IMAD and 336 bytes per product.  A 2^14 subset is checked against
    Python big integers: (a0 + a1 i)(b0 + b1 i) 2^-448 mod p."""
    import torch
    rng = np.random.default_rng(24)
    a = torch.from_numpy(rng.integers(0, 2 ** 63, size=(FP2_MICRO, 14), dtype=np.int64)).to(dev)
    a[:, 6] &= 0x1FFFFFFFFFFFFFFF       # each coordinate < 2^445 < p
    a[:, 13] &= 0x1FFFFFFFFFFFFFFF
    b = torch.roll(a, 1, 0)
    c = torch.empty_like(a)
    for _ in range(2):
        gm.field_mul_array(a, b, op="fp2_mont_mul", out=c)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        gm.field_mul_array(a, b, op="fp2_mont_mul", out=c)
    e1.record()
    torch.cuda.synchronize()
    t = e0.elapsed_time(e1) / reps / 1e3
    P = wl.P_MODULUS
    rinv = pow(1 << 448, -1, P)
    ah = a[:check_n].cpu().numpy().view(np.uint64)
    bh = b[:check_n].cpu().numpy().view(np.uint64)
    ch = c[:check_n].cpu().numpy().view(np.uint64)

    def val(row, k):
        return sum(int(row[7 * k + i]) << (64 * i) for i in range(7))

    ok = 0
    for i in range(check_n):
        a0, a1, b0, b1 = val(ah[i], 0), val(ah[i], 1), val(bh[i], 0), val(bh[i], 1)
        c0 = (a0 * b0 - a1 * b1) * rinv % P
        c1 = (a0 * b1 + a1 * b0) * rinv % P
        ok += (val(ch[i], 0), val(ch[i], 1)) == (c0, c1)
    return {"products_per_s": FP2_MICRO / t, "ms": t * 1e3, "imad_frac": FP2_MICRO * 2394 / t / imad_peak,
            "hbm_gbs": FP2_MICRO * 336 / t / 1e9, "checked": f"{ok}/{check_n}", "all_checked_equal": ok == check_n}


def measure_extra(gm, wl, dev, imad_peak):
    import torch
    out = {}
    # Fp microbench: 2^26 independent fp_mont_mul pairs, Montgomery form
    rng = np.random.default_rng(26)
    a = torch.from_numpy(rng.integers(0, 2 ** 63, size=(FP_MICRO, 7), dtype=np.int64)).to(dev)
    a[:, 6] &= 0x1FFFFFFFFFFFFFFF
    b = torch.roll(a, 1, 0)
    c = torch.empty_like(a)
    for _ in range(2):
        gm.field_mul_array(a, b, op="fp_mont_mul", out=c)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    reps = 5
    for _ in range(reps):
        gm.field_mul_array(a, b, op="fp_mont_mul", out=c)
    e1.record()
    torch.cuda.synchronize()
    t = e0.elapsed_time(e1) / reps / 1e3
    out["fp_mont_mul_2^26"] = {"muls_per_s": FP_MICRO / t, "ms": t * 1e3,
                               "imad_frac": FP_MICRO * 798 / t / imad_peak,
                               "hbm_gbs": FP_MICRO * 168 / t / 1e9}
    del a, b, c
    out["fp2_mont_mul_2^24"] = measure_fp2_micro(gm, wl, dev, imad_peak)
    # G2 2^18
    n2 = 1 << G2_LOG2N
    sc2 = wl.make_scalars(n2, seed=43, one_frac=0.0)
    logs2 = wl.make_base_logs(n2, seed=4343)
    sc2_d = torch.from_numpy(sc2.view(np.int64)).to(dev)
    pts2 = gm.generator_mul_batch(torch.from_numpy(logs2.view(np.int64)).to(dev), group=2)
    o2 = torch.empty(gm.G2P_WORDS, dtype=torch.int64, device=dev)
    gm.msm_device(pts2, sc2_d, group=2, out=o2)
    torch.cuda.synchronize()
    gm.profile_enable(True)
    e0.record()
    reps = 3
    for _ in range(reps):
        gm.msm_device(pts2, sc2_d, group=2, out=o2)
    e1.record()
    torch.cuda.synchronize()
    phases2 = gm.profile_collect()
    gm.profile_enable(False)
    t2 = e0.elapsed_time(e1) / reps / 1e3
    ops2 = wl.msm_roofline_imad(n2, 2)
    acc2 = {}
    for name, v in phases2:
        if name != "start":
            acc2.setdefault(name, []).append(v)
    # the same MSMs round-robin over PIPELINE_STREAMS streams
    main = torch.cuda.current_stream()
    side = [torch.cuda.Stream() for _ in range(PIPELINE_STREAMS)]
    o2s = [torch.empty(gm.G2P_WORDS, dtype=torch.int64, device=dev) for _ in range(PIPELINE_STREAMS)]
    preps = 2 * PIPELINE_STREAMS
    for timed in (False, True):
        e0.record(main)
        for st in side:
            st.wait_stream(main)
        for i in range(preps):
            gm.msm_device(pts2, sc2_d, group=2, out=o2s[i % PIPELINE_STREAMS], stream=side[i % PIPELINE_STREAMS])
        for st in side:
            main.wait_stream(st)
        e1.record(main)
        torch.cuda.synchronize()
    t2p = e0.elapsed_time(e1) / preps / 1e3
    want2 = gm.canonical_affine(gm.to_numpy_proj(o2, 2), 2)
    pipe_ok = all(np.array_equal(gm.canonical_affine(gm.to_numpy_proj(o, 2), 2), want2) for o in o2s)
    out["g2_msm_2^18"] = {"points_per_s": n2 / t2, "ms": t2 * 1e3, "imad_frac": ops2 / t2 / imad_peak,
                          "window_bits": gm.default_window(2, n2, 5),
                          "phases_ms": {k: statistics.mean(v) for k, v in acc2.items()},
                          "pipelined": {"streams": PIPELINE_STREAMS, "ms_per_msm": t2p * 1e3,
                                        "points_per_s": n2 / t2p, "results_equal": bool(pipe_ok)}}
    del pts2, sc2_d
    out["batched_512"] = measure_batched(gm, wl, dev)
    out["serving"] = measure_serving(gm, wl, dev)
    return out


def relation_points(gm, dev, logs_list, group):
    """(s mod r) * G for every s, standard-form canonical affine (numpy), from
    the library's fixed-base generator kernel: a sum of the precomputed
    2^j * G over the set bits of s, which shares no code with the Pippenger
    pipeline under test."""
    import torch

    from gpu_msm_b200 import workload as wl
    if not logs_list:
        return []
    lim = np.stack([wl.int_to_limbs(s, 5) for s in logs_list]).view(np.int64)
    pts = gm.generator_mul_batch(torch.from_numpy(lim).to(dev), group=group)
    aff = gm.to_numpy_points(pts, group)
    return list(gm.from_montgomery(aff, group))


def same_affine(gm, proj, want, group):
    """proj (one projective point, Montgomery) equals want (standard affine)."""
    got = gm.canonical_affine(np.asarray(proj).reshape(1), group)[0]
    return bool(got["infinity"] == want["infinity"] and np.array_equal(got["x"], want["x"])
                and np.array_equal(got["y"], want["y"]))


def check_outputs(gm, dev, outputs, groups, logs_list):
    """Every output against the exact relation MSM = (sum_i k_i t_i mod r) * G
    (the synthetic bases are P_i = t_i * G).  Returns (equal, checked)."""
    want = [None] * len(outputs)
    for g in (1, 2):
        idx = [i for i in range(len(outputs)) if int(groups[i]) == g]
        for i, w in zip(idx, relation_points(gm, dev, [logs_list[i] for i in idx], g)):
            want[i] = w
    ok = sum(same_affine(gm, outputs[i], want[i], int(groups[i])) for i in range(len(outputs)))
    return int(ok), len(outputs)


def measure_serving(gm, wl, dev, loads=(0.5, 1.0, 2.0, 4.0, 8.0), count=1000):
    """Resident tables of 2^20 G1 and 2^18 G2 points carrying fixed-base window
    tables; Poisson arrivals at offered loads relative to the measured
    capacity of plain launches on the SAME tables, 70% G1 / 30% G2, prefix
    lengths floor(2^U) with U ~ U[10, 20] (G1) and U[10, 18] (G2; capped by
    its table), each request with its own scalars.  The same trace is served
    by the continuous-batching server and by plain launches one request at a
    time over the same tables, so the difference is batching and overlap
    alone.  Throughput and p50/p99 latency for both; every result of both arms
    is checked against the exact relation."""
    import torch

    from gpu_msm_b200 import serving
    tables, bare, log_tabs, build_s = {}, {}, {}, 0.0
    for g, log2n, seed in ((1, 20, 8181), (2, 18, 8282)):
        logs = wl.make_base_logs(1 << log2n, seed=seed)
        log_tabs[g] = wl.limbs16(logs)
        pts = gm.generator_mul_batch(torch.from_numpy(logs.view(np.int64)).to(dev), group=g)
        tables[g] = gm.ResidentBases(pts, group=g)
        bare[g] = gm.ResidentBases(pts, group=g)   # no window tables: context only
        t0 = time.perf_counter()
        for c in PRECOMPUTE_SERVE[g]:
            tables[g].precompute(c)
        build_s += time.perf_counter() - t0
        del pts
    pool = wl.make_scalars(1 << 21, seed=8383)
    pool16 = wl.limbs16(pool)
    ranges = {1: (10, 20), 2: (10, 18)}

    def trace(n_req, rate, seed):
        t, g, sizes = serving.poisson_trace(n_req, rate, seed, log2_range=ranges)
        rng = np.random.default_rng(seed)
        starts = [int(rng.integers(0, len(pool) - n)) for n in sizes]
        scs = [pool[s0:s0 + n] for s0, n in zip(starts, sizes)]
        logs = [wl.dot_log(pool16[s0:s0 + n], log_tabs[int(gg)][:n]) for s0, n, gg in zip(starts, sizes, g)]
        return t, g, sizes, scs, logs

    # plain capacity: back-to-back requests of the mix, same tables (and,
    # for context, on tables without fixed-base window tables)
    t, g, sizes, scs, _ = trace(64, 1e9, 1)
    serving.plain_trace(tables, np.zeros(8), g[:8], scs[:8], dev)
    _, _, span = serving.plain_trace(tables, np.zeros(64), g, scs, dev)
    capacity = 64 / span
    _, _, span_b = serving.plain_trace(bare, np.zeros(64), g, scs, dev)
    res = {"plain_capacity_req_s": capacity, "plain_capacity_points_per_s": float(sizes.sum()) / span,
           "plain_no_window_tables_capacity_req_s": 64 / span_b, "requests_per_load": count,
           "window_tables": {f"g{g}": list(v) for g, v in PRECOMPUTE_SERVE.items()}, "table_build_s": build_s,
           "check": "every result of both arms against (sum k_i t_i mod r) * G", "loads": []}
    for k, load in enumerate(loads):
        rate = load * capacity
        t, g, sizes, scs, logs = trace(count, rate, 100 + k)
        server = serving.MsmServer(tables, max_batch=64, max_points=1 << 22, slots=2).start()
        reqs, span_s = serving.serve_trace(server, t, g, scs)
        server.stop()
        lat_p, outs_p, span_p = serving.plain_trace(tables, t, g, scs, dev)
        pts = int(sizes.sum())
        ok_s, n_s = check_outputs(gm, dev, [r.result for r in reqs], g, logs)
        ok_p, n_p = check_outputs(gm, dev, [gm.to_numpy_proj(o, int(gg)) for o, gg in zip(outs_p, g)], g, logs)
        batch_sizes = [b[2] for b in server.batches]
        res["loads"].append({
            "offered_load": load, "rate_req_s": rate, "points": pts,
            "served": {"points_per_s": pts / span_s, **serving.percentiles([r.latency for r in reqs]),
                       "batches": len(batch_sizes), "mean_batch": float(np.mean(batch_sizes)),
                       "max_batch": int(max(batch_sizes))},
            "plain": {"points_per_s": pts / span_p, **serving.percentiles(lat_p)},
            "served_over_plain": span_p / span_s,
            "all_outputs_equal": bool(ok_s == n_s and ok_p == n_p), "checked": f"{ok_s}/{n_s} + {ok_p}/{n_p}"})
    top = max(res["loads"], key=lambda r: r["served"]["points_per_s"])
    res["served_capacity_points_per_s"] = top["served"]["points_per_s"]
    res["served_capacity_over_plain"] = top["served"]["points_per_s"] / res["plain_capacity_points_per_s"]
    for tb in list(tables.values()) + list(bare.values()):
        tb.close()
    return res


def measure_batched(gm, wl, dev, count=512, table_log2=16):
    """512 independent G1 MSMs, sizes floor(2^U) with U ~ U[8, 16] (seeded),
    each over a prefix of one resident 2^16-point table with its own scalars:
    one batch plan (window widths per size class from the autotuner table)
    captured in a CUDA graph, against 512 sequential plain launches.  Every
    output of every arm is checked against the exact relation."""
    import torch
    n_table = 1 << table_log2
    logs = wl.make_base_logs(n_table, seed=7070)
    pts = gm.generator_mul_batch(torch.from_numpy(logs.view(np.int64)).to(dev), group=1)
    table = gm.ResidentBases(pts, group=1)
    sizes = wl.mixed_sizes(count, 8, 16, seed=7)
    total = int(sizes.sum())
    sc_h = wl.make_scalars(total, seed=7171)
    sc = torch.from_numpy(sc_h.view(np.int64)).to(dev)
    want_logs = wl.expected_logs(sizes, sc_h, logs)
    groups = np.ones(count, dtype=np.int64)

    def check(out_t):
        ok, n = check_outputs(gm, dev, list(gm.to_numpy_proj(out_t, 1)), groups, want_logs)
        return {"all_outputs_equal": ok == n, "checked": f"{ok}/{n}"}

    plan = gm.BatchPlan(table, sizes)
    out = torch.empty((count, gm.G1P_WORDS), dtype=torch.int64, device=dev)
    t_batch = time_graph(plan, sc, out)
    out_class = torch.empty_like(out)
    t_class = time_graph(plan.set_queue(False), sc, out_class)
    # sequential plain launches over the same slices
    rows = np.concatenate([[0], np.cumsum(sizes)])
    seq_out = torch.empty((count, gm.G1P_WORDS), dtype=torch.int64, device=dev)
    for i in range(4):
        table.msm(sc[rows[i]:rows[i + 1]], offset=0, out=seq_out[i])
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for i in range(count):
        table.msm(sc[rows[i]:rows[i + 1]], offset=0, window_bits=gm.tuned_window(1, int(sizes[i])), out=seq_out[i])
    e1.record()
    torch.cuda.synchronize()
    t_seq = e0.elapsed_time(e1) / 1e3
    res = {"count": count, "points": total, "classes": plan.classes(),
           "batched_points_per_s": total / t_batch, "batched_ms": t_batch * 1e3,
           "sequential_points_per_s": total / t_seq, "sequential_ms": t_seq * 1e3,
           "speedup": t_seq / t_batch, "graph": "cuda graph replay",
           "batched_check": check(out), "sequential_check": check(seq_out),
           "mode": "every class's accumulation in one persistent launch over a device work queue",
           "per_class_pipelines": {"batched_points_per_s": total / t_class, "batched_ms": t_class * 1e3,
                                   "speedup_vs_sequential": t_seq / t_class, "check": check(out_class)}}
    plan.close()
    # the same batch over fixed-base window tables of the resident set
    t0 = time.perf_counter()
    for c in PRECOMPUTE_BATCH:
        table.precompute(c)
    t_pre = time.perf_counter() - t0
    plan = gm.BatchPlan(table, sizes)
    out_pc = torch.empty_like(out)
    t_pc = time_graph(plan, sc, out_pc)
    out_pclass = torch.empty_like(out)
    t_pclass = time_graph(plan.set_queue(False), sc, out_pclass)
    res["precomputed"] = {"windows": list(PRECOMPUTE_BATCH), "classes": plan.classes(),
                          "build_s": t_pre, "batched_points_per_s": total / t_pc, "batched_ms": t_pc * 1e3,
                          "speedup_vs_sequential": t_seq / t_pc, "check": check(out_pc),
                          "per_class_pipelines": {"batched_points_per_s": total / t_pclass, "batched_ms": t_pclass * 1e3,
                                                  "speedup_vs_sequential": t_seq / t_pclass, "check": check(out_pclass)}}
    plan.close()
    table.close()
    return res


def time_graph(plan, sc, out, reps=5):
    """Capture plan.run in a CUDA graph and time its replays (seconds)."""
    import torch
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        plan.run(sc, out=out)
    torch.cuda.current_stream().wait_stream(s)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        plan.run(sc, out=out)
    g.replay()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        g.replay()
    e1.record()
    torch.cuda.synchronize()
    del g
    return e0.elapsed_time(e1) / reps / 1e3


def main():
    args = parse()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank, world)
        return
    if args.msm_only:
        run_msm_only(args)
        return
    if world > 1:
        import datetime

        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    try:
        run_ours(args, rank, world, local_rank)
    finally:
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()


if __name__ == "__main__":
    main()
