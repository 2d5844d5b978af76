"""Benchmark: FP64 SpGEMM GFLOPS (2 * nnzCub / time) of C = A*A on the
3D 27-point stencil 96^3 (the workload whose HBM-roofline target the
project is measured on), through the library's C ABI.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--workload st27-96|st27-<side>|lap256|rmat<s>-aat|batched|served]
                    [--cpu-seconds S] [--no-e2e] [--no-extras]

One step = one full SpGEMM: CSR A in device memory -> tile conversion ->
step 1 -> step 2 -> numeric -> CSR C in device memory (C is freed after the
step, back into the context's pool).  `value` is timed with CUDA events on
the library's stream; `e2e` repeats the step through the same C ABI with
host operands (pinned) and a host C, the copies inside the timed region.
Under torchrun each rank runs its own replica of the workload (weak scaling)
and rank 0 prints one JSON line with the max time over ranks.

The default line (st27-96, one GPU) also carries the benchmark's other
workloads, each run in a child process after the headline's timing:
`configs` (2D Laplacian 256^2 A*A and R-MAT 2^20 A*A^T, device-resident),
`batched` (4,096 instances in waves, against one call per instance and
numeric-only graph replays) and `served` (the Poisson stream at 2,000
requests/s offered, then at 0.5x and 0.9x of the measured capacity, with
the host link's share of wall time).  `--no-extras` leaves them out.

--impl reference times the reference's own CPU algorithm for the path
(thmkl_dcsrmultcsr, restated in oracle/tsg_oracle.c) on the host cores, on a
bounded sample of rows of the same workload per step.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "FP64 SpGEMM GFLOPS (2*nnzCub/s)"
UNIT = "GFLOP/s"


def make_workload(name: str):
    from tilespgemm_gb300 import matrices as M
    if name == "st27-96":
        return M.stencil_27(96, seed=1), "AA", ("3D 27-point stencil 96^3 (n=884,736), values U[0.5,1.5], "
                                                 "diagonal = row sum, C = A*A")
    if name.startswith("st27-") and name[5:].isdigit() and name != "st27-96":
        side = int(name[5:])
        return M.stencil_27(side, seed=1), "AA", f"3D 27-point stencil {side}^3, values U[0.5,1.5], diagonal = row sum, C = A*A"
    if name == "lap256":
        return M.laplacian_2d(256), "AA", "2D 5-point Laplacian 256x256 (n=65,536), diag 4, off -1, C = A*A"
    if name.startswith("rmat") and name.endswith("-aat") and name[4:-4].isdigit():
        scale = int(name[4:-4])
        return (M.rmat(scale, 16, seed=1), "AAT",
                f"R-MAT 2^{scale} x 16/row (0.57,0.19,0.19,0.05), duplicates merged, values U[-1,1], C = A*A^T")
    raise SystemExit(f"unknown workload {name}")


def operand_b(A, op):
    if op == "AA":
        return A
    from tilespgemm_gb300 import matrices as M
    return M.transpose(A)


def nnzcub(A, B) -> int:
    rp = np.asarray(B.rowptr, np.int64)
    lens = rp[1:] - rp[:-1]
    return int(lens[np.asarray(A.col)].sum())


def algorithmic_bytes(A, B, nnz_c: int) -> dict:
    """Compulsory traffic with int32 indices and FP64 values; B counted even
    when it aliases A; C's row pointer 4 bytes when nnzC < 2^31, else 8."""
    a = 4 * (A.m + 1) + 12 * A.nnz
    b = 4 * (B.m + 1) + 12 * B.nnz
    c = (4 if nnz_c < 2 ** 31 else 8) * (A.m + 1) + 12 * nnz_c
    # the numeric step reads A and B and writes C's columns and values
    return {"total": a + b + c, "numeric": a + b + 12 * nnz_c}


def load_peaks() -> dict:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return json.loads(p.read_text())
        except Exception:
            pass
    return {}


def load_traffic(workload: str):
    p = ROOT / "profiles" / "traffic.json"
    if p.exists():
        try:
            return json.loads(p.read_text()).get(workload)
        except Exception:
            return None
    return None


class ClockSampler:
    """nvidia-smi sampling during the timed region (clocks and throttle reasons)."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.proc = None
        self.f = None

    def __enter__(self):
        try:
            self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "20"],
                                         stdout=self.f, stderr=subprocess.DEVNULL)
            # nvidia-smi takes a while to start: wait (2 s at most) for its
            # first sample, so that short timed regions are sampled too
            t0 = time.perf_counter()
            while time.perf_counter() - t0 < 2.0 and self.proc.poll() is None and os.path.getsize(self.f.name) == 0:
                time.sleep(0.01)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self) -> dict:
        if self.proc is None or self.f is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.f.flush()
        rows = []
        for line in Path(self.f.name).read_text().splitlines():
            parts = [x.strip() for x in line.split(",")]
            if len(parts) >= 9:
                rows.append(parts)
        os.unlink(self.f.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"], "samples": 0}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        reasons = set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            for nm, v in zip(names, r[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(rows)}


def cpu_thmkl_sample(A, B, seconds: float) -> dict:
    """The reference CPU algorithm (thmkl_dcsrmultcsr restated, all host
    threads) on a contiguous block of rows from the middle of the matrix,
    grown until it takes about `seconds`."""
    from oracle import oracle as O
    rp = np.asarray(A.rowptr, np.int64)
    brp = np.asarray(B.rowptr, np.int64)
    blen = brp[1:] - brp[:-1]
    mid = A.m // 2
    rows = 32
    while True:
        r0 = max(0, mid - rows // 2)
        r1 = min(A.m, r0 + rows)
        t0 = time.perf_counter()
        O.thmkl_rows(A, B, r0, r1)
        dt = time.perf_counter() - t0
        if dt >= seconds * 0.5 or r1 - r0 >= A.m:
            break
        rows = int(rows * min(8.0, max(2.0, seconds * 0.6 / max(dt, 1e-3))))
    cub = int(blen[np.asarray(A.col)[rp[r0]:rp[r1]]].sum())
    return {"value": 2.0 * cub / dt / 1e9, "unit": UNIT, "cores": O.max_threads(), "kind": "port",
            "sample": f"rows [{r0},{r1}) of {A.m} ({r1 - r0} rows, {cub} intermediate products, {dt:.2f} s), "
                      "symbolic + numeric as in thmkl_dcsrmultcsr.c:190-210",
            "seconds": dt, "rows": r1 - r0, "r0": r0}


def run_reference(args) -> None:
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    A, op, desc = make_workload(args.workload)
    B = operand_b(A, op)
    from oracle import oracle as O
    cal = cpu_thmkl_sample(A, B, min(args.cpu_seconds, 4.0))
    r0, r1 = cal["r0"], cal["r0"] + cal["rows"]
    rp = np.asarray(A.rowptr, np.int64)
    blen = np.diff(np.asarray(B.rowptr, np.int64))
    cub = int(blen[np.asarray(A.col)[rp[r0]:rp[r1]]].sum())
    for _ in range(args.warmup):
        O.thmkl_rows(A, B, r0, r1)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        O.thmkl_rows(A, B, r0, r1)
    dt = (time.perf_counter() - t0) / args.steps
    val = 2.0 * cub / dt / 1e9
    out = {
        "impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": f"{args.workload}: {desc}", "sample_rows": [r0, r1], "nnz_cub_sample": cub},
        "cpu_baseline": {"value": val, "unit": UNIT, "cores": O.max_threads(), "kind": "port",
                         "sample": cal["sample"]},
        "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(out))


def max_over_ranks(x: float, dist, device: str = "cuda") -> float:
    """The largest x over the ranks of the job (x itself with one rank):
    the whole job takes as long as its slowest replica."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_gflops(world: int, cub_per_rank: int, ms: float) -> float:
    """GFLOPS of the job: every rank does 2 * cub_per_rank flops in ms
    (the slowest rank's time)."""
    return world * 2.0 * cub_per_rank / (ms * 1e6)


def measure_e2e(args, ctx, A, op, stream, nnz_c, barrier, dist):
    """The same SpGEMM through the C ABI with host operands (pinned) and a
    host C: the copies both ways are inside the timed region.  Returns
    (ms per step, H2D bytes per step, D2H bytes per step)."""
    import torch
    from tilespgemm_gb300.api import CSR
    Ah = CSR(A.m, A.n, torch.from_numpy(np.asarray(A.rowptr, np.int32)).pin_memory(),
             torch.from_numpy(np.asarray(A.col, np.int32)).pin_memory(),
             torch.from_numpy(np.asarray(A.val, np.float64)).pin_memory())
    oc, _ = ctx.spgemm_raw(Ah, op=op, out="host")
    c_rowptr_bytes = 4 * (A.m + 1) if oc.rowptr_bits == 32 else 8 * (A.m + 1)
    oc.free()
    barrier()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        oc, _ = ctx.spgemm_raw(Ah, op=op, out="host")
        oc.free()
    e1.record(stream)
    e1.synchronize()
    barrier()
    ms_e2e = max_over_ranks(e0.elapsed_time(e1) / args.steps, dist)
    h2d = 4 * (A.m + 1) + 12 * A.nnz
    d2h = c_rowptr_bytes + 12 * nnz_c
    return ms_e2e, h2d, d2h


def cli_per_call(A, device: int, runs: int = 200) -> dict | None:
    """Per-call time through the plain-C command line (tilespgemm_gb300/_lib/tsg,
    the reference driver's interface over the C ABI): A resident on the
    device, C on the device, the minimum of `runs` calls by the host clock
    around each call -- the library's cost without the Python wrapper."""
    from tilespgemm_gb300 import build
    from tilespgemm_gb300.api import write_mtx
    if not build.CLI.exists():
        return None
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, "a.mtx")
        write_mtx(path, A, exact=True)
        res = subprocess.run([str(build.CLI), "-d", str(device), "--keep-values", "--repeat", str(runs),
                              "--csv", os.path.join(td, "r.csv"), path], capture_output=True, text=True, timeout=300)
    for line in res.stdout.splitlines():
        if "min of" in line and " ms," in line:
            ms = float(line.split("runs =")[1].split("ms")[0])
            return {"ms_min": ms, "runs": runs,
                    "via": "tsg CLI (plain C over the C ABI; A resident on the device, C on the device)"}
    return None


def run_ours(args) -> None:
    import torch
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl")
    torch.cuda.set_device(local)
    from tilespgemm_gb300 import Context
    from tilespgemm_gb300 import _abi
    from tilespgemm_gb300.api import CSR

    A, op, desc = make_workload(args.workload)
    B = operand_b(A, op)
    cub = nnzcub(A, B)
    ctx = Context(local, phase_times=1, count_products=0)   # nnzCub is counted on the host above
    lib = _abi.lib()
    stream = torch.cuda.ExternalStream(lib.tsg_get_stream(ctx.handle), device=torch.device("cuda", local))

    Ad = A.to_device(local)
    Ad.rowptr = Ad.rowptr.to(torch.int32)          # the reference's int row pointers
    for _ in range(args.warmup):
        t_call = time.perf_counter()
        oc, st = ctx.spgemm_raw(Ad, op=op, out="device", stats=True)
        oc.free()
        t_call = time.perf_counter() - t_call
    nnz_c = st["nnz_c"]
    every = t_call >= 1e-3   # per-step statistics cost next to nothing against the call

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    # ---- device-resident value ----
    phases = []
    barrier()
    l0 = lib.tsg_launch_count()
    with ClockSampler(local) as clk:
        ev0 = torch.cuda.Event(enable_timing=True)
        ev1 = torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for i in range(args.steps):   # calls under a millisecond: statistics of the last step only
            oc, st = ctx.spgemm_raw(Ad, op=op, out="device", stats=every or i == args.steps - 1)
            if st is not None:
                phases.append(st)
            oc.free()
        ev1.record(stream)
        ev1.synchronize()
    launches = lib.tsg_launch_count() - l0
    barrier()
    ms = max_over_ranks(ev0.elapsed_time(ev1) / args.steps, dist)
    value = whole_job_gflops(world, cub, ms)

    # ---- e2e through the ABI with host operands ----
    ms_e2e, h2d, d2h = None, 0, 0
    if not args.no_e2e:
        ms_e2e, h2d, d2h = measure_e2e(args, ctx, A, op, stream, nnz_c, barrier, dist)

    if rank != 0:
        ctx.close()
        if dist is not None:
            dist.destroy_process_group()
        return

    peaks = load_peaks()
    hbm_peak = peaks.get("hbm_gbs")
    import ctypes
    fp64 = ctypes.c_double(0.0)
    _abi.check(lib.tsg_measure_fp64_peak(ctx.handle, ctypes.byref(fp64)))
    # the small-product path has no phase events: its dominant kernel
    # (k_small_fill_one) is taken with the call's time and the call's bytes
    small = bool(phases[-1].get("small_path", 0))
    ab = algorithmic_bytes(A, B, nnz_c)
    ms_num = ms if small else statistics.mean(p["ms_step3"] for p in phases)
    kbytes = ab["total"] if small else ab["numeric"]
    achieved = kbytes / (ms_num * 1e6)
    traffic = None if small else load_traffic(args.workload)
    roofline = {
        "kernel": ("k_small_fill_one (small-product path, the whole call: count pass skipped on a repeated shape)"
                   if small else "k_numeric_smem (step 3: FP64 accumulation + CSR write)"),
        "bound": "hbm", "achieved": achieved, "peak": hbm_peak, "unit": "GB/s",
        "frac": (achieved / hbm_peak) if hbm_peak else None,
        "peak_source": "of measured (MEASURED_PEAKS.json hbm_gbs)" if hbm_peak else "of fallback 6800 GB/s",
        "traffic": traffic,
        "algorithmic_bytes_per_launch": kbytes, "ms_per_launch": ms_num,
        "fp64": {"achieved_gflops": 2.0 * cub / (ms_num * 1e6), "peak_gflops": fp64.value,
                 "frac": 2.0 * cub / (ms_num * 1e6) / fp64.value if fp64.value else None,
                 "peak_source": "measured live (tsg_measure_fp64_peak, DFMA-only kernel)"},
        "whole_step": {"achieved_gbs": ab["total"] / (ms * 1e6),
                       "frac": ab["total"] / (ms * 1e6) / hbm_peak if hbm_peak else None,
                       "algorithmic_bytes": ab["total"]},
    }
    if hbm_peak is None:
        roofline["peak"] = 6800.0
        roofline["frac"] = achieved / 6800.0
    cpu = None
    if world == 1 and not args.no_cpu_baseline:
        cpu = cpu_thmkl_sample(A, B, args.cpu_seconds)
        for k in ("seconds", "rows", "r0"):
            cpu.pop(k, None)
    mean = lambda k: statistics.mean(p[k] for p in phases)  # noqa: E731
    out = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded generator, shapes of the named workload)",
        "config": {"workload": f"{args.workload}: {desc}", "n": A.m, "nnz_a": A.nnz, "nnz_cub": cub,
                   "nnz_c": nnz_c, "tiles_a": phases[-1]["tiles_a"], "tiles_c": phases[-1]["tiles_c"],
                   "l2": "inputs larger than L2: A is %.0f MB and C %.0f MB against a 129 MB L2" % (
                       (12 * A.nnz + 4 * A.m) / 1e6, 12 * nnz_c / 1e6),
                   "parallelism": f"one replica per GPU ({world})"},
        "phases_ms": (None if small else
                      {"convert": mean("ms_convert"), "step1": mean("ms_step1"), "step2": mean("ms_step2"),
                       "step3": mean("ms_step3")}),
        "path": "small-product (row by row)" if small else "tiled",
        "host_waits_per_step": phases[-1]["n_syncs"],
        "roofline": roofline,
        "cpu_baseline": cpu,
        "e2e": ({"value": whole_job_gflops(world, cub, ms_e2e), "unit": UNIT, "ms_per_step": ms_e2e,
                 "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h} if ms_e2e is not None else None),
        "gpu_launches": int(launches),
        "gpu_launches_per_step": launches / args.steps,
        "clocks": clk.summary(),
    }
    if world == 1 and args.workload == "lap256":
        out["c_abi_per_call"] = cli_per_call(A, local)
    if out["e2e"] is not None:
        # the host link's share: the bytes each way at the link's measured
        # bandwidth, as if nothing overlapped them
        link = link_gbs()
        floor = h2d / (link["h2d"] * 1e6) + d2h / (link["d2h"] * 1e6)
        out["e2e"].update({"host_link_gbs": link, "link_floor_ms": floor, "beyond_link_floor_ms": ms_e2e - floor})
    ctx.close()
    if world == 1 and not args.no_extras and args.workload == "st27-96":
        out.update(sub_benchmarks(args))
    print(json.dumps(out))
    if dist is not None:
        dist.destroy_process_group()


def run_batched(args) -> None:
    """Batched instances/s (tsg_spgemm_batched, in waves) against the same
    instances computed one call at a time (tsg_spgemm), device operands and
    device results, CUDA events on the library's stream."""
    import torch
    from tilespgemm_gb300 import Context, _abi
    from tilespgemm_gb300 import matrices as M
    count, waves = args.batch_count, max(1, args.batch_waves)
    As = [M.batch_instance(i, seed=1) for i in range(count)]
    cub = sum(int(np.diff(np.asarray(A.rowptr))[np.asarray(A.col)].sum()) for A in As)
    Ad = [A.to_device(0) for A in As]
    ctx = Context(0)
    lib = _abi.lib()
    stream = torch.cuda.ExternalStream(lib.tsg_get_stream(ctx.handle), device=torch.device("cuda", 0))
    per = (count + waves - 1) // waves
    groups = [Ad[w * per:(w + 1) * per] for w in range(waves) if Ad[w * per:(w + 1) * per]]

    def batched_pass():
        nnz = 0
        for g in groups:
            outs, _ = ctx.spgemm_batched_raw(g, op="AA", out="device")
            nnz += sum(o.nnz for o in outs)
            for o in outs:
                o.free()
        return nnz

    def single_pass():
        for A in Ad:
            oc, _ = ctx.spgemm_raw(A, op="AA", out="device")
            oc.free()

    def timed(fn, reps):
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(reps):
            fn()
        e1.record(stream)
        e1.synchronize()
        return e0.elapsed_time(e1) / reps

    for _ in range(args.warmup):
        nnz_c = batched_pass()
    single_pass()
    l0 = lib.tsg_launch_count()
    with ClockSampler(0) as clk:
        ms_b = timed(batched_pass, args.steps)
    launches_b = (lib.tsg_launch_count() - l0) / args.steps
    ms_s = timed(single_pass, 1)
    # numeric-only repeats: one batched plan per wave (symbolic once, tuned),
    # then graph replays of the numeric step on resident values
    ms_r, launches_r = 0.0, 0
    tuned = []
    for grp in groups:
        plan = ctx.plan_batched(grp, op="AA")
        plan.tune()
        tuned.append(plan.settings())
        plan.replay()
        l0 = lib.tsg_launch_count()
        ms_r += timed(plan.replay, args.steps)
        launches_r += (lib.tsg_launch_count() - l0) // args.steps
        plan.close()
    out = {
        "metric": "batched SpGEMM instances/s", "value": count / (ms_b / 1e3), "unit": "instances/s",
        "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_b, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded, batched workload shapes)",
        "config": {"workload": f"batched: {count} x A*A, n log-uniform [64,16384], nnz/row U[2,64], "
                               f"banded (n/8) for even instances, uniform for odd", "waves": len(groups),
                   "nnz_a": int(sum(A.nnz for A in As)), "nnz_cub": cub, "nnz_c": int(nnz_c)},
        "one_at_a_time": {"instances_per_s": count / (ms_s / 1e3), "ms": ms_s},
        "speedup_vs_one_at_a_time": ms_s / ms_b,
        "numeric_replay": {"instances_per_s": count / (ms_r / 1e3), "ms": ms_r, "graph_kernels": launches_r,
                           "note": "same instances, new values: batched plan per wave, tuned, one CUDA graph each"},
        "tuned": tuned,
        "gflops_batched": 2.0 * cub / (ms_b * 1e6),
        "gpu_launches_per_step": launches_b,
        "clocks": clk.summary(),
    }
    print(json.dumps(out))
    ctx.close()


def link_gbs() -> dict:
    """Host-link bandwidth of this machine: the best of eight 2 GiB pinned copies
    each way, timed one by one with CUDA events (the link bounds every
    host-memory result; a mean would carry whatever else the host did)."""
    import torch
    n = 1 << 31
    h = torch.empty(n, dtype=torch.uint8).pin_memory()
    d = torch.empty(n, dtype=torch.uint8, device="cuda")
    out = {}
    for name, dst, src in (("h2d", d, h), ("d2h", h, d)):
        out[name] = 0.0
        for _ in range(9):                      # the first warms up
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            dst.copy_(src, non_blocking=True)
            e1.record()
            e1.synchronize()
            out[name] = max(out[name], n / (e0.elapsed_time(e1) * 1e6))
    del h, d
    return out


def run_served(args) -> None:
    """Served streams through tsg_server_*: p50/p99 latency and throughput.

    1. The configured stream (Poisson, 2,000 requests/s offered) after a
       warm-up on another realization: far above what the GPU and the host
       link complete, so its latencies are the time the backlog takes to
       drain; its completion rate is the capacity.
    2. Streams of the same kind offered at 0.5x and 0.9x of that capacity
       (other seeds and keys), where latency is per-request time, not
       backlog.
    For each: completed requests/s, p50/p99/mean latency, refusals, and the
    share of wall time the host link needed for the results (C's bytes at
    the measured device-to-host bandwidth)."""
    from tilespgemm_gb300.serving import Server, make_stream, run_stream
    procs = max(1, min(16, (os.cpu_count() or 1)))
    scale = (12, args.serve_max_scale)
    reqs = make_stream(args.serve_requests, seed=1, rate=args.serve_rate, rmat_scale=scale, procs=procs)
    warm = make_stream(max(16, args.serve_requests // 4), seed=2, rate=args.serve_rate, rmat_scale=scale,
                       procs=procs, key_base=1 << 40)
    n_sub = max(40, args.serve_requests // 3)
    sub = [make_stream(n_sub, seed=3 + j, rate=1.0, rmat_scale=scale, procs=procs, key_base=(2 + j) << 40)
           for j in range(2)]
    link = link_gbs()

    def summary(st, offered):
        done = [r for r in st["results"] if r is not None]
        lat = [r[1]["latency_ms"] for r in done]
        link_s = sum(12 * r[1]["nnz"] for r in done) / (link["d2h"] * 1e9)
        return {"offered_rps": offered, "requests": st["n"], "completed": st["completed"],
                "throughput_rps": st["throughput_rps"], "p50_ms": st["p50_ms"], "p99_ms": st["p99_ms"],
                "mean_ms": st["mean_ms"], "max_ms": float(max(lat)) if lat else None,
                "refused_over_budget": st["refused"], "numeric_only_requests": st["numeric_only"],
                "wall_s": st["wall_s"], "c_entries_returned": int(sum(r[1]["nnz"] for r in done)),
                "host_link_s": link_s, "host_link_frac_of_wall": link_s / st["wall_s"] if st["wall_s"] else None}

    with Server(workers=args.serve_workers, budget_gb=64.0) as srv:
        run_stream(srv, warm, realtime=False, download=False)
        with ClockSampler(0) as clk:
            st = run_stream(srv, reqs, realtime=True, download=False)
        top = summary(st, args.serve_rate)
        cap = top["throughput_rps"]
        below = []
        for frac, rq in zip((0.5, 0.9), sub):
            rate = frac * cap
            for r in rq:                 # the drawn stream re-timed: gaps scale as 1/rate
                r["t"] = r["t"] / rate
            with ClockSampler(0) as clk2:
                s2 = run_stream(srv, rq, realtime=True, download=False)
            d = summary(s2, rate)
            d["fraction_of_capacity"] = frac
            d["clocks"] = clk2.summary()
            below.append(d)
    out = {
        "metric": "served SpGEMM requests/s with p50/p99 latency", "value": top["throughput_rps"],
        "unit": "requests/s", "n_gpus": 1, "steps": 1, "warmup": 1, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded Poisson stream)",
        "config": {"workload": f"served: {len(reqs)} requests, Poisson {args.serve_rate:.0f}/s, 50/50 Laplacian "
                               f"(side 32-512) / R-MAT (2^12-2^{args.serve_max_scale}, 8-32/row), 50/50 A*A / A*A^T, "
                               "30% numeric-only repeats, 64 GB budget", "workers": args.serve_workers},
        **{k: v for k, v in top.items() if k != "offered_rps"},
        "note": "offered far above capacity: these latencies measure the backlog's drain; see below_capacity",
        "below_capacity": below,
        "host_link_gbs": link,
        "clocks": clk.summary(),
    }
    print(json.dumps(out))


def run_sub(args, workload: str, extra: list) -> dict:
    """One more workload in a child process (its memory -- R-MAT 2^20's
    116 GB C, the served stream's pinned buffers -- goes with it): its JSON
    line, or the reason it has none."""
    cmd = [sys.executable, str(ROOT / "bench.py"), "--workload", workload, "--no-cpu-baseline", "--no-e2e",
           "--no-extras", *extra]
    t0 = time.perf_counter()
    try:
        res = subprocess.run(cmd, capture_output=True, text=True, timeout=args.sub_timeout)
    except subprocess.TimeoutExpired:
        return {"workload": workload, "error": f"timed out after {args.sub_timeout} s"}
    lines = [x for x in res.stdout.splitlines() if x.startswith("{")]
    if res.returncode != 0 or not lines:
        return {"workload": workload, "error": f"exit {res.returncode}: {res.stderr.strip()[-400:]}"}
    d = json.loads(lines[-1])
    d.setdefault("wall_s", time.perf_counter() - t0)
    return d


def sub_benchmarks(args) -> dict:
    """The benchmark's other workloads, each measured on its own (device-
    resident operands and results, CUDA events, their own clock records),
    reported beside the headline and outside its timing."""
    out = {"configs": {}}
    for w, steps in (("lap256", 20), ("rmat20-aat", 3)):
        d = run_sub(args, w, ["--steps", str(steps), "--warmup", "3"])
        if "error" in d:
            out["configs"][w] = d
            continue
        out["configs"][w] = {"workload": d["config"]["workload"], "value": d["value"], "unit": d["unit"],
                             "ms_per_step": d["ms_per_step"], "path": d.get("path"),
                             "c_abi_per_call": d.get("c_abi_per_call"), "phases_ms": d["phases_ms"],
                             "nnz_a": d["config"]["nnz_a"], "nnz_cub": d["config"]["nnz_cub"],
                             "nnz_c": d["config"]["nnz_c"], "host_waits_per_step": d["host_waits_per_step"],
                             "gpu_launches_per_step": d["gpu_launches_per_step"],
                             "whole_step_hbm_frac": d["roofline"]["whole_step"]["frac"],
                             "numeric_fp64_frac": d["roofline"]["fp64"]["frac"], "clocks": d["clocks"]}
    b = run_sub(args, "batched", ["--steps", "5", "--warmup", "3"])
    out["batched"] = b if "error" in b else {k: b[k] for k in (
        "metric", "value", "unit", "ms_per_step", "config", "one_at_a_time", "speedup_vs_one_at_a_time",
        "numeric_replay", "gflops_batched", "gpu_launches_per_step", "tuned", "clocks") if k in b}
    s_ = run_sub(args, "served", [])
    out["served"] = s_ if "error" in s_ else {k: v for k, v in s_.items() if k not in (
        "n_gpus", "steps", "warmup", "higher_is_better", "scaling", "vs_baseline", "dtype", "data")}
    return out


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--workload", default="st27-96")
    ap.add_argument("--cpu-seconds", type=float, default=10.0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true", help="skip the host-operand leg (C of R-MAT 2^20 is 116 GB)")
    ap.add_argument("--no-extras", action="store_true",
                    help="leave the other workloads (lap256, rmat20-aat, batched, served) out of the headline line")
    ap.add_argument("--sub-timeout", type=float, default=600.0)
    ap.add_argument("--batch-count", type=int, default=4096)
    ap.add_argument("--batch-waves", type=int, default=8)
    ap.add_argument("--serve-requests", type=int, default=400)
    ap.add_argument("--serve-rate", type=float, default=2000.0)
    ap.add_argument("--serve-max-scale", type=int, default=18)
    ap.add_argument("--serve-workers", type=int, default=4)
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference(args)
    elif args.workload == "batched":
        run_batched(args)
    elif args.workload == "served":
        run_served(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
