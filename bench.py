#!/usr/bin/env python
"""bench.py -- DDA solve throughput on B200.

Workload (the reference README's GPU-scale case): box 10 x 5 x 5 um, grid
unit 0.1 um (100 x 50 x 50 = 250 000 dipoles, FFT grid 200 x 100 x 100),
refractive index 1.5+0.1i, wavelength 6 um, incidence (0,1,0), LDR couple
constants, BiCGStab to relative residual 1e-5, both polarisations.  One step
is one solve of both polarisations; the metric is solves per second.

  python bench.py [--gpus N --steps K --warmup W] [--impl reference]

Every GPU (one process each under torchrun) solves its own copy: the solves
are independent ("replicas only"), so `value` is the total solves of all
ranks over the slowest rank's device time.
"""
import argparse
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = {
    "workload": "box 10x5x5um d=0.1um m=1.5+0.1i lambda=6um prop=(0,1,0) ldr bicgstab eps=1e-5, both pols",
    "nv": 250000, "grid": [200, 100, 100], "rhs_per_step": 2,
}
EPS = 1e-5
PROP = (0.0, 1.0, 0.0)
METRIC = "solves/s at relative residual 1e-5 (box 10x5x5um, BiCGStab)"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--precision", default="fp32", choices=["fp32", "fp64", "mixed"])
    ap.add_argument("--solver", default="bicgstab")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline sample")
    ap.add_argument("--workload", default="box", choices=["box", "batched", "mixed512", "serve"],
                    help="box: the default line; batched: 128-rhs spheroid; mixed512: 512^3 sphere "
                         "with FP64 refinement; serve: Poisson request stream")
    ap.add_argument("--requests", type=int, default=120, help="serve: requests in the stream")
    ap.add_argument("--rate", type=float, default=50.0, help="serve: mean arrivals per second")
    ap.add_argument("--slots", type=int, default=8, help="serve: concurrent requests")
    ap.add_argument("--no-plain", action="store_true",
                    help="serve: skip the FP64 and straightforward-solve samples of the stream")
    ap.add_argument("--max-iter", type=int, default=0, help="mixed512: iteration cap of each solve (0: none)")
    ap.add_argument("--no-batched", action="store_true",
                    help="default line without the 128-rhs spheroid block beside it")
    ap.add_argument("--matvec-only", type=int, default=0,
                    help="run this many matvecs of the workload and exit (for ncu captures)")
    ap.add_argument("--rhs", type=int, default=0, help="--matvec-only: right-hand sides (0: the workload's)")
    ap.add_argument("--solve-only", type=int, default=0,
                    help="run this many solves of the default workload and exit (for ncu launch lists)")
    return ap.parse_args()


# DRAM traffic of one matvec's y/z passes (dram__bytes_read.sum +
# dram__bytes_write.sum of k_zfwd, k_rows and k_zinv, L2 as the launch before
# left it), from ncu captures of `bench.py --matvec-only`:
#   box:       the default workload, FP32, 2 rhs (the work buffer stays in L2 in
#              part)
#   spheroid:  the 128-rhs block's kernels captured at 8 and 16 rhs: a fixed part
#              (D octant, tables) and a part per rhs
# Summaries with the commands: profiles/yz_passes_box10x5x5_fp32.md,
# profiles/yz_passes_spheroid_fp32.md.
TRAFFIC = {"box": {"fixed": 75313408, "per_rhs": 0, "rhs": 2},
           "spheroid": {"fixed": 23286272, "per_rhs": 197693056}}


def yz_traffic(workload, nrhs):
    t = TRAFFIC.get(workload)
    if t is None or ("rhs" in t and t["rhs"] != nrhs):
        return None
    return int(t["fixed"] + nrhs * t["per_rhs"])


def dist_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("LOCAL_RANK", 0)), \
        int(os.environ.get("WORLD_SIZE", 1))


def max_over_ranks(dist, value, device):
    """The slowest rank's time (every rank calls it, in the same order)."""
    if dist is None:
        return value
    import torch
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_throughput(units_per_rank, world, t_max_ms):
    """Whole-job units per second: every rank does the same work; the job ends
    with the slowest rank."""
    return units_per_rank * world / (t_max_ms / 1000.0)


# ------------------------------------------------------------ clocks ----
class ClockSampler:
    """SM clocks and throttle reasons during the timed region: NVML queries
    taken between timed steps (sample()), plus nvidia-smi polling every
    200 ms as a second source when the region is long enough."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    # NVML clocks-event reason bits (nvml.h): sw power cap 0x4, hw slowdown
    # 0x8, sw thermal 0x20, hw thermal 0x40
    BITS = {"sw_power_cap": 0x4, "hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40}

    def __init__(self, gpu_index):
        self.idx = gpu_index
        self.proc = None
        self.f = None
        self.nv = None
        self.sm, self.mx, self.reasons = [], [], set()

    def start(self):
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nv = (pynvml, pynvml.nvmlDeviceGetHandleByIndex(self.idx))
        except Exception:
            self.nv = None
        try:
            self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.idx), "--query-gpu=" + self.FIELDS,
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def sample(self):
        if self.nv is None:
            return
        nv, h = self.nv
        try:
            self.sm.append(float(nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)))
            self.mx.append(float(nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM)))
            bits = nv.nvmlDeviceGetCurrentClocksEventReasons(h)
            for name, b in self.BITS.items():
                if bits & b:
                    self.reasons.add(name)
        except Exception:
            pass

    def stop(self):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(5)
            except Exception:
                self.proc.kill()
            self.f.flush()
            self.f.seek(0)
            rows = [r.split(",") for r in self.f.read().strip().splitlines() if r.strip()]
            os.unlink(self.f.name)
            names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
            for r in rows:
                try:
                    self.sm.append(float(r[1]))
                    self.mx.append(float(r[2]))
                    for n, v in zip(names, r[5:9]):
                        if v.strip().lower() == "active":
                            self.reasons.add(n)
                except (ValueError, IndexError):
                    pass
        if self.nv is not None:
            try:
                self.nv[0].nvmlShutdown()
            except Exception:
                pass
        if not self.sm:
            return None
        return {"sm_mhz": float(np.median(self.sm)), "sm_max_mhz": float(max(self.mx)),
                "reasons": sorted(self.reasons), "samples": len(self.sm)}


# --------------------------------------------------------- CPU sample ----
def cpu_model():
    try:
        for line in open("/proc/cpuinfo"):
            if line.startswith("model name"):
                return line.split(":", 1)[1].strip()
    except OSError:
        pass
    return None


class CpuArm:
    """The oracle (the C++ restatement of the reference's --cpu path,
    MatVecCpu + BicgStab) on this workload: D matrix built once, then full
    solves to relative residual 1e-5, timed with the host clock.  precision
    "fp32" is the reference's --ftype float path (D, matvec, vectors and
    scalars in float), "fp64" its --ftype double path."""

    def __init__(self, threads=None, precision="fp32"):
        self.precision = precision
        from oracle import oracle as O
        self.O = O
        if threads:
            O.set_threads(threads)
        self.threads = O.max_threads()
        g = O.Geometry.box("10um", "5um", "5um", "0.1um")
        self.p = O.Problem(g, [1.5 + 0.1j], "6um")
        t0 = time.perf_counter()
        self.p.build_dmatrix()
        self.setup_s = time.perf_counter() - t0
        self.einc = {}
        for pol in (1, 2):
            self.p.set_cc(PROP, pol, "ldr")
            self.einc[pol] = self.p.einc(PROP, pol)

    def solve(self, pol):
        """One full solve of polarisation `pol`: (seconds, iterations)."""
        self.p.set_cc(PROP, pol, "ldr")
        t0 = time.perf_counter()
        rc, _, st, _ = self.p.solve(self.einc[pol], "bicgstab", EPS, precision=self.precision)
        dt = time.perf_counter() - t0
        if rc != 0:
            raise RuntimeError("oracle solve failed (%d)" % rc)
        return dt, int(st.iterations)


def cpu_sample(precision="fp32"):
    """The default line's CPU baseline: full solves of both polarisations on
    all host threads at the line's precision (and, for comparison, at the
    other one), then one full solve of polarisation 1 on one thread (the
    reference's --cpu path is single-threaded, LinAlg/FFTWPlan.cpp:82)."""
    arm = CpuArm(precision=precision)
    arm.solve(1)  # first use builds the float D matrix
    res = [arm.solve(pol) for pol in (1, 2)]
    secs = [r[0] for r in res]
    threads = arm.threads
    other = "fp64" if precision == "fp32" else "fp32"
    arm.precision = other
    res_o = [arm.solve(pol) for pol in (1, 2)]
    arm.precision = "fp64"
    arm.O.set_threads(1)
    t1, it1 = arm.solve(1)
    arm.O.set_threads(threads)
    arm.precision = precision
    return {"value": 2.0 / sum(secs), "unit": "solves/s", "cores": threads, "kind": "port",
            "precision": precision,
            "sample": "oracle BiCGStab (%s, the reference's --ftype %s CPU path), full solves of both "
                      "polarisations to 1e-5 (%.1f s; D matrix built beforehand)"
                      % (precision, "float" if precision == "fp32" else "double", sum(secs)),
            "seconds": secs, "iterations": [r[1] for r in res],
            other: {"value": 2.0 / sum(r[0] for r in res_o), "unit": "solves/s", "cores": threads,
                    "seconds": [r[0] for r in res_o], "iterations": [r[1] for r in res_o]},
            "single_thread": {"value": 1.0 / t1, "unit": "solves/s", "cores": 1, "seconds": t1,
                              "iterations": it1, "precision": "fp64",
                              "sample": "oracle BiCGStab, full solve of polarisation 1"},
            "nproc": os.cpu_count(), "cpu_model": cpu_model()}


# ----------------------------------------------------------- our arm ----
def build_problem(precision, max_rhs):
    import dda_b200
    g = dda_b200.Geometry.box_shape("10um", "5um", "5um", "0.1um")
    p = dda_b200.DDAParams(g, [1.5 + 0.1j], "6um")
    mv = dda_b200.CudaMatVec(p, precision, max_rhs=max_rhs)
    ein = []
    for r, pol in enumerate((1, 2)[:max_rhs]):
        mv.set_couple_constants(dda_b200.CoupleConstants(p, PROP, pol, "ldr"), rhs=r)
        ein.append(p.einc(PROP, pol))
    return p, mv, np.concatenate(ein)


def stage_names(mv):
    """The stages of a matvec: x forward, y/z (three kernels or a plane
    kernel), x inverse."""
    return ["x_forward", "yz_passes" if mv.passes else "yz_plane_kernel", "x_inverse"]


def stage_bytes(p, mv, nrhs, s):
    """Algorithmic bytes per matvec of its three stages."""
    gx, gy, gz = p.grid
    bx, by, bz = p.box
    nvs, nv = p.nvs, p.nv
    plane = gx * by * bz
    oct_ = (gx // 2 + 1) * (gy // 2 + 1) * (gz // 2 + 1)
    return dict(zip(stage_names(mv), (nrhs * s * (3 * nvs + 3 * plane) + 13 * nv,
                                      nrhs * s * 6 * plane + s * 6 * oct_,
                                      nrhs * s * (6 * nvs + 3 * plane) + 13 * nv)))


def run_ours(args):
    import torch
    import dda_b200
    rank, local, world = dist_env()
    torch.cuda.set_device(local)
    pg = None
    if world > 1:
        import torch.distributed as dist
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=300))
        pg = dist
    prec = args.precision
    nrhs = 2
    p, mv, einc = build_problem(prec, nrhs)
    solver = dda_b200.CudaSolver(mv, args.solver)
    cdt = torch.complex128 if prec == "fp64" else torch.complex64
    s_bytes = 16 if prec == "fp64" else 8
    einc_dev = torch.from_numpy(einc).to(cdt).cuda()
    pol_dev = torch.zeros_like(einc_dev)
    stream = torch.cuda.ExternalStream(mv.stream)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device="cuda")  # 256 MB > L2
    torch.cuda.synchronize()  # the library's stream does not wait for torch's

    def step():
        solver.get_pol_vec_device(einc_dev.data_ptr(), pol_dev.data_ptr(), nrhs, EPS)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    iters = [st.iterations for st in solver.last_stats]
    if pg:
        pg.barrier()
    torch.cuda.synchronize()
    sampler = ClockSampler(local)
    sampler.start()
    l0 = mv.launches
    total_ms = 0.0
    lat = []
    for _ in range(args.steps):
        with torch.cuda.stream(stream):
            flush.zero_()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
        step()
        e1.record(stream)
        e1.synchronize()
        lat.append(e0.elapsed_time(e1))
        total_ms += lat[-1]
        sampler.sample()
    launches = mv.launches - l0
    torch.cuda.synchronize()
    clocks = sampler.stop()
    t_max = max_over_ranks(pg, total_ms, "cuda")
    value = replica_throughput(nrhs * args.steps, world, t_max)
    ms_per_step = t_max / args.steps

    # e2e: host fields in, host polarisations out, both from / into pinned
    # host memory, in the line's precision: complex64 through dda_solve_f32
    # for FP32 (the vectors of the reference's --ftype float path), complex128
    # through dda_solve for FP64
    hdt = torch.complex64 if prec == "fp32" else torch.complex128
    einc_host = torch.empty(einc.size, dtype=hdt, pin_memory=True).numpy()
    einc_host[:] = einc.reshape(-1)
    pol_host = torch.empty(einc.size, dtype=hdt, pin_memory=True).numpy()
    e2e_ms = 0.0
    for _ in range(args.steps):
        with torch.cuda.stream(stream):
            flush.zero_()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
        solver.get_pol_vec(einc_host, EPS, history_cap=1, out=pol_host)
        e1.record(stream)
        e1.synchronize()
        e2e_ms += e0.elapsed_time(e1)
    e2e_ms = max_over_ranks(pg, e2e_ms, "cuda")
    e2e = {"value": replica_throughput(nrhs * args.steps, world, e2e_ms), "unit": "solves/s",
           "h2d_bytes_per_step": int(einc_host.nbytes), "d2h_bytes_per_step": int(einc_host.nbytes),
           "host_arrays": "complex64 (dda_solve_f32)" if prec == "fp32" else "complex128 (dda_solve)"}

    # matvec stage profile and roofline of the dominant stage
    ms = mv.profile(nrhs=nrhs, reps=20)
    sb = stage_bytes(p, mv, nrhs, s_bytes)
    names = stage_names(mv)
    dom = int(np.argmax(ms[:3]))
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    peak = float(peaks.get("hbm_gbs", 6650.0))
    achieved = sb[names[dom]] / (ms[dom] * 1e-3) / 1e9
    roofline = {"bound": "hbm", "kernel": names[dom], "achieved": achieved, "peak": peak,
                "unit": "GB/s", "frac": achieved / peak,
                "traffic": yz_traffic("box", nrhs) if (prec == "fp32" and names[dom] == "yz_passes") else None,
                "peak_source": "measured" if "hbm_gbs" in peaks else "fallback",
                "algorithmic_bytes_per_matvec": sb[names[dom]], "ms_per_matvec": float(ms[dom])}
    matvec = {"ms": float(ms[3]), "stages_ms": dict(zip(names, map(float, ms[:3]))),
              "GB_per_s": sum(sb.values()) / (ms[3] * 1e-3) / 1e9, "nrhs": nrhs}

    # FP64 single-rhs solves: the two polarisations one after the other
    plain = ours64 = None
    if rank == 0:
        p64, mv64, e64 = build_problem("fp64", 1)
        s64 = dda_b200.CudaSolver(mv64, args.solver)
        ein = [p64.einc(PROP, pol) for pol in (1, 2)]
        import dda_b200 as D

        def plain_step():
            for pol in (1, 2):
                mv64.set_couple_constants(D.CoupleConstants(p64, PROP, pol, "ldr"))
                s64.get_pol_vec(ein[pol - 1], EPS, history_cap=1)

        plain_step()
        st64 = torch.cuda.ExternalStream(mv64.stream)
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        a.record(st64)
        plain_step()
        b.record(st64)
        b.synchronize()
        ours64 = {"value": 2 / (a.elapsed_time(b) / 1000.0), "unit": "solves/s",
                  "iterations": [st.iterations for st in s64.last_stats],
                  "what": "this library's FP64 path, one rhs at a time"}
        # the straightforward restatement (cuFFT through torch, unfused vector
        # operations, host-side scalars): the "plain GPU solve" denominator
        import bench_plain
        solvers = [bench_plain.PlainSolver(mv64, p64, D.CoupleConstants(p64, PROP, pol, "ldr").cc_sqrt)
                   for pol in (1, 2)]
        for sp, e in zip(solvers, ein):  # warm-up (cuFFT plans)
            sp.solve(e, EPS)
        torch.cuda.synchronize()
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        a.record()
        its = [sp.solve(e, EPS)[1] for sp, e in zip(solvers, ein)]
        b.record()
        b.synchronize()
        plain = {"value": 2 / (a.elapsed_time(b) / 1000.0), "unit": "solves/s", "iterations": its,
                 "what": "straightforward FP64 restatement: cuFFT (torch.fft), unfused vector operations, "
                         "host-side scalars, one rhs at a time (bench_plain.py)"}
        del solvers
        mv64.close()

    # the 128-rhs spheroid block beside the box (rank 0, one GPU)
    batched = None
    if rank == 0 and world == 1 and not args.no_batched:
        import bench_workloads
        batched = bench_workloads.batched_block(3, 1, local, cpu=not args.no_cpu)
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        try:
            cpu = cpu_sample("fp64" if prec == "fp64" else "fp32")
        except Exception as ex:  # the CPU baseline is reported, never required
            cpu = {"value": None, "error": str(ex)}
    if rank == 0:
        line = {"metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "c64+f64" if prec != "fp64" else "c128",
                "data": "synthetic (the reference README geometry; generated in-process)",
                "config": dict(WORKLOAD, precision=prec, solver=args.solver,
                               parallelism="replicas x%d" % world),
                "iterations": iters, "l2": "flushed between steps (256 MB write)",
                "e2e": e2e, "gpu_launches": launches, "roofline": roofline, "matvec": matvec,
                "plain_fp64_single_rhs": plain, "ours_fp64_single_rhs": ours64,
                "speedup_vs_plain": value / plain["value"] if plain else None,
                "cpu_baseline": cpu, "clocks": clocks,
                "latency_ms": {"p50": float(np.percentile(lat, 50)), "p99": float(np.percentile(lat, 99)),
                               "per": "solve of both polarisations (one step)", "samples": len(lat)},
                "batched_spheroid_128rhs": batched}
        print(json.dumps(line), flush=True)
    if pg:
        pg.barrier()
        pg.destroy_process_group()


def run_reference(args):
    """The reference arm: the oracle on the host cores, all host threads, at
    the precision of our line; one step is one full solve of both
    polarisations, like a step of our arm."""
    rank, local, world = dist_env()
    if rank != 0:
        return
    prec = args.precision if args.precision in ("fp32", "fp64") else "fp64"
    arm = CpuArm(precision=prec)
    for _ in range(args.warmup):
        arm.solve(1)
        arm.solve(2)
    secs, its = [], []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        its.append([arm.solve(pol)[1] for pol in (1, 2)])
        secs.append(time.perf_counter() - t0)
    total = sum(secs)
    v = 2 * args.steps / total
    cpu = {"value": v, "unit": "solves/s", "cores": arm.threads, "kind": "port",
           "precision": prec,
           "sample": "oracle BiCGStab (the reference's --ftype %s CPU path), full solves of both "
                     "polarisations to 1e-5 per step, D matrix built once beforehand"
                     % ("float" if prec == "fp32" else "double"),
           "iterations": its[-1], "nproc": os.cpu_count(), "cpu_model": cpu_model()}
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "solves/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000.0 * total / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "c64" if prec == "fp32" else "c128",
            "data": "synthetic", "config": dict(WORKLOAD, precision=prec, solver="bicgstab",
                                                 parallelism="replicas x%d" % world),
            "iterations": its[-1], "cpu_baseline": cpu,
            "e2e": {"value": v, "unit": "solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def run_matvec_only(args):
    """Runs args.matvec_only matvecs of the workload's context (FP32 unless
    --precision says otherwise) and exits: the command ncu captures."""
    import torch
    import dda_b200
    torch.cuda.set_device(0)
    prec = args.precision if args.precision != "mixed" else "fp32"
    if args.workload == "batched":
        import bench_workloads
        nrhs = args.rhs or 128
        p, einc, rhs = bench_workloads.spheroid_problem(nrhs)
        mv = dda_b200.CudaMatVec(p, prec, max_rhs=nrhs)
        for r, (prop, pol) in enumerate(rhs):
            mv.set_couple_constants(dda_b200.CoupleConstants(p, prop, pol, "ldr"), rhs=r)
    else:
        nrhs = args.rhs or 2
        p, mv, einc = build_problem(prec, nrhs)
        einc = einc.reshape(nrhs, -1)
    cdt = torch.complex128 if prec == "fp64" else torch.complex64
    x = torch.from_numpy(np.ascontiguousarray(einc[:nrhs])).to(cdt).cuda()
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    torch.cuda.profiler.start()  # ncu --profile-from-start off: capture only these matvecs
    for _ in range(args.matvec_only):
        mv.apply_device(x.data_ptr(), y.data_ptr(), nrhs=nrhs)
    mv.synchronize()
    torch.cuda.profiler.stop()
    print("matvecs", args.matvec_only, "nrhs", nrhs, "grid", p.grid, "layout", mv.layout, flush=True)


def run_solve_only(args):
    """Runs args.solve_only solves of the default workload (both
    polarisations, device-resident fields; with --workload batched the
    128-rhs spheroid block) after one untimed solve, and exits: the command
    ncu's launch list captures (--profile-from-start off)."""
    import torch
    import dda_b200
    torch.cuda.set_device(0)
    prec = args.precision
    if args.workload == "batched":  # the 128-rhs spheroid block, mixed precision, QMR-CS
        import bench_workloads
        nrhs = args.rhs or 128
        p, einc, rhs = bench_workloads.spheroid_problem(nrhs)
        mv = dda_b200.CudaMatVec(p, "mixed", max_rhs=nrhs)
        for r, (prop, pol) in enumerate(rhs):
            mv.set_couple_constants(dda_b200.CoupleConstants(p, prop, pol, "ldr"), rhs=r)
        solver = dda_b200.CudaSolver(mv, "qmr")
        cdt = torch.complex128
    else:
        nrhs = 2
        p, mv, einc = build_problem(prec, 2)
        solver = dda_b200.CudaSolver(mv, args.solver)
        cdt = torch.complex128 if prec == "fp64" else torch.complex64
    e_dev = torch.from_numpy(np.ascontiguousarray(einc)).to(cdt).cuda()
    p_dev = torch.zeros_like(e_dev)
    torch.cuda.synchronize()
    solver.get_pol_vec_device(e_dev.data_ptr(), p_dev.data_ptr(), nrhs, EPS)
    torch.cuda.profiler.start()
    for _ in range(args.solve_only):
        solver.get_pol_vec_device(e_dev.data_ptr(), p_dev.data_ptr(), nrhs, EPS)
    mv.synchronize()
    torch.cuda.profiler.stop()
    print("solves", args.solve_only, "iterations", [st.iterations for st in solver.last_stats], flush=True)


if __name__ == "__main__":
    a = parse()
    if a.matvec_only:
        run_matvec_only(a)
    elif a.solve_only:
        run_solve_only(a)
    elif a.impl == "reference":
        run_reference(a)
    elif a.workload == "box":
        run_ours(a)
    else:
        import bench_workloads
        getattr(bench_workloads, "run_" + a.workload)(a)
