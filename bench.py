#!/usr/bin/env python3
"""Benchmark of the MRHS even-odd Wilson dslash on GB300.

Workload (one "step"): the hopping term D_eo applied to nrhs = 12 right-hand
sides of SU(3) spinors on a 32^3 x 64 lattice (Vh = 1,048,576 output sites),
FP32 storage and arithmetic, antiperiodic time boundaries, seeded random
SU(3) links and Gaussian spinors (synthetic data; the reference publishes no
dataset).  The input field (1.2 GB) and gauge (0.6 GB) exceed the 129 MB L2,
so no flush is needed between steps.

Reported (one JSON line on rank 0; the full tables of sweep, solve, serve,
multi_lattice and colors go to stderr, one JSON line each):
  value      site*RHS/s of the device-resident dslash (CUDA events on the
             library stream around exactly --steps launches)
  e2e        the same metric through the drop-in C ABI (pushBackFermions x 12 +
             startDslash) with pinned host buffers: host->device copy of the
             caller-layout FP64 inputs and device->host copy of the outputs
             inside the timed region
  roofline   algorithmic bytes per launch / mean launch time vs measured HBM
  cpu_baseline  the FP64 OpenMP oracle dslash on this host's cores
  sweep      site*RHS/s and roofline fraction per precision x nrhs
  fma_peaks  measured FP64 / FP32 FMA peaks (the FP64 dslash is FP64-pipe-bound)
  solve      eo-CG to FP64 true residual 1e-10: mixed precision vs plain FP64
  serve      Poisson request stream over 4 resident gauges: p50/p99, solves/s
             vs serial plain-FP64 solves
  colors     16^3x32 SU(N), N = 4, 6, 8, nrhs 16-64 (FP32 / BF16), and a
             masked BiCGStab per N

--impl reference times the reference's CPU path for this operator on the
host cores.  The reference has no CPU implementation (its only code path is
the sm_70-era GPU kernel), so this arm runs the FP64 OpenMP restatement of its
operator (oracle/), on a bounded sample of the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

L_BENCH = (32, 32, 32, 64)
NRHS = 12
NC = 3
FLOPS_PER_SITE_RHS = lambda n: 128 * n * n + 56 * n  # noqa: E731
METRIC = "dslash site\u00b7RHS/s & % HBM roofline; mixed vs FP64 solve time @1e-10; p99"


def workload_config(L, n, nrhs, world, precision):
    """The workload both arms measure; `precision` is the arm's storage
    (ours) or arithmetic (the reference's FP64 CPU path) precision."""
    return {"workload": "MRHS even-odd Wilson dslash D_eo, SU(%d), %s, nrhs=%d, antiperiodic t"
                        % (n, "x".join(map(str, L)), nrhs),
            "lattice": list(L), "nrhs": nrhs, "N": n, "precision": precision,
            "parallelism": "replicas (RHS sets independent)" if world > 1 else "1 GPU",
            "l2": "inputs larger than L2 (1.2 GB field + 0.6 GB gauge at FP32); no flush"}


def bytes_per_site_rhs(prec: int, n: int, nrhs: int) -> float:
    """Compulsory bytes per output site per RHS: 8 links (N^2 complex each,
    amortised over the RHS) + one input and one output spinor (4N complex)
    + the per-(site, RHS) FP32 scale of FP16 storage, read and written
    (BF16 fields are unscaled)."""
    c = {2: 16, 1: 8, 0: 4, 4: 4, 5: 4}[prec]
    nn = 4 if prec == 0 else 0
    return 8 * n * n * c / nrhs + 2 * (4 * n * c + nn)


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as fh:
            d = json.load(fh)
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


def profile_traffic(kernel: str):
    """Per-launch DRAM bytes (dram__bytes_read.sum + dram__bytes_write.sum)
    of exactly this kernel shape on the headline workload, from the committed
    ncu summary (lines "<bytes> <kernel string>"); None when that shape was
    not captured."""
    path = os.path.join(ROOT, "profiles", "dslash_traffic.txt")
    if not os.path.exists(path):
        return None
    with open(path) as fh:
        for line in fh:
            if line.strip() and not line.startswith("#"):
                v, k = line.split(None, 1)
                if k.strip() == kernel:
                    return float(v)
    return None


class ClockSampler:
    """SM clock and clock-event reasons sampled every few ms during the timed
    region, through NVML (read-only queries), with nvidia-smi as a fallback."""

    REASONS = {0x4: "sw_power_cap", 0x8: "hw_slowdown", 0x20: "sw_thermal_slowdown",
               0x40: "hw_thermal_slowdown", 0x80: "hw_power_brake_slowdown"}

    def __init__(self, index: int, period_s: float = 0.005):
        self.index = index
        self.period = period_s
        self.sm, self.reasons, self.max_mhz = [], set(), None
        self._stop = threading.Event()
        self._nvml = None
        self._thread = None

    def _open(self):
        import ctypes
        try:
            lib = ctypes.CDLL("libnvidia-ml.so.1")
        except OSError:
            return None
        if lib.nvmlInit_v2() != 0:
            return None
        h = ctypes.c_void_p()
        vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
        idx = int(vis.split(",")[self.index]) if vis and vis.split(",")[0].isdigit() else self.index
        if lib.nvmlDeviceGetHandleByIndex_v2(ctypes.c_uint(idx), ctypes.byref(h)) != 0:
            return None
        mx = ctypes.c_uint()
        if lib.nvmlDeviceGetMaxClockInfo(h, ctypes.c_int(1), ctypes.byref(mx)) == 0:
            self.max_mhz = float(mx.value)
        return lib, h

    def _run(self):
        import ctypes
        lib, h = self._nvml
        clk = ctypes.c_uint()
        rs = ctypes.c_ulonglong()
        get_r = getattr(lib, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
            lib.nvmlDeviceGetCurrentClocksThrottleReasons
        while not self._stop.is_set():
            if lib.nvmlDeviceGetClockInfo(h, ctypes.c_int(1), ctypes.byref(clk)) == 0:
                self.sm.append(float(clk.value))
            if get_r(h, ctypes.byref(rs)) == 0:
                for bit, name in self.REASONS.items():
                    if rs.value & bit:
                        self.reasons.add(name)
            self._stop.wait(self.period)

    def __enter__(self):
        self._nvml = self._open()
        if self._nvml is not None:
            self._thread = threading.Thread(target=self._run, daemon=True)
            self._thread.start()
        return self

    def __exit__(self, *a):
        self._stop.set()
        if self._thread is not None:
            self._thread.join(timeout=2)
        if not self.sm:  # fallback: one nvidia-smi reading right after the region
            try:
                out = subprocess.run(["nvidia-smi", "-i", str(self.index), "--query-gpu=clocks.sm,clocks.max.sm",
                                      "--format=csv,noheader,nounits"], capture_output=True, text=True,
                                     timeout=20).stdout.split(",")
                self.sm.append(float(out[0]))
                self.max_mhz = float(out[1])
            except (OSError, ValueError, IndexError, subprocess.TimeoutExpired):
                pass

    def summary(self):
        med = float(np.median(self.sm)) if self.sm else None
        return {"sm_mhz": med, "sm_max_mhz": self.max_mhz, "reasons": sorted(self.reasons),
                "samples": len(self.sm), "source": "nvml" if self._nvml is not None else "nvidia-smi"}


def dist_setup():
    """One process per GPU under torchrun; replicas of the workload (the RHS
    sets are independent, so no data-path collective exists)."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("gloo")
        return world, rank, local, dist
    return 1, 0, 0, None


def job_throughput(units_per_rank: float, world: int, ms_max: float) -> float:
    """Whole-job units per second: every rank processes units_per_rank in
    its step; the step time is the maximum over ranks."""
    return units_per_rank * world / (ms_max * 1e-3)


def barrier(dist):
    if dist is not None:
        dist.barrier()


def max_over_ranks(dist, v: float) -> float:
    if dist is None:
        return v
    import torch
    t = torch.tensor([v], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def make_inputs(torch, L, n, nrhs, seed_g=0, seed_p=1):
    """Seeded SU(N) gauge and Gaussian spinors, generated on the GPU with the
    phase-fixed QR construction (Gram-Schmidt, then det^(-1/N))."""
    from mrhs_qcu_gb300 import synthetic as S
    vh = S.half_volume(L)
    gen = torch.Generator(device="cuda").manual_seed(seed_g)
    g = S.random_sun_torch(4 * 2 * vh, n, gen).view(4, 2, vh, n, n)
    genp = torch.Generator(device="cuda").manual_seed(seed_p)
    psi = torch.complex(torch.randn((nrhs, vh, 4, n), generator=genp, device="cuda", dtype=torch.float64),
                        torch.randn((nrhs, vh, 4, n), generator=genp, device="cuda", dtype=torch.float64)) * (0.5 ** 0.5)
    return g, psi


def time_resident(torch, Q, L, n, nrhs, prec, steps, warmup, g_dev, psi_dev, count_launches=True):
    """Device-resident dslash: pack once, then time `steps` MRHS launches."""
    from mrhs_qcu_gb300 import synthetic as S
    vh = S.half_volume(L)
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    Q.set_stream(torch.cuda.current_stream().cuda_stream)
    Q.loadQcuGauge(g_dev.data_ptr())
    Q.getDslash(Q.DSLASH_WILSON, 0.0, n, nrhs, prec)
    db, nb = Q.field_bytes(prec, nrhs)
    fin = torch.empty(db // 8 + 2, dtype=torch.float64, device="cuda")
    fout = torch.empty(db // 8 + 2, dtype=torch.float64, device="cuda")
    nin = torch.empty(max(nb, 16) // 4, dtype=torch.float32, device="cuda") if nb else None
    nout = torch.empty(max(nb, 16) // 4, dtype=torch.float32, device="cuda") if nb else None
    ptrs = [psi_dev[r % psi_dev.shape[0]].data_ptr() for r in range(nrhs)]
    Q.pack_fermions(fin.data_ptr(), nin.data_ptr() if nin is not None else None, ptrs, Q.QCU_SRC_EO_HALF, 1, prec)
    args = (fout.data_ptr(), nout.data_ptr() if nout is not None else None, fin.data_ptr(),
            nin.data_ptr() if nin is not None else None, nrhs, 0, 0, prec)
    Q.tune_dslash(nrhs, prec)
    for _ in range(max(warmup, 1)):
        Q.dslash_mrhs(*args)
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        Q.dslash_mrhs(*args)
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / steps
    Q.set_stream(None)
    return ms, vh * nrhs


def run_gpu(args):
    import torch

    import mrhs_qcu_gb300 as Q
    from mrhs_qcu_gb300 import synthetic as S

    world, rank, local, dist = dist_setup()
    torch.cuda.set_device(local)
    L = tuple(int(v) for v in args.lattice.split(","))
    n, nrhs, prec = args.ncolors, args.nrhs, args.precision
    pname = {0: "fp16", 1: "fp32", 2: "fp64", 4: "bf16", 5: "bf16-site"}[prec]
    vh = S.half_volume(L)
    g_dev, psi_dev = make_inputs(torch, L, n, nrhs, seed_g=0, seed_p=1 + rank)

    # ---- device-resident headline --------------------------------------
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    stream = torch.cuda.current_stream()
    Q.set_stream(stream.cuda_stream)
    Q.loadQcuGauge(g_dev.data_ptr())
    Q.getDslash(Q.DSLASH_WILSON, 0.0, n, nrhs, prec)
    db, nb = Q.field_bytes(prec, nrhs)
    fin = torch.empty(db // 8 + 2, dtype=torch.float64, device="cuda")
    fout = torch.empty(db // 8 + 2, dtype=torch.float64, device="cuda")
    nin = torch.empty(max(nb, 16) // 4, dtype=torch.float32, device="cuda") if nb else None
    nout = torch.empty(max(nb, 16) // 4, dtype=torch.float32, device="cuda") if nb else None
    nin_p = nin.data_ptr() if nin is not None else None
    nout_p = nout.data_ptr() if nout is not None else None
    ptrs = [psi_dev[r].data_ptr() for r in range(nrhs)]
    Q.pack_fermions(fin.data_ptr(), nin_p, ptrs, Q.QCU_SRC_EO_HALF, 1, prec)
    R, block, minb, pk, stages, recon, linktma = Q.tune_dslash(nrhs, prec)
    for _ in range(args.warmup):
        Q.dslash_mrhs(fout.data_ptr(), nout_p, fin.data_ptr(), nin_p, nrhs, 0, 0, prec)
    torch.cuda.synchronize()
    barrier(dist)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clk:
        torch.cuda.synchronize()
        e0.record(stream)
        for _ in range(args.steps):
            Q.dslash_mrhs(fout.data_ptr(), nout_p, fin.data_ptr(), nin_p, nrhs, 0, 0, prec)
        e1.record(stream)
        torch.cuda.synchronize()
    barrier(dist)
    ms_local = e0.elapsed_time(e1) / args.steps
    ms = max_over_ranks(dist, ms_local)
    units = vh * nrhs
    value = job_throughput(units, world, ms)
    peak, peak_kind = measured_peaks()
    bpu = bytes_per_site_rhs(prec, n, nrhs)
    achieved = bpu * units / (ms_local * 1e-3) / 1e9
    tcs_rings = {4: (4, 3), 6: (5, 2), 7: (8, 2), 8: (6, 2)}  # (TMA stages, B buffers) of variants 4, 6-8
    kernel = ("wilson_mma_kernel<%s,N=%d> (register-fragment mma.sync)" % (pname, n) if stages == -5 else
              ("wilson_tcs_kernel<N=%d,stages=%d,bbufs=%d> (tcgen05, %s)"
               % ((n,) + tcs_rings[-stages] + ("site-major" if prec == 5 else "component-major",)))
              if stages <= -4 else
              ("wilson_tc_kernel<%s,N=%d> (tcgen05)" % (pname, n)) if stages < 0 else
              ("wilson_tma_kernel<%s,N=%d,R=%d,stages=%d>" % (pname, n, R, stages)) if stages else
              ("wilson_tmalink_kernel<%s,N=%d,R=%d,reg_cap=%d,recon=%d> row CTA"
               % (pname, n, R, minb, recon)) if linktma else
              ("wilson_mrhs_kernel<%s,N=%d,R=%d,reg_cap=%d,PK=%d,recon=%d> block %d"
               % (pname, n, R, minb, pk, recon, block)))
    roof = {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
            "frac": round(achieved / peak, 4), "peak_kind": peak_kind,
            "algorithmic_bytes_per_launch": bpu * units,
            # measured DRAM bytes of exactly this kernel shape on this workload (profiles/dslash_traffic.txt)
            "traffic": profile_traffic(kernel)
            if (tuple(L) == L_BENCH and nrhs == NRHS and prec == 1 and n == NC) else None,
            "kernel": kernel,
            "gflops": round(FLOPS_PER_SITE_RHS(n) * units / (ms_local * 1e-3) / 1e9, 1)}
    rel_err = headline_error(torch, Q, L, n, nrhs, prec, fout, nout_p, psi_dev, g_dev)
    Q.set_stream(None)

    # ---- end to end through the drop-in ABI with host buffers -----------
    e2e = None
    if not args.skip_e2e:
        # Pinned host buffers in and out; every step uploads its 12 sources,
        # runs the drop-in ABI (pushBackFermions x 12, startDslash) and
        # downloads its 12 results.  Device buffers are triple buffered and the
        # copies run on their own streams, so step k+1's upload and step k-1's
        # download overlap step k (the two directions of the host link run
        # concurrently), and the next upload does not wait for step k's
        # compute: with two buffers both directions of the link stood idle
        # while a step computed.
        host_in = [torch.empty((vh, 4, n), dtype=torch.complex128).pin_memory() for _ in range(nrhs)]
        for r in range(nrhs):
            host_in[r].copy_(psi_dev[r])
        host_out = [torch.empty((vh, 4, n), dtype=torch.complex128).pin_memory() for _ in range(nrhs)]
        nbuf = 3
        dev_in = [[torch.empty((vh, 4, n), dtype=torch.complex128, device="cuda") for _ in range(nrhs)]
                  for _ in range(nbuf)]
        dev_out = [[torch.empty((vh, 4, n), dtype=torch.complex128, device="cuda") for _ in range(nrhs)]
                   for _ in range(nbuf)]
        s_up, s_down, s_comp = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
        up_done = [torch.cuda.Event() for _ in range(nbuf)]
        comp_done = [torch.cuda.Event() for _ in range(nbuf)]
        down_done = [torch.cuda.Event() for _ in range(nbuf)]
        Q.set_stream(s_comp.cuda_stream)

        def upload(k):
            b = k % nbuf
            s_up.wait_event(comp_done[b])  # step k - nbuf has read dev_in[b]
            with torch.cuda.stream(s_up):
                for r in range(nrhs):
                    dev_in[b][r].copy_(host_in[r], non_blocking=True)
            up_done[b].record(s_up)

        def compute(k):
            b = k % nbuf
            s_comp.wait_event(up_done[b])
            s_comp.wait_event(down_done[b])  # step k - nbuf's results have left dev_out[b]
            for r in range(nrhs):
                Q.pushBackFermions(dev_out[b][r].data_ptr(), dev_in[b][r].data_ptr())
            Q.startDslash(0, 0)
            comp_done[b].record(s_comp)

        def download(k):
            b = k % nbuf
            s_down.wait_event(comp_done[b])
            with torch.cuda.stream(s_down):
                for r in range(nrhs):
                    host_out[r].copy_(dev_out[b][r], non_blocking=True)
            down_done[b].record(s_down)

        def run(k_steps, f0=None, f1=None):
            if f0 is not None:
                f0.record(s_up)
            upload(0)
            for k in range(k_steps):
                if k + 1 < k_steps:
                    upload(k + 1)
                compute(k)
                download(k)
            if f1 is not None:
                f1.record(s_down)

        run(max(2, args.warmup // 2))
        torch.cuda.synchronize()
        # the same K steps as the device-resident line: the pipeline's first upload and last
        # download, which nothing overlaps, are part of the timed region
        e2e_steps = max(2, args.steps)
        barrier(dist)
        f0 = torch.cuda.Event(enable_timing=True)
        f1 = torch.cuda.Event(enable_timing=True)
        run(e2e_steps, f0, f1)
        torch.cuda.synchronize()
        ems = max_over_ranks(dist, f0.elapsed_time(f1) / e2e_steps)
        # the downloaded results equal one untimed call of the same ABI on device buffers
        for r in range(nrhs):
            Q.pushBackFermions(dev_out[0][r].data_ptr(), dev_in[1][r].data_ptr())
        Q.startDslash(0, 0)
        torch.cuda.synchronize()
        e2e_same = all(torch.equal(host_out[r], dev_out[0][r].cpu()) for r in range(nrhs))
        bytes_io = nrhs * vh * 4 * n * 16
        link = host_link_peaks(torch, host_in, host_out, dev_in[0], dev_out[0])
        # the step moves bytes_io each way over the host link: its bound is the slowest of the
        # two directions alone and of both directions at once
        link_ms = max(bytes_io / link["h2d_gbs"], bytes_io / link["d2h_gbs"], 2 * bytes_io / link["both_gbs"]) / 1e6
        e2e = {"value": job_throughput(units, world, ems), "unit": "site*RHS/s", "h2d_bytes_per_step": bytes_io,
               "d2h_bytes_per_step": bytes_io, "ms_per_step": round(ems, 3), "steps": e2e_steps,
               "host_link": link, "link_bound_ms_per_step": round(link_ms, 3),
               "frac_of_link_bound": round(link_ms / ems, 4),
               "path": "pinned host -> upload stream -> pushBackFermions x12 + startDslash -> download stream -> "
                       "pinned host (FP64 caller layout); device buffers triple buffered so step k+1's upload "
                       "and step k-1's download overlap step k",
               "results_equal_device_path": e2e_same}
        Q.set_stream(None)
        del host_in, host_out, dev_in, dev_out

    del fin, fout
    torch.cuda.empty_cache()

    # ---- sweep of precisions x nrhs ------------------------------------
    sweep = []
    fma = None
    if not args.skip_sweep and rank == 0:
        # FMA pipe peaks: FP64 bounds the FP64 dslash (1320 flop vs 480 B per site*RHS at nrhs 12)
        fma = {"fp64_tflops": round(Q.measure_fma_rate(Q.QCU_DOUBLE_PRECISION), 2),
               "fp32_tflops": round(Q.measure_fma_rate(Q.QCU_SINGLE_PRECISION), 2),
               "how": "8 independent FMA chains per thread, 8 blocks of 256 per SM, CUDA events"}
        for p, sname in ((2, "fp64"), (1, "fp32"), (0, "fp16"), (4, "bf16")):
            for nr in (1, 4, 12, 24):
                if p == 2 and nr == 24:
                    continue
                ms_s, u = time_resident(torch, Q, L, n, nr, p, 5 if p != 2 else 2, 2, g_dev, psi_dev)
                ach = bytes_per_site_rhs(p, n, nr) * u / (ms_s * 1e-3) / 1e9
                sweep.append({"precision": sname, "nrhs": nr, "ms": round(ms_s, 4),
                              "site_rhs_per_s": round(u / (ms_s * 1e-3)),
                              "gbs": round(ach, 1), "hbm_frac": round(ach / peak, 4),
                              "gflops": round(FLOPS_PER_SITE_RHS(n) * u / (ms_s * 1e-3) / 1e9, 1)})
                if p == 2:
                    sweep[-1]["fp64_pipe_frac"] = round(sweep[-1]["gflops"] / (1e3 * fma["fp64_tflops"]), 4)
        torch.cuda.empty_cache()

    # ---- CPU baseline (oracle, FP64, host cores) -----------------------
    cpu = None
    if rank == 0 and not args.skip_cpu:
        cpu = cpu_baseline(g_dev, psi_dev, L, n, budget_s=args.cpu_seconds)

    # ---- solver: mixed vs FP64 ----------------------------------------
    solve = None
    if rank == 0 and not args.skip_solve:
        solve = solve_bench(torch, Q)

    # ---- one launch over several lattices vs one launch per lattice ------
    multi = None
    if rank == 0 and not args.skip_serve:
        multi = multi_lattice_bench(torch, Q)

    # ---- serving stream: continuous batching over resident gauges -------
    serve = None
    if rank == 0 and not args.skip_serve:
        serve = serve_bench(torch, Q)

    # ---- SU(N), N = 4..8, large nrhs ----------------------------------------
    colors = None
    if rank == 0 and not args.skip_colors:
        colors = colors_bench(torch, Q, peak, fma)

    if rank == 0:
        line = {
            "metric": METRIC,
            "value": value, "unit": "site*RHS/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": round(ms, 4), "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": {"fp32": "f32", "fp64": "f64", "fp16": "f16", "bf16": "bf16", "bf16-site": "bf16"}[pname], "data": "synthetic (seeded SU(3) links, Gaussian spinors)",
            "config": workload_config(L, n, nrhs, world, pname),
            "roofline": roof, "rel_err": rel_err, "clocks": clk.summary(), "gpu_launches": args.steps,
            "e2e": e2e, "cpu_baseline": cpu, "sweep": sweep, "fma_peaks": fma, "solve": solve, "serve": serve,
            "multi_lattice": multi, "colors": colors,
        }
        line, tables = split_line(line)
        for name, table in tables.items():
            print(json.dumps({name: table}), file=sys.stderr)
        print(json.dumps(line))
    if dist is not None:
        dist.destroy_process_group()


def host_link_peaks(torch, host_in, host_out, dev_in, dev_out, reps=3):
    """Copy-engine bandwidth between pinned host memory and the GPU with the
    e2e leg's own buffers: host->device alone, device->host alone, and both
    directions at once on two streams (GB/s, best of `reps`)."""
    s_up, s_down = torch.cuda.Stream(), torch.cuda.Stream()
    nbytes = sum(t.numel() * t.element_size() for t in host_in)

    def run(up, down):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        if up:
            with torch.cuda.stream(s_up):
                for h, d in zip(host_in, dev_in):
                    d.copy_(h, non_blocking=True)
        if down:
            with torch.cuda.stream(s_down):
                for h, d in zip(host_out, dev_out):
                    h.copy_(d, non_blocking=True)
        torch.cuda.synchronize()
        return time.perf_counter() - t0

    out = {}
    for name, up, down, moved in (("h2d_gbs", 1, 0, nbytes), ("d2h_gbs", 0, 1, nbytes),
                                  ("both_gbs", 1, 1, 2 * nbytes)):
        best = min(run(up, down) for _ in range(reps))
        out[name] = round(moved / best / 1e9, 1)
    out["how"] = "pinned host <-> device copies of the e2e buffers, best of %d, wall clock" % reps
    return out


def headline_error(torch, Q, L, n, nrhs, prec, fout, nout_p, psi_dev, g_dev, checked=2):
    """Relative L2 error of the benchmarked result against the FP64 oracle:
    the timed launches' output field, unpacked to the caller layout, for the
    first `checked` RHS (the oracle runs on the host cores)."""
    from mrhs_qcu_gb300 import synthetic as S
    from oracle import oracle as O
    checked = min(checked, nrhs)
    vh = S.half_volume(L)
    dsts = [torch.empty((vh, 4, n), dtype=torch.complex128, device="cuda") for _ in range(nrhs)]
    Q.unpack_fermions([d.data_ptr() for d in dsts], fout.data_ptr(), nout_p, Q.QCU_SRC_EO_HALF, 0, prec)
    torch.cuda.synchronize()
    got = np.stack([dsts[r].cpu().numpy() for r in range(checked)])
    del dsts
    ref = O.dslash(psi_dev[:checked].cpu().numpy(), g_dev.cpu().numpy(), L, 0, 0, True)
    errs = [float(np.linalg.norm(got[r] - ref[r]) / np.linalg.norm(ref[r])) for r in range(checked)]
    tol = {2: 1e-13, 1: 1e-6, 0: 5e-3, 4: 5e-3, 5: 5e-3}[prec]
    return {"max": max(errs), "per_rhs": errs, "rhs_checked": checked, "tolerance": tol,
            "within_tolerance": max(errs) < tol,
            "against": "FP64 OpenMP oracle on the host, same inputs (D_eo, antiperiodic t)"}


def cpu_baseline(g_dev, psi_dev, L, n, budget_s=12.0):
    """FP64 OpenMP oracle dslash on the host cores, on a bounded sample of the
    workload: the full 32^3x64 gauge and the benchmark field's RHS, one RHS per
    call, cycling over the RHS until about budget_s of host work is done."""
    from oracle import oracle as O
    g = g_dev.cpu().numpy()
    threads = O.num_threads()
    from mrhs_qcu_gb300 import synthetic as S
    vh = S.half_volume(L)
    done = 0
    t0 = time.perf_counter()
    elapsed = 0.0
    r = 0
    host = [psi_dev[k:k + 1].cpu().numpy() for k in range(psi_dev.shape[0])]
    while elapsed < budget_s:
        psi = host[r % len(host)]
        t1 = time.perf_counter()
        O.dslash(psi, g, L, 0, 0, True)
        elapsed += time.perf_counter() - t1
        done += vh
        r += 1
    return {"value": done / elapsed, "unit": "site*RHS/s", "cores": threads, "kind": "port",
            "sample": "%d single-RHS D_eo applications (cycling over the %d RHS) of the 32^3x64 SU(3) "
                      "workload, FP64, %.1f s" % (r, len(host), elapsed),
            "wall_s": round(time.perf_counter() - t0, 2)}


def solve_bench(torch, Q):
    """eo-CG on Mhat^dag Mhat to FP64 true residual 1e-10, 24^3x48, SU(3),
    nrhs=12, kappa=0.12, point sources: FP32 / FP16 inner with FP64 reliable
    updates vs the plain FP64 MRHS CG."""
    from mrhs_qcu_gb300 import synthetic as S
    L, n, nrhs, kappa = (24, 24, 24, 48), 3, 12, 0.12
    g_dev, _ = make_inputs(torch, L, n, 1, seed_g=5)
    b = S.point_sources(L, n, nrhs, seed=6)
    db = [torch.from_numpy(b[r]).cuda() for r in range(nrhs)]
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    Q.loadQcuGauge(g_dev.data_ptr())
    out = {"workload": "24^3x48 SU(3) nrhs=12 kappa=0.12 point sources, tol 1e-10 (FP64 true residual)"}
    for name, inner in (("fp32_inner", 1), ("fp16_inner", 0), ("fp64_plain", 2)):
        res = {}
        for phase in ("cold", "warm"):  # the cold solve tunes kernels and captures graphs
            dx = [torch.zeros_like(x) for x in db]
            p = Q.solver_params(kappa=kappa, tol=1e-10, inner_precision=inner, max_iter=20000)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            Q.invert([x.data_ptr() for x in dx], [x.data_ptr() for x in db], p, raise_on_error=False)
            torch.cuda.synchronize()
            res[phase] = time.perf_counter() - t0
        out[name] = {"seconds": round(res["warm"], 4), "seconds_cold": round(res["cold"], 4),
                     "iterations": p.iterations, "reliable_updates": p.reliable_updates,
                     "max_true_residual": max(p.true_residual[r] for r in range(nrhs)),
                     "all_converged": all(p.converged[r] for r in range(nrhs))}
    if out["fp64_plain"]["seconds"] > 0:
        out["speedup_fp32_inner_vs_fp64"] = round(out["fp64_plain"]["seconds"] / out["fp32_inner"]["seconds"], 2)
        out["speedup_fp16_inner_vs_fp64"] = round(out["fp64_plain"]["seconds"] / out["fp16_inner"]["seconds"], 2)
    return out


def colors_bench(torch, Q, peak, fma):
    """16^3x32, SU(N) N = 4, 6, 8, nrhs 16 / 32 / 64, FP32 and BF16 storage
    (FP32 arithmetic): dslash throughput against the HBM roofline and the FP32
    FMA peak (at N = 8 the CUDA-core kernel is compute-bound), and one
    BiCGStab solve per N with per-RHS masks (one source 1e-4 times smaller,
    one zero) to 1e-8."""
    from mrhs_qcu_gb300 import synthetic as S
    L = (16, 16, 16, 32)
    vh = S.half_volume(L)
    rows, solves = [], []
    for n in (4, 6, 8):
        g_dev, psi = make_inputs(torch, L, n, 64, seed_g=300 + n, seed_p=301)
        # FP32: the autotuned CUDA-core kernel; BF16: CUDA cores (register kernel, R = 2) and the
        # tensor-core (tcgen05) kernels, each pinned (spinor-operand variants 4 and 6: rings of 4 and
        # 5 stages), and the autotuner's choice on site-major fields
        for p, pname, kernel, pin in ((1, "fp32", "cuda_core", None), (4, "bf16", "cuda_core", "2,64,1,0"),
                                      (4, "bf16", "tensor_core_projected", "1,0,0,0,0,0,1"),
                                      (4, "bf16", "tensor_core_projected_tma", "1,0,0,0,0,0,2"),
                                      (4, "bf16", "tensor_core_spinor", "1,0,0,0,0,0,4"),
                                      (4, "bf16", "tensor_core_spinor_ring5", "1,0,0,0,0,0,6"),
                                      (5, "bf16-site", "tensor_core_spinor", "1,0,0,0,0,0,4"),
                                      (5, "bf16-site", "tensor_core_spinor_ring5", "1,0,0,0,0,0,6"),
                                      (5, "bf16-site", "tensor_core_tuned", None)):
            for nr in (16, 32, 64):
                if pin:
                    os.environ["QCU_DSLASH_CONFIG"] = pin
                try:
                    ms_s, u = time_resident(torch, Q, L, n, nr, p, 10, 3, g_dev, psi)
                finally:
                    os.environ.pop("QCU_DSLASH_CONFIG", None)
                rate = u / (ms_s * 1e-3)
                gbs = bytes_per_site_rhs(p, n, nr) * rate / 1e9
                tf = FLOPS_PER_SITE_RHS(n) * rate / 1e12
                rows.append({"N": n, "precision": pname, "kernel": kernel, "nrhs": nr, "ms": round(ms_s, 4),
                             "site_rhs_per_s": round(rate), "gbs": round(gbs, 1), "hbm_frac": round(gbs / peak, 4),
                             "tflops": round(tf, 2),
                             "fp32_fma_frac": round(tf / fma["fp32_tflops"], 4) if fma else None})
        # BiCGStab with masks: 16 RHS, FP32 inner
        nr = 16
        b = torch.complex(torch.randn((nr, 2, vh, 4, n), device="cuda", dtype=torch.float64,
                                      generator=torch.Generator(device="cuda").manual_seed(302)),
                          torch.randn((nr, 2, vh, 4, n), device="cuda", dtype=torch.float64,
                                      generator=torch.Generator(device="cuda").manual_seed(303)))
        b[1] *= 1e-4
        b[2] = 0
        x = torch.zeros_like(b)
        Q.initGridSize(L, n)
        Q.set_antiperiodic_t(True)
        Q.loadQcuGauge(g_dev.data_ptr())
        # FP32 inner (CUDA-core dslash), BF16 inner (the autotuner's dslash: tensor cores where they win)
        # and site-major BF16 inner (the tensor-core dslash)
        for inner, iname in ((Q.QCU_SINGLE_PRECISION, "fp32"), (Q.QCU_BF16_PRECISION, "bf16"),
                             (Q.QCU_BF16_SITE_PRECISION, "bf16-site")):
            prm = Q.solver_params(kappa=0.11, tol=1e-8, inner_precision=inner,
                                  solver=Q.QCU_SOLVER_BICGSTAB, max_iter=5000)
            for phase in ("cold", "warm"):
                x.zero_()
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                Q.invert([x[r].data_ptr() for r in range(nr)], [b[r].data_ptr() for r in range(nr)], prm,
                         raise_on_error=False)
                torch.cuda.synchronize()
                sec = time.perf_counter() - t0
            st_bf = Q.tune_dslash(nr, inner)[4]
            solves.append({"N": n, "nrhs": nr, "inner": iname, "seconds": round(sec, 4),
                           "iterations": prm.iterations, "reliable_updates": prm.reliable_updates,
                           "inner_dslash": ("tensor_core_variant_%d" % -st_bf) if st_bf < 0 else "cuda_core",
                           "max_true_residual": max(prm.true_residual[r] for r in range(nr)),
                           "all_converged": all(prm.converged[r] for r in range(nr))})
        del g_dev, psi, b, x
        torch.cuda.empty_cache()
    return {"workload": "16^3x32 SU(N) dslash: FP32 storage on CUDA cores; BF16 storage on CUDA cores (FP32 "
                        "arithmetic) and on the tensor cores (tcgen05, BF16 operands, FP32 accumulation), "
                        "component-major and site-major (bf16-site) fields; BiCGStab kappa 0.11, FP32, BF16 and "
                        "site-major BF16 inner, 16 RHS (one 1e-4 smaller, one zero) to 1e-8",
            "dslash": rows, "bicgstab": solves}


def multi_lattice_bench(torch, Q, reps=20):
    """The hop term on a mix of lattices (the serving workload's 8^4,
    16^3x32 and 24^3x48 SU(3), FP32, various RHS counts, plus sixteen small
    8^4 segments): one qcuDslashSegments launch over the whole work list
    against one launch per lattice (each with its own tuned shape), timed with
    CUDA events on one stream."""
    from mrhs_qcu_gb300 import synthetic as S
    n = 3
    mixes = {"serving_lattices": [((8, 8, 8, 8), 4), ((16, 16, 16, 32), 12), ((24, 24, 24, 48), 24),
                                  ((16, 16, 16, 32), 8)],
             "sixteen_8^4": [((8, 8, 8, 8), 4)] * 16}
    stream = torch.cuda.current_stream()
    out = {"workload": "D_eo, SU(3), FP32, antiperiodic t; one launch over the work list vs one per lattice"}
    gen = torch.Generator(device="cuda").manual_seed(77)
    for name, mix in mixes.items():
        segs, keep, units = [], [], 0
        for L, nrhs in mix:
            vh = S.half_volume(L)
            g = S.random_sun_torch(4 * 2 * vh, n, gen).view(4, 2, vh, n * n).permute(0, 1, 3, 2)
            gc = g.to(torch.complex64).contiguous()
            vp = (vh + 31) // 32 * 32  # two-row links in groups of 32 sites: [4][2][Vp/32][6][32]
            t12 = torch.zeros((4, 2, 6, vp), dtype=gc.dtype, device=gc.device)
            t12[..., :vh] = gc[:, :, :6, :]
            g12 = t12.view(4, 2, 6, vp // 32, 32).permute(0, 1, 3, 2, 4).contiguous()
            fin = torch.randn(4 * n * vh * nrhs * 2, generator=gen, device="cuda", dtype=torch.float32)
            fout = torch.empty_like(fin)
            keep += [gc, g12, fin, fout]
            segs.append({"lattice": L, "gauge": gc.data_ptr(), "gauge_two_row": g12.data_ptr(),
                         "in_": fin.data_ptr(), "out": fout.data_ptr(), "nrhs": nrhs, "antiperiodic_t": True})
            units += vh * nrhs
        h = stream.cuda_stream

        def batched():
            Q.dslash_segments(segs, n, 1, h)

        def separate():
            for sg in segs:
                Q.dslash_segments([sg], n, 1, h)

        res = {}
        for arm, fn in (("one_launch", batched), ("per_lattice", separate)):
            for _ in range(3):
                fn()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(reps):
                fn()
            e1.record(stream)
            torch.cuda.synchronize()
            ms = e0.elapsed_time(e1) / reps
            res[arm] = {"ms": round(ms, 4), "site_rhs_per_s": round(units / (ms * 1e-3))}
        res["speedup"] = round(res["per_lattice"]["ms"] / res["one_launch"]["ms"], 3)
        res["segments"] = len(mix)
        res["lattices"] = ["%s nrhs %d" % ("x".join(map(str, L)), r) for L, r in mix[:4]] + (
            ["..."] if len(mix) > 4 else [])
        out[name] = res
        del keep
    torch.cuda.empty_cache()
    return out


def serve_bench(torch, Q, n_requests=48, rates=(5.0, 10.0, 20.0, 60.0, 200.0), serial_budget_s=8.0):
    """Serving stream: the same seeded request set arriving by a Poisson
    process at each rate into a server with 4 resident gauges; p50/p99 latency
    and solves/s per rate, next to serial plain-FP64 solves of the same
    requests (one at a time, a bounded sample)."""
    from mrhs_qcu_gb300 import synthetic as S
    gauges = [((8, 8, 8, 8), 3), ((16, 16, 16, 32), 3), ((24, 24, 24, 48), 3), ((16, 16, 16, 32), 4)]
    srv = Q.Server(160 << 30, max_slots=24, inner_precision=Q.QCU_SINGLE_PRECISION)
    dgs = []
    for gid, (L, n) in enumerate(gauges):
        g, _ = make_inputs(torch, L, n, 1, seed_g=100 + gid)
        dgs.append(g)
        srv.add_gauge(gid, L, n, g.data_ptr(), antiperiodic_t=True)
    rng = np.random.default_rng(7)
    gaps = rng.exponential(1.0, n_requests)  # unit-rate Poisson gaps, scaled per rate
    reqs = []
    for i in range(n_requests):
        gid = int(rng.integers(len(gauges)))
        L, n = gauges[gid]
        nrhs = int(rng.integers(1, 25))
        kappa = float(rng.uniform(0.10, 0.125))
        tol = float(rng.choice([1e-8, 1e-10, 1e-12]))
        vh = S.half_volume(L)
        gen = torch.Generator(device="cuda").manual_seed(1000 + i)
        b = torch.complex(torch.randn((nrhs, 2, vh, 4, n), generator=gen, device="cuda", dtype=torch.float64),
                          torch.randn((nrhs, 2, vh, 4, n), generator=gen, device="cuda", dtype=torch.float64))
        x = torch.zeros_like(b)
        reqs.append((gid, kappa, tol, b, x))
    torch.cuda.synchronize()
    # warm-up: one request per gauge (kernel tuning, graph capture)
    for gid, (L, n) in enumerate(gauges):
        vh = S.half_volume(L)
        b = torch.ones((1, 2, vh, 4, n), dtype=torch.complex128, device="cuda")
        x = torch.zeros_like(b)
        srv.wait(srv.submit(gid, 0.11, 1e-8, [x[0].data_ptr()], [b[0].data_ptr()]))
    per_rate = []
    for rate in rates:
        for _, _, _, _, x in reqs:
            x.zero_()
        torch.cuda.synchronize()
        arrivals = np.cumsum(gaps / rate)
        ids = []
        t0 = time.perf_counter()
        for (gid, kappa, tol, b, x), t_arr in zip(reqs, arrivals):
            delay = t_arr - (time.perf_counter() - t0)
            if delay > 0:
                time.sleep(delay)
            ids.append(srv.submit(gid, kappa, tol, [x[r].data_ptr() for r in range(x.shape[0])],
                                  [b[r].data_ptr() for r in range(b.shape[0])]))
        infos = [srv.wait(i) for i in ids]
        wall = time.perf_counter() - t0
        lat = sorted(inf.latency_s for inf in infos)
        per_rate.append({
            "rate_req_s": rate, "p50_s": round(float(np.percentile(lat, 50)), 4),
            "p99_s": round(float(np.percentile(lat, 99)), 4), "mean_s": round(float(np.mean(lat)), 4),
            "queue_mean_s": round(float(np.mean([inf.queue_s for inf in infos])), 4),
            "solves_per_s": round(n_requests / wall, 2),
            "rhs_per_s": round(sum(r[3].shape[0] for r in reqs) / wall, 1), "wall_s": round(wall, 3),
            "all_ok": all(inf.status == 0 for inf in infos),
            "max_true_residual_over_tol": max(inf.max_true_residual / reqs[k][2] for k, inf in enumerate(infos))})
    mid = per_rate[len(per_rate) // 2]
    out = {"workload": "%d requests, Poisson arrivals at %s req/s, 4 resident gauges (8^4, 16^3x32, 24^3x48 "
                       "SU(3); 16^3x32 SU(4)), nrhs U[1,24], kappa U[0.10,0.125], tol {1e-8,1e-10,1e-12}, FP32 "
                       "inner + FP64 reliable updates" % (n_requests, "/".join("%g" % r for r in rates)),
           "rates": per_rate,
           "p50_s": mid["p50_s"], "p99_s": mid["p99_s"], "solves_per_s": mid["solves_per_s"],
           "all_ok": all(r["all_ok"] for r in per_rate)}
    srv.close()
    # serial plain FP64: each request alone through qcuInvert, a bounded sample
    t_ser, n_ser = 0.0, 0
    cur = None
    for gid, kappa, tol, b, x in reqs:
        if t_ser > serial_budget_s:
            break
        L, n = gauges[gid]
        if cur != gid:
            Q.initGridSize(L, n)
            Q.set_antiperiodic_t(True)
            Q.loadQcuGauge(dgs[gid].data_ptr())
            cur = gid
        x.zero_()
        p = Q.solver_params(kappa=kappa, tol=tol, inner_precision=Q.QCU_DOUBLE_PRECISION, max_iter=20000)
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        Q.invert([x[r].data_ptr() for r in range(x.shape[0])], [b[r].data_ptr() for r in range(b.shape[0])], p,
                 raise_on_error=False)
        torch.cuda.synchronize()
        t_ser += time.perf_counter() - t1
        n_ser += 1
    out["serial_fp64_solves_per_s"] = round(n_ser / t_ser, 2) if t_ser > 0 else None
    out["serial_fp64_sample"] = "%d of the %d requests, one at a time, plain FP64 CG" % (n_ser, n_requests)
    return out


TABLES = ("sweep", "solve", "serve", "multi_lattice", "colors")


def split_line(full):
    """The result line, short enough for a reader that keeps the last 3 KB of the output, and the tables that go to
    stderr: the line has the main figures of solve and serve under the same names."""
    line = {k: v for k, v in full.items() if k not in TABLES}
    tables = {k: full[k] for k in TABLES if full.get(k)}
    if "solve" in tables:
        t = tables["solve"]
        line["solve"] = {"workload": t["workload"],
                         "seconds": {k: v["seconds"] for k, v in t.items() if isinstance(v, dict)},
                         **{k: v for k, v in t.items() if k.startswith("speedup")},
                         "all_converged": all(v["all_converged"] for v in t.values() if isinstance(v, dict))}
    if "serve" in tables:
        t = tables["serve"]
        line["serve"] = {k: t.get(k) for k in ("p50_s", "p99_s", "solves_per_s", "serial_fp64_solves_per_s", "all_ok")}
    return line, tables


def run_reference(args):
    """The reference's CPU path for this operator: FP64 OpenMP restatement
    (the reference itself has no CPU implementation), all host threads."""
    world, rank, local, dist = dist_setup()
    if rank != 0:
        return
    from mrhs_qcu_gb300 import synthetic as S
    from oracle import oracle as O
    L, n, nrhs = L_BENCH, NC, NRHS
    g = S.random_gauge(L, n, seed=0)
    vh = S.half_volume(L)
    rng = np.random.default_rng(1)
    psi = (rng.standard_normal((1, vh, 4, n)) + 1j * rng.standard_normal((1, vh, 4, n))) * np.sqrt(0.5)
    for _ in range(args.warmup):
        O.dslash(psi, g, L, 0, 0, True)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        O.dslash(psi, g, L, 0, 0, True)
    dt = (time.perf_counter() - t0) / args.steps
    value = vh / dt
    line = {"impl": "reference", "metric": METRIC,
            "value": value, "unit": "site*RHS/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": round(dt * 1e3, 3), "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic (seeded SU(3) links, Gaussian spinors)",
            "config": workload_config(L, n, nrhs, world, "fp64"),
            "cpu_baseline": {"value": value, "unit": "site*RHS/s", "cores": O.num_threads(), "kind": "port",
                             "sample": "one RHS of the 32^3x64 SU(3) workload per step (1/12 of a step), FP64"},
            "e2e": {"value": value, "unit": "site*RHS/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


def profile_solve(inner):
    """The config-2 solve alone: one cold solve (tuning, graph capture), then
    a warm one inside the NVTX range 'warm_solve'; prints its wall time."""
    import torch

    import mrhs_qcu_gb300 as Q
    from mrhs_qcu_gb300 import synthetic as S
    L, n, nrhs, kappa = (24, 24, 24, 48), 3, 12, 0.12
    g_dev, _ = make_inputs(torch, L, n, 1, seed_g=5)
    b = S.point_sources(L, n, nrhs, seed=6)
    db = [torch.from_numpy(b[r]).cuda() for r in range(nrhs)]
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    Q.loadQcuGauge(g_dev.data_ptr())
    for phase in ("cold", "warm"):
        dx = [torch.zeros_like(x) for x in db]
        p = Q.solver_params(kappa=kappa, tol=1e-10, inner_precision=inner, max_iter=20000)
        torch.cuda.synchronize()
        if phase == "warm":
            torch.cuda.nvtx.range_push("warm_solve")
        t0 = time.perf_counter()
        Q.invert([x.data_ptr() for x in dx], [x.data_ptr() for x in db], p, raise_on_error=False)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
        if phase == "warm":
            torch.cuda.nvtx.range_pop()
        print(json.dumps({"solve": phase, "inner_precision": inner, "seconds": round(dt, 4),
                          "iterations": p.iterations, "reliable_updates": p.reliable_updates}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--skip-sweep", action="store_true")
    ap.add_argument("--skip-solve", action="store_true")
    ap.add_argument("--skip-serve", action="store_true")
    ap.add_argument("--skip-colors", action="store_true")
    ap.add_argument("--skip-cpu", action="store_true")
    ap.add_argument("--skip-e2e", action="store_true")
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--lattice", default="32,32,32,64", help="X,Y,Z,T of the headline workload")
    ap.add_argument("--nrhs", type=int, default=NRHS)
    ap.add_argument("--ncolors", type=int, default=NC, help="N of SU(N) for the headline kernel (profiling)")
    ap.add_argument("--precision", type=int, default=1, help="0 fp16, 1 fp32, 2 fp64, 4 bf16")
    ap.add_argument("--profile", action="store_true",
                    help="headline kernel only (no e2e, sweep, CPU or solve legs), for ncu captures")
    ap.add_argument("--profile-solve", type=int, default=None, metavar="INNER",
                    help="only the 24^3x48 mixed solve with this inner precision (0 fp16, 1 fp32, 2 fp64): "
                         "a cold solve, then a warm one inside the NVTX range 'warm_solve', for ncu captures")
    args = ap.parse_args()
    if args.profile_solve is not None:
        profile_solve(args.profile_solve)
        return
    if args.profile:
        args.skip_sweep = args.skip_solve = args.skip_serve = args.skip_colors = args.skip_cpu = True
        args.skip_e2e = True
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference(args)
    else:
        run_gpu(args)


if __name__ == "__main__":
    main()
