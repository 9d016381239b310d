#!/usr/bin/env python
"""Benchmark: filtered stochastic orbitals/s on the 512-atom Si workload.

One step = one Chebyshev Fermi-operator filter (order L) of the rank's
stochastic orbitals plus their density contribution (the unit of the
metric: one orbital taken through all L polynomial steps incl. its share of
H.psi, accumulation and density).  Default workload: 4x4x4 Si supercell
(512 atoms, a = 41.04 bohr), 96^3 grid, 512 orbitals, L = 512, mixed
precision; mu from FP64 bisection on the Chebyshev moments of the same
noise (setup, untimed).  Inputs are synthetic (seeded), larger than L2.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Multi-GPU (torchrun): every rank filters its own 512 orbitals (state
parallel, weak scaling); the density is summed across ranks with one NCCL
all-reduce per step.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

PEAKS_FALLBACK = {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0}


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return d, "measured"
    return PEAKS_FALLBACK, "fallback"


class Clocks:
    """nvidia-smi sampler running during the timed region."""

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except FileNotFoundError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, reasons, power = [], None, set(), []
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax = float(f[2])
                power.append(float(f[3]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        load = [x for x in sm if x > 0.5 * (smax or 1)] or sm
        return {"sm_mhz": statistics.median(load) if load else None, "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples": len(sm),
                "power_w_max": max(power) if power else None}


def setup_system(cfg_name, rank):
    import __graft_entry__ as g
    wl = g.load_workload()
    cfg = wl.CONFIGS[cfg_name]
    s = wl.make_system(cfg["nrep"], cfg["grid"])
    return wl, cfg, s


def algorithmic(kind, s, nsto, csz, digits):
    """Compulsory bytes (or flops) of one launch of `kind` over nsto orbitals
    (digits: the KB GEMMs are INT8 digit GEMMs, not FP64).

    stage A: read the orbitals (16 B/coef) + write the column scratch;
    stage B: read + write the column scratch + V_KS once;
    stage C: read the scratch, c and T_{k-2}, write T_k (FP64 orbitals);
    read FNL (FP32 from the digit GEMMs, FP64 otherwise); the filter sum is
    read and written every other step (one orbital block per step on
    average); it also packs the next step's columns (write one column scratch)
    in place of a stage A launch;
    GEMMs: 2*P*nsto*2*ncoef flops."""
    npairs = (nsto + 1) // 2
    n1, n2, n3 = s["grid"]
    ncoef = s["ncoef"]
    ncols = s["_ncols"]
    xb = npairs * n3 * ncols * csz
    vec = nsto * ncoef * 16
    if kind == "stage_a_pack_cfft":
        return "hbm", vec + xb
    if kind == "stage_b_plane_fft_vks":
        return "hbm", 2 * xb + n1 * n2 * n3 * (csz // 2)
    if kind == "stage_c_cfft_unpack_recur":
        return "hbm", 2 * xb + (4.5 if digits else 5) * vec
    if kind in ("kb_proj_gemm", "kb_back_gemm"):
        return "tensor", 2.0 * s["_P"] * nsto * 2 * ncoef
    if kind == "density_planes":
        return "hbm", xb + npairs * n1 * n2 * n3 * 8
    return "hbm", None


# DRAM bytes from ncu captures (profiles/): kf_stage_b<float,96,96> and
# kf_stage_c<float,96,8,0> per orbital pair (136.5 + 73.6 MB, and the mean of
# 509.1 + 303.9 and 401.9 + 203.6 MB with and without the filter sum, for 64
# pairs, scaled by pairs); the KB GEMMs
# per launch at 512 orbitals (full-size capture, mean of the projection
# 1.14 GB + 63.8 MB and the back projection 865.8 + 398.0 MB)
PROFILED_TRAFFIC = {("kf_stage_b", (96, 96, 96), True): (136.5e6 + 73.6e6) / 64,
                    ("kf_stage_c", (96, 96, 96), True): (509.1e6 + 303.9e6 + 401.9e6 + 203.6e6) / 128}
PROFILED_GEMM_TRAFFIC = {((96, 96, 96), True, 512): (1.14e9 + 63.8e6 + 865.8e6 + 398.0e6) / 2}

# What bounds the HBM-class kernels that sit well below the copy bandwidth,
# from their ncu captures (profiles/)
PROFILED_LIMITER = {
    "kf_stage_b": "shared-memory pipe (l1tex 76.6 % of peak, issue 67 %; ten plane-sized shared passes per plane)",
    "kf_stage_c": "latency (long-scoreboard stalls lead, then barriers; DRAM 54 to 60 % on a 64-pair capture)",
}

KERNEL_OF = {"stage_a_pack_cfft": "kf_stage_a", "stage_b_plane_fft_vks": "kf_stage_b",
             "stage_c_cfft_unpack_recur": "kf_stage_c", "kb_proj_gemm": "kb_gemm", "kb_back_gemm": "kb_gemm",
             "density_planes": "kf_density"}


def fp64_gemm_peak(local):
    """Measured FP64 tensor-core (DMMA) rate of this GPU: cuBLAS DGEMM
    (torch.matmul, float64) 8192^3, best of 5 by CUDA events; TFLOP/s."""
    import torch
    dev = f"cuda:{local}"
    n = 8192
    a = torch.randn(n, n, dtype=torch.float64, device=dev)
    b = torch.randn(n, n, dtype=torch.float64, device=dev)
    torch.matmul(a, b)
    best = None
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        torch.matmul(a, b)
        e1.record()
        e1.synchronize()
        ms = e0.elapsed_time(e1)
        best = ms if best is None else min(best, ms)
    del a, b
    return 2.0 * n ** 3 / (best * 1e-3) / 1e12


def rooflines(timing, s, nsto, mixed, back_products=10, fp64_peak=None, digits=None):
    """Roofline of every kernel function with an algorithmic model, largest
    total time first.  Tensor: the KB GEMMs (projection and back projection,
    one kernel) -- digit GEMMs (digits; mixed contexts with enough projection work): int8 tcgen05 ops (10 digit products per FP64-
    equivalent multiply-add) against 2 x the measured bf16 burst peak (B200's
    dense int8 rate is twice its bf16 rate); FP64: DMMA flops against the
    FP64 tensor (DMMA) rate measured by fp64_gemm_peak (fp64_peak), else the
    nominal 40 TFLOP/s.  HBM: algorithmic bytes (algorithmic())
    against the measured copy bandwidth.  back_products: int8 digit products
    of the back projection (10, or 6 with the 24-bit digits of mixed_fast)."""
    pk, src = peaks()
    csz = 8 if mixed else 16
    digits = mixed if digits is None else digits
    agg = {}
    for kind, (ms, n) in timing.items():
        kern = KERNEL_OF.get(kind)
        if kern is None or n == 0:
            continue
        bound, work = algorithmic(kind, s, nsto, csz, digits)
        a = agg.setdefault(kern, [bound, 0.0, 0, 0.0, 0.0])
        a[1] += ms
        a[2] += n
        a[3] += work * n
        if bound == "tensor":  # int8 products executed
            a[4] += work * n * (back_products if kind == "kb_back_gemm" else 10)
    out = []
    for kern, (bound, ms, n, work, ops8) in sorted(agg.items(), key=lambda kv: -kv[1][1]):
        t = ms / 1e3
        if bound == "hbm":
            ach = work / t / 1e9
            peak = pk["hbm_gbs"]
            tr = PROFILED_TRAFFIC.get((kern, tuple(s["grid"]), mixed))
            out.append({"kernel": kern, "bound": "hbm", "achieved": ach, "peak": peak, "unit": "GB/s",
                        "frac": ach / peak, "traffic": tr * ((nsto + 1) // 2) if tr else None,
                        "peak_source": src, "ms_total": ms, "launches": n})
            if kern in PROFILED_LIMITER:
                out[-1]["limiter"] = PROFILED_LIMITER[kern]
        else:
            if digits:
                ach = ops8 / t / 1e12
                peak = 2.0 * pk["bf16_tflops"]
                psrc = f"int8 dense = 2 x {src} bf16 burst ({pk['bf16_tflops']})"
                name = "kb_gemm (k_gemm_oz8, int8 tcgen05)"
            else:
                ach = work / t / 1e12
                peak = fp64_peak or 40.0
                psrc = ("measured cuBLAS DGEMM 8192^3 (torch.matmul float64, best of 5) on this GPU"
                        if fp64_peak else "nominal FP64 tensor (DMMA) rate")
                name = "kb_gemm (k_gemm_nt_f64, DMMA)"
            out.append({"kernel": name, "bound": "tensor", "achieved": ach, "peak": peak, "unit": "TFLOP/s",
                        "frac": ach / peak, "traffic": PROFILED_GEMM_TRAFFIC.get((tuple(s["grid"]), digits, nsto)),
                        "peak_source": psrc, "ms_total": ms, "launches": n,
                        "fp64_equivalent_tflops": work / t / 1e12})
            if digits and pk.get("bf16_tflops_sustained"):
                # the same against the sustained bf16 loop (its clocks sat near 1.33 GHz under the
                # power cap; this step runs near 1.75-1.8 GHz, so the burst figure is the stricter one)
                out[-1]["frac_vs_sustained"] = ach / (2.0 * pk["bf16_tflops_sustained"])
    return out


def ncols_of(s):
    ka, kb = s["ka"][:-1], s["kb"][:-1]
    cols = set(zip(ka.tolist(), kb.tolist()))
    return 2 * len([c for c in cols if c != (0, 0)]) + 1


def run_ours(args):
    import torch
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
    torch.cuda.set_device(local)
    import __graft_entry__ as g
    pkg = g.load_package()
    wl, cfg, s = setup_system(args.config, rank)
    s["_ncols"] = ncols_of(s)
    s["_P"] = 4 * s["natm"]
    nsto = cfg["nsto"] if args.nsto is None else args.nsto
    L = cfg["L"] if args.L is None else args.L
    prec = {"mixed": pkg.SDFT_PREC_MIXED, "mixed_fast": pkg.SDFT_PREC_MIXED_FAST, "fp64": pkg.SDFT_PREC_FP64}[args.prec]
    ctx = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=prec, max_states=nsto, device=local)
    ctx.set_vks(s["vks"])
    ctx.set_kb(s["kb_desc"])
    if args.plane_threads != "tuned" and prec != pkg.SDFT_PREC_FP64:
        ctx.set_plane_threads(int(args.plane_threads))
    t0 = time.time()
    emin, emax = ctx.lanczos_bounds(20, seed=15, margin=0.1)[:2]  # 20 device Lanczos steps
    ediff, emean = emax - emin, 0.5 * (emin + emax)
    scale = 2.0 / ediff
    # noise of this state rank (np_states = world): host copy kept for the e2e leg
    t1 = time.time()
    chi_h = ctx.genNoiseOrbitalReal(nsto, seed=10.0, np_states=world, myid=rank)
    noise_s = time.time() - t1
    # launch shapes from the autotuner (tile width and split-K of the KB GEMMs,
    # plane-stage CTA size), timed on these resident noise orbitals
    tuned = None
    if args.plane_threads == "tuned" and prec != pkg.SDFT_PREC_FP64:
        tn = __import__(pkg.__name__ + ".tuner", fromlist=["Tuner"]).Tuner(pkg)
        tn.tune(ctx, nsto, s["_P"], scale, emean)
        entry = tn.cache[tn.key(ctx, nsto, s["_P"])]
        tuned = {"gemm_bn": entry.get("gemm_bn"), "gemm_split": entry["split"],
                 "plane_threads": entry.get("plane_threads")}
    # chemical potential from the moments (calcChemPotCheby), summed over ranks
    states = __import__(pkg.__name__ + ".states", fromlist=["StateGroup"])
    grp = states.StateGroup(dist, device=f"cuda:{local}")
    mom = ctx.moments_dev(nsto, L, scale, emean)
    mu, ne = grp.chem_pot(pkg, mom, nsto * world, L, ediff, emean, wl.BETA, wl.OCC, s["num_elec"], 0.2, 0.05)
    ec = pkg.calcChebyCoeff(L, ediff, emean, wl.BETA, mu, fun_flag=2)
    setup_s = time.time() - t0
    occ_over = wl.OCC / (nsto * world)
    ext = torch.cuda.ExternalStream(pkg.lib.sdft_ctx_stream(ctx._p), device=f"cuda:{local}")
    rho_t = torch.zeros(int(np.prod(s["grid"])), dtype=torch.float64, device=f"cuda:{local}")

    def step():
        ctx.filter_cheby_dev(nsto, ec, 1, scale, emean)
        if dist:
            # this rank's density into a device buffer, then the path's one
            # exchange step: the sum of the density over the state ranks
            ctx.density_dev(nsto, 0, occ_over, out_ptr=rho_t.data_ptr())
            grp.sum_tensor_(rho_t)
        else:
            ctx.density_dev(nsto, 0, occ_over, want=False)

    for _ in range(args.warmup):
        step()
    ctx.sync()
    launches0 = ctx.launches
    ctx.read_timing()
    ctx.set_timing(True)
    clk = Clocks(local)
    if rank == 0:
        clk.start()
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    ctx.sync()
    evs = []
    cur = torch.cuda.current_stream()
    for _ in range(args.steps):
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        a.record(ext)
        step()
        if dist:
            b.record(cur)  # after the all-reduce (the current stream waits for NCCL)
        else:
            b.record(ext)
        evs.append((a, b))
    ctx.sync()
    torch.cuda.synchronize()
    step_ms = [a.elapsed_time(b) for a, b in evs]
    tot_ms = sum(step_ms)
    if dist:
        t = torch.tensor([tot_ms], device=f"cuda:{local}")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        tot_ms = float(t.item())
    clocks = None
    launches = ctx.launches - launches0
    timing = ctx.read_timing()
    ctx.set_timing(False)
    eager = {"orbitals_per_s": args.steps * nsto * world / (tot_ms / 1e3), "ms_per_step": tot_ms / args.steps,
             "launches_per_step": launches / args.steps, "note": "per-kernel event timing on"}
    # ---- the same step as one CUDA-graph launch (sdft_batch of this context);
    # the small configurations are launch-bound when issued kernel by kernel
    graph = None
    if world == 1 and not args.no_graph:
        bt = pkg.Batch([ctx], [nsto], [L], [ec], [scale], [emean], [occ_over])
        gst = torch.cuda.ExternalStream(bt.stream_ptr, device=f"cuda:{local}")
        for _ in range(args.warmup):
            bt.launch()
        bt.sync()
        gevs = []
        for _ in range(args.steps):
            a = torch.cuda.Event(enable_timing=True)
            b = torch.cuda.Event(enable_timing=True)
            a.record(gst)
            bt.launch()
            b.record(gst)
            gevs.append((a, b))
        bt.sync()
        g_ms = [a.elapsed_time(b) for a, b in gevs]
        graph = {"ms": g_ms, "kernels_per_launch": bt.kernels_per_launch}
        bt.close()
    if rank == 0:
        clocks = clk.stop()
    if graph:
        step_ms = graph["ms"]
        tot_ms = sum(step_ms)
        launches = graph["kernels_per_launch"] * args.steps
    value = args.steps * nsto * world / (tot_ms / 1e3)

    # ---- e2e: the public host-buffer API, H2D of chi and D2H of results
    e2e = None
    if not args.no_e2e:
        pin = lambda n: torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
        chi_re, chi_im = pin(nsto * s["ncoef"]), pin(nsto * s["ncoef"])
        chi_re[:] = chi_h[0]
        chi_im[:] = chi_h[1]
        out_re, out_im = pin(nsto * s["ncoef"]), pin(nsto * s["ncoef"])
        rho_h = pin(int(np.prod(s["grid"])))
        import ctypes as C
        dp = C.POINTER(C.c_double)
        pr = (dp * 1)(out_re.ctypes.data_as(dp))
        pi = (dp * 1)(out_im.ctypes.data_as(dp))
        ecd = np.ascontiguousarray(ec)

        def e2e_step():
            rc = pkg.lib.sdft_filter_cheby(ctx._p, nsto, chi_re.ctypes.data_as(dp), chi_im.ctypes.data_as(dp), L, 1,
                                           ecd.ctypes.data_as(dp), scale, emean, pr, pi, None)
            pkg._chk(rc)
            pkg._chk(pkg.lib.sdft_density_dev(ctx._p, nsto, 0, occ_over, rho_h.ctypes.data_as(dp)))

        e2e_step()
        if dist:
            dist.barrier()
        ks = max(1, min(args.steps, 2))
        t1 = time.perf_counter()
        for _ in range(ks):
            e2e_step()
        el = time.perf_counter() - t1
        if dist:
            t = torch.tensor([el], device=f"cuda:{local}")
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            el = float(t.item())
        e2e = {"value": ks * nsto * world / el, "unit": "orbitals/s",
               "h2d_bytes_per_step": 2 * nsto * s["ncoef"] * 8,
               "d2h_bytes_per_step": 2 * nsto * s["ncoef"] * 8 + int(np.prod(s["grid"])) * 8}
        launches_e2e = None

    # ---- FP64 arm and accuracy of the mixed arm (rank 0 data)
    fp64 = None
    if prec != pkg.SDFT_PREC_FP64 and not args.no_fp64:
        c64 = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=pkg.SDFT_PREC_FP64,
                          max_states=nsto, device=local)
        c64.set_vks(s["vks"])
        c64.set_kb(s["kb_desc"])
        c64.upload(*chi_h)
        ctx.upload(*chi_h)
        # timed the same way as the mixed step (one graph launch, or eager)
        if graph:
            b64 = pkg.Batch([c64], [nsto], [L], [ec], [scale], [emean], [occ_over])
            ext64 = torch.cuda.ExternalStream(b64.stream_ptr, device=f"cuda:{local}")
            run64 = b64.launch
        else:
            b64 = None
            ext64 = torch.cuda.ExternalStream(pkg.lib.sdft_ctx_stream(c64._p), device=f"cuda:{local}")

            def run64():
                c64.filter_cheby_dev(nsto, ec, 1, scale, emean)
                c64.density_dev(nsto, 0, occ_over, want=False)
        run64()  # warm-up
        c64.sync()
        if b64:
            b64.sync()
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        a.record(ext64)
        run64()
        b.record(ext64)
        if b64:
            b64.sync()
            b64.close()
        c64.sync()
        ms64 = a.elapsed_time(b)
        # the FP64 step once more, issued eagerly with per-kernel event timing:
        # the kernel table and rooflines of the plain form (the denominator of
        # the mixed speed-up), its DMMA GEMM against the measured DGEMM rate
        c64.read_timing()
        c64.set_timing(True)
        c64.filter_cheby_dev(nsto, ec, 1, scale, emean)
        c64.density_dev(nsto, 0, occ_over, want=False)
        c64.sync()
        t64 = c64.read_timing()
        c64.set_timing(False)
        f64peak = fp64_gemm_peak(local)
        roof64 = rooflines(t64, s, nsto, False, fp64_peak=f64peak)
        tot64 = max(1e-9, sum(x[0] for x in t64.values()))
        ktab64 = {k: {"ms_total": v[0], "launches": v[1], "share": v[0] / tot64} for k, v in t64.items() if v[1]}
        rho64 = c64.density_dev(nsto, 0, occ_over)
        ctx.filter_cheby_dev(nsto, ec, 1, scale, emean)
        rhom = ctx.density_dev(nsto, 0, occ_over)
        fr, fi = c64.download_filtered(nsto)
        mr, mi = ctx.download_filtered(nsto)
        # energy of the filtered orbitals: occ/Nsto sum_s <psi_s|H|psi_s> (H from the FP64 context)
        def band_energy(cr, ci):
            e = 0.0
            nc = s["ncoef"]
            for k in range(0, nsto, 64):
                sl = slice(k * nc, min(nsto, k + 64) * nc)
                hr, hi = c64.calc_coef_force(cr[sl], ci[sl])
                hr, hi = -0.25 * hr, -0.25 * hi
                ns = (sl.stop - sl.start) // nc
                hr2 = hr.reshape(ns, nc)
                hr2[:, -1] *= 2.0
                e += sum(wl.half_dot(nc, cr[sl].reshape(ns, nc)[j], ci[sl].reshape(ns, nc)[j], hr2[j],
                                     hi.reshape(ns, nc)[j]) for j in range(ns))
            return e * wl.OCC / (nsto * world)
        e64, em = band_energy(fr, fi), band_energy(mr, mi)

        # nonlocal atomic forces of the same filtered orbitals (calcEnergyForce's
        # KB part: four projection GEMMs), device time of one call per precision
        def force_ms(c):
            st = torch.cuda.ExternalStream(pkg.lib.sdft_ctx_stream(c._p), device=f"cuda:{local}")
            c.nl_force_dev(nsto, 0, occ=wl.OCC, nsto_total=nsto * world)  # warm-up (allocates Z scratch)
            ea, eb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            ea.record(st)
            f, _ = c.nl_force_dev(nsto, 0, occ=wl.OCC, nsto_total=nsto * world)
            eb.record(st)
            eb.synchronize()
            return f, ea.elapsed_time(eb)
        f64f, fms64 = force_ms(c64)
        fmxf, fmsmx = force_ms(ctx)
        # four projections (c and i G_d c, d = x, y, z), each 2 P S (2 ncoef) FP64-equivalent flops;
        # digit GEMMs execute 10 int8 products per FP64-equivalent multiply-add
        pk, psrc = peaks()
        f_flops = 4 * 2.0 * s["_P"] * nsto * 2 * s["ncoef"]
        nl_force = {"natm": int(f64f.shape[0]), "ms_fp64": fms64, "ms_mixed": fmsmx,
                    "max_abs_err_mixed_vs_fp64_over_max_force":
                        float(np.abs(fmxf - f64f).max() / max(1e-300, np.abs(f64f).max())) if f64f.size else 0.0,
                    "fp64_equiv_tflops_mixed": f_flops / (fmsmx * 1e-3) / 1e12}
        if ctx.digit_gemms:
            nl_force.update(
                frac_of_int8_peak_mixed=10.0 * f_flops / (fmsmx * 1e-3) / 1e12 / (2.0 * pk["bf16_tflops"]),
                peak_source=f"int8 dense = 2 x {psrc} bf16 burst ({pk['bf16_tflops']})")
        fp64 = {"orbitals_per_s": nsto * world / (ms64 / 1e3), "ms_per_step": ms64,
                "mixed_speedup": (nsto * world / (ms64 / 1e3)) and value / (nsto * world / (ms64 / 1e3)),
                "density_rel_l2_mixed_vs_fp64": float(np.linalg.norm(rhom - rho64) / np.linalg.norm(rho64)),
                "band_energy_fp64": e64, "band_energy_mixed": em,
                "energy_rel_err_mixed_vs_fp64": abs(em - e64) / abs(e64),
                "num_elec_density": float(rho64.sum() / rho64.size), "nl_force": nl_force,
                "kernels": ktab64, "roofline_kernels": roof64, "fp64_dgemm_tflops_measured": f64peak}
        c64.close()

    # ---- roofline: per kernel function, the dominant one first
    roof_all = rooflines(timing, s, nsto, prec != pkg.SDFT_PREC_FP64,
                         back_products=6 if prec == pkg.SDFT_PREC_MIXED_FAST else 10, digits=ctx.digit_gemms)
    roof = roof_all[0] if roof_all else None
    kernel_table = {k: {"ms_total": v[0], "launches": v[1], "share": v[0] / max(1e-9, sum(x[0] for x in
                    timing.values()))} for k, v in timing.items() if v[1]}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:  # reported at N=1 only
        cpu = cpu_baseline(s, nsto, L, scale, emean, ec, args)
    lat = sorted(step_ms)
    out = {
        "metric": "filtered stochastic orbitals/s (512-atom Si, mixed vs FP64 GPU); p50/p99 latency",
        "value": value, "unit": "orbitals/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": tot_ms / args.steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": ("f64" if prec == pkg.SDFT_PREC_FP64 else
                  "mixed(fp32 fft, fp64 kb gemm, fp64 recurrence)" if not ctx.digit_gemms else
                  "mixed(fp32 fft, int8-ozaki kb gemm, fp64 recurrence)" if prec == pkg.SDFT_PREC_MIXED else
                  "mixed_fast(fp32 fft, int8-ozaki kb gemm with 24-bit back projection, fp64 recurrence)"),
        "data": "synthetic (seeded Si supercell, Gaussian V_loc, Gaussian s+p KB, +-1 noise)",
        "config": {"workload": f"{args.config}: {s['natm']}-atom Si, grid {s['grid'][0]}x{s['grid'][1]}x{s['grid'][2]}, "
                               f"{nsto} orbitals/GPU, Chebyshev L={L}, ncoef={s['ncoef']}, P={s['_P']}",
                   "orbitals_per_gpu": nsto, "L": L, "precision": args.prec, "mu": mu, "num_elec": ne,
                   "emin": emin, "emax": emax, "l2": "inputs (orbitals 0.43 GB/GPU) larger than L2; no flush",
                   "setup_s": setup_s, "noise_host_s": noise_s, "parallelism": f"state-parallel x{world}",
                   "launch_shapes": tuned if tuned is not None else f"plane threads {args.plane_threads}"},
        "latency_ms": {"p50": lat[len(lat) // 2], "p99": lat[min(len(lat) - 1, int(math.ceil(0.99 * len(lat))) - 1)]},
        "e2e": e2e, "gpu_launches": launches, "roofline": roof, "roofline_kernels": roof_all,
        "kernels": kernel_table, "eager": eager, "step_launch": "one CUDA graph" if graph else "eager", "fp64": fp64,
        "cpu_baseline": cpu, "clocks": clocks,
    }
    ctx.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if rank == 0:
        print(json.dumps(out))


def _workload_standalone():
    """workload.py (the seeded synthetic Si builder; numpy only) loaded on
    its own, without the package, so that the reference's CPU arm maps none
    of the product's libraries."""
    import importlib.util
    name = "sdft_synthetic_si"
    if name in sys.modules:
        return sys.modules[name]
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)),
                        "stochastic-density-functional-theory-piny_b200", "workload.py")
    spec = importlib.util.spec_from_file_location(name, path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    sys.modules[name] = mod
    return mod


def _ref_gvec(hmat, ecut, kmax):
    """The half G sphere from the reference's own setkvec3d_sm (oracle/_ref),
    its length counted by the oracle; the oracle's list where the reference
    build is absent."""
    from oracle import oracle as O
    from oracle import ref as R
    og = O.gvec(hmat, ecut, kmax)
    return R.gvec(hmat, ecut, kmax, len(og[0])) if R.available() else og


def ref_setup_system(cfg_name):
    """setup_system for the reference arm: the same seeded workload, built
    without the product library."""
    wl = _workload_standalone()
    cfg = wl.CONFIGS[cfg_name]
    return wl, cfg, wl.make_system(cfg["nrep"], cfg["grid"], gvec=_ref_gvec)


def _ref_worker_init(cfg_name):
    """Worker of the reference CPU arm: silence the reference's own timer
    printouts (stdout) and build the system once."""
    devnull = os.open(os.devnull, os.O_WRONLY)
    os.dup2(devnull, 1)
    global _W
    wl, _, s = ref_setup_system(cfg_name)
    _W = {"s": s, "wl": wl}


def _ref_worker_run(task):
    """k Chebyshev steps of 2 orbitals through the reference's own compiled
    filterChebyPolyHerm (oracle/_ref); returns seconds."""
    seed, k, scale, emean, ec, kind = task
    s = _W["s"]
    nc = s["ncoef"]
    rng = np.random.default_rng(seed)
    cr = rng.standard_normal(2 * nc)
    ci = rng.standard_normal(2 * nc)
    ci.reshape(2, nc)[:, -1] = 0.0
    if kind == "reference":
        from oracle import ref as R
        r = R.RefSys(s, 2)
        t = time.perf_counter()
        r.filter(True, cr, ci, np.asarray(ec[:k + 1]), 1, scale, emean)
    else:
        from oracle import oracle as O
        r = O.OracleSys(s)
        t = time.perf_counter()
        r.filter_cheby(cr, ci, np.asarray(ec[:k + 1]), 1, scale, emean)
    return time.perf_counter() - t


class RefCpu:
    """The reference's CPU path on all host cores: one process per core, each
    filtering its own 2 orbitals (the reference spreads stochastic orbitals
    over MPI ranks, filter.c / gen-stodft-wf.c), k polynomial steps per
    call, extrapolated linearly to order L."""

    def __init__(self, cfg_name, cores=None):
        import multiprocessing as mp
        from oracle import ref as R
        self.kind = "reference" if R.available() else "port"
        self.cores = cores or len(os.sched_getaffinity(0))
        self.pool = mp.get_context("spawn").Pool(self.cores, initializer=_ref_worker_init, initargs=(cfg_name,))

    def rate(self, L, k, scale, emean, ec, seed0=0):
        tasks = [(seed0 + i, k, scale, emean, list(ec[:k + 1]), self.kind) for i in range(self.cores)]
        secs = self.pool.map(_ref_worker_run, tasks)
        return sum(2.0 / (t * L / k) for t in secs)

    def close(self):
        self.pool.close()
        self.pool.join()


def cpu_baseline(s, nsto, L, scale, emean, ec, args):
    """Reference CPU path (oracle/_ref, else the oracle port) timed on every
    host core on a bounded sample: 2 orbitals x k steps per core."""
    try:
        rc = RefCpu(args.config)
        try:
            k = args.cpu_steps
            v = rc.rate(L, k, scale, emean, ec)
        finally:
            rc.close()
        return {"value": v, "unit": "orbitals/s", "cores": rc.cores, "kind": rc.kind,
                "sample": f"{rc.cores} processes x 2 orbitals x {k} Chebyshev steps of {args.config}, "
                          f"extrapolated linearly to L={L}"}
    except Exception as e:  # the baseline is reported, never required
        return {"value": None, "unit": "orbitals/s", "cores": None, "kind": "reference", "sample": f"failed: {e}"}


def run_reference(args):
    """--impl reference: the reference's own CPU implementation of the path
    (its C sources compiled into oracle/_ref) on all host cores, same metric
    and workload; each step is a bounded sample (k polynomial steps of two
    orbitals per core, extrapolated to the full order L)."""
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    if rank != 0:
        return
    # nothing of the product is loaded on this arm: the workload comes from
    # the numpy builder with the reference's setkvec3d_sm, the coefficients
    # from the reference's calcChebyCoeff (stodft/coeff.c:1093), both in oracle/_ref
    from oracle import oracle as O
    from oracle import ref as R
    wl, cfg, s = ref_setup_system(args.config)
    nsto = cfg["nsto"] if args.nsto is None else args.nsto
    L = cfg["L"] if args.L is None else args.L
    # spectral window and coefficients as the GPU arm uses (Lanczos bounds of
    # this workload; mu only changes coefficient values, not the cost)
    emin, emax = -0.9735, 9.8349
    ediff, emean = emax - emin, 0.5 * (emin + emax)
    scale = 2.0 / ediff
    ec = (R.cheby_coeff(L, ediff, emean, wl.BETA, -0.677, 2) if R.available()
          else O.cheby_coeff(L, ediff, emean, wl.BETA, -0.677, 2))
    rc = RefCpu(args.config)
    k = args.cpu_steps
    vals, ms = [], []
    try:
        for i in range(args.warmup + args.steps):
            t = time.perf_counter()
            v = rc.rate(L, k, scale, emean, ec, seed0=100 * i)
            if i >= args.warmup:
                vals.append(v)
                ms.append(1e3 * (time.perf_counter() - t))  # the sample's own wall time
    finally:
        rc.close()
    v = statistics.median(vals)
    out = {"impl": "reference",
           "metric": "filtered stochastic orbitals/s (512-atom Si, mixed vs FP64 GPU); p50/p99 latency",
           "value": v, "unit": "orbitals/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
           "ms_per_step": statistics.median(ms), "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "f64", "data": "synthetic (seeded Si supercell, Gaussian V_loc, Gaussian s+p KB, random orbitals)",
           "config": {"workload": f"{args.config}: {s['natm']}-atom Si, grid {s['grid'][0]}x{s['grid'][1]}x{s['grid'][2]}, "
                                  f"{nsto} orbitals, Chebyshev L={L}, ncoef={s['ncoef']}, P={4 * s['natm']}",
                      "orbitals": nsto, "L": L, "implementation": "reference C sources (filter.c, normh.c, "
                      "energy-wrapper-scf.c, cp-energy-*-stodft.c, fft_package.c ...) compiled in oracle/_ref",
                      "fft": "project mixed-radix FFT behind the FFTW API (FFTW absent)"},
           "cpu_baseline": {"value": v, "unit": "orbitals/s", "cores": rc.cores, "kind": rc.kind,
                            "sample": f"per step {rc.cores} processes x 2 orbitals x {k} Chebyshev steps, "
                                      f"extrapolated linearly to L={L}"},
           "step": (f"one bounded sample ({rc.cores} x 2 orbitals x {k} steps); ms_per_step is its wall time, "
                    f"value the rate extrapolated to the full order (the full {nsto}-orbital step would take "
                    f"{nsto / v:.0f} s)"),
           "e2e": {"value": v, "unit": "orbitals/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(out))


def _modules(pkg):
    serve = __import__(pkg.__name__ + ".serve", fromlist=["prepare"])
    tuner = __import__(pkg.__name__ + ".tuner", fromlist=["Tuner"])
    return serve, tuner


def run_batch(args):
    """Batched uneven systems: 32 seeded Si supercells (8..216 atoms, +-2 %
    strain, 0.05 bohr displacements, grids 24..72 per axis, 16..256 orbitals,
    order 128..512), mixed precision, split-K per system from the autotuner,
    all filters + densities in one CUDA graph replayed with one launch."""
    import torch
    import __graft_entry__ as g
    pkg = g.load_package()
    wl = g.load_workload()
    serve, tuner_mod = _modules(pkg)
    prec = {"mixed": pkg.SDFT_PREC_MIXED, "mixed_fast": pkg.SDFT_PREC_MIXED_FAST, "fp64": pkg.SDFT_PREC_FP64}[args.prec]
    specs = wl.batch_specs()
    t0 = time.time()
    tuner = tuner_mod.Tuner(pkg)
    preps, systems = [], []
    for i, sp in enumerate(specs):
        s = wl.build_spec(sp)
        systems.append(s)
        preps.append(serve.prepare(pkg, wl, s, sp["nsto"], sp["L"], prec, seed=10.0 + i, tuner=tuner))
        if args.plane_threads != "tuned":  # one fixed plane-stage CTA size for every system
            try:
                preps[-1]["ctx"].set_plane_threads(int(args.plane_threads))
            except pkg.SdftError:
                pass
    setup_s = time.time() - t0
    nsto = [sp["nsto"] for sp in specs]
    total = sum(nsto)
    # eager: every system in turn through the per-call API (same kernels)
    torch.cuda.synchronize()
    t1 = time.perf_counter()
    for p, sp in zip(preps, specs):
        p["ctx"].filter_cheby_dev(sp["nsto"], p["ec"], 1, p["scale"], p["emean"])
        p["ctx"].density_dev(sp["nsto"], 0, p["occ_over"], want=False)
    for p in preps:
        p["ctx"].sync()
    eager_s = time.perf_counter() - t1
    rho_eager = [p["ctx"].download_density() for p in preps]
    t2 = time.time()
    b = pkg.Batch([p["ctx"] for p in preps], nsto, [sp["L"] for sp in specs], [p["ec"] for p in preps],
                  [p["scale"] for p in preps], [p["emean"] for p in preps], [p["occ_over"] for p in preps])
    capture_s = time.time() - t2
    ext = torch.cuda.ExternalStream(b.stream_ptr)
    for _ in range(args.warmup):
        b.launch()
    b.sync()
    clk = Clocks(0)
    clk.start()
    evs = []
    for _ in range(args.steps):
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(ext)
        b.launch()
        e1.record(ext)
        evs.append((e0, e1))
    b.sync()
    clocks = clk.stop()
    ms = [x.elapsed_time(y) for x, y in evs]
    same = max(float(np.linalg.norm(p["ctx"].download_density() - r) / np.linalg.norm(r))
               for p, r in zip(preps, rho_eager))
    # e2e: fresh noise orbitals uploaded from pinned host memory every replay,
    # densities read back
    host = []
    for p, sp in zip(preps, specs):
        cr = torch.empty(sp["nsto"] * p["ctx"].ncoef, dtype=torch.float64, pin_memory=True).numpy()
        ci = torch.empty_like(torch.from_numpy(cr)).pin_memory().numpy()
        rng = np.random.default_rng(len(host))
        cr[:] = rng.standard_normal(cr.size)
        ci[:] = rng.standard_normal(ci.size)
        host.append((cr, ci))
    ks = max(1, min(args.steps, 2))
    t3 = time.perf_counter()
    h2d = d2h = 0
    for _ in range(ks):
        for p, (cr, ci) in zip(preps, host):
            p["ctx"].upload(cr, ci)
            h2d += cr.nbytes + ci.nbytes
        b.launch()
        b.sync()
        for p in preps:
            rho = p["ctx"].download_density()
            d2h += rho.nbytes
    e2e_s = (time.perf_counter() - t3) / ks
    tot_ms = sum(ms)
    lat = sorted(ms)
    out = {
        "metric": "filtered stochastic orbitals/s, 32 batched uneven Si systems in one CUDA-graph launch",
        "value": total * args.steps / (tot_ms / 1e3), "unit": "orbitals/s", "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": tot_ms / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "mixed(fp32 fft, int8-ozaki kb gemm, fp64 recurrence)" if prec else "f64",
        "data": "synthetic (seeded Si supercells, Gaussian V_loc, Gaussian s+p KB, +-1 noise)",
        "config": {"workload": f"cfg4: {len(specs)} systems, {sum(s['natm'] for s in systems)} atoms, "
                               f"{total} orbitals, grids 24..72 per axis, orders 128..512",
                   "plane_threads": args.plane_threads,
                   "systems": [{"atoms": s["natm"], "grid": list(s["grid"]), "orbitals": sp["nsto"], "L": sp["L"],
                                "gemm_split": tuner.cache[tuner.key(p["ctx"], sp["nsto"], 4 * s["natm"])]["split"],
                                "plane_threads": tuner.cache[tuner.key(p["ctx"], sp["nsto"], 4 * s["natm"])].get(
                                    "plane_threads"),
                                "gemm_bn": tuner.cache[tuner.key(p["ctx"], sp["nsto"], 4 * s["natm"])].get("gemm_bn")}
                               for s, sp, p in zip(systems, specs, preps)],
                   "setup_s": setup_s, "capture_s": capture_s, "l2": "per-system orbitals in HBM; no flush"},
        "latency_ms": {"p50": lat[len(lat) // 2], "p99": lat[-1]},
        "eager_sequential": {"orbitals_per_s": total / eager_s, "s": eager_s},
        "graph_vs_eager_density_rel_l2": same,
        "e2e": {"value": total / e2e_s, "unit": "orbitals/s", "h2d_bytes_per_step": h2d // ks,
                "d2h_bytes_per_step": d2h // ks},
        "gpu_launches": b.kernels_per_launch * args.steps, "graph_launches": args.steps, "clocks": clocks,
    }
    b.close()
    for p in preps:
        p["ctx"].close()
    print(json.dumps(out))


def run_serve(args):
    """Serving: seeded Poisson stream (50 req/s) of filter + density requests
    from the batch distribution with 10 % 512-atom systems; admission by
    free slot and a 150 GB HBM budget; continuous batching (requests admitted
    while others run); mixed precision and the same stream in FP64."""
    import __graft_entry__ as g
    pkg = g.load_package()
    wl = g.load_workload()
    serve, tuner_mod = _modules(pkg)
    reqs = serve.poisson_requests(wl, args.requests, 50.0, seed=5, big_fraction=0.1)
    out_runs = {}
    recs = {}
    for name, prec in (("mixed", pkg.SDFT_PREC_MIXED), ("fp64", pkg.SDFT_PREC_FP64)):
        srv = serve.Server(pkg, wl, prec, hbm_budget=150e9, slots=args.slots, workers=args.workers,
                           priorities=not args.no_priorities, graph=not args.serve_eager)
        srv.run([dict(r, arrival=0.0) for r in reqs[:2]])  # warm-up (module loads, first-use attributes)
        # FP64 serves the same stream with the mixed run's mu, so the density
        # difference is the precision alone (the moments are still computed)
        rq = reqs if name == "mixed" else [dict(r, mu=recs["mixed"][i]["mu"]) for i, r in enumerate(reqs)]
        rec, summ = srv.run(rq)
        out_runs[name] = summ
        recs[name] = rec
    errs = [float(np.linalg.norm(a["density"] - b["density"]) / np.linalg.norm(b["density"]))
            for a, b in zip(recs["mixed"], recs["fp64"])]
    m = out_runs["mixed"]
    # saturation: the mix's service rate with every request queued at once;
    # then a sustained Poisson stream at 85 % of it (mixed precision)
    srv = serve.Server(pkg, wl, pkg.SDFT_PREC_MIXED, hbm_budget=150e9, slots=args.slots, workers=args.workers,
                       priorities=not args.no_priorities, graph=not args.serve_eager)
    sat_reqs = serve.poisson_requests(wl, args.sat_requests, 1.0, seed=7, big_fraction=0.1)
    _, sat = srv.run([dict(r, arrival=0.0) for r in sat_reqs], keep_density=False)
    sat_rate = sat["requests_per_s"]
    sus_reqs = serve.poisson_requests(wl, args.sustained_requests, 0.85 * sat_rate, seed=9, big_fraction=0.1)
    _, sus = srv.run(sus_reqs, keep_density=False)
    lat_small = [r["latency"] for r in recs["mixed"] if r["natm"] < 512]
    lat_big = [r["latency"] for r in recs["mixed"] if r["natm"] >= 512]
    out = {
        "metric": "serving: filtered stochastic orbitals/s with p50/p99 request latency (Poisson 50 req/s)",
        "value": m["orbitals_per_s"], "unit": "orbitals/s", "n_gpus": 1, "steps": 1, "warmup": 1,
        "ms_per_step": m["span_s"] * 1e3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "mixed(fp32 fft, int8-ozaki kb gemm, fp64 recurrence)",
        "data": "synthetic (seeded Poisson arrivals; Si supercells 8..216 atoms + 10 % 512-atom)",
        "config": {"workload": f"cfg5: {len(reqs)} requests at 50 req/s, slots {args.slots}, "
                               f"{args.workers} host workers, HBM budget 150 GB",
                   "stream_priorities": "by request work (serve.request_priority)" if not args.no_priorities
                   else "off",
                   "request_launch": "kernels on the request stream" if args.serve_eager else "captured CUDA graph",
                   "requests": len(reqs), "orbitals": m["orbitals"],
                   "atoms": [int(8 * np.prod(r["spec"]["nrep"])) for r in reqs]},
        "latency_ms": {"p50": m["p50_ms"], "p99": m["p99_ms"], "mean": m["mean_ms"],
                       "p50_below_512_atoms": float(np.percentile(lat_small, 50) * 1e3) if lat_small else None,
                       "max_512_atoms": float(max(lat_big) * 1e3) if lat_big else None},
        "mixed": m, "fp64": out_runs["fp64"],
        "saturation": {"requests": len(sat_reqs), "requests_per_s": sat_rate,
                       "orbitals_per_s": sat["orbitals_per_s"], "note": "all requests queued at t = 0"},
        "sustained": {"rate_req_per_s": 0.85 * sat_rate, "fraction_of_saturation": 0.85, "requests": len(sus_reqs),
                      "completed": sus["completed"], "refused": sus["refused"], "failed": sus["failed"],
                      "p50_ms": sus.get("p50_ms"), "p99_ms": sus.get("p99_ms"), "mean_ms": sus.get("mean_ms"),
                      "orbitals_per_s": sus.get("orbitals_per_s")},
        "mixed_speedup": m["orbitals_per_s"] / out_runs["fp64"]["orbitals_per_s"],
        "density_rel_l2_mixed_vs_fp64": {"max": max(errs), "median": float(np.median(errs)),
                                         "per_request": [[int(recs["mixed"][i]["natm"]), int(reqs[i]["nsto"]),
                                                          int(reqs[i]["L"]), float(e)] for i, e in enumerate(errs)]},
    }
    print(json.dumps(out))


def run_forces(args):
    """The nonlocal atomic forces alone (sdft_nl_force_dev) on the config's
    system: seeded random orbitals taken as the filtered ones (coefficients
    [1, 0]), then `steps` timed calls after `warmup` untimed ones.  One JSON
    line; a small, fixed command for profiling the force path."""
    import torch
    import __graft_entry__ as g
    pkg = g.load_package()
    wl, cfg, s = setup_system(args.config, 0)
    nsto = cfg["nsto"] if args.nsto is None else args.nsto
    prec = {"mixed": pkg.SDFT_PREC_MIXED, "mixed_fast": pkg.SDFT_PREC_MIXED_FAST, "fp64": pkg.SDFT_PREC_FP64}[args.prec]
    ctx = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=prec, max_states=nsto)
    ctx.set_vks(s["vks"])
    ctx.set_kb(s["kb_desc"])
    rng = np.random.default_rng(3)
    cr = rng.standard_normal(nsto * s["ncoef"])
    ci = rng.standard_normal(nsto * s["ncoef"])
    ci.reshape(nsto, -1)[:, -1] = 0.0
    ctx.upload(cr, ci)
    ctx.filter_cheby_dev(nsto, np.array([1.0, 0.0]), 1, 0.1, 0.0)
    st = torch.cuda.ExternalStream(pkg.lib.sdft_ctx_stream(ctx._p))
    for _ in range(args.warmup):
        ctx.nl_force_dev(nsto, 0, occ=wl.OCC, nsto_total=nsto)
    ms = []
    for _ in range(args.steps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(st)
        f, e = ctx.nl_force_dev(nsto, 0, occ=wl.OCC, nsto_total=nsto)
        b.record(st)
        b.synchronize()
        ms.append(a.elapsed_time(b))
    ctx.close()
    print(json.dumps({"metric": "nonlocal atomic forces of filtered orbitals (ms per call)", "value": min(ms),
                      "unit": "ms", "higher_is_better": False, "steps": args.steps, "warmup": args.warmup,
                      "config": {"workload": args.config, "orbitals": nsto, "natm": int(f.shape[0]),
                                 "precision": args.prec}, "energy_pnl": e}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--config", default="cfg3")
    ap.add_argument("--prec", default="mixed", choices=["mixed", "mixed_fast", "fp64"])
    ap.add_argument("--nsto", type=int, default=None)
    ap.add_argument("--L", type=int, default=None)
    ap.add_argument("--cpu-steps", type=int, default=2)
    ap.add_argument("--no-fp64", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-graph", action="store_true", help="time the eager step only")
    ap.add_argument("--requests", type=int, default=48, help="cfg5: number of requests")
    ap.add_argument("--slots", type=int, default=16, help="cfg5: concurrent requests")
    ap.add_argument("--plane-threads", default="tuned", choices=["tuned", "256", "128"],
                    help="plane-stage CTA size: the autotuner's choice (tuned: with the KB GEMM tile width and "
                         "split-K, per system in cfg4) or one size for all (the GEMM shapes then per call)")
    ap.add_argument("--sat-requests", type=int, default=64,
                    help="cfg5: requests queued at once to measure the saturation rate")
    ap.add_argument("--sustained-requests", type=int, default=200,
                    help="cfg5: requests of the Poisson stream at 85 %% of the saturation rate")
    ap.add_argument("--workers", type=int, default=16, help="cfg5: host threads preparing requests")
    ap.add_argument("--no-priorities", action="store_true", help="cfg5: all request streams at default priority")
    ap.add_argument("--serve-eager", action="store_true",
                    help="cfg5: issue each request's kernels directly instead of as a captured CUDA graph")
    ap.add_argument("--forces-only", action="store_true",
                    help="time sdft_nl_force_dev alone on the config's system (profiling the force path)")
    args = ap.parse_args()
    if args.forces_only:
        run_forces(args)
    elif args.impl == "reference":
        run_reference(args)
    elif args.config == "cfg4":
        run_batch(args)
    elif args.config == "cfg5":
        run_serve(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
