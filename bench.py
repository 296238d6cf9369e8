#!/usr/bin/env python
"""Benchmark: batched BEM solves/s and adjoint grads/s at N=2048 panels on B200.

Workload (one "step" = one pass of the hot path over one batch): a
hemisphere of radius 1 m meshed at resolution 64 x 64 (2048 panels), 64
frequencies omega = linspace(0.3, 3.0), heave and surge radiating and
influenced, one incident heading (beta = 0), Rankine + reflected Rankine +
tabulated Guevel-Delhommeau wave term, direct formulation; mixed precision
(FP16 tensor-core LU updates with FP32 panels, FP64 refinement to
max|r|/max|b| <= 1e-8, two sweeps).  A solve is one (mesh, frequency) problem
with all its right-hand sides and outputs (A, B, F, FK).

  value  solves/s with the mesh already resident on the device
  e2e    the same through the C ABI from pinned host buffers: mesh upload,
         batch call, outputs back to the host, every step
  grads  adjoint grads/s: one grad = one (mesh, frequency) problem solved
         forward, its adjoint solve and the tangent contraction, giving the
         cotangents of every mesh field and of omega for a scalar objective
         J = sum(wA A) + sum(wB B) + Re sum(conj(wF) F) (seeded weights), and
         from them dJ/dR through the exact mesh tangent
  grads_two_body
         the two-body power objective (two 1024-panel hemispheres 5 m apart,
         Wu, indirect, omega = 1.03) and dJ/d(r1, dx1, omega), end to end
         through two_body_power(grad=True)

Also reported: the FP64 GPU path batched the same way (the denominator of
the mixed path's speed-up) and one frequency at a time; the error of the
mixed outputs against the FP64 oracle's exact-quadrature fixture at all 64
frequencies; per-phase times measured with CUDA events on the library's
stream; the roofline of the LU phase and of the wave pass; clocks sampled
during the timed region; and the CPU oracle baseline.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]
"""
from __future__ import annotations

import argparse
import ctypes
import datetime
import importlib.util
import json
import os
import pathlib
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = pathlib.Path(__file__).resolve().parent
METRIC = "BEM solves/s + adjoint grads/s, N=2048 panels: mixed vs FP64 GPU at 1e-6 err"
WORKLOAD = "hemisphere_2048p_64omega_heave_surge_diffraction_delhommeau_direct"


def load_package():
    name = "marinehydro_b200"
    if name in sys.modules:
        return sys.modules[name]
    pkg_dir = ROOT / "marinehydro.jl_b200"
    spec = importlib.util.spec_from_file_location(
        name, pkg_dir / "__init__.py", submodule_search_locations=[str(pkg_dir)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules[name] = mod
    spec.loader.exec_module(mod)
    return mod


def workload(mh, res, n_omega):
    mesh = mh.mesh_hemisphere(1.0, (0.0, 0.0, 0.0), tuple(res))
    body = mh.FloatingBody.rigid(mesh, ["Heave", "Surge"])
    dofs = list(body.dofs.values())
    omegas = np.linspace(0.3, 3.0, n_omega)
    betas = [0.0]
    gfs = (mh.Rankine(), mh.RankineReflected(), mh.ExactGuevelDelhommeau())
    return mesh, dofs, omegas, betas, gfs


def config_dict(mesh, omegas, args):
    return {"workload": WORKLOAD, "panels": int(mesh.nfaces), "resolution": list(args.res),
            "n_omega": int(len(omegas)), "omega_range": [float(omegas[0]), float(omegas[-1])],
            "dofs": ["Heave", "Surge"], "headings": [0.0],
            "green_functions": "Rankine+RankineReflected+ExactGuevelDelhommeau(table)",
            "formulation": "direct",
            "precision": ("mixed: FP16 tcgen05 trailing update / FP32 LU, FP64 refinement"
                          if args.lu == "tcgen05" else "mixed: FP32 LU, FP64 refinement")
            + {0: "; wave series FP64", 1: "; wave-pass Horner series FP32, the rest of the assembly FP64",
               2: "; wave-pass series and alpha contraction FP32, the rest of the assembly FP64"}[args.wave_level],
            "lu_backend": args.lu,
            "tol": args.tol, "solve": "one (mesh, omega) problem, 3 right-hand sides",
            "l2": "working set ~11 GB per step, larger than the 126 MB L2 (no flush needed)"}


# --------------------------------------------------------------------------
# clocks during the timed region
# --------------------------------------------------------------------------

class ClockSampler:
    """SM clock and clock-event reasons of the bench's GPU while the timed
    region runs.  Read-only NVML queries from a background thread every
    5 ms (the library calls release the GIL), so a timed region of tens of
    milliseconds still gets a few dozen samples; without NVML, nvidia-smi
    polls every 50 ms into a temporary file.  Nothing is changed on the GPU."""

    REASONS = (("hw_slowdown", "nvmlClocksEventReasonHwSlowdown"),
               ("hw_thermal_slowdown", "nvmlClocksEventReasonHwThermalSlowdown"),
               ("sw_thermal_slowdown", "nvmlClocksEventReasonSwThermalSlowdown"),
               ("sw_power_cap", "nvmlClocksEventReasonSwPowerCap"))
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: str, device: int = 0):
        import threading

        self.sm, self.mx, self.reasons = [], None, set()
        self.proc = self.thread = None
        self.stop_flag = threading.Event()
        try:
            import pynvml as nv
            import torch

            nv.nvmlInit()
            prop = torch.cuda.get_device_properties(device)
            bus = f"{prop.pci_domain_id:08x}:{prop.pci_bus_id:02x}:{prop.pci_device_id:02x}.0"
            try:
                h = nv.nvmlDeviceGetHandleByPciBusId(bus.encode())
            except nv.NVMLError:
                h = nv.nvmlDeviceGetHandleByIndex(int(gpu_index))
            self.mx = float(nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM))
            bits = [(name, getattr(nv, attr)) for name, attr in self.REASONS]

            def run():
                while not self.stop_flag.is_set():
                    try:
                        self.sm.append(float(nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)))
                        r = nv.nvmlDeviceGetCurrentClocksEventReasons(h)
                        self.reasons.update(name for name, bit in bits if r & bit)
                    except nv.NVMLError:
                        return
                    self.stop_flag.wait(0.005)

            self.thread = threading.Thread(target=run, daemon=True)
            self.thread.start()
            return
        except Exception:  # noqa: BLE001 - no NVML: fall back to nvidia-smi
            self.thread = None
        try:
            import tempfile

            self.fh = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "50", "-i", gpu_index], stdout=self.fh, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self):
        if self.thread is not None:
            self.stop_flag.set()
            self.thread.join(timeout=5)
        elif self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
            self.fh.flush()
            self.fh.seek(0)
            names = [nm for nm, _ in self.REASONS]
            for r in (x.split(",") for x in self.fh.read().splitlines() if x.strip()):
                r = [x.strip() for x in r]
                if len(r) < 9:
                    continue
                try:
                    self.sm.append(float(r[1]))
                    self.mx = float(r[2])
                except ValueError:
                    continue
                self.reasons.update(nm for nm, v in zip(names, r[5:9]) if v.lower().startswith("active"))
            self.fh.close()
            os.unlink(self.fh.name)
        else:
            return None
        if not self.sm:
            return None
        return {"sm_mhz": statistics.median(self.sm), "sm_max_mhz": self.mx, "reasons": sorted(self.reasons),
                "samples": len(self.sm), "source": "nvml" if self.thread is not None else "nvidia-smi"}


# --------------------------------------------------------------------------
# CPU baseline (the FP64 CPU oracle; test infrastructure, timed as the baseline)
# --------------------------------------------------------------------------

def cpu_threads() -> int:
    """Host threads this process may use: the affinity mask, capped by the
    cgroup CPU quota when one is set (a container may see more cores than
    its quota lets it run)."""
    n = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
    try:
        quota, period = open("/sys/fs/cgroup/cpu.max").read().split()[:2]
        if quota != "max":
            n = max(1, min(n, int(int(quota) // int(period))))
    except (OSError, ValueError):
        pass
    return n


def exact_matrices(mesh, omegas):
    """S and D of the middle frequency by the oracle's exact quadrature, all
    columns (untimed set-up of the CPU legs' LAPACK timing)."""
    sys.path.insert(0, str(ROOT))
    import oracle

    w = float(omegas[len(omegas) // 2])
    return oracle.assemble(mesh, w * w / 9.81,
                           oracle.GF_RANKINE | oracle.GF_RANKINE_REFLECTED | oracle.GF_DELHOMMEAU, True,
                           cpu_threads())


def cpu_baseline(mh, mesh, dofs, omegas, betas, columns: int, offset: int = 0, SD=None):
    """One (mesh, frequency) solve of the FP64 CPU oracle at the middle
    frequency: exact-quadrature Delhommeau assembly of the `columns` source
    columns from `offset` (wrapping), scaled to all n columns, plus LAPACK
    zgetrf/zgetrs, the right-hand sides and the forces on the full matrices
    SD = (S, D) of that frequency (exact_matrices)."""
    sys.path.insert(0, str(ROOT))
    import oracle
    import scipy.linalg as sla

    oracle.lib()
    threads = cpu_threads()
    n = mesh.nfaces
    w = float(omegas[len(omegas) // 2])
    k = w * w / 9.81
    mask = oracle.GF_RANKINE | oracle.GF_RANKINE_REFLECTED | oracle.GF_DELHOMMEAU
    j0 = offset % n
    spans = [(j0, min(n, j0 + columns))]
    if j0 + columns > n:
        spans.append((0, j0 + columns - n))
    t0 = time.perf_counter()
    for a, b in spans:
        oracle.assemble(mesh, k, mask, True, threads, columns=(a, b))
    t_asm = (time.perf_counter() - t0) * n / columns
    S, D = SD if SD is not None else exact_matrices(mesh, omegas)
    t0 = time.perf_counter()
    lu = sla.lu_factor(D, check_finite=False)
    bcs = [oracle.radiation_bc(mesh.normals, d, w) for d in dofs]
    bcs += [oracle.airy_bc(mesh.centers, mesh.normals, w, b) for b in betas]
    phi = sla.lu_solve(lu, S @ np.stack(bcs, axis=1), check_finite=False)
    for q in range(phi.shape[1]):
        for d in dofs:
            oracle.integrate_pressure(mesh.normals, mesh.areas, 1j * 1000.0 * w * phi[:, q], d)
    t_lu = time.perf_counter() - t0
    per_solve = t_asm + t_lu
    return {"value": 1.0 / per_solve, "unit": "solves/s", "cores": threads, "kind": "port",
            "extrapolated": True, "columns": [j0, columns], "assembly_scale": n / columns,
            "sample": (f"1 frequency (omega={w:.3f}): FP64 exact-quadrature Delhommeau assembly of "
                       f"source columns {j0}..{(j0 + columns - 1) % n} ({columns} of {n}) scaled "
                       f"x{n / columns:g} ({t_asm:.2f} s), plus LAPACK zgetrf/zgetrs on the exact-quadrature "
                       f"D (assembled once, untimed) + 3 right-hand sides + forces ({t_lu:.3f} s)")}


def reference_config(mesh, omegas, args):
    c = config_dict(mesh, omegas, args)
    c.update(green_functions="Rankine+RankineReflected+ExactGuevelDelhommeau (adaptive quadrature per pair)",
             precision="FP64 (CPU oracle, the C restatement of the reference's path) + LAPACK",
             lu_backend="LAPACK zgetrf (scipy)", tol=None,
             solve="one (mesh, omega) problem, 3 right-hand sides; assembly timed on a window of "
                   "source columns per step and scaled to all columns")
    return c


# --------------------------------------------------------------------------
# reference arm: the CPU implementation of the path (oracle port)
# --------------------------------------------------------------------------

def run_reference(args):
    """The CPU implementation of the path (the oracle) on the host cores.
    One step is a bounded sample of one (mesh, frequency) solve: the
    exact-quadrature assembly of the next window of source columns (the
    window advances every step) plus the LAPACK factorisation, solves and
    forces.  ms_per_step is the wall time of that sample; value (solves/s) is
    the full solve it extrapolates to, the assembly scaled to all columns."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    mh = load_package()
    mesh, dofs, omegas, betas, gfs = workload(mh, args.res, args.n_omega)
    solve_s, step_s = [], []
    base = None
    SD = exact_matrices(mesh, omegas)
    for step in range(args.warmup + args.steps):
        t0 = time.perf_counter()
        base = cpu_baseline(mh, mesh, dofs, omegas, betas, args.cpu_columns, step * args.cpu_columns, SD)
        dt = time.perf_counter() - t0
        if step >= args.warmup:
            solve_s.append(1.0 / base["value"])
            step_s.append(dt)
    per = float(np.mean(solve_s))
    v = 1.0 / per
    n = mesh.nfaces
    timed_cols = min(n, args.steps * args.cpu_columns)
    line = {"metric": METRIC, "value": v, "unit": "solves/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": float(np.mean(step_s)) * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": reference_config(mesh, omegas, args), "impl": "reference",
            "extrapolated": True, "sampled_columns": timed_cols, "ms_per_solve_extrapolated": per * 1e3,
            "note": (f"a step is a bounded sample: the exact-quadrature assembly of {args.cpu_columns} source "
                     f"columns (the window advances every step; the {args.steps} timed steps cover {timed_cols} "
                     f"distinct columns of {n}) plus the LAPACK LU, solves and forces on the exact-quadrature "
                     f"S and D (assembled once before the steps); ms_per_step is its wall "
                     f"time; value is the full solve it extrapolates to (assembly x{n / args.cpu_columns:g})"),
            "cpu_baseline": {"value": v, "unit": "solves/s", "cores": base["cores"],
                             "kind": "port", "sample": base["sample"], "extrapolated": True},
            "e2e": {"value": v, "unit": "solves/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


# --------------------------------------------------------------------------
# our arm
# --------------------------------------------------------------------------

def _pinned(a: np.ndarray, torch):
    t = torch.from_numpy(np.ascontiguousarray(a)).pin_memory()
    return t


def e2e_step(mh, ctx, host, omegas_p, dofs_p, betas_p, out_p, args, mask, info):
    """Mesh upload + batch + outputs to host through the C ABI."""
    N = mh.native
    L = N.lib()
    h = N._P()
    dp = lambda t: ctypes.cast(t.data_ptr(), N._D)
    N.check(L.mh_mesh_create(ctx.handle, host["n"], host["nv"], dp(host["vertices"]),
                             ctypes.cast(host["faces"].data_ptr(), N._I64), dp(host["centers"]),
                             dp(host["normals"]), dp(host["areas"]), dp(host["radii"]),
                             ctypes.byref(h)), ctx.handle)
    try:
        N.check(L.mh_hydro_batch(ctx.handle, h, omegas_p.numel(), dp(omegas_p), args.n_dof,
                                 dp(dofs_p), betas_p.numel(), dp(betas_p), 1000.0, 9.81, mask, 1,
                                 N.MH_PRECISION_MIXED, args.tol, args.max_iter, dp(out_p[0]),
                                 dp(out_p[1]), dp(out_p[2]), dp(out_p[3]), ctypes.byref(info)),
                ctx.handle)
    finally:
        L.mh_mesh_destroy(ctx.handle, h)


def e2e_grad_step(mh, ctx, host, omegas_p, dofs_p, betas_p, bars_p, grads_p, args, mask, info):
    """Mesh upload + forward/adjoint batch + cotangents to host through the C ABI."""
    N = mh.native
    L = N.lib()
    h = N._P()
    dp = lambda t: ctypes.cast(t.data_ptr(), N._D) if t is not None else None
    N.check(L.mh_mesh_create(ctx.handle, host["n"], host["nv"], dp(host["vertices"]),
                             ctypes.cast(host["faces"].data_ptr(), N._I64), dp(host["centers"]),
                             dp(host["normals"]), dp(host["areas"]), dp(host["radii"]),
                             ctypes.byref(h)), ctx.handle)
    try:
        N.check(L.mh_hydro_batch_vjp(
            ctx.handle, h, omegas_p.numel(), dp(omegas_p), args.n_dof, dp(dofs_p), betas_p.numel(),
            dp(betas_p), 1000.0, 9.81, mask, 1, N.MH_PRECISION_MIXED, args.tol, args.max_iter,
            dp(bars_p[0]), dp(bars_p[1]), dp(bars_p[2]), None, None, None, None, None,
            dp(grads_p[0]), dp(grads_p[1]), dp(grads_p[2]), dp(grads_p[3]), None, dp(grads_p[4]),
            None, ctypes.byref(info)), ctx.handle)
    finally:
        L.mh_mesh_destroy(ctx.handle, h)


def grad_weights(nd, nw, nb):
    rng = np.random.default_rng(2024)
    return (rng.normal(size=(nd, nd, nw)), rng.normal(size=(nd, nd, nw)),
            rng.normal(size=(nd, nw, nb)) + 1j * rng.normal(size=(nd, nw, nb)))


def run_grads(mh, ctx, mesh, dofs, omegas, betas, gfs, args, stream, barrier, dist, world, torch):
    """Adjoint grads/s (mixed) with the FP64 GPU path and the agreement of
    the two; each step one mh_hydro_batch_vjp over all frequencies."""
    nd, nw, nb = len(dofs), len(omegas), len(betas)
    wA, wB, wF = grad_weights(nd, nw, nb)
    tan = mh.hemisphere_tangents(1.0, (0.0, 0.0, 0.0), tuple(args.res))["radius"]

    def gstep():
        r = mh.hydro_batch_vjp(mesh, omegas, dofs, betas, wA, wB, wF, None, green_functions=gfs,
                               precision="mixed", tol=args.tol, max_iter=args.max_iter, ctx=ctx)
        return r, r.mesh.dot(tan)

    for _ in range(args.warmup):
        r, dR = gstep()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    ctx.set_profiling(True)
    l0 = ctx.kernel_launches()
    barrier()
    ev0.record(stream)
    for _ in range(args.steps):
        r, dR = gstep()
    ev1.record(stream)
    barrier()
    launches = ctx.kernel_launches() - l0
    phases = ctx.phase_times()
    ctx.set_profiling(False)
    ms = ev0.elapsed_time(ev1)
    if dist is not None:
        t = torch.tensor([ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    out = {"value": world * nw * args.steps / (ms / 1e3), "unit": "grads/s",
           "ms_per_step": ms / args.steps, "gpu_launches": launches,
           "objective": "J = sum(wA A) + sum(wB B) + Re sum(conj(wF) Fd), seeded weights",
           "outputs": "cotangents of vertices, centers, normals, areas, radii, omegas; dJ/dR",
           "dJ_dR": dR, "phases_ms_per_step": {k: v[0] / args.steps for k, v in phases.items() if v[1]}}
    # e2e through the C ABI
    host = host_mesh(mesh, torch)
    omegas_p = _pinned(omegas, torch)
    betas_p = _pinned(np.asarray(betas, dtype=np.float64), torch)
    dofs_p = _pinned(np.concatenate([np.asfortranarray(d).reshape(-1, order="F") for d in dofs]), torch)
    bars_p = [_pinned(np.asfortranarray(wA).reshape(-1, order="F"), torch),
              _pinned(np.asfortranarray(wB).reshape(-1, order="F"), torch),
              _pinned(np.asfortranarray(wF).reshape(-1, order="F").view(np.float64), torch)]
    grads_p = [torch.zeros(3 * mesh.nvertices, dtype=torch.float64).pin_memory(),
               torch.zeros(3 * mesh.nfaces, dtype=torch.float64).pin_memory(),
               torch.zeros(3 * mesh.nfaces, dtype=torch.float64).pin_memory(),
               torch.zeros(mesh.nfaces, dtype=torch.float64).pin_memory(),
               torch.zeros(nw, dtype=torch.float64).pin_memory()]
    cinfo = mh.bodies._Info()
    mask = mh.gf_mask(gfs)
    e2e_grad_step(mh, ctx, host, omegas_p, dofs_p, betas_p, bars_p, grads_p, args, mask, cinfo)
    barrier()
    ev0.record(stream)
    for _ in range(args.steps):
        e2e_grad_step(mh, ctx, host, omegas_p, dofs_p, betas_p, bars_p, grads_p, args, mask, cinfo)
    ev1.record(stream)
    barrier()
    ms_e2e = ev0.elapsed_time(ev1)
    if dist is not None:
        t = torch.tensor([ms_e2e], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms_e2e = float(t.item())
    h2d = sum(int(v.numel() * v.element_size()) for k, v in host.items() if k not in ("n", "nv"))
    h2d += int(omegas_p.numel() * 8 + betas_p.numel() * 8 + dofs_p.numel() * 8)
    h2d += sum(int(t.numel() * t.element_size()) for t in bars_p)
    out["e2e"] = {"value": world * nw * args.steps / (ms_e2e / 1e3), "unit": "grads/s",
                  "h2d_bytes_per_step": h2d,
                  "d2h_bytes_per_step": sum(int(t.numel() * t.element_size()) for t in grads_p),
                  "ms_per_step": ms_e2e / args.steps}
    if args.no_fp64:
        return out
    # FP64 GPU path batched the same way (the denominator), all frequencies
    fcall = lambda om_, s_, prec: mh.hydro_batch_vjp(mesh, om_, dofs, betas, wA[:, :, s_], wB[:, :, s_], wF[:, s_],
                                                      None, green_functions=gfs, precision=prec, tol=args.tol,
                                                      max_iter=args.max_iter, ctx=ctx)
    allz = np.arange(nw)
    fcall(omegas[:8], allz[:8], "fp64_batched")  # warm-up
    torch.cuda.synchronize()
    ev0.record(stream)
    res64 = fcall(omegas, allz, "fp64_batched")
    ev1.record(stream)
    torch.cuda.synchronize()
    ms64 = ev0.elapsed_time(ev1)
    resmx = r
    out["fp64_gpu"] = {"value": nw / (ms64 / 1e3), "unit": "grads/s", "ms_per_step": ms64,
                       "mode": "FP64 forward + adjoint batched like the mixed path (cuSOLVER getrf/getrs per "
                               "frequency on four streams)"}
    # and one frequency at a time: per-call cost a + b * n_omega fitted on two subsample sizes
    sub = np.arange(0, nw, max(1, nw // args.fp64_omegas))[:args.fp64_omegas]
    fcall(omegas[sub[:1]], sub[:1], "fp64")  # warm-up
    times = {}
    for cnt in (2, len(sub)):
        s_ = sub[:cnt]
        torch.cuda.synchronize()
        ev0.record(stream)
        fcall(omegas[s_], s_, "fp64")
        ev1.record(stream)
        torch.cuda.synchronize()
        times[cnt] = ev0.elapsed_time(ev1)
    b = (times[len(sub)] - times[2]) / (len(sub) - 2)
    a = times[2] - 2 * b
    per = (a + nw * b) / nw
    out["fp64_gpu_per_frequency"] = {"value": 1e3 / per, "unit": "grads/s", "ms_per_grad_at_n_omega": per,
                                     "mode": "FP64 forward + adjoint one frequency at a time",
                                     "fit_ms": {"per_call": a, "per_omega": b},
                                     "omegas_timed": [2, int(len(sub))]}
    out["speedup_vs_fp64_gpu"] = out["value"] / out["fp64_gpu"]["value"]
    out["speedup_vs_fp64_gpu_per_frequency"] = out["value"] / out["fp64_gpu_per_frequency"]["value"]
    acc = {}
    for f in ("vertices", "centers", "normals", "areas"):
        x, y = getattr(resmx.mesh, f), getattr(res64.mesh, f)
        acc[f] = float(np.max(np.abs(x - y)) / np.max(np.abs(y)))
    acc["omegas"] = float(np.max(np.abs(resmx.omegas - res64.omegas)) / np.max(np.abs(res64.omegas)))
    acc["dJ_dR"] = abs(resmx.mesh.dot(tan) - res64.mesh.dot(tan)) / abs(res64.mesh.dot(tan))
    acc["note"] = "max abs difference / max abs value, mixed vs batched FP64 GPU gradients, all frequencies"
    out["accuracy"] = acc
    return out


def host_mesh(mesh, torch):
    return {"n": mesh.nfaces, "nv": mesh.nvertices,
            "vertices": _pinned(np.asfortranarray(mesh.vertices).reshape(-1, order="F"), torch),
            "faces": _pinned(np.asfortranarray(mesh.faces).reshape(-1, order="F"), torch),
            "centers": _pinned(np.asfortranarray(mesh.centers).reshape(-1, order="F"), torch),
            "normals": _pinned(np.asfortranarray(mesh.normals).reshape(-1, order="F"), torch),
            "areas": _pinned(mesh.areas, torch), "radii": _pinned(mesh.radii, torch)}


def run_ours(args):
    import torch

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300),
                                device_id=torch.device("cuda", local))
    else:
        torch.cuda.set_device(local)
    mh = load_package()
    ctx = mh.Context(local)
    ctx.set_lu_backend(args.lu)
    ctx.set_wave_series_fp32(args.wave_level)
    stream = torch.cuda.ExternalStream(ctx.stream())
    mesh, dofs, omegas, betas, gfs = workload(mh, args.res, args.n_omega)
    mask = mh.gf_mask(gfs)
    args.n_dof = len(dofs)
    dm = mh.device_mesh(mesh, ctx)

    def step():
        return mh.hydro_batch(mesh, omegas, dofs, betas, green_functions=gfs, precision="mixed",
                              tol=args.tol, max_iter=args.max_iter, ctx=ctx)

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    for _ in range(args.warmup):
        out = step()
    # ---- timed region (resident inputs) ----
    vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
    gpu_index = vis.split(",")[local] if vis and vis.split(",")[local].strip().isdigit() else str(local)
    sampler = ClockSampler(gpu_index, local)
    ctx.set_profiling(True)
    launches0 = ctx.kernel_launches()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    barrier()
    ev0.record(stream)
    for _ in range(args.steps):
        out = step()
    ev1.record(stream)
    barrier()
    launches = ctx.kernel_launches() - launches0
    phases = ctx.phase_times()
    ctx.set_profiling(False)
    clocks = sampler.stop()
    ms = ev0.elapsed_time(ev1)
    if dist is not None:
        t = torch.tensor([ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    value = world * args.n_omega * args.steps / (ms / 1e3)
    A, B, Fd, Fk, info = out

    # ---- e2e through the C ABI from pinned host buffers ----
    host = host_mesh(mesh, torch)
    omegas_p = _pinned(omegas, torch)
    betas_p = _pinned(np.asarray(betas, dtype=np.float64), torch)
    dofs_p = _pinned(np.concatenate([np.asfortranarray(d).reshape(-1, order="F") for d in dofs]),
                     torch)
    nd, nw, nb = len(dofs), len(omegas), len(betas)
    out_p = [torch.zeros(nd * nd * nw, dtype=torch.float64).pin_memory(),
             torch.zeros(nd * nd * nw, dtype=torch.float64).pin_memory(),
             torch.zeros(2 * nd * nw * nb, dtype=torch.float64).pin_memory(),
             torch.zeros(2 * nd * nw * nb, dtype=torch.float64).pin_memory()]
    cinfo = mh.bodies._Info()
    e2e_step(mh, ctx, host, omegas_p, dofs_p, betas_p, out_p, args, mask, cinfo)
    barrier()
    ev0.record(stream)
    for _ in range(args.steps):
        e2e_step(mh, ctx, host, omegas_p, dofs_p, betas_p, out_p, args, mask, cinfo)
    ev1.record(stream)
    barrier()
    ms_e2e = ev0.elapsed_time(ev1)
    if dist is not None:
        t = torch.tensor([ms_e2e], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms_e2e = float(t.item())
    h2d = sum(int(v.numel() * v.element_size()) for k, v in host.items() if k not in ("n", "nv"))
    h2d += int(omegas_p.numel() * 8 * 2 + betas_p.numel() * 8 + dofs_p.numel() * 8)
    d2h = sum(int(t.numel() * t.element_size()) for t in out_p)
    e2e = {"value": world * args.n_omega * args.steps / (ms_e2e / 1e3), "unit": "solves/s",
           "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
           "ms_per_step": ms_e2e / args.steps}

    line = {"metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": ("f64+f32+f16 (FP64 matrices and residuals, FP32 LU panels, FP16 tensor-core "
                      "updates)" if args.lu == "tcgen05" else "f64+f32"), "data": "synthetic",
            "config": config_dict(mesh, omegas, args), "e2e": e2e, "gpu_launches": launches,
            "refinement": {"iterations": info.refine_iterations, "fallbacks": info.n_fallback,
                           "max_rel_residual": info.max_rel_residual}}
    if clocks:
        line["clocks"] = clocks
    per_phase = {k: v[0] / args.steps for k, v in phases.items() if v[1]}
    line["phases_ms_per_step"] = per_phase
    line["roofline"] = roofline(per_phase, mesh.nfaces, args)

    if not args.no_grads:
        line["grads"] = run_grads(mh, ctx, mesh, dofs, omegas, betas, gfs, args, stream, barrier, dist,
                                  world, torch)
    acc = oracle_accuracy(omegas, (A, B, Fd, Fk), args)
    if acc is not None:
        line["accuracy"] = acc
    if rank == 0 and not args.no_fp64:
        line["fp64_gpu"], line["accuracy_vs_fp64_gpu"] = fp64_baseline(mh, ctx, mesh, dofs, omegas, betas, gfs,
                                                                       (A, B, Fd, Fk), args)
        line["speedup_vs_fp64_gpu"] = value / line["fp64_gpu"]["batched"]["value"]
        line["speedup_vs_fp64_gpu_per_frequency"] = value / line["fp64_gpu"]["table"]["value"]
    if rank == 0 and not args.no_grads and not args.no_two_body:
        line["grads_two_body"] = run_two_body(mh, ctx, args, torch)
    if rank == 0 and not args.no_design:
        line["design_batch"] = run_design_batch(mh, args, torch)
    if rank == 0 and not args.no_cpu:
        line["cpu_baseline"] = cpu_baseline(mh, mesh, dofs, omegas, betas, args.cpu_columns)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    ctx.close()
    return 0


def _peaks():
    try:
        peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
        return peaks, "measured"
    except (OSError, ValueError):
        return {}, "fallback"


# DRAM bytes (read + write) per pair-frequency of k_wave_delh_allw from an
# ncu capture (hemisphere 1024 panels, 64 frequencies, the solve step's
# launch without tape: (dram__bytes_read.sum + dram__bytes_write.sum) /
# (n^2 * 64)); traffic grows with the pairs and frequencies a launch
# processes, so it is scaled by them.
WAVE_DRAM_BYTES_PER_PAIR_FREQ = 39.4
# FP64 operations of k_wave_delh_allw counted from its source (an FMA is 2,
# any other arithmetic operation or library call 1): per pair, the geometry and
# the factors of S and D (36), the Chebyshev values (24) and the alpha contraction
# of the four polar functions (15 rows x 22 terms x 4 functions FMAs = 2640; the
# matrix instruction's padding is not counted); per pair and frequency, R and u
# (3), the four degree-14 Horner series (14 x 4 FMAs = 112), G, G_r, G_z from
# them (14) and the scaling into S and D (15).
WAVE_FLOPS_PER_PAIR = 2700.0
WAVE_FLOPS_PER_PAIR_FREQ = 144.0
# Nominal FP64 and FP32 (CUDA-core) peaks of a B200: 148 SMs x 64 FP64 or
# 128 FP32 FMA per clock x 2 x 1.965 GHz; neither is measured on this pool.
FP64_PEAK_TFLOPS = 37.2
FP32_PEAK_TFLOPS = 74.5
# Of the per pair-frequency operations, the Horner series (112) runs in FP32
# at the mixed path's default series level (1), the rest (32) in FP64.
WAVE_FP32_FLOPS_PER_PAIR_FREQ = 112.0
# DRAM bytes of the LU phase per matrix of 2048, from an ncu capture of its
# kernels over one factorisation of 20 matrices of 2048 with the schedule of 64
# (2 groups x 8 panels per outer step): 3.710 GB / 20 = 185.5 MB per matrix (11.9
# GB per 64).  Reads with cold caches per launch; writes leave L2 after a kernel
# ends and hardly appear.
LU_DRAM_BYTES_PER_MATRIX_2048 = 3.710e9 / 20


def roofline(per_phase, n, args):
    """Dominant phase of the solve step: the low-precision LU (k_lu_diag64 +
    k_lu_trsm_tc + k_lu_update_tc), tensor bound, (8/3) n^3 real flops per
    matrix, timed by its phase events on the library's streams; against the
    measured dense bf16 tensor peak (the burst figure, the sustained one
    beside it).  The wave pass k_wave_delh_allw beside it, against the FP64
    issue rate with its flops counted from the source, and its HBM bytes."""
    peaks, src = _peaks()
    hbm = float(peaks.get("hbm_gbs", 6650.0))
    tensor = float(peaks.get("bf16_tflops", 1590.0))
    tensor_sus = float(peaks.get("bf16_tflops_sustained", 1400.0))
    if "lu" not in per_phase:
        return None
    nn = float(n) * n
    fl = 8.0 / 3.0 * float(n) ** 3 * args.n_omega
    ach = fl / (per_phase["lu"] / 1e3) / 1e12
    out = {"kernel": "LU phase: k_lu_update_tc (tcgen05) + k_lu_diag64 + k_lu_trsm_tc", "bound": "tensor",
           "achieved": ach, "peak": tensor, "unit": "TFLOP/s", "frac": ach / tensor,
           "frac_of_sustained_peak": ach / tensor_sus, "peak_source": src,
           "traffic": (LU_DRAM_BYTES_PER_MATRIX_2048 * args.n_omega * (n / 2048.0) ** 2
                       if LU_DRAM_BYTES_PER_MATRIX_2048 else None),
           "ms_per_step": per_phase["lu"], "algorithmic_flops_per_step": fl,
           "note": ("achieved = (8/3) n^3 real flops x matrices / LU phase time; traffic from ncu "
                    "(scaled by n^2 from 2048); the algorithmic bytes (each FP32 matrix read and "
                    "written once) are 8 n^2 x 2 per matrix")}
    if "wave" in per_phase:
        ms = per_phase["wave"]
        alg = nn * (16.0 + 40.0 * args.n_omega)
        flops = nn * (WAVE_FLOPS_PER_PAIR + WAVE_FLOPS_PER_PAIR_FREQ * args.n_omega)
        f32 = nn * WAVE_FP32_FLOPS_PER_PAIR_FREQ * args.n_omega if args.wave_level >= 1 else 0.0
        f64 = flops - f32
        # issue-bound roofline: the time the FP64 and FP32 work take at their peaks
        ideal_ms = (f64 / FP64_PEAK_TFLOPS + f32 / FP32_PEAK_TFLOPS) / 1e9
        out["wave"] = {"kernel": "k_wave_delh_allw", "bound": "fp64+fp32 issue",
                       "achieved": flops / (ms / 1e3) / 1e12, "unit": "TFLOP/s",
                       "frac": ideal_ms / ms, "ideal_ms": ideal_ms,
                       "peak": {"fp64": FP64_PEAK_TFLOPS, "fp32": FP32_PEAK_TFLOPS},
                       "peak_source": "nominal (148 SMs x 64 FP64 / 128 FP32 FMA per clock x 2 x 1.965 GHz)",
                       "flops_per_launch": {"fp64": f64, "fp32": f32}, "flops_per_pair": WAVE_FLOPS_PER_PAIR,
                       "flops_per_pair_freq": WAVE_FLOPS_PER_PAIR_FREQ, "ms_per_launch": ms,
                       "series_level": args.wave_level,
                       "hbm": {"achieved": alg / (ms / 1e3) / 1e9, "peak": hbm, "unit": "GB/s",
                               "frac": alg / (ms / 1e3) / 1e9 / hbm, "algorithmic_bytes_per_launch": alg,
                               "traffic": WAVE_DRAM_BYTES_PER_PAIR_FREQ * nn * args.n_omega}}
    return out


def fp64_baseline(mh, ctx, mesh, dofs, omegas, betas, gfs, mixed, args):
    """The FP64 GPU path, timed with CUDA events on the library's stream:
    batched (MH_PRECISION_FP64_BATCHED: Rankine part once, the
    frequency-batched FP64 wave pass, cuSOLVER zgetrf/zgetrs per frequency)
    over all frequencies, the denominator of the mixed path's speed-up; and
    one frequency at a time (FP64 assembly with the table and with exact
    quadrature) on a subsample."""
    import torch

    stream = torch.cuda.ExternalStream(ctx.stream())
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    res = {}

    def timed(om, prec):
        torch.cuda.synchronize()
        ev0.record(stream)
        o = mh.hydro_batch(mesh, om, dofs, betas, green_functions=gfs, precision=prec, ctx=ctx)
        ev1.record(stream)
        torch.cuda.synchronize()
        return o, ev0.elapsed_time(ev1) / 1e3

    mh.hydro_batch(mesh, omegas[:kAllw_warm], dofs, betas, green_functions=gfs, precision="fp64_batched",
                   ctx=ctx)
    o_b, dt = timed(omegas, "fp64_batched")
    res["batched"] = {"value": len(omegas) / dt, "unit": "solves/s", "omegas": int(len(omegas)),
                      "ms_per_solve": dt / len(omegas) * 1e3}
    sub = np.arange(0, len(omegas), max(1, len(omegas) // args.fp64_omegas))[:args.fp64_omegas]
    for method in ("table", "exact"):
        ctx.set_delhommeau_method(method)
        om = omegas[sub] if method == "table" else omegas[sub[:2]]
        mh.hydro_batch(mesh, om[:1], dofs, betas, green_functions=gfs, precision="fp64", ctx=ctx)
        _, dt = timed(om, "fp64")
        res[method] = {"value": len(om) / dt, "unit": "solves/s", "omegas": int(len(om)),
                       "ms_per_solve": dt / len(om) * 1e3, "mode": "one frequency at a time"}
    ctx.set_delhommeau_method("table")
    A, B, Fd, Fk = mixed
    acc = {}
    for name, a, b in (("A", A, o_b[0]), ("B", B, o_b[1]), ("F", Fd, o_b[2]), ("FK", Fk, o_b[3])):
        acc[name] = float(np.max(np.abs(a - b)) / np.max(np.abs(b)))
    acc["note"] = "max abs difference / max abs value, mixed vs batched FP64 GPU path, all frequencies"
    return res, acc


kAllw_warm = 8  # frequencies of the warm-up call (the frequency-batched wave pass needs >= 6)


def oracle_accuracy(omegas, mixed, args):
    """The mixed outputs against the FP64 oracle's fixture of this workload
    (tests/golden/hemisphere_2048p_delhommeau.npz: exact-quadrature assembly,
    LAPACK; written by tests/golden/make_fixtures.py), every frequency."""
    path = ROOT / "tests" / "golden" / "hemisphere_2048p_delhommeau.npz"
    if not path.exists() or tuple(args.res) != (64, 64):
        return None
    fx = np.load(path)
    if fx["omegas"].shape != omegas.shape or not np.allclose(fx["omegas"], omegas, rtol=0, atol=1e-14):
        return None
    A, B, Fd, Fk = mixed
    out = {}
    for name, a, key in (("A", A, "added_mass"), ("B", B, "damping"), ("F", Fd, "diffraction"),
                         ("FK", Fk, "froude_krylov")):
        ref = fx[key]
        out[name] = float(np.max(np.abs(a - ref)) / np.max(np.abs(ref)))
    out["note"] = ("max abs difference / max abs value over all 64 frequencies, mixed path vs the FP64 "
                   "oracle (exact-quadrature Delhommeau, LAPACK)")
    return out


def run_two_body(mh, ctx, args, torch):
    """Grads of the two-body power objective (paper/Power.jl:13-83): two
    1024-panel hemispheres 5 m apart, Wu, indirect, omega = 1.03; one grad =
    J and dJ/d(r1, dx1, omega) through two_body_power(grad=True) (meshes
    generated on the device, forward + adjoint batch, the mesh cotangent
    pulled back to the parameters on the device), timed end to end; against
    the oracle's central differences."""
    kw = dict(resolution=(32, 64), direct=False, tol=args.tol, ctx=ctx)

    def call(prec):
        return mh.two_body_power(1.0, 4.0, 1.03, precision=prec, grad=True, **kw)

    call("mixed")
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        J, g = call("mixed")
    torch.cuda.synchronize()
    dt = (time.perf_counter() - t0) / args.steps
    call("fp64")
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    J64, g64 = call("fp64")
    torch.cuda.synchronize()
    dt64 = time.perf_counter() - t0
    out = {"value": 1.0 / dt, "unit": "grads/s", "ms_per_grad": dt * 1e3,
           "workload": "two_hemispheres_2x1024p_wu_indirect_power_grad", "panels": 2048,
           "timing": "host wall clock around the public call (meshes generated on the device, forward, adjoint, parameter pull-back)",
           "J": J, "grad": g, "fp64_gpu": {"value": 1.0 / dt64, "unit": "grads/s", "ms_per_grad": dt64 * 1e3}}
    path = ROOT / "tests" / "golden" / "two_hemispheres_2048p_wu.npz"
    if path.exists():
        fx = np.load(path)
        out["accuracy_vs_oracle_fd"] = {k: abs(g[k] - float(fx[f"fd_{k}"])) / abs(float(fx[f"fd_{k}"]))
                                        for k in ("r1", "dx1", "omega")}
        out["accuracy_vs_oracle_fd"]["J"] = abs(J - float(fx["power"])) / abs(float(fx["power"]))
        out["accuracy_vs_oracle_fd"]["note"] = ("relative difference to central differences (h = 1e-6) of "
                                                "the FP64 oracle")
    return out


def run_design_batch(mh, args, torch):
    """The uneven design population: 48 seeded hemispheres (radius ~ U(0.5, 2),
    n_theta ~ U{8..40}, n_phi = 2 n_theta: 64 to 1640 panels, 34968 in all),
    16 frequencies in [0.3, 3.0], heave, Delhommeau, mixed; each design's A, B
    and forward-mode dA/dR, dB/dR at every frequency (one
    hydro_batch_jvp call per design), the designs dealt largest first over
    eight library contexts on their own host threads.  Timed end to end on
    the host clock around the public call; one solve = one (design,
    frequency) problem with its radius tangent."""
    pop = mh.designs(0, 48)
    om = np.linspace(0.3, 3.0, 16)
    ctxs = [mh.Context(0) for _ in range(8)]
    try:
        mh.design_batch(pop, om, precision="mixed", tol=args.tol, contexts=ctxs)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            res = mh.design_batch(pop, om, precision="mixed", tol=args.tol, contexts=ctxs)
        torch.cuda.synchronize()
        dt = (time.perf_counter() - t0) / args.steps
        t0 = time.perf_counter()
        res64 = mh.design_batch(pop, om, precision="fp64", contexts=ctxs)
        torch.cuda.synchronize()
        dt64 = time.perf_counter() - t0
    finally:
        for c in ctxs:
            c.close()
    acc = max(float(np.max(np.abs(a.d_added_mass_dR - b.d_added_mass_dR)) / np.max(np.abs(b.d_added_mass_dR)))
              for a, b in zip(res, res64))
    nprob = len(pop) * len(om)
    return {"value": nprob / dt, "unit": "solves/s (each with dA/dR, dB/dR)", "ms_per_batch": dt * 1e3,
            "workload": "design_population_48_hemispheres_64_to_1640p_16omega_heave_delhommeau",
            "panels_total": int(sum(r.nfaces for r in res)), "contexts": len(ctxs),
            "timing": "host wall clock around design_batch (meshes and radius tangents generated on the device, forward + tangent)",
            "fp64_gpu": {"value": nprob / dt64, "unit": "solves/s", "ms_per_batch": dt64 * 1e3,
                         "mode": "FP64 path one frequency at a time, same contexts"},
            "accuracy_dA_dR_vs_fp64": acc}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--res", type=int, nargs=2, default=[64, 64])
    ap.add_argument("--n-omega", type=int, default=64)
    # relative residual of the FP64 refinement; 1e-8 takes two sweeps and leaves A, B, F within
    # 4e-10 and the gradients within 2e-8 of the FP64 path (the metric asks 1e-6 and 1e-5)
    ap.add_argument("--tol", type=float, default=1e-8)
    ap.add_argument("--max-iter", type=int, default=30)
    ap.add_argument("--fp64-omegas", type=int, default=8)
    ap.add_argument("--cpu-columns", type=int, default=64)
    ap.add_argument("--lu", default="tcgen05", choices=["tcgen05", "simt"])
    ap.add_argument("--no-fp64", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-grads", action="store_true")
    ap.add_argument("--no-two-body", action="store_true")
    ap.add_argument("--no-design", action="store_true")
    # precision level of the wave pass's series (0 FP64, 1 the default FP32 Horner series, 2 also the
    # FP32 alpha contraction)
    ap.add_argument("--wave-level", type=int, default=1, choices=[0, 1, 2])
    args = ap.parse_args()
    if args.impl == "reference":
        return run_reference(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
