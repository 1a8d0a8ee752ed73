#!/usr/bin/env python
"""Benchmark of the KPM hot path: Chebyshev moments of an ELL Hamiltonian.

Workload (default, one GPU): nearest-neighbour graphene on 2048 x 2048
primitive cells (8,388,608 sites), t = -2.7 eV, Anderson disorder W = 1 eV
(W(2U-1), seed 1234), ELL width 4 (on-site + 3 bonds), spectrum rescaled by
the Gershgorin bound x 1.01, M = 2048 moments for R = 8 random-phase vectors
advanced together, complex128.  A step is one full recursion (all M moments
for the R vectors): N * R * (M - 1) site-steps.  Inputs are device-resident
in the timed region and larger than L2 (one vector set is 1.07 GB).

Reported on one JSON line: site-steps/s (value), the roofline of the
dominant kernel (the fused Chebyshev step) against measured HBM bandwidth,
its FP64 ceiling (measured live), an end-to-end figure through the
reference-facing host-pointer call, the CPU baseline (jclsquant's own
kernels, compiled from its sources, or the C restatement), and SM clocks
sampled during the timed region.

--impl reference times jclsquant's CPU path on the host cores instead, or says that it is
unavailable where its sources are absent.
Multi-GPU (torchrun): replicas, each rank runs its own R vectors on the same
lattice (weak scaling), no data-path collective.
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

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "site-steps/s & HBM GB/s: batched c64 vs plain c128 KPM at ≤1e-6 DOS error"
UNIT = "site-steps/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--cells", type=int, default=2048, help="lattice side in primitive cells")
    ap.add_argument("--M", type=int, default=2048)
    ap.add_argument("--R", type=int, default=8)
    ap.add_argument("--W", type=float, default=1.0)
    ap.add_argument("--dtype", default="c128", choices=["c128", "c64"])
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-clocks", action="store_true")
    ap.add_argument("--cpu-seconds", type=float, default=12.0, help="target CPU-baseline sample length")
    ap.add_argument("--no-batched", action="store_true", help="skip the batched complex64 ensemble measurement")
    ap.add_argument("--batch-inst", type=int, default=256)
    ap.add_argument("--batch-M", type=int, default=1024)
    ap.add_argument("--batch-R", type=int, default=2)
    ap.add_argument("--batch-side-max", type=int, default=512)
    ap.add_argument("--no-adjoint", action="store_true", help="skip the differentiable-DOS measurement")
    ap.add_argument("--adj-cells", type=int, default=512)
    ap.add_argument("--adj-M", type=int, default=1024)
    ap.add_argument("--adj-fd", type=int, default=64, help="parameters checked by central differences")
    ap.add_argument("--no-setup", action="store_true", help="skip the operator-construction measurement")
    ap.add_argument("--no-sigma", action="store_true", help="skip the time-domain Kubo (for_time_sigma) measurement")
    ap.add_argument("--no-driven", action="store_true", help="skip the light-pulse operator update measurement")
    ap.add_argument("--sigma-cells", type=int, default=1024)
    ap.add_argument("--sigma-M", type=int, default=512, help="Fermi-Dirac (commutator series) terms")
    ap.add_argument("--sigma-len-t", type=int, default=32)
    ap.add_argument("--no-time", action="store_true", help="skip the time-evolution (for_time) measurement")
    ap.add_argument("--time-M", type=int, default=64, help="series terms per time step")
    ap.add_argument("--time-len", type=int, default=8, help="time steps per timed step")
    ap.add_argument("--time-dt", type=float, default=16.0, help="time step in units of 1/a (scaled H)")
    ap.add_argument("--no-kubo", action="store_true", help="skip the Kubo-Greenwood mu_nm measurement")
    ap.add_argument("--kubo-cells", type=int, default=1024)
    ap.add_argument("--kubo-Nm", type=int, default=256)
    ap.add_argument("--kubo-R", type=int, default=4)
    ap.add_argument("--no-config1", action="store_true", help="skip the 8192-site DOS configuration")
    ap.add_argument("--no-adjoint-kubo", action="store_true", help="skip the differentiable conductivity")
    ap.add_argument("--adjk-cells", type=int, default=512)
    ap.add_argument("--adjk-Nm", type=int, default=256)
    ap.add_argument("--adjk-fd", type=int, default=4, help="parameters checked by central differences")
    ap.add_argument("--e2e-max-steps", type=int, default=6, help="host-pointer passes timed for e2e")
    return ap.parse_args()


# ---------------------------------------------------------------------------
def build_problem(cells, W, seed=1234):
    from minijclsquant_gb300 import lattice
    from minijclsquant_gb300.ell_matrix import gershgorin_bounds_ell
    from minijclsquant_gb300.modifiers import modifier_bounds

    arr = lattice.honeycomb_arrays(cells, cells, t=-2.7, W=W, seed=seed, with_geometry=False)
    bounds = gershgorin_bounds_ell(arr["data"], arr["indices"], arr["n"], factor=1.01)

    class _H:
        pass

    H = _H()
    H.data, H.indices, H.bounds = arr["data"], arr["indices"], bounds
    H.valid_row_values, H.len_row, H.shape = arr["valid"], arr["len_row"], (arr["n"], arr["n"])
    data_kpm = modifier_bounds(H)
    return dict(n=arr["n"], L=arr["len_row"], data_kpm=np.ascontiguousarray(data_kpm),
                indices=np.ascontiguousarray(arr["indices"]), bounds=bounds)


def random_vectors(n, R, seed0):
    from minijclsquant_gb300.observables import random_vector_generator

    return np.stack([random_vector_generator(n, seed0 + r) for r in range(R)])


# ---------------------------------------------------------------------------
class ClockSampler:
    """nvidia-smi samples during the timed region (read-only queries)."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index, enabled=True):
        self.enabled = enabled
        self.idx = device_index
        self.proc = None
        self.path = None

    def __enter__(self):
        if not self.enabled:
            return self
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.idx), "--query-gpu=" + self.FIELDS,
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.enabled or self.proc is None or not self.path:
            return None
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                rows.append((float(parts[1]), float(parts[2]), parts[5:9], float(parts[3])))
            except ValueError:
                continue
        os.unlink(self.path)
        if not rows:
            return None
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for _, _, fl, _ in rows for i, f in enumerate(fl) if f.lower().startswith("active")})
        return {"sm_mhz": statistics.median(r[0] for r in rows), "sm_max_mhz": max(r[1] for r in rows),
                "reasons": reasons, "power_w": statistics.median(r[3] for r in rows), "samples": len(rows)}


# ---------------------------------------------------------------------------
def cpu_reference_kernels():
    """jclsquant's own aAxby / vdot compiled from its .pyx (oracle/_ref), or None."""
    try:
        from oracle import build as ob

        built = ob.build_reference(names=("blas_funs",))
        path = built.get("blas_funs")
        if not path:
            return None
        import importlib.util

        spec = importlib.util.spec_from_file_location("blas_funs", path)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        return mod
    except Exception:
        return None


def cpu_rec_A_tab(M, prob, v, threads, want_moments=False):
    """One CPU recursion of M moments; returns (seconds, kind), or (seconds, kind, moments)
    with want_moments."""
    blas = cpu_reference_kernels()
    n, L = prob["n"], prob["L"]
    if blas is not None:
        # the loop of jclsquant/recurrence_functions.py:9-40 over jclsquant's own kernels
        data, idx = prob["data_kpm"], prob["indices"]
        t0 = time.perf_counter()
        A_vec = np.zeros(M, dtype=np.complex128)
        T0 = np.copy(v)
        T1 = np.zeros(n, dtype=np.complex128)
        blas.aAxby(1 + 0j, 0 + 0j, v, T1, data, idx, L, n, threads)
        A_vec[0] = blas.vdot(1 + 0j, v, v, n, threads)
        A_vec[1] = blas.vdot(1 + 0j, v, T1, n, threads)
        for m in range(2, M):
            blas.aAxby(2.0 + 0j, -1 + 0j, T1, T0, data, idx, L, n, threads)
            T0, T1 = T1, T0
            A_vec[m] = blas.vdot(1 + 0j, v, T1, n, threads)
        dt = time.perf_counter() - t0
        return (dt, "reference", A_vec) if want_moments else (dt, "reference")
    from oracle import oracle

    t0 = time.perf_counter()
    A_vec = oracle.rec_A_tab(M, prob["data_kpm"], prob["indices"], L, v, threads=threads)
    dt = time.perf_counter() - t0
    return (dt, "port", A_vec) if want_moments else (dt, "port")


def cpu_model():
    """The host CPU as lscpu names it (model name, or vendor and model for Arm cores)."""
    try:
        out = subprocess.run(["lscpu"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True,
                             timeout=10).stdout
        kv = {}
        for line in out.splitlines():
            if ":" in line:
                k, v = line.split(":", 1)
                kv.setdefault(k.strip(), v.strip())
        name = kv.get("Model name") or kv.get("BIOS Model name")
        vendor = kv.get("Vendor ID", "")
        if name:
            return (vendor + " " + name).strip()
    except (OSError, subprocess.SubprocessError):
        pass
    import platform

    return platform.processor() or platform.machine()


def moment_parity(mu, ref, rel=1e-10, floor_frac=1e-6):
    """Per-order parity against the reference's moments: max_m |mu_m - ref_m| /
    max(|ref_m|, floor_frac |ref_0|), with the order where it is largest."""
    mu, ref = np.asarray(mu), np.asarray(ref)
    scale = np.maximum(np.abs(ref), floor_frac * np.abs(ref[0]))
    r = np.abs(mu[: len(ref)] - ref) / scale
    return {"orders": int(len(ref)), "max_rel": float(np.max(r)), "at_order": int(np.argmax(r)),
            "max_abs_over_mu0": float(np.max(np.abs(mu[: len(ref)] - ref)) / abs(ref[0])), "tolerance": rel,
            "pass": bool(np.max(r) <= rel)}


def cpu_time_evolve(M2, prob, vs, threads):
    """One time step of U and U_c on the CPU: the loop of jclsquant/recurrence_functions.py:114-143
    (aAxby + axpy2 per order) over jclsquant's own kernels, else the oracle.  (seconds, kind)."""
    from minijclsquant_gb300.kernel_and_moments import moments_U

    blas = cpu_reference_kernels()
    n, L = prob["n"], prob["L"]
    c = moments_U(1.0, M2).astype(np.complex128)
    if blas is not None:
        data, idx = prob["data_kpm"], prob["indices"]
        t0 = time.perf_counter()
        for v in vs:
            T0 = np.copy(v)
            T1 = np.zeros(n, dtype=np.complex128)
            blas.aAxby(1 + 0j, 0 + 0j, v, T1, data, idx, L, n, threads)
            acc = c[0] * v
            acc += c[1] * T1
            for m in range(2, M2):
                blas.aAxby(2.0 + 0j, -1 + 0j, T1, T0, data, idx, L, n, threads)
                T0, T1 = T1, T0
                blas.axpy2(c[m], 1 + 0j, T1, acc, n, threads)
        return time.perf_counter() - t0, "reference"
    from oracle import oracle

    t0 = time.perf_counter()
    for v in vs:
        oracle.rec_A_vec(M2, prob["data_kpm"], prob["indices"], L, c, v, threads=threads)
    return time.perf_counter() - t0, "port"


def run_time_evolution(a, op, n, L, prob, hbm_peak, world):
    """for_time (obv.cu:93-122) on the DOS lattice: U and U_c, one group of two vectors,
    advanced len_t times by the series of exp(-i H dt) with M2 terms.  Value: site-steps/s,
    N * 2 * (M2 - 1) * len_t per timed step.  The dominant kernel is the series step:
    T_{m+1} = 2H T_m - T_{m-1} and series += c_m T_{m+1}, algorithmic bytes per row
    L (value + index) + 2 vectors x 5 x 16 B (T_m gathered once, T_{m-1} read, T_{m+1}
    written, the series read and written)."""
    import ctypes

    import torch

    from minijclsquant_gb300 import _capi, device
    from minijclsquant_gb300.kernel_and_moments import moments_U

    lib = _capi.lib()
    stream = torch.cuda.current_stream()
    M2, len_t, R2 = a.time_M, a.time_len, 2
    c = torch.from_numpy(moments_U(a.time_dt, M2).astype(np.complex128)).cuda()
    uv = torch.from_numpy(random_vectors(n, R2, 4242)).cuda()
    for _ in range(max(1, a.warmup)):
        out = device.time_evolve(op, M2, c, 1, uv)  # the first call also tunes the series step
    torch.cuda.synchronize()
    loop_ms, launches, rows = ctypes.c_double(), ctypes.c_int64(), ctypes.c_int64()
    lib.kpm_ell_profile(op.handle, 1)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(a.steps):
        out = device.time_evolve(op, M2, c, len_t, uv)
    e1.record(stream)
    torch.cuda.synchronize()
    _capi.check(lib.kpm_ell_profile_read(op.handle, ctypes.byref(loop_ms), ctypes.byref(launches),
                                         ctypes.byref(rows)))
    lib.kpm_ell_profile(op.handle, 0)
    ms = max_over_ranks(e0.elapsed_time(e1), world) / a.steps
    n0 = torch.linalg.vector_norm(uv, dim=1)
    drift = float(torch.max(torch.abs(torch.linalg.vector_norm(out, dim=1) - n0) / n0))
    val_bytes = 8 if op.is_real else 16
    bytes_per_row = L * (val_bytes + 4) + R2 * 5 * 16
    step_s = loop_ms.value * 1e-3 / max(1, launches.value)
    gbs = float(n) * bytes_per_row / step_s / 1e9
    kind, rpt, grid, us = ctypes.c_int(), ctypes.c_int(), ctypes.c_int(), ctypes.c_float()
    _capi.check(lib.kpm_ell_series_config(op.handle, _capi.KPM_C128, R2, ctypes.byref(kind), ctypes.byref(rpt),
                                          ctypes.byref(grid), ctypes.byref(us)))
    kname = ("cheb_next_ws_kernel<SER> (producer warp, %d row(s)/thread%s)"
             % (rpt.value, ", two sub-tiles per stage" if kind.value == 3 else "") if kind.value in (2, 3)
             else "cheb_step_kernel (grid-stride, MODE_NEXT STORE|SERIES)")
    blk = {"value": float(n) * R2 * (M2 - 1) * len_t * world / (ms * 1e-3), "unit": UNIT, "ms_per_step": ms,
           "config": {"vectors": "U, U_c", "M2": M2, "len_t": len_t, "dt": a.time_dt, "sites": n},
           "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm_peak, "unit": "GB/s", "frac": gbs / hbm_peak,
                        "kernel": kname, "grid": grid.value, "algorithmic_bytes_per_launch": float(n) * bytes_per_row,
                        "avg_launch_ms": step_s * 1e3},
           "norm_drift": drift,
           "gpu_launches": len_t * (M2 + 1) * a.steps,
           "note": "exp(-i H dt) by its Chebyshev series (moments_U); norm_drift = max |(|U(t)| - |U(0)|)| / |U(0)|"}
    # the same workload in float-float complex128 (KPM_C128F, FP32 pipe), same memory streams
    out_f = device.time_evolve(op, M2, c, 1, uv, dtype="c128f")  # tunes the float-float series step
    torch.cuda.synchronize()
    lib.kpm_ell_profile(op.handle, 1)
    f0 = torch.cuda.Event(enable_timing=True)
    f1 = torch.cuda.Event(enable_timing=True)
    f0.record(stream)
    for _ in range(a.steps):
        out_f = device.time_evolve(op, M2, c, len_t, uv, dtype="c128f")
    f1.record(stream)
    torch.cuda.synchronize()
    _capi.check(lib.kpm_ell_profile_read(op.handle, ctypes.byref(loop_ms), ctypes.byref(launches),
                                         ctypes.byref(rows)))
    lib.kpm_ell_profile(op.handle, 0)
    ms_f = max_over_ranks(f0.elapsed_time(f1), world) / a.steps
    step_f = loop_ms.value * 1e-3 / max(1, launches.value)
    gbs_f = float(n) * bytes_per_row / step_f / 1e9
    blk["c128f"] = {"value": float(n) * R2 * (M2 - 1) * len_t * world / (ms_f * 1e-3), "ms_per_step": ms_f,
                    "roofline": {"bound": "hbm", "achieved": gbs_f, "peak": hbm_peak, "unit": "GB/s",
                                 "frac": gbs_f / hbm_peak, "kernel": "ff_next_kernel<SER> (float-float series step)",
                                 "avg_launch_ms": step_f * 1e3},
                    "max_abs_diff_vs_c128_over_max": float(torch.max(torch.abs(out_f - out)) / torch.max(torch.abs(out))),
                    "note": "dtype KPM_C128F: every real as a float pair (~48 bits), FP32 pipe; opt-in"}
    if not a.no_cpu and world == 1:
        threads = os.cpu_count() or 1
        vs = random_vectors(n, R2, 4242)
        dt, kind_s = cpu_time_evolve(M2, prob, vs, threads)
        blk["cpu_baseline"] = {"value": float(n) * R2 * (M2 - 1) / dt, "unit": UNIT, "cores": threads,
                               "kind": kind_s, "sample": "one time step of U and U_c (M2=%d) on the full %d-site "
                               "operator in %.2f s" % (M2, n, dt)}
    return blk


def run_setup(a, prob, host_s, hbm_peak):
    """Operator construction for the DOS lattice: the host route (numpy builder, Gershgorin
    bound, modifier_bounds, upload and kpm_ell_create; host_s) against the device builder
    (on-site energies on the host, then kpm_honeycomb_ell, kpm_ell_gershgorin_partner,
    kpm_ell_scale_values and kpm_ell_create from device arrays), both to a ready handle.
    The generator kernel is timed alone with CUDA events: it writes data (16 B), column
    (4 B), valid (4 B) and partner (8 B) per slot and reads one on-site energy per site."""
    import torch

    from minijclsquant_gb300 import _capi, lattice

    kw = dict(t=-2.7, W=a.W, seed=1234, bounds_factor=1.01)
    lattice.honeycomb_device(64, 64, **kw)  # first launches, allocator warm-up
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    g = lattice.honeycomb_device(a.cells, a.cells, **kw)
    torch.cuda.synchronize()
    dev_s = time.perf_counter() - t0
    same = bool(np.array_equal(g.bounds, prob["bounds"])) and bool(
        torch.equal(g.data_kpm, torch.from_numpy(prob["data_kpm"]).cuda())) and bool(
        torch.equal(g.indices, torch.from_numpy(prob["indices"]).cuda()))
    n, L = g.n, g.len_row
    eps = torch.from_numpy(lattice._onsite_energies(n, a.W, 1234, 0.0, None)[0]).cuda()
    disp = np.ascontiguousarray(lattice._bond_displacements(lattice.A_CC).reshape(-1))
    lib = _capi.lib()
    stream = torch.cuda.current_stream()
    sp = ctypes_stream(stream)
    reps = 5
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(reps):
        _capi.check(lib.kpm_honeycomb_ell(a.cells, a.cells, 1, -2.7, eps.data_ptr(), L, disp.ctypes.data,
                                          g.data.data_ptr(), g.indices.data_ptr(), g.valid.data_ptr(), None, None,
                                          g.partner.data_ptr(), sp), "kpm_honeycomb_ell")
    e1.record(stream)
    torch.cuda.synchronize()
    k_s = e0.elapsed_time(e1) * 1e-3 / reps
    bytes_k = float(n) * (L * (16 + 4 + 4 + 8) + 8)
    gbs = bytes_k / k_s / 1e9
    del g
    torch.cuda.empty_cache()
    return {"sites": n, "host_route_s": host_s, "device_route_s": dev_s, "speedup": host_s / dev_s,
            "bit_identical": same,
            "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm_peak, "unit": "GB/s", "frac": gbs / hbm_peak,
                         "kernel": "honeycomb_kernel", "algorithmic_bytes_per_launch": bytes_k,
                         "avg_launch_ms": k_s * 1e3},
            "note": "host route: honeycomb_arrays + gershgorin_bounds_ell + modifier_bounds + DeviceELL upload; "
                    "device route: lattice.honeycomb_device (both end at a ready operator handle)"}


def run_time_sigma(a, hbm_peak, world):
    """Time-domain Kubo correlator sigma(t_j) = <U_c(t_j)|V1 U(t_j)> (for_time_sigma,
    obv.cu:124-176; the historical kpm_sigma_time_gpu): U_c(0) = the commutator series of
    the Fermi-Dirac moments (M terms, V2 = H o dx / a), then U and U_c advanced len_t - 1
    times by the exp(-i H dt) series (M2 terms, truncated where |c_m| <= 1e-15) and
    correlated with V1 = -i H o dy.  One random-phase vector, as the reference calls it.
    Value: site-steps/s counting N per commutator order and N per series order of each of
    U and U_c: N ((M - 1) + 2 (M2 - 1)(len_t - 1))."""
    import torch

    from minijclsquant_gb300 import device, lattice
    from minijclsquant_gb300.constants import hbar_fs
    from minijclsquant_gb300.kernel_and_moments import JacksonKernel, moments_FD_T0, moments_U
    from minijclsquant_gb300.modifiers import modifier_bounds, modifier_velocity, modifier_velocity_bounds
    from minijclsquant_gb300.observables import random_vector_generator

    H = lattice.honeycomb(a.sigma_cells, a.sigma_cells, t=-2.7, W=a.W, seed=1234)
    n, L = H.shape[0], H.len_row
    M, len_t = a.sigma_M, a.sigma_len_t
    t_vec = np.linspace(0, 5 * hbar_fs * M / (np.pi * H.bounds[1]), 500)
    dt_kpm = t_vec[1] * H.bounds[1] / hbar_fs
    cu = moments_U(dt_kpm, M)
    M2 = 0
    while np.abs(cu[M2]) > 1e-15 and M2 < M - 1:
        M2 += 1
    cu = moments_U(dt_kpm, M2).astype(np.complex128)
    cfd = (moments_FD_T0(0.0, M) * JacksonKernel(M)).astype(np.complex128)
    Hk = device.DeviceELL(modifier_bounds(H), H.indices, L)
    V1 = device.DeviceELL(modifier_velocity(H, "y"), H.indices, L)
    V2 = device.DeviceELL(modifier_velocity_bounds(H, "x"), H.indices, L)
    v = torch.from_numpy(random_vector_generator(n, 77)).cuda()
    for _ in range(max(1, a.warmup)):
        sig = device.time_sigma(Hk, V1, V2, cu, M2, cfd, M, 2, v)
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(a.steps):
        sig = device.time_sigma(Hk, V1, V2, cu, M2, cfd, M, len_t, v)
    e1.record(stream)
    torch.cuda.synchronize()
    ms = max_over_ranks(e0.elapsed_time(e1), world) / a.steps
    site_steps = float(n) * ((M - 1) + 2 * (M2 - 1) * (len_t - 1))
    # the same call in float-float complex128 (KPM_C128F): commutator series, series and
    # correlator on the FP32 pipe
    sig_f = device.time_sigma(Hk, V1, V2, cu, M2, cfd, M, 2, v, dtype="c128f")
    torch.cuda.synchronize()
    f0 = torch.cuda.Event(enable_timing=True)
    f1 = torch.cuda.Event(enable_timing=True)
    f0.record(stream)
    for _ in range(a.steps):
        sig_f = device.time_sigma(Hk, V1, V2, cu, M2, cfd, M, len_t, v, dtype="c128f")
    f1.record(stream)
    torch.cuda.synchronize()
    ms_f = max_over_ranks(f0.elapsed_time(f1), world) / a.steps
    blk = {"value": site_steps * world / (ms * 1e-3), "unit": UNIT, "ms_per_step": ms,
           "config": {"lattice": "honeycomb %dx%d cells (%d sites), W=%g" % (a.sigma_cells, a.sigma_cells, n, a.W),
                      "M": M, "M2": M2, "len_t": len_t, "dt_kpm": dt_kpm, "vectors": 1},
           "gpu_launches": (M + 1) + (len_t - 1) * (M2 + 2) + 2 * len_t,
           "sigma_0": [float(np.real(sig.cpu().numpy()[0])), float(np.imag(sig.cpu().numpy()[0]))],
           "note": "U and U_c advance as one set of two vectors through the autotuned series step",
           "c128f": {"value": site_steps * world / (ms_f * 1e-3), "ms_per_step": ms_f,
                     "max_abs_diff_vs_c128_over_max": float(torch.max(torch.abs(sig_f - sig)) / torch.max(torch.abs(sig))),
                     "note": "dtype KPM_C128F: float pairs (~48 bits) on the FP32 pipe; opt-in"}}
    if not a.no_cpu and world == 1:
        from oracle import oracle

        threads = os.cpu_count() or 1
        lt = 2
        t0 = time.perf_counter()
        oracle.for_time_sigma(modifier_bounds(H), modifier_velocity(H, "y"), modifier_velocity_bounds(H, "x"),
                              H.indices, L, cu, cfd, lt, v.cpu().numpy(), M, M2, threads=threads)
        dt = time.perf_counter() - t0
        blk["cpu_baseline"] = {"value": float(n) * ((M - 1) + 2 * (M2 - 1) * (lt - 1)) / dt, "unit": UNIT,
                               "cores": threads, "kind": "port",
                               "sample": "for_time_sigma restated in C (oracle), len_t=%d, same lattice and M, M2 "
                                         "(%.2f s)" % (lt, dt)}
    del Hk, V1, V2
    torch.cuda.empty_cache()
    return blk


def run_driven(a, hbm_peak):
    """The operator of a light-driven system, H(t) = H0 o exp(i A0 (cos wt dx + sin wt dy) / ch)
    (the circular pulse form of light_modifier_cython, Extra_funs.pyx:301-317), written into
    the operator's values on the device once per time step (kpm_ell_light_update), on the DOS
    lattice with its bond vectors.  Algorithmic bytes per slot: H0, dx, dy read and the
    stored value written, 4 x 16 B."""
    import torch

    from minijclsquant_gb300 import device, lattice
    from minijclsquant_gb300.observables import random_vector_generator

    g = lattice.honeycomb_device(a.cells, a.cells, t=-2.7, W=a.W, seed=1234, geometry=True)
    op = device.DeviceELL(g.data_kpm, g.indices, g.len_row, complex_values=True)
    prm = (2.0, 1.7, "r", 0.8)
    op.light_update(g.data_kpm, g.dx, g.dy, "circle_packed", prm, 0.5)  # warm-up
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream()
    reps = 10
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for k in range(reps):
        op.light_update(g.data_kpm, g.dx, g.dy, "circle_packed", prm, 0.5 + 0.01 * k)
    e1.record(stream)
    torch.cuda.synchronize()
    # the Hermiticity check is lazy: it runs on the first read of the flag below, not per update
    ms = e0.elapsed_time(e1) / reps
    slots = float(g.n) * g.len_row
    gbs = slots * 64 / (ms * 1e-3) / 1e9
    herm = bool(op.hermitian)
    v = torch.from_numpy(random_vector_generator(g.n, 3)).cuda()
    mu = device.cheb_moments(op, 64, v)
    blk = {"sites": g.n, "ms_per_update": ms, "hermitian_after_update": herm,
           "mu0_over_n": float(abs(mu[0].item()) / g.n),
           "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm_peak, "unit": "GB/s", "frac": gbs / hbm_peak,
                        "kernel": "light_update_kernel", "algorithmic_bytes_per_update": slots * 64,
                        "limiter": "FP64 pipe: per bond slot one table-driven sin/cos and two complex products"},
           "note": "kpm_ell_light_update: H(t) into the operator's stored values, once per time step"}
    del op, g
    torch.cuda.empty_cache()
    return blk


def ctypes_stream(stream):
    import ctypes

    return ctypes.c_void_p(int(stream.cuda_stream))


def cpu_baseline(prob, target_s):
    """The reference's rec_A_tab loop on the host cores for vector seed 1000 (the GPU's vector 0
    on rank 0); returns (block, moments) so the caller can check parity on the same input."""
    threads = os.cpu_count() or 1
    v = random_vectors(prob["n"], 1, 1000)[0]
    dt, kind = cpu_rec_A_tab(4, prob, v, threads)  # calibration (also warms caches)
    per_step = max(dt / 3, 1e-6)
    M = int(min(512, max(8, target_s / per_step)))
    dt, kind, mu = cpu_rec_A_tab(M, prob, v, threads, want_moments=True)
    steps = prob["n"] * (M - 1)
    return {"value": steps / dt, "unit": UNIT, "cores": threads, "kind": kind, "cpu_model": cpu_model(),
            "sample": "rec_A_tab loop, 1 vector (seed 1000), M=%d on the full %d-site operator (%d site-steps in "
                      "%.2f s)" % (M, prob["n"], steps, dt)}, mu


# ---------------------------------------------------------------------------
def dist_init():
    import torch

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    elif torch.cuda.is_available():
        torch.cuda.set_device(0)
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist

        dist.barrier()


def max_over_ranks(x, world):
    if world == 1:
        return x
    import torch
    import torch.distributed as dist

    t = torch.tensor([x], dtype=torch.float64, device="cuda")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def workload_desc(a, n):
    return ("plain %s KPM moments: honeycomb %dx%d cells (%d sites), t=-2.7 eV, W=%g eV, ELL width 4, "
            "M=%d, R=%d vectors per launch" % (a.dtype, a.cells, a.cells, n, a.W, a.M, a.R))


def run_reference_arm(a):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    if cpu_reference_kernels() is None:
        # a restatement of the recursion in this repository is not the reference's arm
        print(json.dumps({"impl": "reference", "unavailable": "jclsquant's kernels (blas_funs.pyx) are not built here: "
                          "its sources are absent"}), flush=True)
        return
    prob = build_problem(a.cells, a.W)
    threads = os.cpu_count() or 1
    v = random_vectors(prob["n"], 1, 1000)[0]
    dt, kind = cpu_rec_A_tab(4, prob, v, threads)
    per_step = max(dt / 3, 1e-6)
    M = int(min(256, max(8, 10.0 / per_step)))
    for _ in range(a.warmup):
        cpu_rec_A_tab(M, prob, v, threads)
    times = []
    for _ in range(a.steps):
        dt, kind = cpu_rec_A_tab(M, prob, v, threads)
        times.append(dt)
    tot = sum(times)
    value = prob["n"] * (M - 1) * a.steps / tot
    sample = ("each step: rec_A_tab loop (aAxby + vdot per order), 1 vector, M=%d on the full %d-site operator"
              % (M, prob["n"]))
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": a.steps, "warmup": a.warmup,
            "ms_per_step": 1e3 * tot / a.steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic", "impl": "reference",
            "config": {"workload": "plain c128 KPM moments on the %d-site honeycomb operator of the GPU arm "
                                   "(%dx%d cells, W=%g eV, ELL width 4); sampled at M=%d moments and R=1 "
                                   "vector per step (the GPU arm runs M=%d, R=%d; the unit, site-steps/s, is "
                                   "per site, vector and order)" % (prob["n"], a.cells, a.cells, a.W, M, a.M, a.R),
                       "sites": prob["n"], "M": M, "R": 1, "gpu_arm_M": a.M, "gpu_arm_R": a.R},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": kind, "sample": sample,
                             "cpu_model": cpu_model()},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def executed_steps(M, doubled):
    """Recursion steps after the first one: M - 2 (direct) or ceil(M/2) - 1 (doubled)."""
    return (M + 1) // 2 - 1 if doubled else max(0, M - 2)


def launches_per_recursion(M, R, doubled=False):
    groups = []
    r = R
    while r > 0:
        g = 8 if r >= 8 else 4 if r >= 4 else 2 if r >= 2 else 1
        groups.append(g)
        r -= g
    steps = executed_steps(M, doubled)
    # step launches (operators beyond the one-launch form): packing with mu_0, first step, their reduction,
    # the steps, their chunked reductions; doubled: packing (2), half norms, first step and its reduction,
    # the steps, their reductions, the assembly of the moments
    per_group = 2 + 1 + steps + (steps + 1 + 127) // 128 + 3 if doubled else 3 + steps + (steps + 127) // 128
    return per_group * len(groups)


def load_traffic(kernel_tag):
    """DRAM bytes per launch from the committed ncu summary, if present."""
    path = os.path.join(ROOT, "profiles", kernel_tag + ".md")
    if not os.path.exists(path):
        return None
    for line in open(path):
        if line.strip().startswith("traffic_bytes_per_launch:"):
            try:
                return float(line.split(":", 1)[1].strip().split()[0])
            except ValueError:
                return None
    return None


def run_batched(a, hbm_peak, steps, warmup):
    """The batched mixed-precision configuration: uneven honeycomb instances (side
    32..side_max cells, W ~ U[0, 2] eV, own seed each), R vectors per instance, M
    moments; complex64 recursion with FP64 moment accumulation, timed against the
    same ensemble in complex128; DOS error of every instance against complex128."""
    import torch

    from minijclsquant_gb300 import batched

    t0 = time.perf_counter()
    datas, idxs, L, bnds, prm = batched.honeycomb_ensemble(a.batch_inst, side_range=(32, a.batch_side_max),
                                                           W_range=(0.0, 2.0), seed=42)
    B = batched.BatchedELL(datas, idxs, L)
    setup_s = time.perf_counter() - t0
    cpu_sample = [(datas[k], idxs[k]) for k in range(min(16, len(datas)))]
    del datas, idxs
    R, M = a.batch_R, a.batch_M
    v = torch.from_numpy(batched.ensemble_vectors(B.rows, R)).cuda()
    stream = torch.cuda.current_stream()

    def timed(dtype, k_steps, w_steps):
        for _ in range(w_steps):
            mu = B.moments(M, v, dtype=dtype)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(k_steps):
            mu = B.moments(M, v, dtype=dtype)
        e1.record(stream)
        torch.cuda.synchronize()
        return mu, e0.elapsed_time(e1) / k_steps

    doubled = bool(B.doubling)  # the direct recursion unless doubling was requested
    mu64, ms64 = timed("c64", steps, warmup)
    mu128, ms128 = timed("c128", 1, 1)
    cfg64, cfg128 = B.step_config("c64", R), B.step_config("c128", R)
    # the opt-in doubled moments of the same ensemble, both precisions
    B.set_doubling(True)
    mu64x, ms64x = timed("c64", 1, 1)
    mu128x, ms128x = timed("c128", 1, 1)
    B.set_doubling(doubled)
    mu64 = mu64.cpu().numpy()
    mu128d = mu128.cpu().numpy()  # errors are taken against direct complex128, the reference's algorithm
    mu64x = mu64x.cpu().numpy()
    d64x = batched.batched_dos(mu64x, bnds, M)
    site_steps = float(B.n_total) * R * (M - 1)  # per moment delivered
    val64 = site_steps / (ms64 * 1e-3)
    val128 = site_steps / (ms128 * 1e-3)
    d64 = batched.batched_dos(mu64, bnds, M)
    d128 = batched.batched_dos(mu128d, bnds, M)
    dos_err = max(float(np.max(np.abs(x[:, 1] - y[:, 1])) / np.max(np.abs(y[:, 1]))) for x, y in zip(d64, d128))
    dos_err_x = max(float(np.max(np.abs(x[:, 1] - y[:, 1])) / np.max(np.abs(y[:, 1]))) for x, y in zip(d64x, d128))
    mom_err = np.abs(mu64 - mu128d) / np.abs(mu128d[:, :, :1])
    per_order = mom_err.max(axis=(0, 1))
    # bytes per executed site-step: split-float value (8 B) + index per slot, T_m, T_{m-1},
    # T_{m+1}, and v_l (direct) or |v|^2/2 (doubled)
    bytes_per_site_step = L * (8 + 4) / R + 3 * 8 + (4 if doubled else 8)
    exec_steps = executed_steps(M, doubled) + 1
    exec_rate = float(B.n_total) * R * exec_steps / (ms64 * 1e-3)
    ach = bytes_per_site_step * exec_rate / 1e9
    cpu = None
    if not a.no_cpu:
        # the reference's way through an ensemble: one rec_A_tab per instance and vector
        # (jclsquant/recurrence_functions.py:9-40 over its own aAxby / vdot), on the first
        # instances of the ensemble at reduced M, per site-step
        threads = os.cpu_count() or 1
        Mc, site_steps_c, t_c, kind_c = 512, 0.0, 0.0, "port"
        vcpu = batched.ensemble_vectors(np.array([d.size // L for d, _ in cpu_sample]), R)
        off = 0
        for d, ix in cpu_sample:
            nk = d.size // L
            prob_k = {"n": nk, "L": L, "data_kpm": np.ascontiguousarray(d), "indices": np.ascontiguousarray(ix)}
            for r in range(R):
                dt_k, kind_c = cpu_rec_A_tab(Mc, prob_k, np.ascontiguousarray(vcpu[r, off:off + nk]), threads)
                t_c += dt_k
                site_steps_c += nk * (Mc - 1)
            off += nk
        cpu = {"value": site_steps_c / t_c, "unit": UNIT, "cores": threads, "kind": kind_c,
               "sample": "rec_A_tab loop per instance and vector, the first %d instances (%d sites), R=%d, M=%d "
                         "(%.2f s)" % (len(cpu_sample), int(sum(d.size // L for d, _ in cpu_sample)), R, Mc, t_c),
               "gpu_c64_over_cpu": val64 / (site_steps_c / t_c)}
    return {"workload": "%d honeycomb instances, sides U{32..%d} cells (%d sites total), W~U[0,2] eV, R=%d, M=%d"
                        % (B.n_inst, a.batch_side_max, B.n_total, R, M),
            "cpu_baseline": cpu,
            "value": val64, "unit": UNIT, "ms_per_step": ms64, "dtype": "c64 recursion, f64 moment accumulation",
            "hbm_gbs": ach, "roofline": {"bound": "hbm", "achieved": ach, "peak": hbm_peak, "unit": "GB/s",
                                         "frac": ach / hbm_peak, "bytes_per_site_step": bytes_per_site_step},
            "c128_same_ensemble": {"value": val128, "ms_per_step": ms128},
            "speedup_c64_vs_c128": val64 / val128,
            "doubling": {"used_above": doubled,
                         "note": "opt-in; ceil(M/2)-1 steps; values count site-steps per moment delivered",
                         "c64": {"value": site_steps / (ms64x * 1e-3), "ms_per_step": ms64x,
                                 "dos_error_max_over_instances": dos_err_x},
                         "c128": {"value": site_steps / (ms128x * 1e-3), "ms_per_step": ms128x}},
            "dos_error_max_over_instances": dos_err,
            "moment_error_vs_c128": {"max_rel_mu0": float(per_order.max()),
                                     "by_order": {str(m): float(per_order[m]) for m in (1, 10, 100, 500, M - 1) if m < M}},
            "setup_s": setup_s, "graph": "one CUDA graph launch per recursion",
            "graph_vs_step_sum": {
                "step_kernel_us": cfg64["step_us"], "step_launches": executed_steps(M, doubled),
                "steps_sum_ms": executed_steps(M, doubled) * cfg64["step_us"] * 1e-3, "graph_ms": ms64,
                "other_ms_frac": (ms64 - executed_steps(M, doubled) * cfg64["step_us"] * 1e-3) / ms64,
                "note": "time of the graph replay not spent in the step kernel (first step, reductions, launch "
                        "gaps): the most a single persistent launch could save"},
            "step_kernel": {"c64": cfg64, "c128": cfg128},
            "gpu_launches_per_step": 1 + executed_steps(M, doubled) + (M + 127) // 128 + (3 if doubled else 0)}


def run_adjoint(a, steps, warmup):
    """The differentiable DOS configuration: 512 x 512 cells (524,288 sites), learnable
    FP64 on-site potentials U[-0.5, 0.5] eV and per-bond hoppings -2.7 + U[-0.1, 0.1] eV,
    L2 loss against the DOS of another disorder draw on 512 energies, M = 1024, R = 4,
    checkpoints every 32 orders.  Reports forward and forward+backward times (their
    ratio is the adjoint cost) and the gradient against central differences
    (h = 1e-6) on 64 seeded random parameters."""
    import torch

    from minijclsquant_gb300 import adjoint

    cells, M, R = a.adj_cells, a.adj_M, 4
    n = 2 * cells * cells
    rng = np.random.default_rng(5)
    on0 = rng.uniform(-0.5, 0.5, n)
    hop0 = None
    plan = adjoint.DosPlan(cells, cells, M=M, R=R, n_energies=512, ckpt=32, onsite0=on0)
    hop0 = -2.7 + rng.uniform(-0.1, 0.1, plan.n_bonds)
    onsite = torch.tensor(on0, dtype=torch.float64, device="cuda", requires_grad=True)
    hop = torch.tensor(hop0, dtype=torch.float64, device="cuda", requires_grad=True)
    rng_t = np.random.default_rng(6)
    with torch.no_grad():
        target = adjoint.kpm_dos(torch.tensor(rng_t.uniform(-0.5, 0.5, n), device="cuda"),
                                 torch.tensor(-2.7 + rng_t.uniform(-0.1, 0.1, plan.n_bonds), device="cuda"), plan)

    def fwd():
        with torch.no_grad():
            return adjoint.dos_l2_loss(onsite, hop, plan, target)

    def fwd_bwd():
        onsite.grad = None
        hop.grad = None
        loss = adjoint.dos_l2_loss(onsite, hop, plan, target)
        loss.backward()
        return loss

    def timeit(fn, k):
        for _ in range(warmup):
            fn()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(k):
            fn()
        torch.cuda.synchronize()
        return (time.perf_counter() - t0) / k

    from minijclsquant_gb300 import _capi

    t_f = timeit(fwd, steps)
    t_fb = timeit(fwd_bwd, steps)  # float-float backward (the plan's default)
    go, gh = onsite.grad.detach().cpu().numpy(), hop.grad.detach().cpu().numpy()
    plan.backward_dtype = _capi.KPM_C128  # the same pass in FP64 arithmetic
    t_fb64 = timeit(fwd_bwd, steps)
    go64, gh64 = onsite.grad.detach().cpu().numpy(), hop.grad.detach().cpu().numpy()
    plan.backward_dtype = _capi.KPM_C128F
    pick = np.random.default_rng(7)
    half = a.adj_fd // 2
    params = [("onsite", int(i)) for i in pick.choice(n, half, replace=False)] + \
             [("hopping", int(i)) for i in pick.choice(plan.n_bonds, a.adj_fd - half, replace=False)]
    h = 1e-6
    worst = 0.0
    scale = max(np.max(np.abs(go)), np.max(np.abs(gh)))
    with torch.no_grad():
        for which, i in params:
            p = onsite if which == "onsite" else hop
            old = p[i].item()
            p[i] = old + h
            lp = fwd().item()
            p[i] = old - h
            lm = fwd().item()
            p[i] = old
            fd = (lp - lm) / (2 * h)
            an = (go if which == "onsite" else gh)[i]
            worst = max(worst, abs(an - fd) / scale)
        # the same gradient against a fourth-order stencil at h = 1e-4: the rounding noise of
        # the loss difference (~1e-6 of the gradient at h = 1e-6) drops by 100, truncation is O(h^4)
        h4 = 1e-4
        worst4 = 0.0
        for which, i in params[: min(16, len(params))]:
            p = onsite if which == "onsite" else hop
            old = p[i].item()
            vals = []
            for k in (2, 1, -1, -2):
                p[i] = old + k * h4
                vals.append(fwd().item())
            p[i] = old
            fd4 = (-vals[0] + 8 * vals[1] - 8 * vals[2] + vals[3]) / (12 * h4)
            an = (go if which == "onsite" else gh)[i]
            worst4 = max(worst4, abs(an - fd4) / scale)
    return {"workload": "differentiable DOS: %dx%d cells (%d sites), M=%d, R=%d, 512 energies, checkpoints every 32"
                        % (cells, cells, n, M, R),
            "forward_ms": 1e3 * t_f, "forward_backward_ms": 1e3 * t_fb, "backward_over_forward": (t_fb - t_f) / t_f,
            "fwd_plus_bwd_over_fwd": t_fb / t_f,
            "backward": "float-float (KPM_C128F) adjoint, recompute and gradient; FP64 forward and checkpoints",
            "fp64_backward": {"forward_backward_ms": 1e3 * t_fb64, "fwd_plus_bwd_over_fwd": t_fb64 / t_f,
                              "max_abs_diff_vs_float_float_over_max_grad": float(
                                  max(np.max(np.abs(go - go64)), np.max(np.abs(gh - gh64)))
                                  / max(np.max(np.abs(go64)), np.max(np.abs(gh64))))},
            "fd_check": {"params": len(params), "h": h, "max_abs_err_over_max_grad": worst,
                         "stencil4_h1e-4": {"params": min(16, len(params)), "max_abs_err_over_max_grad": worst4}}}


def run_adjoint_kubo(a, steps):
    """The differentiable Kubo-Greenwood conductivity: honeycomb cells x cells, learnable FP64
    on-site potentials U[-0.5, 0.5] eV and per-bond hoppings -2.7 + U[-0.1, 0.1] eV, V_x =
    -i H o dx, Nm moments, R = 4 vectors, sigma(E) on 64 energies in [-0.9 a, 0.9 a], loss = L2
    against sigma of another disorder draw.  Everything complex128; the moment matrix and the
    two mixing products of the backward are exact digit products on the tensor cores.  Reports forward and
    forward+backward times (their ratio is the adjoint cost) and central differences
    (h = 1e-6) on a few seeded parameters."""
    import torch

    from minijclsquant_gb300 import adjoint

    cells, Nm, R = a.adjk_cells, a.adjk_Nm, 4
    n = 2 * cells * cells
    rng = np.random.default_rng(21)
    on0 = rng.uniform(-0.5, 0.5, n)
    hop0 = -2.7 + rng.uniform(-0.1, 0.1, 3 * cells * cells)
    t0 = time.perf_counter()
    plan = adjoint.KuboPlan(cells, cells, Nm, R=R, n_energies=64, onsite0=on0, hopping0=hop0)
    setup_s = time.perf_counter() - t0
    rng_t = np.random.default_rng(22)
    with torch.no_grad():
        target = adjoint.kpm_sigma(torch.tensor(rng_t.uniform(-0.5, 0.5, n), device="cuda"),
                                   torch.tensor(-2.7 + rng_t.uniform(-0.1, 0.1, plan.n_bonds), device="cuda"), plan)
    onsite = torch.tensor(on0, dtype=torch.float64, device="cuda", requires_grad=True)
    hop = torch.tensor(hop0, dtype=torch.float64, device="cuda", requires_grad=True)

    def fwd():
        with torch.no_grad():
            return adjoint.sigma_l2_loss(onsite, hop, plan, target)

    def fwd_bwd():
        onsite.grad = None
        hop.grad = None
        loss = adjoint.sigma_l2_loss(onsite, hop, plan, target)
        loss.backward()
        return loss

    def timeit(fn, k):
        fn()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(k):
            fn()
        torch.cuda.synchronize()
        return (time.perf_counter() - t0) / k

    k = max(1, min(steps, 2))
    torch.cuda.reset_peak_memory_stats()
    t_f = timeit(fwd, k)
    t_fb = timeit(fwd_bwd, k)
    peak_gb = torch.cuda.max_memory_allocated() / 1e9
    go, gh = onsite.grad.detach().cpu().numpy(), hop.grad.detach().cpu().numpy()
    scale = max(np.max(np.abs(go)), np.max(np.abs(gh)))
    pick = np.random.default_rng(23)
    half = a.adjk_fd // 2
    params = [("onsite", int(i)) for i in pick.choice(n, half, replace=False)] + \
             [("hopping", int(i)) for i in pick.choice(plan.n_bonds, a.adjk_fd - half, replace=False)]
    h = 1e-6
    worst = 0.0
    with torch.no_grad():
        for which, i in params:
            p = onsite if which == "onsite" else hop
            old = p[i].item()
            p[i] = old + h
            lp = fwd().item()
            p[i] = old - h
            lm = fwd().item()
            p[i] = old
            an = (go if which == "onsite" else gh)[i]
            worst = max(worst, abs(an - (lp - lm) / (2 * h)) / scale)
        # a fourth-order stencil at h = 1e-4: the loss difference's rounding noise (~1e-6 of
        # the gradient at h = 1e-6) drops by 100 while the truncation error is O(h^4)
        h4 = 1e-4
        worst4 = 0.0
        for which, i in params:
            p = onsite if which == "onsite" else hop
            old = p[i].item()
            vals = []
            for kk in (2, 1, -1, -2):
                p[i] = old + kk * h4
                vals.append(fwd().item())
            p[i] = old
            fd4 = (-vals[0] + 8 * vals[1] - 8 * vals[2] + vals[3]) / (12 * h4)
            worst4 = max(worst4, abs((go if which == "onsite" else gh)[i] - fd4) / scale)
    gemm_flops = 8.0 * Nm * Nm * n * R  # the forward's moment-matrix GEMM (complex MACs x 8)
    del plan
    torch.cuda.empty_cache()
    return {"workload": "differentiable Kubo-Greenwood sigma_xx(E): honeycomb %dx%d cells (%d sites), learnable on-site "
                        "and per-bond hoppings, V_x = -i H o dx, Nm=%d, R=%d, 64 energies, L2 loss against another "
                        "disorder draw" % (cells, cells, n, Nm, R),
            "forward_ms": 1e3 * t_f, "forward_backward_ms": 1e3 * t_fb, "fwd_plus_bwd_over_fwd": t_fb / t_f,
            "steps": k, "setup_s": setup_s, "peak_device_gb": peak_gb,
            "forward_gemm_fp64_tflops": gemm_flops / t_f / 1e12,
            "fd_check": {"params": len(params), "h": h, "max_abs_err_over_max_grad": worst,
                         "stencil4_h1e-4": {"params": len(params), "max_abs_err_over_max_grad": worst4}},
            "note": "complex128 throughout; tables of every order per vector (the moment matrix couples all "
                    "orders), exact digit products on the tensor cores for mu_nm and the backward's C T products "
                    "(forward_gemm_fp64_tflops: the FP64 products that the forward's stand for, over its whole time)"}


def _fp64_mu_block(Hd, Vd, idx, L, v, sel):
    """FP64 mu[n][m] = <v| V T_n(H) V T_m(H) |v> for n, m in `sel`, from plain torch gathers
    on the device (complex128 ELL products): L_n = T_n(H) V v, R_m = V T_m(H) v."""
    import torch

    n = v.shape[0]
    d = torch.from_numpy(Hd.reshape(n, L)).cuda()
    dv = torch.from_numpy(Vd.reshape(n, L)).cuda()
    ix = torch.from_numpy(idx.reshape(n, L).astype(np.int64)).cuda()

    def mv(a, x):
        return (a * x[ix]).sum(1)

    def chebs(x0, keep):
        out, prev, cur = {}, None, x0
        for m in range(max(keep) + 1):
            if m in keep:
                out[m] = cur
            nxt = mv(d, cur) if m == 0 else 2 * mv(d, cur) - prev
            prev, cur = cur, nxt
        return out

    keep = set(sel)
    vt = torch.from_numpy(v).cuda()
    Ls = chebs(mv(dv, vt), keep)
    Rs = {m: mv(dv, t) for m, t in chebs(vt, keep).items()}
    Lm = torch.stack([Ls[k] for k in sel])
    Rm = torch.stack([Rs[k] for k in sel])
    return (Lm.conj() @ Rm.T).cpu().numpy()


def run_kubo(a, peaks, steps, warmup):
    """The Kubo-Greenwood configuration: honeycomb cells x cells, W = 1 eV, V_x as a second
    ELL operator, mu_nm for Nm = 256 with R random vectors (complex64 recursions, 3xTF32
    tensor-core contraction).  Reports the whole mu_nm time, the contraction alone
    (tensor TFLOP/s against the TF32 dense rate, half the measured bf16 rate), and the
    error of a 16 x 16 sub-block (n, m = 0, 17, .., 255) against an FP64 product."""
    import torch

    from minijclsquant_gb300 import _capi, device, lattice
    from minijclsquant_gb300.modifiers import modifier_bounds, modifier_velocity
    from minijclsquant_gb300.observables import random_vector_generator

    cells, Nm, R = a.kubo_cells, a.kubo_Nm, a.kubo_R
    t0 = time.perf_counter()
    H = lattice.honeycomb(cells, cells, t=-2.7, W=1.0, seed=11)
    Hk = H.modifier(modifier_bounds)
    Vx = H.modifier(modifier_velocity, "x")
    Vk = np.ascontiguousarray(Vx.data / H.bounds[1])
    n = int(H.shape[0])
    hop = device.DeviceELL(Hk.data, Hk.indices, Hk.len_row)
    vop = device.DeviceELL(Vk, Hk.indices, Hk.len_row)
    vs = np.stack([random_vector_generator(n, 3000 + r) for r in range(R)])
    tv = torch.from_numpy(vs).cuda()
    mu = torch.empty((Nm, Nm), dtype=torch.complex128, device="cuda")
    setup_s = time.perf_counter() - t0
    lib = _capi.lib()
    stream = torch.cuda.current_stream()
    sp = int(stream.cuda_stream)

    def call(rr, out):
        _capi.check(lib.kpm_mu_nm(hop.handle, vop.handle, rr, Nm, tv.data_ptr(), out.data_ptr(), sp), "kpm_mu_nm")

    def timed(fn, k, w):
        for _ in range(w):
            fn()
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(k):
            fn()
        e1.record(stream)
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / k

    ms = timed(lambda: call(R, mu), steps, max(1, warmup // 3))
    # the contraction alone, on operands of the same shape (256 x 2 n_pad floats per vector)
    n_pad = ((n + 511) // 512) * 512
    g = torch.Generator(device="cuda").manual_seed(5)
    A = torch.randn((256, 2 * n_pad), device="cuda", generator=g, dtype=torch.float32)
    B = torch.randn((256, 2 * n_pad), device="cuda", generator=g, dtype=torch.float32)
    mc = torch.empty((256, 256), dtype=torch.complex128, device="cuda")

    def contract():
        _capi.check(lib.kpm_mu_contract(A.data_ptr(), B.data_ptr(), 2 * n_pad, 2 * n_pad, 256, 1.0, 0,
                                        mc.data_ptr(), sp), "kpm_mu_contract")

    ms_c = timed(contract, max(3, steps), 3)
    del A, B
    mma_flops = 3 * 2 * 2 * 256 * 256 * (2 * n_pad)  # 3 split products x (Re, Im) x 2 flops x N x M x K
    tf32_peak = peaks.get("bf16_tflops", 1900.0) / 2
    ach = mma_flops / (ms_c * 1e-3) / 1e12
    # error of a sub-block against FP64 (vector 0 alone)
    sel = list(range(0, 256, 17))[:16]
    sel = [s for s in sel if s < Nm]
    mu1 = torch.empty((Nm, Nm), dtype=torch.complex128, device="cuda")
    call(1, mu1)
    got = mu1.cpu().numpy()[np.ix_(sel, sel)]
    ref = _fp64_mu_block(Hk.data, Vk, Hk.indices, Hk.len_row, vs[0], sel)
    err = float(np.max(np.abs(got - ref)) / np.max(np.abs(ref)))
    rec_site_steps = float(n) * R * 3 * Nm  # L and R recursions plus the V products, per vector
    path = lib.kpm_mu_gemm_path()  # bit 0: TMA-fed operand tiles, bit 1: 64-byte-swizzled layout
    gemm = ("mu_gemm_tma_kernel" if path & 1 else "mu_gemm_kernel") + (" (swizzled" if path & 2 else " (no-swizzle")
    return {"workload": "Kubo-Greenwood mu_nm: honeycomb %dx%d cells (%d sites), W=1 eV, V_x, Nm=%d, R=%d"
                        % (cells, cells, n, Nm, R),
            "ms_per_mu_nm": ms, "site_steps_per_s": rec_site_steps / (ms * 1e-3), "setup_s": setup_s,
            "contraction": {"ms_per_vector": ms_c, "mma_flops_per_vector": mma_flops,
                            "roofline": {"bound": "tensor", "achieved": ach, "peak": tf32_peak, "unit": "TFLOP/s",
                                         "frac": ach / tf32_peak,
                                         "peak_source": "TF32 dense = half of MEASURED_PEAKS.json bf16_tflops"},
                            "kernel": gemm + " layout; tcgen05.mma kind::tf32, 3xTF32, TMEM accumulators)"},
            "fp64_check": {"block": "n, m in %s, vector 0" % sel, "max_abs_err_over_max": err}}


def run_fp64_products(a, op, v, M, R, n, bytes_per_launch, hbm_peak, fma_peak, rec_fma, world, mu_default):
    """The headline recursion with every moment product in FP64 (KPM_MOMENTS_FP64=1, read by
    the library at each call): value, roofline of its step kernel, FP64 FMA rate, and the
    per-order difference from the default (float-float products).  Returns (block, moments)."""
    import ctypes

    import torch

    from minijclsquant_gb300 import _capi, device

    lib = _capi.lib()
    stream = torch.cuda.current_stream()
    os.environ["KPM_MOMENTS_FP64"] = "1"
    try:
        mu = device.cheb_moments(op, M, v, dtype="c128")  # tunes the FP64-products step once
        torch.cuda.synchronize()
        k = max(1, min(a.steps, 3))
        lib.kpm_ell_profile(op.handle, 1)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(k):
            mu = device.cheb_moments(op, M, v, dtype="c128")
        e1.record(stream)
        torch.cuda.synchronize()
        loop_ms, launches, rows = ctypes.c_double(), ctypes.c_int64(), ctypes.c_int64()
        _capi.check(lib.kpm_ell_profile_read(op.handle, ctypes.byref(loop_ms), ctypes.byref(launches),
                                             ctypes.byref(rows)))
        lib.kpm_ell_profile(op.handle, 0)
        kind, rpt, grid, us = ctypes.c_int(), ctypes.c_int(), ctypes.c_int(), ctypes.c_float()
        _capi.check(lib.kpm_ell_step_config(op.handle, _capi.KPM_C128, R, ctypes.byref(kind), ctypes.byref(rpt),
                                            ctypes.byref(grid), ctypes.byref(us)))
    finally:
        del os.environ["KPM_MOMENTS_FP64"]
    ms = max_over_ranks(e0.elapsed_time(e1), world) / k
    launch_s = loop_ms.value * 1e-3 / max(1, launches.value)
    gbs = bytes_per_launch / launch_s / 1e9
    fma = (rec_fma + 4) * float(n) * R / launch_s
    mu_h = mu.cpu().numpy()
    d = np.abs(mu_h - mu_default) / np.maximum(np.abs(mu_h), 1e-6 * np.abs(mu_h[:, :1]))
    blk = {"value": float(n) * R * (M - 1) * world / (ms * 1e-3), "unit": UNIT, "ms_per_step": ms, "steps": k,
           "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm_peak, "unit": "GB/s", "frac": gbs / hbm_peak,
                        "kernel": "%s (FP64 moment products, %d row(s)/thread)"
                                  % ({0: "cheb_step_kernel", 1: "cheb_next_staged_kernel",
                                      2: "cheb_next_ws_kernel", 3: "cheb_next_ws_kernel (two sub-tiles per stage)"}
                                     .get(kind.value, "?"), rpt.value),
                        "grid": grid.value, "avg_launch_ms": launch_s * 1e3},
           "fp64": {"achieved_fma_per_s": fma, "peak_fma_per_s": fma_peak, "frac": fma / fma_peak,
                    "fma_per_site_step": rec_fma + 4},
           "default_vs_fp64_products": {"max_rel_per_order": float(d.max()),
                                        "max_abs_over_mu0": float(np.max(np.abs(mu_h - mu_default))
                                                                  / np.max(np.abs(mu_h[:, 0])))},
           "note": "KPM_MOMENTS_FP64=1: the all-FP64 complex128 recursion and moment products (strict form)"}
    return blk, mu_h


def run_config1(a, world):
    """The CPU-runnable DOS configuration: honeycomb 64 x 64 cells (8,192 sites), W = 0.5 eV
    (seed 1234), Gershgorin bound x 1.01, M = 512, R = 4 vectors (seeds 1000..1003), DOS on 1024
    energies.  L2-resident, so launch- and latency-bound: reported as recursion steps/s and
    site-steps/s (moments on the device, CUDA events), the host DOS reconstruction time, and the
    whole drop-in call (numpy vectors in, DOS out) beside the reference's CPU path in the same
    run: its rec_A_tab loop over jclsquant's own aAxby/vdot for the four vectors and its DOS
    loop (jclsquant/observables.py:49-52: one moments_delta and one dot per energy)."""
    import torch

    from minijclsquant_gb300 import device
    from minijclsquant_gb300.kernel_and_moments import JacksonKernel, moments_delta
    from minijclsquant_gb300.observables import dos_from_moments

    prob = build_problem(64, 0.5)
    n, L = prob["n"], prob["L"]
    M, R, n_e = 512, 4, 1024
    vs = random_vectors(n, R, 1000)
    op = device.DeviceELL(prob["data_kpm"], prob["indices"], L)
    v = torch.from_numpy(vs).cuda()
    for _ in range(max(3, a.warmup)):
        mu = device.cheb_moments(op, M, v)
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream()
    k = max(10, a.steps)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(k):
        mu = device.cheb_moments(op, M, v)
    e1.record(stream)
    torch.cuda.synchronize()
    ms = max_over_ranks(e0.elapsed_time(e1), world) / k
    mu_h = mu.cpu().numpy()
    t0 = time.perf_counter()
    dos = dos_from_moments(mu_h, prob["bounds"], M, n_e)
    dos_s = time.perf_counter() - t0
    # the whole call as a user makes it: host vectors in, moments back, DOS on the host
    t0 = time.perf_counter()
    for _ in range(k):
        dos_e2e = dos_from_moments(device.cheb_moments(op, M, vs), prob["bounds"], M, n_e)
    e2e_s = (time.perf_counter() - t0) / k
    blk = {"workload": "honeycomb 64x64 cells (%d sites), W=0.5 eV, Gershgorin x 1.01, M=%d, R=%d, DOS on %d "
                       "energies" % (n, M, R, n_e),
           "value": float(n) * R * (M - 1) / (ms * 1e-3), "unit": UNIT, "ms_per_recursion": ms,
           "recursion_steps_per_s": (M - 1) / (ms * 1e-3), "dos_reconstruction_ms": dos_s * 1e3,
           "e2e": {"ms_per_dos": e2e_s * 1e3, "value": float(n) * R * (M - 1) / e2e_s, "unit": UNIT,
                   "path": "device.cheb_moments(numpy [R, N]) + dos_from_moments (host FP64)"},
           "bound": "launch/latency (8192 sites x R=4 stay in L2)",
           "same_dos_twice": bool(np.array_equal(dos, dos_e2e))}
    if not a.no_cpu and world == 1:
        blas = cpu_reference_kernels()
        threads = os.cpu_count() or 1
        t0 = time.perf_counter()
        mus = [cpu_rec_A_tab(M, prob, vs[r], threads, want_moments=True)[2] for r in range(R)]
        cpu_rec_s = time.perf_counter() - t0
        kind = "reference" if blas is not None else "port"
        mu_c = np.mean(np.stack(mus), axis=0)
        # the reference's DOS loop: per energy, moments_delta(E~) * Jackson, then its blas dot
        b = prob["bounds"]
        a_ = 0.5 * (b[1] - b[0])
        Ef = np.linspace(b[0] + 1e-3, b[1] - 1e-3, n_e)
        kern = JacksonKernel(M).astype(np.complex128)
        t0 = time.perf_counter()
        rho = np.empty(n_e)
        for i in range(n_e):
            md = moments_delta(Ef[i] / a_ - 0.5 * (b[1] + b[0]) / a_, M).astype(np.complex128) * kern
            rho[i] = np.real(blas.dot(1 + 0j, md, mu_c, M, threads) if blas is not None else md @ mu_c)
        cpu_dos_s = time.perf_counter() - t0
        blk["cpu_reference"] = {"value": float(n) * R * (M - 1) / cpu_rec_s, "unit": UNIT, "cores": threads,
                                "kind": kind, "recursion_ms": cpu_rec_s * 1e3, "dos_loop_ms": cpu_dos_s * 1e3,
                                "ms_per_dos": (cpu_rec_s + cpu_dos_s) * 1e3,
                                "sample": "the full configuration: 4 vectors x M=512, then the DOS loop"}
        blk["gpu_over_cpu_e2e"] = (cpu_rec_s + cpu_dos_s) / e2e_s
        per_vec = [moment_parity(mu_h[r], mus[r]) for r in range(R)]
        blk["parity_vs_reference"] = max(per_vec, key=lambda d: d["max_rel"])
        blk["parity_vs_reference"]["vectors"] = R
        blk["dos_max_abs_diff_over_max"] = float(np.max(np.abs(dos[:, 1] - rho)) / np.max(np.abs(rho)))
    del op, v
    return blk


def run_ours(a):
    import ctypes

    import torch

    from minijclsquant_gb300 import _capi, device, obv_gpu

    world, rank, local = dist_init()
    _capi.load(build_if_missing=False)
    t_build = time.perf_counter()
    prob = build_problem(a.cells, a.W)
    n, L, M, R = prob["n"], prob["L"], a.M, a.R
    op = device.DeviceELL(prob["data_kpm"], prob["indices"], L)
    torch.cuda.synchronize()
    host_build_s = time.perf_counter() - t_build
    vs_host = random_vectors(n, R, 1000 + rank * R)
    v = torch.from_numpy(vs_host).cuda()
    op.reserve(a.dtype, R, M)
    lib = _capi.lib()
    stream = torch.cuda.current_stream()

    def step():
        return device.cheb_moments(op, M, v, dtype=a.dtype)

    for _ in range(a.warmup):
        mu = step()
    torch.cuda.synchronize()
    # timed region
    lib.kpm_ell_profile(op.handle, 1)
    barrier(world)
    torch.cuda.synchronize()
    with ClockSampler(local, enabled=not a.no_clocks) as clk:
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(a.steps):
            mu = step()
        e1.record(stream)
        torch.cuda.synchronize()
    barrier(world)
    ms = e0.elapsed_time(e1)
    loop_ms = ctypes.c_double()
    launches = ctypes.c_int64()
    rows = ctypes.c_int64()
    _capi.check(lib.kpm_ell_profile_read(op.handle, ctypes.byref(loop_ms), ctypes.byref(launches), ctypes.byref(rows)))
    lib.kpm_ell_profile(op.handle, 0)
    ms_max = max_over_ranks(ms, world)
    site_steps = float(n) * R * (M - 1) * a.steps
    value = site_steps * world / (ms_max * 1e-3)
    doubled = bool(op.doubling)

    # sanity: mu_0 = N for unit-modulus vectors
    mu_h = mu.cpu().numpy()
    assert np.allclose(mu_h[:, 0].real, n, rtol=1e-6), "moment check failed"

    # roofline of the dominant kernel (the fused step, MODE_NEXT)
    s_v = 16 if a.dtype == "c128" else 8
    # complex128: FP64 values; complex64: exact float pairs (hi, lo) -- 8 B real, 16 B complex either way
    val_bytes = 8 if op.is_real else 16
    # per executed step: T_m gathered once, T_{m-1}, T_{m+1}, and v_l (direct) or |v|^2/2 (doubled)
    bytes_per_row = L * (val_bytes + 4) + R * (3 * s_v + (s_v // 4 if doubled else s_v))
    bytes_per_launch = float(n) * bytes_per_row
    avg_launch_s = (loop_ms.value * 1e-3) / max(1, launches.value)
    achieved_gbs = bytes_per_launch / avg_launch_s / 1e9
    peaks = {}
    pk_path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(pk_path):
        peaks = json.load(open(pk_path))
    hbm_peak = peaks.get("hbm_gbs")
    peak_src = "MEASURED_PEAKS.json hbm_gbs (measured)"
    if not hbm_peak:
        hbm_peak, peak_src = 6800.0, "fallback 6.8 TB/s"
    tag = "cheb_step_%s_r%d_%dx%d" % (a.dtype, R, a.cells, a.cells)
    traffic = load_traffic(tag)
    kind, rpt, grid, us = ctypes.c_int(), ctypes.c_int(), ctypes.c_int(), ctypes.c_float()
    _capi.check(lib.kpm_ell_step_config(op.handle, _capi.dtype_code(a.dtype), R, ctypes.byref(kind), ctypes.byref(rpt),
                                        ctypes.byref(grid), ctypes.byref(us)))
    kname = {1: "cheb_next_staged_kernel (bulk-copy staged, %d row(s)/thread)" % rpt.value,
             2: "cheb_next_ws_kernel (bulk-copy staged, producer warp, %d row(s)/thread)" % rpt.value,
             3: "cheb_next_ws_kernel (bulk-copy staged, producer warp, %d row(s)/thread, two sub-tiles per stage)"
                % rpt.value}.get(
        kind.value, "cheb_step_kernel (grid-stride, MODE_NEXT STORE|MOM1)")
    roofline = {"bound": "hbm", "achieved": achieved_gbs, "peak": hbm_peak, "unit": "GB/s",
                "frac": achieved_gbs / hbm_peak, "traffic": traffic, "peak_source": peak_src,
                "kernel": kname, "grid": grid.value,
                "algorithmic_bytes_per_launch": bytes_per_launch, "avg_launch_ms": avg_launch_s * 1e3}
    fma_rate = ctypes.c_double()
    _capi.check(lib.kpm_measure_fp64_fma_rate(ctypes.byref(fma_rate), ctypes.c_void_p(int(stream.cuda_stream))))
    # FP64 FMAs per site-step: the recursion's 2L (real values) or 4L, plus the moment's 4 unless
    # the producer-warp kernel forms the moment products in float-float arithmetic (the default
    # for one moment set; KPM_MOMENTS_FP64=1 turns it off)
    ff_products = (a.dtype == "c128" and not doubled and kind.value in (2, 3)
                   and os.environ.get("KPM_MOMENTS_FP64", "") in ("", "0"))
    rec_fma = 2 * L if op.is_real else 4 * L
    fma_per_site_step = rec_fma + (6 if doubled else (0 if ff_products else 4))
    fp64 = None
    if a.dtype == "c128":
        ach = fma_per_site_step * float(n) * R / avg_launch_s
        fp64 = {"achieved_fma_per_s": ach, "peak_fma_per_s": fma_rate.value, "frac": ach / fma_rate.value,
                "fma_per_site_step": fma_per_site_step, "peak_source": "measured live (independent FP64 FMA chains)",
                "moment_products": ("float-float on the FP32 pipe (2^-49 per product), FP64 sums" if ff_products
                                    else "FP64")}

    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": a.steps, "warmup": a.warmup,
            "ms_per_step": ms_max / a.steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64" if a.dtype == "c128" else "f32 (f64 moment accumulation)", "data": "synthetic",
            "config": {"workload": workload_desc(a, n), "sites": n, "M": M, "R": R, "len_row": L, "W": a.W,
                       "bounds": "Gershgorin x 1.01", "l2": "inputs larger than L2 (vector set %.2f GB)"
                       % (n * R * s_v / 1e9), "parallelism": "replicas x%d" % world},
            "roofline": roofline, "fp64": fp64, "gpu_launches": launches_per_recursion(M, R, doubled) * a.steps,
            "hbm_gbs": achieved_gbs}
    # the opt-in doubled moments on the same handle (H is Hermitian): the same M moments
    # from ceil(M/2) - 1 recursion steps; value counts site-steps per moment delivered
    if op.hermitian and not doubled and a.dtype == "c128":
        op.set_doubling(True)
        step()
        torch.cuda.synchronize()
        d0 = torch.cuda.Event(enable_timing=True)
        d1 = torch.cuda.Event(enable_timing=True)
        d0.record(stream)
        for _ in range(a.steps):
            mu_dbl = step()
        d1.record(stream)
        torch.cuda.synchronize()
        op.set_doubling(False)
        ms_d = max_over_ranks(d0.elapsed_time(d1), world) / a.steps
        dk = ctypes.c_int()
        _capi.check(lib.kpm_ell_props(op.handle, None, ctypes.byref(dk)))
        line["doubling"] = {
            "value": float(n) * R * (M - 1) * world / (ms_d * 1e-3), "ms_per_step": ms_d,
            "executed_steps_per_recursion": executed_steps(M, True) + 1, "moments_per_recursion": M,
            "fma_per_executed_site_step": rec_fma + 6,
            "max_abs_diff_vs_direct_over_mu0": float(np.max(np.abs(mu_dbl.cpu().numpy() - mu_h))
                                                     / np.max(np.abs(mu_h[:, 0]))),
            "note": "opt-in (KPM_FLAG_DOUBLING); value counts site-steps per moment delivered, N R (M-1)"}
    if a.dtype == "c128":
        # complex128 accuracy in float-float arithmetic on the FP32 pipe (dtype c128f), same
        # handle, same memory streams (16 B per complex, 8 B per value)
        op.reserve("c128f", R, M)
        device.cheb_moments(op, M, v, dtype="c128f")
        torch.cuda.synchronize()
        lib.kpm_ell_profile(op.handle, 1)
        f0 = torch.cuda.Event(enable_timing=True)
        f1 = torch.cuda.Event(enable_timing=True)
        f0.record(stream)
        for _ in range(a.steps):
            mu_f = device.cheb_moments(op, M, v, dtype="c128f")
        f1.record(stream)
        torch.cuda.synchronize()
        _capi.check(lib.kpm_ell_profile_read(op.handle, ctypes.byref(loop_ms), ctypes.byref(launches),
                                             ctypes.byref(rows)))
        lib.kpm_ell_profile(op.handle, 0)
        ms_f = max_over_ranks(f0.elapsed_time(f1), world) / a.steps
        f_launch_s = (loop_ms.value * 1e-3) / max(1, launches.value)
        f_gbs = bytes_per_launch / f_launch_s / 1e9
        line["c128f"] = {
            "value": float(n) * R * (M - 1) * world / (ms_f * 1e-3), "ms_per_step": ms_f,
            "roofline": {"bound": "hbm", "achieved": f_gbs, "peak": hbm_peak, "unit": "GB/s", "frac": f_gbs / hbm_peak,
                         "kernel": "ff_next_kernel (float-float, bulk-copy staged, producer warp)",
                         "avg_launch_ms": f_launch_s * 1e3},
            "max_abs_diff_vs_c128_over_mu0": float(np.max(np.abs(mu_f.cpu().numpy() - mu_h))
                                                   / np.max(np.abs(mu_h[:, 0]))),
            "note": "dtype KPM_C128F: every real as a float pair (~48 bits), FP32 pipe; opt-in"}
    mu_fp64 = None
    if a.dtype == "c128" and ff_products:
        # the same recursion with every moment product in FP64 (KPM_MOMENTS_FP64=1): the strict
        # all-FP64 form beside the default, timed on the same handle and vectors
        blk, mu_fp64 = run_fp64_products(a, op, v, M, R, n, bytes_per_launch, hbm_peak, fma_rate.value, rec_fma,
                                         world, mu_h)
        line["c128_fp64_products"] = blk
    if a.dtype == "c128" and not a.no_time:
        line["time_evolution"] = run_time_evolution(a, op, n, L, prob, hbm_peak, world)
    if not a.no_setup:
        line["setup"] = run_setup(a, prob, host_build_s, hbm_peak)
    if not a.no_sigma:
        line["time_sigma"] = run_time_sigma(a, hbm_peak, world)
    if not a.no_driven:
        line["driven"] = run_driven(a, hbm_peak)
    clocks = clk.summary()
    if clocks is not None:
        line["clocks"] = clocks

    # end to end through the reference-facing host-pointer call (rec_A_tab_gpu per vector, as
    # jclsquant's kpm_dos_gpu issues it): operator and vector uploads inside the timed region.
    if not a.no_e2e and a.dtype == "c128":
        data_p = torch.from_numpy(prob["data_kpm"]).pin_memory().numpy()
        idx_p = torch.from_numpy(prob["indices"]).pin_memory().numpy()
        vs_p = torch.from_numpy(vs_host).pin_memory().numpy()
        out = torch.zeros((R, M), dtype=torch.complex128).pin_memory().numpy()
        obv_gpu.rec_A_tab_gpu(data_p, idx_p, L, np.ascontiguousarray(vs_p[0]), out[0], 16)  # warm-up
        torch.cuda.synchronize()
        barrier(world)
        with ClockSampler(local, enabled=not a.no_clocks) as clk_e2e:
            t0 = time.perf_counter()
            # each pass is one step of the workload (all R vectors through the host-pointer call);
            # at about 3.4 s a pass, the passes are capped so the run stays within a few minutes
            e2e_steps = max(1, min(a.steps, a.e2e_max_steps))
            for _ in range(e2e_steps):
                for r in range(R):
                    obv_gpu.rec_A_tab_gpu(data_p, idx_p, L, vs_p[r], out[r], M)
            torch.cuda.synchronize()
            dt = max_over_ranks(time.perf_counter() - t0, world)
        assert np.allclose(out[:, 0].real, n, rtol=1e-6)
        line["e2e"] = {"value": float(n) * R * (M - 1) * e2e_steps * world / dt, "unit": UNIT,
                       "steps": e2e_steps, "ms_per_step": 1e3 * dt / e2e_steps,
                       "h2d_bytes_per_step": int(R * (prob["data_kpm"].nbytes + prob["indices"].nbytes + n * 16)),
                       "d2h_bytes_per_step": int(R * M * 16),
                       "path": "obv_gpu.rec_A_tab_gpu -> exported rec_A_tab (host pointers, one vector per call)"}
        ce = clk_e2e.summary()
        if ce is not None:
            line["e2e"]["clocks"] = ce
    if not a.no_batched:
        del op, v
        torch.cuda.empty_cache()
        line["batched_c64"] = run_batched(a, hbm_peak, a.steps, a.warmup)
    if not a.no_adjoint:
        torch.cuda.empty_cache()
        line["adjoint"] = run_adjoint(a, a.steps, a.warmup)
    if not a.no_kubo:
        torch.cuda.empty_cache()
        line["kubo"] = run_kubo(a, peaks, a.steps, a.warmup)
    if not a.no_adjoint_kubo:
        torch.cuda.empty_cache()
        line["adjoint_kubo"] = run_adjoint_kubo(a, a.steps)
    if not a.no_config1:
        torch.cuda.empty_cache()
        line["config1_dos"] = run_config1(a, world)
    if rank == 0 and world == 1 and not a.no_cpu:
        line["cpu_baseline"], mu_cpu = cpu_baseline(prob, a.cpu_seconds)
        # parity at this configuration: the reference's own recursion on the host (same operator,
        # same vector, seed 1000) against the GPU's vector 0, per order
        line["parity_vs_reference"] = dict(moment_parity(mu_h[0], mu_cpu), vector="seed 1000 (GPU vector 0)",
                                           kind=line["cpu_baseline"]["kind"],
                                           gpu_path=line["fp64"]["moment_products"] if line.get("fp64") else a.dtype)
        if mu_fp64 is not None:
            line["c128_fp64_products"]["parity_vs_reference"] = moment_parity(mu_fp64[0], mu_cpu)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()


def main():
    a = parse()
    if a.impl == "reference":
        run_reference_arm(a)
    else:
        run_ours(a)


if __name__ == "__main__":
    main()
