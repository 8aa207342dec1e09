#!/usr/bin/env python
"""Benchmark of the per-energy NEGF hot path on B200.

Workload (one GPU): 32 diagonal blocks of 256x256, 1024 energies in
[-3, 3] (complex128, FP64 arithmetic). One *energy point* = assembly of
A(E), both-contact Sancho-Rubio OBC to 1e-12 with the OBCSystem refinement
step and the boundary self-energies, RGF selected solve (G^R diagonal,
G^< and G^> diagonal + off-diagonal blocks, Meir-Wingreen current), Caroli
transmission and density. A *step* is one batch of energies
(default 128); steps cycle through the energy grid, which is split evenly
across ranks (independent energies: weak scaling, no collective in the
data path).

``python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]``
prints one JSON line on rank 0.
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

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "RGF energy-points/s at 256x256 blocks (FP64)"
UNIT = "energy-points/s"
WORKLOAD = ("32 blocks of 256x256, 1024 energies in [-3,3], complex128: both-contact Sancho-Rubio "
            "(tol 1e-12) + OBC refinement + selected_solve (G^R, G^<, G^>, current) + Caroli "
            "transmission + density per energy point")


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=7)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--batch", type=int, default=148)
    p.add_argument("--energies", type=int, default=1024)
    p.add_argument("--e2e-batch", type=int, default=64, help="energies per end-to-end step (host memory: "
                   "six pinned block-tridiagonal stacks of this many energies, ~38 GB at 64)")
    p.add_argument("--e2e-subbatch", type=int, default=16, help="RGF max_batch_size of the end-to-end leg")
    p.add_argument("--e2e-steps", type=int, default=2)
    p.add_argument("--cpu-energies", type=int, default=2)
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu", action="store_true")
    p.add_argument("--no-peak", action="store_true", help="skip the cuBLAS peak measurements")
    p.add_argument("--precision", choices=["fp64", "mixed", "emulated", "both"], default="both",
                   help="fp64 is the headline value; mixed (and emulated) are reported beside it. cfg1 also "
                        "accepts 'emulated' alone (FP64 with int8-emulated products as the main line)")
    p.add_argument("--emulated-slices", type=int, default=5,
                   help="with --precision both: also time the FP64 path with the selected solve's complex128 "
                        "products emulated on the int8 tensor cores from this many digit planes (0: skip). "
                        "5 (default) is the fastest setting inside the transmission-error target of 1e-6; "
                        "6 gives FP64-class accuracy (the library default)")
    p.add_argument("--workload", choices=["cfg1", "cfg2", "cfg3", "cfg4", "kernels", "inverse", "w"], default="cfg1",
                   help="cfg1 (default): the headline line. cfg2: 64 blocks of 512x512, mixed vs FP64. "
                        "cfg3: eight uneven devices on one GPU. cfg4: the serving loop. inverse: the batched "
                        "inverse of --batch blocks of --block-size on the selected --inverse-path. w: the "
                        "screened-interaction (W) solve of a Coulomb-screening step")
    p.add_argument("--block-size", type=int, default=256, help="block size of the inverse workload")
    p.add_argument("--cfg3-energies", type=int, default=32, help="energies per device of the uneven batch")
    p.add_argument("--budget-gb", type=float, default=150.0, help="HBM budget of the resident solvers")
    p.add_argument("--cfg4-catalogue", choices=["small", "cfg3"], default="small",
                   help="serving catalogue: 8 devices with (N, b) drawn as in cfg3 with b in {128, 256} "
                        "(small) or b in {128, ..., 768} (cfg3)")
    p.add_argument("--cfg4-rate", type=float, default=None,
                   help="arrivals per second (default: --cfg4-load of the measured capacity)")
    p.add_argument("--cfg4-duration", type=float, default=60.0)
    p.add_argument("--cfg4-load", type=float, default=0.5,
                   help="arrival rate as a fraction of the capacity measured per lane")
    p.add_argument("--graph", action="store_true",
                   help="replay each batch through one captured CUDA graph (device-side Sancho-Rubio loop)")
    p.add_argument("--inverse-path", choices=["auto", "single", "wide", "cluster", "split"], default="auto",
                   help="inverse kernels: automatic choice, one CTA per matrix, multi-CTA panels, one "
                        "thread-block cluster per matrix, or the one-CTA kernel column-split over a cluster")
    return p.parse_args()


# ---------------------------------------------------------------------------
def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


class ClockSampler:
    """nvidia-smi clock / throttle-reason samples during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_id: str):
        self.gpu_id = gpu_id
        self.proc = None
        self.lines: list[str] = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits", "-lms", "200",
                 "-i", self.gpu_id], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except (OSError, FileNotFoundError):
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, power, reasons = [], [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [x.strip() for x in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
                power.append(float(parts[3]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "power_w_max": max(power) if power else None, "samples": len(sm), "reasons": sorted(reasons)}


def measured_tf32_peak(torch, device) -> float:
    """cuBLAS FP32 GEMM with TF32 tensor cores, 8192^3, best of 5 (TFLOP/s)."""
    old = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    n = 8192
    a = torch.randn((n, n), dtype=torch.float32, device=device)
    b = torch.randn((n, n), dtype=torch.float32, device=device)
    torch.matmul(a, b)
    torch.cuda.synchronize()
    best = 1e30
    for _ in range(5):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        torch.matmul(a, b)
        e.record()
        e.synchronize()
        best = min(best, s.elapsed_time(e))
    torch.backends.cuda.matmul.allow_tf32 = old
    del a, b
    torch.cuda.empty_cache()
    return 2.0 * n ** 3 / (best * 1e-3) / 1e12


def measured_int8_peak(torch, device) -> float:
    """cuBLASLt int8 GEMM (int32 accumulation), 8192^3, best of 5 (TOPS)."""
    n = 8192
    a = torch.randint(-128, 127, (n, n), dtype=torch.int8, device=device)
    b = torch.randint(-128, 127, (n, n), dtype=torch.int8, device=device).t().contiguous().t()
    torch._int_mm(a, b)
    torch.cuda.synchronize()
    best = 1e30
    for _ in range(5):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        torch._int_mm(a, b)
        e.record()
        e.synchronize()
        best = min(best, s.elapsed_time(e))
    del a, b
    torch.cuda.empty_cache()
    return 2.0 * n ** 3 / (best * 1e-3) / 1e12


def measured_fp64_peak(torch, device) -> dict:
    """cuBLAS FP64 throughput on this GPU (best of 5): DGEMM 8192^3 and
    ZGEMM 4096^3; the larger figure is the FP64 roofline denominator."""
    res = {}
    for name, dtype, n, per in (("dgemm", torch.float64, 8192, 2.0), ("zgemm", torch.complex128, 4096, 8.0)):
        a = torch.randn((n, n), dtype=dtype, device=device)
        b = torch.randn((n, n), dtype=dtype, device=device)
        torch.matmul(a, b)
        torch.cuda.synchronize()
        best = 1e30
        for _ in range(5):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record()
            torch.matmul(a, b)
            e.record()
            e.synchronize()
            best = min(best, s.elapsed_time(e))
        res[name] = per * n ** 3 / (best * 1e-3) / 1e12
        del a, b
    torch.cuda.empty_cache()
    res["peak"] = max(res["dgemm"], res["zgemm"])
    return res


def cpu_baseline(num: int) -> dict:
    """The oracle (NumPy restatement of the reference path) on a bounded
    sample of the workload, all host cores."""
    from oracle import negf_oracle as o
    from quatrex_b200 import synthetic

    dev = synthetic.cfg1()
    idx = np.linspace(100, 900, num).astype(int)
    e = dev.energies[idx]
    diag, upper, lower = dev.system_blocks(e)
    t0 = time.perf_counter()
    o.energy_point_solve(diag, upper, lower, dev.fermi_left(e), dev.fermi_right(e))
    dt = time.perf_counter() - t0
    return {"value": num / dt, "unit": UNIT, "cores": os.cpu_count(), "kind": "port",
            "sample": f"{num} energies of the 1024-point grid (indices {idx.tolist()}), one batch",
            "seconds": dt, "blas_threads": _blas_threads()}


def _blas_threads():
    try:
        from threadpoolctl import threadpool_info

        return [d.get("num_threads") for d in threadpool_info()]
    except Exception:  # noqa: BLE001 - informational only
        return None


# ---------------------------------------------------------------------------
def run_reference(args, world, rank):
    if rank != 0:
        return
    from oracle import negf_oracle as o
    from quatrex_b200 import synthetic

    dev = synthetic.cfg1(args.energies)
    times = []
    for step in range(args.warmup + args.steps):
        i = (137 * step + 11) % args.energies
        e = dev.energies[i:i + 1]
        diag, upper, lower = dev.system_blocks(e)
        t0 = time.perf_counter()
        o.energy_point_solve(diag, upper, lower, dev.fermi_left(e), dev.fermi_right(e))
        dt = time.perf_counter() - t0
        if step >= args.warmup:
            times.append(dt)
    total = sum(times)
    value = len(times) / total
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * total / len(times),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "c128", "data": "synthetic",
        "config": {"workload": WORKLOAD, "step": "1 energy point per step (bounded CPU sample)",
                   "parallelism": "host BLAS threads"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": os.cpu_count(), "kind": "port",
                         "sample": f"{len(times)} single-energy steps of the 1024-point grid",
                         "blas_threads": _blas_threads()},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------
def e2e_leg(torch, device, dev, energies, steps, sub=8):
    """The reference-facing plugin path with pinned HOST buffers: the caller's
    DSDBCOO stacks live in host memory; OBCSystem(SanchoRubio) and
    RGF.selected_solve copy them in and the results out in every step."""
    import scipy.sparse as sps

    from quatrex_b200 import RGF, DSDBCOO, OBCBlocks, OBCSystem, SanchoRubio, contact_self_energy
    from quatrex_b200 import observables

    n, b = dev.num_blocks, dev.block_size
    B = energies.size
    rows, cols = [], []
    for i in range(n):
        for j in (i - 1, i, i + 1):
            if 0 <= j < n:
                r, c = np.meshgrid(np.arange(b) + i * b, np.arange(b) + j * b, indexing="ij")
                rows.append(r.ravel())
                cols.append(c.ravel())
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    pattern = sps.coo_matrix((np.ones(rows.size, dtype=np.complex128), (rows, cols)), shape=(n * b, n * b))
    proto = DSDBCOO.from_sparray(pattern, dev.block_sizes, (1,))

    def host(m=None):
        d = torch.zeros((B, proto.nnz), dtype=torch.complex128).pin_memory()
        return DSDBCOO(d, proto.rows, proto.cols, proto.block_sizes, _layout=proto._layout)

    A, SL, SG, XL, XG, XR = (host() for _ in range(6))
    diag, upper, lower = dev.system_blocks(energies)
    for i in range(n):
        A.blocks[i, i] = torch.from_numpy(diag[i])
        if i + 1 < n:
            A.blocks[i, i + 1] = torch.from_numpy(upper[i])
            A.blocks[i + 1, i] = torch.from_numpy(lower[i])
    fl, fr = dev.fermi_left(energies), dev.fermi_right(energies)
    obc_sys = OBCSystem(SanchoRubio(convergence_tol=1e-12, per_energy=True), memoization_mode="off")
    solver = RGF(max_batch_size=min(sub, B))

    phase = {"obc": 0.0, "solve": 0.0, "density": 0.0}

    def step():
        t0 = time.perf_counter()
        ob = OBCBlocks(n)
        a00, a01, a10 = A.blocks[0, 0], A.blocks[0, 1], A.blocks[1, 0]
        g, *_ = obc_sys((a00, a01, a10), contact="left")
        ob.retarded[0], ob.lesser[0], ob.greater[0] = contact_self_energy(a01, a10, g, fl)
        ann, an1, a1n = A.blocks[n - 1, n - 1], A.blocks[n - 1, n - 2], A.blocks[n - 2, n - 1]
        g, *_ = obc_sys((ann, an1, a1n), contact="right")
        ob.retarded[-1], ob.lesser[-1], ob.greater[-1] = contact_self_energy(an1, a1n, g, fr)
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        cur = solver.selected_solve(A, SL, SG, obc_blocks=ob, out=(XL, XG, XR), return_retarded=True,
                                    return_current=True)
        t2 = time.perf_counter()
        dens = observables.density(XL)
        t3 = time.perf_counter()
        phase["obc"] += t1 - t0
        phase["solve"] += t2 - t1
        phase["density"] += t3 - t2
        return cur, dens

    from quatrex_b200 import _interop

    step()  # warm-up
    torch.cuda.synchronize()
    for k in phase:
        phase[k] = 0.0
    _interop.transfer_bytes.update(h2d=0, d2h=0)
    t0 = time.perf_counter()
    for _ in range(steps):
        cur, dens = step()
    torch.cuda.synchronize()
    dt = time.perf_counter() - t0
    # bytes the plugin moved between the host containers and the GPU (counted
    # from the tensors it copied): A in full, the diagonal and upper blocks of
    # Sigma^< / Sigma^> (the only ones the solve reads), the contact blocks,
    # X^< / X^> in full, the diagonal blocks of X^R, surface Green's functions,
    # self-energies, current and density
    h2d = _interop.transfer_bytes["h2d"] / steps
    d2h = _interop.transfer_bytes["d2h"] / steps
    return {"value": steps * B / dt, "unit": UNIT, "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h),
            "energies": steps * B, "seconds": dt,
            "seconds_per_step": {k: v / steps for k, v in phase.items()},
            "path": "RGF.selected_solve + OBCSystem(SanchoRubio) + contact_self_energy on pinned host DSDBCOO "
                    f"stacks, {B} energies per step (RGF max_batch_size {min(sub, B)}), {steps} steps"}


def host_link(torch, device, nbytes=1 << 30, reps=5) -> dict:
    """Pinned host <-> device copy bandwidth on this GPU: H2D alone, D2H alone
    and both directions at once on two streams (GB/s, best of `reps`, CUDA
    events). The roofline of the end-to-end leg, whose every step uploads its
    inputs and downloads its results."""
    h_src = torch.empty(nbytes, dtype=torch.uint8).pin_memory()
    h_dst = torch.empty(nbytes, dtype=torch.uint8).pin_memory()
    d_a = torch.empty(nbytes, dtype=torch.uint8, device=device)
    d_b = torch.empty(nbytes, dtype=torch.uint8, device=device)
    s1, s2 = torch.cuda.Stream(device), torch.cuda.Stream(device)

    def timed(fn):
        best = None
        for _ in range(reps):
            torch.cuda.synchronize()
            ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            ev0.record()
            fn()
            ev1.record()
            torch.cuda.synchronize()
            ms = ev0.elapsed_time(ev1)
            best = ms if best is None else min(best, ms)
        return best * 1e-3

    def duplex():
        cur = torch.cuda.current_stream(device)
        s1.wait_stream(cur)
        s2.wait_stream(cur)
        with torch.cuda.stream(s1):
            d_a.copy_(h_src, non_blocking=True)
        with torch.cuda.stream(s2):
            h_dst.copy_(d_b, non_blocking=True)
        cur.wait_stream(s1)
        cur.wait_stream(s2)

    h2d = nbytes / timed(lambda: d_a.copy_(h_src, non_blocking=True)) / 1e9
    d2h = nbytes / timed(lambda: h_dst.copy_(d_b, non_blocking=True)) / 1e9
    dup = 2 * nbytes / timed(duplex) / 1e9
    del h_src, h_dst, d_a, d_b
    return {"h2d_gbs": h2d, "d2h_gbs": d2h, "duplex_gbs": dup, "bytes_per_copy": nbytes,
            "how": f"pinned host <-> device copies of {nbytes >> 20} MiB, best of {reps}, CUDA events"}


def run_ours(args, world, rank, local):
    import torch
    import torch.distributed as dist

    from quatrex_b200 import EnergyPointSolver, _native, synthetic
    from quatrex_b200.utils import get_section_sizes

    torch.cuda.set_device(local)
    device = torch.device("cuda", local)
    if world > 1:
        import datetime

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600), device_id=device)
    dev = synthetic.cfg1(args.energies)
    sizes, _ = get_section_sizes(args.energies, world)
    offs = np.concatenate(([0], np.cumsum(sizes)))
    mine = np.arange(offs[rank], offs[rank + 1])
    B = min(args.batch, mine.size)
    batches = [mine[i:i + B] for i in range(0, mine.size - B + 1, B)] or [mine]
    fl_all, fr_all = dev.fermi_left(), dev.fermi_right()
    lib = _native.load()
    peak = {"peak": None} if args.no_peak else measured_fp64_peak(torch, device)
    tf32_peak = None if (args.no_peak or args.precision in ("fp64", "emulated")) else measured_tf32_peak(torch, device)
    emulate = args.precision == "emulated" or (args.precision == "both" and args.emulated_slices > 0)
    if emulate and not 3 <= args.emulated_slices <= 8:
        raise SystemExit("--emulated-slices must be 3-8 for the emulated leg")
    int8_peak = measured_int8_peak(torch, device) if (emulate and not args.no_peak) else None
    props = torch.cuda.get_device_properties(device)
    gpu_id = str(getattr(props, "uuid", local))
    if gpu_id and not gpu_id.startswith("GPU-") and len(gpu_id) > 8:
        gpu_id = "GPU-" + gpu_id

    def timed(precision):
        solver = EnergyPointSolver(dev.h_diag, dev.coupling, eta=dev.eta, sr_tol=1e-12, per_energy=True,
                                   device=device, precision=precision, device_loop=args.graph,
                                   slices=args.emulated_slices if precision == "emulated" else 6)

        def step(k):
            idx = batches[k % len(batches)]
            if args.graph:
                return solver.solve_graph(dev.energies[idx], fl_all[idx], fr_all[idx])
            return solver.solve(dev.energies[idx], fl_all[idx], fr_all[idx])

        for k in range(args.warmup):
            step(k)
        torch.cuda.synchronize()
        clocks = ClockSampler(gpu_id)
        lib.qtx_profile_reset()
        lib.qtx_profile_enable(1)
        sr_iters = []
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()
        clocks.start()
        t_start = torch.cuda.Event(enable_timing=True)
        t_end = torch.cuda.Event(enable_timing=True)
        marks = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
        t_start.record()
        for k in range(args.steps):
            r = step(args.warmup + k)
            if not args.graph:
                sr_iters.append(r.sr_iterations)
            marks[k].record()
        t_end.record()
        torch.cuda.synchronize()
        per_step = [t_start.elapsed_time(marks[0])] + [marks[k - 1].elapsed_time(marks[k])
                                                         for k in range(1, args.steps)]
        if args.graph:
            # graph replays record no per-launch profile: one eager step after
            # the timed region gives the kernel-class breakdown
            it = solver.sr_status(B)[0]
            sr_iters = [(it, it)] * args.steps
            lib.qtx_profile_reset()
            t_a = torch.cuda.Event(enable_timing=True)
            t_b = torch.cuda.Event(enable_timing=True)
            t_a.record()
            idx = batches[0]
            solver.solve(dev.energies[idx], fl_all[idx], fr_all[idx])
            t_b.record()
            torch.cuda.synchronize()
            prof_ms = t_a.elapsed_time(t_b)
        if world > 1:
            dist.barrier()
        clk = clocks.stop()
        lib.qtx_profile_enable(0)
        ms = t_start.elapsed_time(t_end)
        prof_ref_ms = prof_ms if args.graph else ms  # the time the launch profile covers
        prof = {name: _native.profile_read(kind) for name, kind in _native.KERNEL_CLASSES.items()}
        prof["all"] = _native.profile_read(-1)

        lib.qtx_profile_reset()
        # a fixed probe batch for cross-precision error reporting
        probe = batches[0]
        rp = solver.solve(dev.energies[probe], fl_all[probe], fr_all[probe])
        torch.cuda.synchronize()
        probe_out = (rp.transmission.cpu().numpy().copy(), rp.density.cpu().numpy().copy())
        del solver
        torch.cuda.empty_cache()
        return ms, prof, clk, sr_iters, probe_out, per_step, prof_ref_ms

    res = {}
    precs = ((["fp64", "mixed"] + (["emulated"] if emulate else [])) if args.precision == "both"
             else [args.precision])
    for prec in precs:
        res[prec] = timed(prec)
    main_prec = precs[0]
    ms, prof, clk, sr_iters, _, per_step, pms = res[main_prec]
    gemm_ms, gemm_flops, gemm_n = prof[{"fp64": "zgemm", "mixed": "cgemm", "emulated": "zgemm_emu"}[main_prec]]
    inv_ms, inv_flops, inv_n = prof["zinv"]
    all_ms, _, all_n = prof["all"]

    t = torch.tensor([ms], dtype=torch.float64, device=device)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_max = float(t.item())
    done = sum(batches[(args.warmup + k) % len(batches)].size for k in range(args.steps))
    total = torch.tensor([done], dtype=torch.float64, device=device)
    if world > 1:
        dist.all_reduce(total)
    value = float(total.item()) / (ms_max * 1e-3)

    mixed_line = None
    if "mixed" in res and main_prec == "fp64":
        mms, mprof, mclk, _, mprobe, mper, mpms = res["mixed"]
        tm = torch.tensor([mms], dtype=torch.float64, device=device)
        if world > 1:
            dist.all_reduce(tm, op=dist.ReduceOp.MAX)
        cg_ms, cg_flops, cg_n = mprof["cgemm"]
        ach = (cg_flops / cg_n) / ((cg_ms / cg_n) * 1e-3) / 1e12 if cg_n else None
        fprobe = res["fp64"][4]
        terr = np.abs(mprobe[0] - fprobe[0]) / np.abs(fprobe[0])
        mixed_line = {
            "value": float(total.item()) / (float(tm.item()) * 1e-3), "unit": UNIT,
            "ms_per_step": float(tm.item()) / args.steps,
            "speedup_vs_fp64": ms_max / float(tm.item()),
            "dtype": "c64 storage; tcgen05 split-TF32 products, FP32 accumulation; FP64 inverses and OBC",
            "roofline": {"bound": "tensor", "kernel": "cgemm_tc (tcgen05 kind::tf32, six MMAs of N = 128 per complex K step)",
                         "achieved": ach, "peak": tf32_peak, "unit": "TFLOP/s (complex as-written 8mnk)",
                         "frac": (ach / tf32_peak) if (ach and tf32_peak) else None,
                         "peak_source": "measured cuBLAS FP32 GEMM with TF32 tensor cores 8192^3 on this GPU",
                         "launches": cg_n, "avg_launch_ms": cg_ms / cg_n if cg_n else None,
                         "share_of_step_time": cg_ms / mpms if mpms else None,
                         "zinv_ms_share": mprof["zinv"][0] / mpms if mpms else None,
                         "class_shares": {k: round(v[0] / mpms, 4) for k, v in mprof.items()
                                          if k != "all" and mpms}},
            "error_vs_fp64": {"transmission_max_rel": float(terr.max()),
                              "transmission_median_rel": float(np.median(terr)),
                              "density_rel": float(np.linalg.norm(mprobe[1] - fprobe[1]) / np.linalg.norm(fprobe[1])),
                              "probe": f"{batches[0].size} energies of the grid"},
            "gpu_launches": mprof["all"][2] * (args.steps if args.graph else 1), "clocks": mclk,
            "latency_ms": _latency(mper, B),
        }

    emulated_line = None
    if "emulated" in res and main_prec == "fp64":
        ems, eprof, eclk, _, eprobe, eper, epms = res["emulated"]
        te = torch.tensor([ems], dtype=torch.float64, device=device)
        if world > 1:
            dist.all_reduce(te, op=dist.ReduceOp.MAX)
        S = args.emulated_slices
        pairs = S * (S + 1) // 2
        eg_ms, eg_work, eg_n = eprof["zgemm_emu"]
        sp_ms, sp_bytes, sp_n = eprof["split"]
        int8_tops = eg_work * pairs / (eg_ms * 1e-3) / 1e12 if eg_n else None
        fprobe = res["fp64"][4]
        terr = np.abs(eprobe[0] - fprobe[0]) / np.abs(fprobe[0])
        emulated_line = {
            "value": float(total.item()) / (float(te.item()) * 1e-3), "unit": UNIT,
            "ms_per_step": float(te.item()) / args.steps,
            "speedup_vs_fp64": ms_max / float(te.item()),
            "dtype": f"c128 storage; complex128 products from {S} int8 digit planes per operand "
                     "(tcgen05 kind::i8, exact int32 sums, FP64 combination); FP64 inverses",
            "slices": S,
            "roofline": {"bound": "tensor", "kernel": "oz_gemm_kernel (tcgen05 kind::i8, M=128, N<=256)",
                         "achieved": int8_tops, "peak": int8_peak, "unit": "int8 TOPS (2 x int8 MACs)",
                         "frac": (int8_tops / int8_peak) if (int8_tops and int8_peak) else None,
                         "peak_source": "measured cuBLASLt int8 GEMM 8192^3 (torch._int_mm) on this GPU",
                         "launches": eg_n, "avg_launch_ms": eg_ms / eg_n if eg_n else None,
                         "share_of_step_time": eg_ms / epms if epms else None,
                         "split_share_of_step_time": sp_ms / epms if epms else None,
                         "class_shares": {k: round(v[0] / epms, 4) for k, v in eprof.items()
                                          if k != "all" and epms}},
            "error_vs_fp64": {"transmission_max_rel": float(terr.max()),
                              "transmission_median_rel": float(np.median(terr)),
                              "density_rel": float(np.linalg.norm(eprobe[1] - fprobe[1]) / np.linalg.norm(fprobe[1])),
                              "probe": f"{batches[0].size} energies of the grid"},
            "gpu_launches": eprof["all"][2] * (args.steps if args.graph else 1), "clocks": eclk,
            "latency_ms": _latency(eper, B),
        }

    e2e = None
    cpu = None
    if not args.no_e2e:
        # Every rank runs the plugin path on its own energy shard; the batch
        # per rank shrinks with N so that the pinned host stacks of all ranks
        # stay near those of one rank at N = 1 (~38 GB).
        nb = args.e2e_batch if world == 1 else max(8, args.e2e_batch // world)
        pick = mine[np.linspace(0, mine.size - 1, min(nb, mine.size)).astype(int)]
        if world > 1:
            dist.barrier()
        e2e = e2e_leg(torch, device, dev, dev.energies[pick], args.e2e_steps, min(args.e2e_subbatch, pick.size))
        if world > 1:
            agg = torch.tensor([e2e["energies"], e2e["h2d_bytes_per_step"], e2e["d2h_bytes_per_step"]],
                               dtype=torch.float64, device=device)
            dist.all_reduce(agg)
            tmax = torch.tensor([e2e["seconds"]], dtype=torch.float64, device=device)
            dist.all_reduce(tmax, op=dist.ReduceOp.MAX)
            e2e["value"] = float(agg[0].item()) / float(tmax.item())
            e2e["h2d_bytes_per_step"] = int(agg[1].item())
            e2e["d2h_bytes_per_step"] = int(agg[2].item())
            e2e["path"] += f"; {world} ranks, {pick.size} energies per rank, max time over ranks"
        link = host_link(torch, device)
        secs = e2e["seconds"] if world == 1 else float(tmax.item())
        moved = (e2e["h2d_bytes_per_step"] + e2e["d2h_bytes_per_step"]) * args.e2e_steps / secs / 1e9
        e2e["link_gbs"] = link["duplex_gbs"] * world
        e2e["link_frac"] = moved / e2e["link_gbs"]
        e2e["link"] = dict(link, achieved_gbs=moved, note="achieved = (h2d + d2h bytes per step) x steps / "
                           "time; link_gbs = simultaneous H2D + D2H bandwidth x ranks")
    if rank == 0 and world == 1 and not args.no_cpu:
        cpu = cpu_baseline(args.cpu_energies)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    if rank != 0:
        return

    achieved = (gemm_flops / gemm_n) / ((gemm_ms / gemm_n) * 1e-3) / 1e12 if gemm_n else None
    if main_prec == "fp64":
        roofline = {"bound": "tensor",
                    "kernel": "zgemm (batched complex128 DMMA, 3M: three real MMAs per complex multiply-add)",
                    "achieved": achieved, "peak": peak["peak"], "unit": "TFLOP/s (complex as-written 8mnk)",
                    "frac": (achieved / peak["peak"]) if achieved and peak["peak"] else None,
                    "executed_frac": (0.75 * achieved / peak["peak"]) if achieved and peak["peak"] else None,
                    "executed_note": "achieved counts the reference's 8 real flops per complex multiply-add; the "
                                     "3M (Gauss) form executes 6 of them on the DMMA pipe, so the executed-work "
                                     "rate is 0.75 x achieved (executed_frac, of the same measured peak)",
                    "peak_source": "measured cuBLAS FP64 (max of DGEMM 8192^3, ZGEMM 4096^3) on this GPU; "
                                   "no FP64 entry in MEASURED_PEAKS.json",
                    "peak_detail": peak, "traffic": _ncu_traffic(),
                    "traffic_source": "stored ncu capture of one launch of one product per entry of a full batch "
                                      "(profiles/zgemm_traffic.txt: dram__bytes_read.sum + dram__bytes_write.sum; "
                                      "the timed launches hold up to four products), not measured in this run",
                    "launches": gemm_n}
    elif main_prec == "emulated":
        S = args.emulated_slices
        tops = achieved * (S * (S + 1) // 2) if achieved else None  # int8 ops = 8mnk x digit pairs
        roofline = {"bound": "tensor", "kernel": "oz_gemm_kernel (tcgen05 kind::i8, M=128, N<=256)",
                    "achieved": tops, "peak": int8_peak, "unit": "int8 TOPS (2 x int8 MACs)",
                    "frac": (tops / int8_peak) if tops and int8_peak else None,
                    "peak_source": "measured cuBLASLt int8 GEMM 8192^3 (torch._int_mm) on this GPU",
                    "fp64_equivalent_tflops": achieved, "traffic": None, "launches": gemm_n}
    else:
        roofline = {"bound": "tensor", "kernel": "cgemm_tc (tcgen05 kind::tf32, six MMAs of N = 128 per complex K step)",
                    "achieved": achieved, "peak": tf32_peak, "unit": "TFLOP/s (complex as-written 8mnk)",
                    "frac": (achieved / tf32_peak) if achieved and tf32_peak else None,
                    "peak_source": "measured cuBLAS FP32 GEMM with TF32 tensor cores 8192^3 on this GPU",
                    "traffic": None, "launches": gemm_n}
    roofline.update({"avg_launch_ms": gemm_ms / gemm_n if gemm_n else None,
                     "share_of_step_time": gemm_ms / pms if pms else None,
                     "zinv_ms_share": inv_ms / pms if pms else None,
                     "class_shares": {k: round(v[0] / pms, 4) for k, v in prof.items() if k != "all" and pms},
                     "profiled": "the timed steps" if not args.graph else
                                 "one eager step after the timed graph replays"})
    from quatrex_b200.negf import flops_per_energy

    its = np.mean(np.array(sr_iters), axis=0) if sr_iters else (0, 0)
    fl = flops_per_energy(32, 256, tuple(float(x) for x in its))
    line = {
        "metric": {"fp64": METRIC, "mixed": METRIC.replace("(FP64)", "(mixed)"),
                   "emulated": METRIC.replace("(FP64)", "(FP64, int8-emulated products)")}[main_prec],
        "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_max / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None,
        "dtype": {"fp64": "f64 (complex128)", "mixed": "c64 storage, split-TF32 products",
                  "emulated": f"f64 (complex128); products from {args.emulated_slices} int8 digit planes"}[main_prec],
        "data": "synthetic",
        "config": {"workload": WORKLOAD, "batch": B, "energies": args.energies,
                   "parallelism": f"energy sharding x{world}", "inverse_path": args.inverse_path,
                   "l2": "inputs exceed L2 (resident batch state "
                   f"~{B * 0.45:.0f} GB)", "sr_iterations_mean": [float(x) for x in its]},
        "roofline": roofline,
        "as_written_tflops": value * fl["total"] / 1e12,
        "cpu_baseline": cpu,
        "e2e": e2e,
        "gpu_launches": all_n * (args.steps if args.graph else 1),
        "clocks": clk,
        "latency_ms": _latency(per_step, B),
        "mixed": mixed_line,
        "emulated": emulated_line,
    }
    print(json.dumps(line), flush=True)


def _latency(per_step, batch) -> dict:
    """Solve latency of one batch (device time between consecutive step
    ends on the solving stream)."""
    x = np.asarray(per_step, dtype=np.float64)
    return {"p50": float(np.percentile(x, 50)), "p99": float(np.percentile(x, 99)), "max": float(x.max()),
            "batch": int(batch), "samples": int(x.size), "unit": "ms per batch"}


def _ncu_traffic():
    f = ROOT / "profiles" / "zgemm_traffic.txt"
    if not f.exists():
        return None
    for ln in f.read_text().splitlines():
        if ln.startswith("bytes_per_launch_full_batch:"):
            try:
                return float(ln.split(":", 1)[1])
            except ValueError:
                return None
    return None


def _timed_batches(torch, solver, energies, fl, fr, B, steps, warmup):
    """Device time of `steps` batches of B energies (cycling through the
    grid) after `warmup` batches; returns (seconds, clocks)."""
    nb = max(1, energies.size // B)

    def step(k):
        i = (k % nb) * B
        solver.solve(energies[i:i + B], fl[i:i + B], fr[i:i + B])

    for k in range(warmup):
        step(k)
    torch.cuda.synchronize()
    gpu = str(getattr(torch.cuda.get_device_properties(solver.device), "uuid", ""))
    clocks = ClockSampler(gpu if gpu.startswith("GPU-") else "GPU-" + gpu if gpu else "0")
    clocks.start()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0.record()
    for k in range(steps):
        step(warmup + k)
    t1.record()
    torch.cuda.synchronize()
    return t0.elapsed_time(t1) * 1e-3, clocks.stop()


def run_cfg2(args, local):
    """64 blocks of 512x512 (complex64 storage on the mixed path), 2048
    energies: mixed energy-points/s beside FP64 on the same grid, and the
    mixed path's errors in G^R, T and density against FP64."""
    import torch

    from quatrex_b200 import EnergyPointSolver, synthetic
    from quatrex_b200.negf import flops_per_energy
    from quatrex_b200.uneven import jobs_from_devices, plan_batches

    device = torch.device("cuda", local)
    torch.cuda.set_device(device)
    ne = args.energies if args.energies != 1024 else 2048
    dev = synthetic.cfg2(ne)
    job = jobs_from_devices([dev])[0]
    fl, fr = dev.fermi_left(), dev.fermi_right()
    out = {}
    emu = ("emulated",) if args.emulated_slices > 0 else ()
    for prec in ("mixed", "fp64") + emu:
        B = plan_batches([job], args.budget_gb * 1e9, prec)[0]
        s = EnergyPointSolver(dev.h_diag, dev.coupling, eta=dev.eta, sr_tol=1e-12, per_energy=True, device=device,
                              precision=prec, device_loop=True, store_blocks=False,
                              slices=max(args.emulated_slices, 3))
        sec, clk = _timed_batches(torch, s, dev.energies, fl, fr, B, args.steps, min(args.warmup, 1))
        it = s.sr_status(B)[0]
        out[prec] = {"value": args.steps * B / sec, "batch": B, "seconds": sec, "clocks": clk, "sr_iterations": it}
        del s
        torch.cuda.empty_cache()
    # Error probe: 4 energies with all blocks kept, both precisions.
    idx = np.linspace(0, ne - 1, 4).astype(int)
    probe = {}
    for prec in ("fp64", "mixed") + emu:
        s = EnergyPointSolver(dev.h_diag, dev.coupling, eta=dev.eta, sr_tol=1e-12, per_energy=True, device=device,
                              precision=prec, slices=max(args.emulated_slices, 3))
        r = s.solve(dev.energies[idx], fl[idx], fr[idx])
        probe[prec] = (r.transmission.cpu().numpy().copy(), r.density.cpu().numpy().copy(),
                       r.blocks["xr_diag"].to(torch.complex128).cpu().numpy())
        del s, r
        torch.cuda.empty_cache()
    f, m = probe["fp64"], probe["mixed"]
    rel = lambda a, b: float(np.linalg.norm(a - b) / np.linalg.norm(b))  # noqa: E731
    # The complex128 oracle (the reference algorithm on the host cores) on one
    # probe energy: errors of both GPU paths against it.
    oracle_err = None
    if not args.no_cpu:
        from oracle import negf_oracle as o

        k = 1  # probe energy index idx[1]
        e1 = dev.energies[idx[k:k + 1]]
        d1, u1, l1 = dev.system_blocks(e1)
        t0 = time.perf_counter()
        ref = o.energy_point_solve(d1, u1, l1, dev.fermi_left(e1), dev.fermi_right(e1))
        osec = time.perf_counter() - t0
        oxr = np.stack([x[0] for x in ref["xr_diag"]]) if "xr_diag" in ref else None
        oracle_err = {"energy": float(e1[0]), "oracle_seconds": osec}
        for name, pr in [("fp64", f), ("mixed", m)] + [(e, probe[e]) for e in emu]:
            e = {"transmission_rel": float(abs(pr[0][k] - ref["transmission"][0]) / abs(ref["transmission"][0])),
                 "density_rel": rel(pr[1][k], ref["density"][0])}
            if oxr is not None:
                e["g_retarded_diag_rel"] = rel(pr[2][:, k], oxr)
            oracle_err[name] = e
    fl_e = flops_per_energy(64, 512, (out["mixed"]["sr_iterations"],) * 2)["total"]
    line = {
        "metric": "RGF energy-points/s at 512x512 blocks (mixed)", "value": out["mixed"]["value"],
        "unit": UNIT, "n_gpus": 1, "steps": args.steps, "warmup": min(args.warmup, 1),
        "higher_is_better": True, "dtype": "c64 storage, split-TF32 products; FP64 inverses and OBC",
        "data": "synthetic",
        "config": {"workload": f"64 blocks of 512x512, {ne} energies in [-3,3], observables only",
                   "batch_mixed": out["mixed"]["batch"], "batch_fp64": out["fp64"]["batch"],
                   "budget_gb": args.budget_gb},
        "fp64": out["fp64"], "mixed": out["mixed"],
        "speedup_vs_fp64": out["mixed"]["value"] / out["fp64"]["value"],
        "as_written_tflops": {k: v["value"] * fl_e / 1e12 for k, v in out.items()},
        "error_vs_fp64": {"transmission_max_rel": float(np.max(np.abs(m[0] - f[0]) / np.abs(f[0]))),
                          "density_rel": rel(m[1], f[1]), "g_retarded_diag_rel": rel(m[2], f[2]),
                          "probe": f"energies {idx.tolist()}"},
        "error_vs_oracle": oracle_err,
    }
    if emu:
        em = probe["emulated"]
        line["emulated"] = dict(out["emulated"], slices=args.emulated_slices,
                                speedup_vs_fp64=out["emulated"]["value"] / out["fp64"]["value"],
                                error_vs_fp64={"transmission_max_rel": float(np.max(np.abs(em[0] - f[0]) / np.abs(f[0]))),
                                               "density_rel": rel(em[1], f[1]), "g_retarded_diag_rel": rel(em[2], f[2])})
    print(json.dumps(line), flush=True)


def run_cfg3(args, local):
    """Eight devices with (N, b) drawn by synthetic.uneven_devices, solved
    together on one GPU: one captured graph per device, replays on one
    stream per device, batch sizes planned under the HBM budget."""
    import torch

    from quatrex_b200 import synthetic
    from quatrex_b200.uneven import UnevenBatchRunner, jobs_from_devices

    device = torch.device("cuda", local)
    torch.cuda.set_device(device)
    ne = args.cfg3_energies
    shapes = synthetic.uneven_devices()
    devs = [synthetic.make_device(N, b, np.linspace(-2.0, 2.0, ne), seed=0, name=f"dev{k}")
            for k, (N, b) in enumerate(shapes)]
    jobs = jobs_from_devices(devs)
    work = sum(j.flops(19.0) for j in jobs)
    res, obs = {}, {}
    precs = ["fp64", "mixed"] if args.precision == "both" else [args.precision]
    for prec in precs:
        runner = UnevenBatchRunner(jobs, precision=prec, budget_bytes=args.budget_gb * 1e9, device=device,
                                   autotune=True)
        runner.prepare()  # tunes batch sizes, then captures every device's graph (one eager pass each)
        tc = time.perf_counter()
        whole = runner.capture_all()  # the whole uneven batch as one graph
        capture_s = time.perf_counter() - tc
        gpu = str(getattr(torch.cuda.get_device_properties(device), "uuid", ""))
        clocks = ClockSampler(gpu if gpu.startswith("GPU-") else "GPU-" + gpu if gpu else "0")
        clocks.start()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        whole.replay()  # one launch
        t1.record()
        torch.cuda.synchronize()
        sec = t0.elapsed_time(t1) * 1e-3
        # the same schedule as per-device graph replays on concurrent streams
        t2, t3 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t2.record()
        runner.enqueue()
        t3.record()
        torch.cuda.synchronize()
        sec_streams = t2.elapsed_time(t3) * 1e-3
        res[prec] = {"value": len(jobs) * ne / sec, "seconds": sec, "as_written_tflops": work / sec / 1e12,
                     "devices": runner.summary(), "sr_converged": all(runner.sr_converged().values()),
                     "tuning": runner.tuning, "one_graph_capture_seconds": capture_s,
                     "per_device_replays_value": len(jobs) * ne / sec_streams,
                     "clocks": clocks.stop()}
        obs[prec] = {k: v["transmission"].cpu().numpy().copy() for k, v in runner.results().items()}
        del whole, runner
        torch.cuda.empty_cache()
    line = {
        "metric": "RGF energy-points/s, uneven batch of 8 devices", "value": res[precs[0]]["value"],
        "unit": UNIT, "n_gpus": 1, "steps": 1, "warmup": 1, "higher_is_better": True,
        "dtype": precs[0], "data": "synthetic",
        "config": {"workload": f"8 devices (N, b) = {shapes}, {ne} energies each in [-2,2], observables only",
                   "budget_gb": args.budget_gb,
                   "step": "every energy of every device: one launch of the graph of the whole schedule",
                   "warmup": "the capture pass of each device's graph"},
        "results": res,
    }
    if len(precs) == 2:
        line["speedup_mixed_vs_fp64"] = res["mixed"]["value"] / res["fp64"]["value"]
        line["mixed_transmission_max_rel_vs_fp64"] = max(
            float(np.max(np.abs(obs["mixed"][k] - obs["fp64"][k]) / np.abs(obs["fp64"][k]))) for k in obs["fp64"])
    print(json.dumps(line), flush=True)


def run_cfg4(args, local):
    """The serving loop: Poisson arrivals of requests (one catalogue device,
    64-512 of its 512 grid energies each), continuous batching per device
    lane, HBM-budget admission, resident OBC warm starts. Reports p50/p99
    request latency (host clock, arrival to completion) and served
    energy-points/s, FP64 and mixed on the same request trace."""
    import torch

    from quatrex_b200 import synthetic
    from quatrex_b200.negf import flops_per_energy
    from quatrex_b200.serving import EnergyServer, Request, latency_stats, poisson_requests, slowdown_stats
    from quatrex_b200.uneven import jobs_from_devices

    device = torch.device("cuda", local)
    torch.cuda.set_device(device)
    bsz = (128, 256) if args.cfg4_catalogue == "small" else (128, 256, 384, 512, 768)
    shapes = synthetic.uneven_devices(block_sizes=bsz)
    grid = 512
    devs = [synthetic.make_device(N, b, np.linspace(-2.0, 2.0, grid), seed=0, name=f"dev{k}")
            for k, (N, b) in enumerate(shapes)]
    cat = jobs_from_devices(devs)
    mean_n = (64 + 512) / 2
    req_flops = np.mean([flops_per_energy(N, b, (19, 19))["total"] * mean_n for N, b in shapes])
    spec_shapes = synthetic.uneven_devices()
    spec_req_flops = np.mean([flops_per_energy(N, b, (19, 19))["total"] * mean_n for N, b in spec_shapes])
    precs = ["fp64", "mixed"] if args.precision == "both" else [args.precision]
    out, rate = {}, args.cfg4_rate
    for prec in precs:
        srv = EnergyServer(cat, precision=prec, budget_bytes=args.budget_gb * 1e9, warm_start=True,
                           device=device)
        if rate is None:  # a fraction of the capacity measured on one cold replay per lane, lanes back to back
            per_energy = []
            for ln in srv.lanes:
                t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                with torch.cuda.stream(ln.stream):
                    t0.record()
                    ln.graphs[False].replay()
                    t1.record()
                torch.cuda.synchronize()
                per_energy.append(t0.elapsed_time(t1) * 1e-3 / ln.B)
            rate = args.cfg4_load / (mean_n * float(np.mean(per_energy)))
        reqs = poisson_requests(rate, args.cfg4_duration, [grid] * len(cat), (64, 512), seed=0)
        gpu = str(getattr(torch.cuda.get_device_properties(device), "uuid", ""))
        clocks = ClockSampler(gpu if gpu.startswith("GPU-") else "GPU-" + gpu if gpu else "0")
        clocks.start()
        stats = srv.run(reqs)
        stats["clocks"] = clocks.stop()
        mixed_lat = {r.rid: r.latency for r in reqs}
        del srv
        torch.cuda.empty_cache()
        # Isolated solve time: each request served alone on an idle server
        # with the same lanes and no warm starts.
        solo = EnergyServer(cat, precision=prec, budget_bytes=args.budget_gb * 1e9, warm_start=False,
                            device=device)
        alone = {}
        for r in reqs:
            q = Request(r.rid, r.device, r.grid_index)
            t0 = time.perf_counter()
            solo.solve_now(q)
            alone[r.rid] = time.perf_counter() - t0
        stats["isolated_latency"] = latency_stats(list(alone.values()))
        stats["slowdown_vs_isolated"] = slowdown_stats(mixed_lat, alone)
        del solo
        srv = None
        stats["as_written_tflops"] = stats["energies"] * req_flops / mean_n / stats["wall_s"] / 1e12
        out[prec] = stats
        del srv
        torch.cuda.empty_cache()
    main = out[precs[0]]
    line = {
        "metric": "serving: energy-points/s and p50/p99 request latency", "value": main["energies_per_s"],
        "unit": UNIT, "n_gpus": 1, "steps": 1, "warmup": 0, "higher_is_better": True, "dtype": precs[0],
        "data": "synthetic",
        "config": {"workload": f"Poisson arrivals at {rate:.3g} req/s for {args.cfg4_duration:g} s, seed 0; "
                               f"catalogue of 8 devices (N, b) = {shapes}, 512-point grids on [-2,2]; "
                               "64-512 grid energies per request",
                   "rate_rule": "given" if args.cfg4_rate else f"{args.cfg4_load} of the capacity measured per lane",
                   "budget_gb": args.budget_gb, "warm_starts": True,
                   "latency_clock": "host wall clock, arrival to completion"},
        "p50_s": main["latency"].get("p50_s"), "p99_s": main["latency"].get("p99_s"),
        "p99_over_isolated_p99": (main["latency"].get("p99_s") / main["isolated_latency"]["p99_s"]
                                  if main["isolated_latency"].get("p99_s") else None),
        "results": out,
        "offered_load_note": {
            "spec_rate_req_s": 200, "spec_mean_request_tflop": spec_req_flops / 1e12,
            "spec_demand_pflops": 200 * spec_req_flops / 1e15,
            "this_catalogue_mean_request_tflop": req_flops / 1e12},
    }
    if len(precs) == 2:
        line["speedup_mixed_vs_fp64"] = out["mixed"]["energies_per_s"] / out["fp64"]["energies_per_s"]
    print(json.dumps(line), flush=True)


def run_w(args, local):
    """The screened-interaction (W) solve of a Coulomb-screening step
    (CoulombScreeningSolver.solve): 24 small blocks of 128 in superblocks of
    three (8 superblocks of 384), 64 energies per step in batches of 32,
    synthetic polarizations (quatrex_b200.synthetic.screened_device).
    GPU energy-points/s (CUDA events over --steps solves after --warmup),
    the oracle's restatement of the reference on the host cores on a
    2-energy sample beside it, and the assembly / selected-solve flops."""
    import torch

    from oracle import negf_oracle as o
    from quatrex_b200 import synthetic
    from quatrex_b200.negf import flops_per_energy
    from quatrex_b200.screening import CoulombScreeningSolve

    device = torch.device("cuda", local)
    torch.cuda.set_device(device)
    ns, b, nc, ne = 24, 128, 3, 64
    d = synthetic.screened_device(ns, b, ne, seed=7)
    energies = np.linspace(0.05, 1.0, ne)

    def dev(t):
        return tuple([torch.from_numpy(np.ascontiguousarray(x)).to(device) for x in lst] for lst in t)

    pl, pg, prh = dev(d["p_lesser"]), dev(d["p_greater"]), dev(d["p_retarded_hermitian"])
    solver = CoulombScreeningSolve(d["v"], nc, energies, filtering_iteration_limit=0, max_batch_size=32,
                                   device=device)
    for _ in range(max(args.warmup, 1)):
        solver.solve(pl, pg, prh)
    torch.cuda.synchronize()
    gpu = str(getattr(torch.cuda.get_device_properties(device), "uuid", ""))
    clocks = ClockSampler(gpu if gpu.startswith("GPU-") else "GPU-" + gpu if gpu else "0")
    clocks.start()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0.record()
    for _ in range(args.steps):
        solver.solve(pl, pg, prh)
    t1.record()
    torch.cuda.synchronize()
    sec = t0.elapsed_time(t1) * 1e-3
    clk = clocks.stop()
    value = args.steps * ne / sec
    # as-written flops per energy: the small-block products of M and L (9 + 2 x 24
    # per block row, 8 b^3 each) and the selected solve on the superblocks
    n_sup, bs = ns // nc, nc * b
    fl = (9 + 48) * ns * 8.0 * b ** 3 + flops_per_energy(n_sup, bs)["solve"]
    cpu = None
    if not args.no_cpu:
        import os
        import time

        sub = lambda lst: [x[:2] for x in lst]  # noqa: E731
        args_cpu = [tuple(sub(lst) for lst in d[k]) for k in ("p_lesser", "p_greater", "p_retarded_hermitian")]
        t = time.perf_counter()
        o.w_solve(d["v"], *args_cpu, nc, energies[:2], lambda x: o.obc_system_solve(x[0], x[1], x[2], 100, 1e-12)[0],
                  lambda bb, q: o.lyapunov_system_solve(bb, q)[0])
        cs = time.perf_counter() - t
        cpu = {"value": 2 / cs, "unit": "energy-points/s", "cores": os.cpu_count(), "kind": "port",
               "sample": "2 energies of the 64 (one batch)", "seconds": cs}
    print(json.dumps({
        "metric": "W energy-points/s (Coulomb-screening step)", "value": value, "unit": "energy-points/s",
        "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec / args.steps * 1e3,
        "higher_is_better": True, "dtype": "f64 (complex128)", "data": "synthetic",
        "config": {"workload": f"{ns} small blocks of {b} in superblocks of {nc} ({n_sup} of {bs}), {ne} energies "
                               "per step in batches of 32: P^R assembly, I - V P^R and V P^< V, V P^> V with the "
                               "contact spillover, Lyapunov boundary conditions, selected solve"},
        "as_written_tflops": value * fl / 1e12, "flops_per_energy": fl, "cpu_baseline": cpu, "clocks": clk}),
        flush=True)


def run_inverse(args, local):
    """The batched complex128 inverse alone (qtx_zinv_batched_ws, the call the
    RGF and Sancho-Rubio drivers make): --batch blocks of --block-size,
    diagonally shifted random matrices, inputs resident, CUDA-event timed
    over --steps launches after --warmup."""
    import ctypes

    import torch

    from quatrex_b200 import _native
    from quatrex_b200._interop import mat

    device = torch.device("cuda", local)
    torch.cuda.set_device(device)
    lib = _native.load()
    n, B = args.block_size, args.batch
    g = torch.Generator(device=device).manual_seed(0)
    a = (torch.randn((B, n, n), dtype=torch.complex128, device=device, generator=g)
         + n * torch.eye(n, dtype=torch.complex128, device=device))
    x = torch.empty_like(a)
    info = torch.zeros(B, dtype=torch.int32, device=device)
    ws = torch.empty(lib.qtx_zinv_workspace(n, B), dtype=torch.uint8, device=device)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def launch():
        _native.check(lib.qtx_zinv_batched_ws(n, B, mat(a), mat(x), info.data_ptr(), ws.data_ptr(), ws.numel(),
                                              stream))

    for _ in range(max(args.warmup, 3)):
        launch()
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(args.steps):
        launch()
    e.record()
    torch.cuda.synchronize()
    ms = s.elapsed_time(e) / args.steps
    print(json.dumps({"metric": "batched inverse (complex flops 8n^3)", "unit": "TFLOP/s",
                      "value": 8.0 * n ** 3 * B / (ms * 1e-3) / 1e12, "ms_per_launch": ms, "block_size": n,
                      "batch": B, "inverse_path": args.inverse_path, "steps": args.steps}), flush=True)


def run_kernels(args, local):
    """Kernel-level rooflines at the cfg1 block shape: batched complex GEMMs
    (ours and cuBLAS through torch on the same shapes) and batched inverses
    (ours, both paths, and torch.linalg.inv), CUDA-event timed, inputs
    resident (batch x 3 blocks of 1 MiB each > L2 for batch 148)."""
    import ctypes

    import torch

    from quatrex_b200 import _native
    from quatrex_b200._interop import mat

    device = torch.device("cuda", local)
    torch.cuda.set_device(device)
    lib = _native.load()
    n, B = 256, args.batch
    stream = lambda: ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)  # noqa: E731
    g = torch.Generator(device=device).manual_seed(0)

    def rnd(dt):
        return torch.randn((B, n, n), dtype=dt, device=device, generator=g)

    def timeit(fn, reps=max(args.steps, 3)):
        for _ in range(max(args.warmup, 3)):
            fn()
        torch.cuda.synchronize()
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        for _ in range(reps):
            fn()
        e.record()
        torch.cuda.synchronize()
        return s.elapsed_time(e) / reps * 1e-3

    flops = 8.0 * n ** 3 * B
    out = {}
    a, b, c = rnd(torch.complex128), rnd(torch.complex128), torch.empty((B, n, n), dtype=torch.complex128,
                                                                         device=device)
    z = _native.NULL_MAT
    out["zgemm_ours"] = flops / timeit(lambda: _native.check(lib.qtx_zgemm_batched(
        n, n, n, B, 1.0, 0.0, mat(a), 0, mat(b), 0, 0.0, 0.0, z, 0, mat(c), stream()))) / 1e12
    out["zgemm_cublas_bmm"] = flops / timeit(lambda: torch.bmm(a, b, out=c)) / 1e12
    d2 = rnd(torch.complex128)
    out["zgemm_ours_plus_ct_addend"] = flops / timeit(lambda: _native.check(lib.qtx_zgemm_batched(
        n, n, n, B, 1.0, 0.0, mat(a), 0, mat(b), 0, 1.0, 0.0, mat(d2), 1, mat(c), stream()))) / 1e12
    out["zgemm_ours_plus_addend"] = flops / timeit(lambda: _native.check(lib.qtx_zgemm_batched(
        n, n, n, B, 1.0, 0.0, mat(a), 0, mat(b), 0, 1.0, 0.0, mat(d2), 0, mat(c), stream()))) / 1e12
    out["zgemm_ours_b_conj_trans"] = flops / timeit(lambda: _native.check(lib.qtx_zgemm_batched(
        n, n, n, B, 1.0, 0.0, mat(a), 0, mat(b), 1, 0.0, 0.0, z, 0, mat(c), stream()))) / 1e12
    del d2
    a32, b32, c32 = a.to(torch.complex64), b.to(torch.complex64), c.to(torch.complex64)
    out["cgemm_ours_split_tf32"] = flops / timeit(lambda: _native.check(lib.qtx_cgemm_batched(
        n, n, n, B, 1.0, 0.0, mat(a32), 0, mat(b32), 0, 0.0, 0.0, z, 0, mat(c32), None, stream()))) / 1e12
    old = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    out["cgemm_cublas_bmm_tf32_allowed"] = flops / timeit(lambda: torch.bmm(a32, b32, out=c32)) / 1e12
    torch.backends.cuda.matmul.allow_tf32 = old
    del a32, b32, c32
    # Complex128 products emulated on the int8 tensor cores (digit planes).
    from quatrex_b200.emulation import workspace_bytes, zgemm_emulated

    _native.check(lib.qtx_zgemm_batched(n, n, n, B, 1.0, 0.0, mat(a), 0, mat(b), 0, 0.0, 0.0, z, 0, mat(c),
                                        stream()))
    ref = c.clone()
    emu = {}
    for S in (5, 6, 7):
        wsS = torch.empty(workspace_bytes(n, n, n, B, S), dtype=torch.uint8, device=device)
        t = timeit(lambda: zgemm_emulated(a, b, slices=S, out=c, workspace=wsS))
        lib.qtx_profile_reset()
        lib.qtx_profile_enable(1)
        zgemm_emulated(a, b, slices=S, out=c, workspace=wsS)
        torch.cuda.synchronize()
        gm, sp = _native.profile_read(6), _native.profile_read(7)
        lib.qtx_profile_enable(0)
        emu[f"slices_{S}"] = {
            "fp64_equivalent_tflops": flops / t / 1e12, "speedup_vs_zgemm_ours": (flops / t / 1e12) / out["zgemm_ours"],
            "gemm_ms": gm[0], "split_ms": sp[0],
            "gemm_int8_tops": gm[1] * (S * (S + 1) // 2) / (gm[0] * 1e-3) / 1e12 if gm[0] else None,
            "rel_err_vs_dmma": float(torch.linalg.norm(c - ref) / torch.linalg.norm(ref))}
        del wsS
    out["zgemm_emulated_int8"] = emu
    del ref
    # The same at 512x512 blocks, batch 74 (twice the K per output tile).
    n2, B2 = 512, min(74, B)
    flops2 = 8.0 * n2 ** 3 * B2
    a2 = torch.randn((B2, n2, n2), dtype=torch.complex128, device=device, generator=g)
    b2 = torch.randn((B2, n2, n2), dtype=torch.complex128, device=device, generator=g)
    c2 = torch.empty_like(a2)
    t_d = timeit(lambda: _native.check(lib.qtx_zgemm_batched(n2, n2, n2, B2, 1.0, 0.0, mat(a2), 0, mat(b2), 0, 0.0,
                                                             0.0, z, 0, mat(c2), stream())))
    emu2 = {"zgemm_ours_tflops": flops2 / t_d / 1e12}
    for S in (5, 6, 7):
        wsS = torch.empty(workspace_bytes(n2, n2, n2, B2, S), dtype=torch.uint8, device=device)
        t = timeit(lambda: zgemm_emulated(a2, b2, slices=S, out=c2, workspace=wsS))
        emu2[f"slices_{S}"] = {"fp64_equivalent_tflops": flops2 / t / 1e12, "speedup_vs_zgemm_ours": t_d / t}
        del wsS
    out["zgemm_emulated_int8_512_b74"] = emu2
    del a2, b2, c2
    eye = torch.eye(n, dtype=torch.complex128, device=device)
    w = (a + n * eye).contiguous()  # well conditioned
    info = torch.zeros(B, dtype=torch.int32, device=device)
    ws = torch.empty(lib.qtx_zinv_workspace(n, B), dtype=torch.uint8, device=device)
    for name, mode in (("zinv_ours_one_cta_per_matrix", 1), ("zinv_ours_multi_cta", 2),
                       ("zinv_ours_cluster", 3), ("zinv_ours_column_split", 4), ("zinv_ours_automatic", 0)):
        _native.check(lib.qtx_set_inverse_path(mode))
        out[name] = flops / timeit(lambda: _native.check(lib.qtx_zinv_batched_ws(
            n, B, mat(w), mat(c), info.data_ptr(), ws.data_ptr(), ws.numel(), stream()))) / 1e12
    _native.check(lib.qtx_set_inverse_path(0))
    out["zinv_torch_linalg_inv"] = flops / timeit(lambda: torch.linalg.inv(w)) / 1e12
    # Inverse paths against the batch size (the automatic choice's crossover).
    sweep = {}
    for nb in (4, 8, 16, 32, 64, 96, 148, 296):
        for nn in (128, 256, 384, 512):
            if nb > B:
                continue
            wn = (torch.randn((nb, nn, nn), dtype=torch.complex128, device=device, generator=g)
                  + nn * torch.eye(nn, dtype=torch.complex128, device=device))
            cn = torch.empty_like(wn)
            wsn = torch.empty(lib.qtx_zinv_workspace(nn, nb), dtype=torch.uint8, device=device)
            row = {}
            for name, mode in (("one_cta", 1), ("multi_cta", 2), ("cluster", 3), ("column_split", 4),
                               ("automatic", 0)):
                if (mode == 3 and nn > 256) or (mode == 4 and nn > 400):
                    continue
                _native.check(lib.qtx_set_inverse_path(mode))
                row[name] = 8.0 * nn ** 3 * nb / timeit(lambda: _native.check(lib.qtx_zinv_batched_ws(
                    nn, nb, mat(wn), mat(cn), info.data_ptr(), wsn.data_ptr(), wsn.numel(), stream()))) / 1e12
            sweep[f"n{nn}_b{nb}"] = row
    _native.check(lib.qtx_set_inverse_path(0))
    out["zinv_path_sweep_tflops"] = sweep
    peak = None if args.no_peak else measured_fp64_peak(torch, device)["peak"]
    tf32 = None if args.no_peak else measured_tf32_peak(torch, device)
    line = {"metric": "kernel throughput at 256x256 blocks (complex flops 8n^3)", "unit": "TFLOP/s",
            "batch": B, "results": out, "fp64_peak_measured": peak, "tf32_peak_measured": tf32,
            "note": "inverse flops counted as 8n^3 like a GEMM; cuBLAS/cuSOLVER legs are library references"}
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    world, rank, local = dist_setup()
    if args.impl == "reference":
        run_reference(args, world, rank)
        return
    from quatrex_b200 import _native

    _native.check(_native.load().qtx_set_inverse_path({"auto": 0, "single": 1, "wide": 2, "cluster": 3, "split": 4}[args.inverse_path]))
    if args.workload != "cfg1":
        if rank == 0:
            {"cfg2": run_cfg2, "cfg3": run_cfg3, "cfg4": run_cfg4, "kernels": run_kernels,
             "inverse": run_inverse, "w": run_w}[args.workload](args, local)
        return
    run_ours(args, world, rank, local)


if __name__ == "__main__":
    main()
