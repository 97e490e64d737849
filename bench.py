"""Throughput of the NICAM-DC dynamics step on B200: gl08 z40 cell-level-steps/s,
mixed-FP32 form against the float64 form, with the mixed form's error stated
against float64.

Workload: the Jablonowski-Williamson baroclinic wave (balanced jet + 1 m/s
perturbation) on the grid-level-8 icosahedral grid (rlevel 1: 40 regions of
128x128 cells plus halo, 655,362 cells), 40 ULLRICH14 layers to 30 km,
dtl = 150 s, RK3 HEVI with [2, 3, 6] acoustic steps, DIRECT lap_order-2
hyperdiffusion and divergence damping (2.5e13), MIURA2004 tracer advection with
Thuburn limiters (nq = 1).  Grid, metrics and state are generated by
``icogrid`` (the reference's prep and setup chain restated).

A step is one large step ``Dyn.dynamics_step`` of the whole globe.  Both forms
run from the same initial state: float64 (bit for bit the reference's numpy
arithmetic) and mixed (float32 work fields, metrics and stencil arithmetic;
float64 tridiagonal elimination and matrix, pressure / density deviations and
mass sums).  ``value`` is the mixed form: K steps on the device-resident
state (CUDA graph replay, events on the library's stream); the float64 form is
timed the same way under ``fp64``.  ``e2e`` times the mixed form through the
reference-facing call sequence per step: marshal-in from pinned host memory
(float64, the reference's host layout), one step, marshal-out to pinned host
memory.  Every 3-D field is 114 MB (float32) or 227 MB (float64), larger than
L2, so no flush is needed.  ``error_vs_fp64`` compares the two forms' states
after the same steps (relative L2 per prognostic and of the surface pressure).

Multi-GPU: the path does not shard (one global step per device); with N ranks
each GPU runs an independent replica and ``value`` sums them.
"""
from __future__ import annotations

import argparse
import importlib
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "gl08 z40 cell-level-steps/s"
UNIT = "cell-level-steps/s"
# The reference's best published figures for this metric and workload, gl08 z40 on
# four GH200 with its resident, fused JAX stack and time-loop fusion
# (README.md:227-229 of pyNICAM-DC): float64 0.190 s and float32 0.100 s per step.
PUBLISHED_F64 = 26_214_480 / 0.190
PUBLISHED_F32 = 26_214_480 / 0.100

# DRAM bytes (dram__bytes_read.sum + dram__bytes_write.sum) per 3-D point of one
# launch, from ncu captures of the present kernels on gl06 z40 (1,942,080 points,
# profiles/vi_col_path1_dd3d_gl06_ncu.md; every launch's fields exceed L2); the
# traffic of a launch grows with its points, so the bench scales this to its own
# grid.  Kernels without a capture report null.
NCU_TRAFFIC_PER_POINT = {"float64": {"path1": 205.4, "dd3d": 113.1, "vi_solve": 471.0},
                         "mixed": {"path1": 100.6, "dd3d": 51.3, "vi_solve": 225.5}}


def _pkg():
    return importlib.import_module("pynicam-dc_b200")


def make_case(glevel: int, vlayer: int = 40, device: str = "cuda"):
    ig = importlib.import_module("pynicam-dc_b200.icogrid")
    dtl = {3: 1200.0, 4: 900.0, 5: 600.0, 6: 300.0, 7: 200.0, 8: 150.0}[glevel]
    gamma = {3: 7.68e17, 4: 9.6e16, 5: 1.2e16, 6: 1.5e15, 7: 2.0e14, 8: 2.5e13}[glevel]
    t = time.time()
    g = ig.Grid(glevel, vlayer=vlayer, ztop=30000.0, device=device)
    t1 = time.time()
    geo = g.setup(dtl=dtl, gamma=gamma, nq=1)
    prg, prg_pl = g.jw_state(nq=1)
    t2 = time.time()
    info = dict(setup_s=t2 - t, spring_iterations=g.spring_iters, dtl=dtl, gamma=gamma)
    print(f"[bench] gl{glevel:02d} grid+metrics {t1 - t:.1f} s, state {t2 - t1:.1f} s, "
          f"spring iterations {g.spring_iters}", file=sys.stderr, flush=True)
    del g
    return geo, prg, prg_pl, info


def cached_case(glevel: int, cache: str, device: str = "cuda"):
    """make_case, saved to / loaded from a directory of .npy files (lets a
    profiler run the step without the grid-generation launches before it)"""
    meta = os.path.join(cache, "meta.json") if cache else None
    if meta and os.path.exists(meta):
        with open(meta) as f:
            info = json.load(f)
        geo = {k: np.load(os.path.join(cache, "geo." + k + ".npy")) for k in info.pop("keys")}
        prg = np.load(os.path.join(cache, "prg.npy"))
        prg_pl = np.load(os.path.join(cache, "prg_pl.npy"))
        return geo, prg, prg_pl, info
    geo, prg, prg_pl, info = make_case(glevel, 40, device=device)
    if cache:
        os.makedirs(cache, exist_ok=True)
        for k, v in geo.items():
            np.save(os.path.join(cache, "geo." + k + ".npy"), v)
        np.save(os.path.join(cache, "prg.npy"), prg)
        np.save(os.path.join(cache, "prg_pl.npy"), prg_pl)
        with open(meta, "w") as f:
            json.dump(dict(info, keys=list(geo)), f)
    return geo, prg, prg_pl, info


def cell_levels(geo) -> int:
    G, L = int(geo["gall_1d"]), int(geo["lall"])
    return (L * (G - 2) ** 2 + 2) * (int(geo["kall"]) - 2)


class Clocks:
    """nvidia-smi sampling of SM clock and throttle reasons while running"""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.rows = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.th = threading.Thread(target=self._read, daemon=True)
            self.th.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([c.strip() for c in line.split(",")])

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.th.join(timeout=2)
        sm = [float(r[1]) for r in self.rows if len(r) >= 9 and r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if len(r) >= 9 and r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[n] for r in self.rows if len(r) >= 9 for n in range(4) if r[5 + n] == "Active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(sm)}


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        for k in ("hbm_gbs", "hbm_GBs", "hbm_gb_s"):
            if k in d:
                return float(d[k]), "measured"
    return 6650.0, "fallback"


def cpu_baseline(sample_glevel: int = 5, steps: int = 1) -> dict:
    """The numpy oracle (float64 restatement of the reference's numpy step) on
    one host core: ``steps`` large steps of the same JW case at a smaller grid
    level, in cell-level-steps/s."""
    from oracle import nicam_step as O
    geo, prg, prg_pl, _ = make_case(sample_glevel, 40, device="cpu")
    G = O.Geo(geo)
    O.dynamics_step(G, prg, prg_pl)        # warm the allocator/caches once
    t = time.time()
    s, sp = prg, prg_pl
    for _ in range(steps):
        s, sp = O.dynamics_step(G, s, sp)
    dt = time.time() - t
    return {"value": cell_levels(geo) * steps / dt, "unit": UNIT, "cores": 1, "kind": "port",
            "sample": f"{steps} large step(s) of the same JW case at gl0{sample_glevel} z40 "
                      f"({cell_levels(geo)} cell-levels), numpy float64 oracle, 1 process, {dt:.1f} s"}


def max_over_ranks(x: float, world: int, device: str) -> float:
    """the largest value of x over the ranks of the default process group
    (every rank calls it at the same point; no-op for one rank)"""
    if world <= 1:
        return float(x)
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_throughput(cell_levels_per_step: int, steps: int, world: int, ms: float) -> float:
    """whole-job cell-level-steps/s of `world` independent replicas that each
    ran `steps` steps, timed by the slowest rank (ms)"""
    return cell_levels_per_step * steps * world / (ms / 1e3)


_REF = {}


def _ref_worker(barrier, warmup, steps):
    """one host process of the reference arm: warm-up steps, then the timed
    steps between two barriers shared with the parent"""
    from oracle import nicam_step as O
    G, s, sp = _REF["G"], _REF["s"], _REF["sp"]
    for _ in range(warmup):
        s, sp = O.dynamics_step(G, s, sp)
    barrier.wait()
    barrier.wait()
    for _ in range(steps):
        s, sp = O.dynamics_step(G, s, sp)


def _host_processes(per_proc_bytes: int = 1 << 30, cap: int = 64) -> int:
    """host processes for the reference arm: every core this process may use,
    bounded by the available memory (about 1 GB per gl05 process) and a cap"""
    try:
        cores = len(os.sched_getaffinity(0))
    except AttributeError:
        cores = os.cpu_count() or 1
    try:
        import psutil
        mem = int(psutil.virtual_memory().available * 0.6 // per_proc_bytes)
    except Exception:
        mem = cores
    return max(1, min(cores, mem, cap))


def run_reference(args, rank, world):
    """The reference's CPU implementation of the step (the oracle restatement)
    on the host cores: one gl05 z40 JW case built once, then P forked
    processes each run W warm-up and K timed large steps of it concurrently;
    value = P * cell-levels * K / (time of the K steps of all processes)."""
    if rank != 0:
        return
    import multiprocessing as mp
    from oracle import nicam_step as O
    geo, prg, prg_pl, _ = make_case(5, 40, device="cpu")
    _REF.update(G=O.Geo(geo), s=prg, sp=prg_pl)
    nproc = _host_processes()
    ctx = mp.get_context("fork")   # no CUDA context exists in this process
    barrier = ctx.Barrier(nproc + 1)
    procs = [ctx.Process(target=_ref_worker, args=(barrier, args.warmup, args.steps)) for _ in range(nproc)]
    for pr in procs:
        pr.start()
    barrier.wait()                  # every process has finished its warm-up steps
    t0 = time.time()
    barrier.wait()                  # ... and starts its timed steps now
    for pr in procs:
        pr.join()
    dt = time.time() - t0
    if any(pr.exitcode != 0 for pr in procs):
        raise RuntimeError("a reference-arm process failed")
    n_cl = cell_levels(geo)
    value = nproc * n_cl * args.steps / dt
    sample = (f"gl05 z40 JW case (same physics and configuration as gl08, {n_cl} cell-levels per step), "
              f"numpy float64 restatement of the reference step; {nproc} concurrent processes x "
              f"({args.warmup} warm-up + {args.steps} timed) large steps")
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * dt / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic (analytic JW initial state)",
            "impl": "reference",
            "config": {"workload": "JW baroclinic wave, sampled at gl05 z40 on the host", "glevel": 5, "vlayer": 40,
                       "host_processes": nproc},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": nproc, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def time_steps(core, stream, steps: int, world: int, barrier) -> float:
    """device time (ms) of `steps` graph-replayed steps, max over ranks"""
    import torch
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    barrier()
    e0.record(stream)
    core.step(steps)
    e1.record(stream)
    barrier()
    return max_over_ranks(e0.elapsed_time(e1), world, "cuda")


def profile_step(core, precision: str, npt: int, npt2: int, halo_points: int, ms_per_step: float, peak: float,
                 peak_kind: str, profile_steps: int, sstep, nq: int) -> tuple:
    """per-kernel event times of eager profiled steps; the roofline of the top
    kernel and of the whole step (algorithmic bytes from roofline.py)"""
    rf = importlib.import_module("pynicam-dc_b200.roofline")
    core.profile(True)
    core.step(profile_steps)
    stats = core.kernel_stats()
    core.profile(False)
    total = sum(v[0] for v in stats.values())
    kern = {k: {"ms": round(v[0] / profile_steps, 3), "launches": v[1] // profile_steps, "share": round(v[0] / total, 4)}
            for k, v in sorted(stats.items(), key=lambda kv: -kv[1][0])}
    for k, v in kern.items():
        if k in rf.KERNELS:
            byts = rf.kernel_bytes(k, npt, npt2, precision)
            v["gbs"] = round(byts / (v["ms"] / v["launches"] / 1e3) / 1e9, 1)
            v["frac"] = round(v["gbs"] / peak, 3)
    top = max((k for k in stats if k in rf.KERNELS), key=lambda k: stats[k][0])
    avg_ms = stats[top][0] / stats[top][1]
    byts = rf.kernel_bytes(top, npt, npt2, precision)
    ach = byts / (avg_ms / 1e3) / 1e9
    tpp = NCU_TRAFFIC_PER_POINT.get(precision, {}).get(top)
    roof = {"kernel": top, "bound": "hbm", "achieved": ach, "peak": peak, "unit": "GB/s", "frac": ach / peak,
            "peak_kind": peak_kind, "traffic": (tpp * npt if tpp else None), "algorithmic_bytes_per_launch": byts,
            "avg_launch_ms": avg_ms, "share": stats[top][0] / total}
    sb = rf.step_bytes(npt, npt2, halo_points, sstep=sstep, nq=nq, precision=precision)
    step = {"algorithmic_bytes": sb["total"], "achieved": sb["total"] / (ms_per_step / 1e3) / 1e9, "peak": peak,
            "unit": "GB/s", "frac": sb["total"] / (ms_per_step / 1e3) / 1e9 / peak,
            "field_passes_f64_equiv": round(rf.field_passes(sstep, nq, npt // npt2), 1)}
    return roof, step, kern


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="cuda", choices=["cuda", "reference"])
    ap.add_argument("--glevel", type=int, default=8)
    ap.add_argument("--precision", default="both", choices=["both", "mixed", "float64"],
                    help="both: the mixed form is the headline, float64 beside it")
    ap.add_argument("--accuracy-steps", type=int, default=0,
                    help="also run this many steps of both forms from the initial state and state the error")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--profile-steps", type=int, default=1)
    ap.add_argument("--case-cache", default="", help="directory to save/load the generated case")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank, world)

    import torch
    import torch.distributed as dist
    torch.cuda.set_device(local)
    if world > 1:
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=600))

    pkg = _pkg()
    dg = importlib.import_module("pynicam-dc_b200.diagnostics")
    geo, prg, prg_pl, info = cached_case(args.glevel, args.case_cache, device="cuda")
    forms = {"both": ("mixed", "float64"), "mixed": ("mixed",), "float64": ("float64",)}[args.precision]
    cores = {f: pkg.NicamCuda(geo, graph=True, precision=f) for f in forms}
    head = forms[0]
    core = cores[head]
    n_cl = cell_levels(geo)
    sfc = {k: geo[k] for k in geo if k.startswith("sfc_") or k in ("kmin", "kmax", "GRAV", "Rdry", "Rvap", "CVdry", "CVW",
                                                                    "VMTR_GSGAM2", "VMTR_GSGAM2_pl")}
    halo_points = int(core._tab["halo_r_dst"].size + core._tab["halo_p_dst"].size)
    sstep = tuple(int(x) for x in np.asarray(geo["sstep"]))
    nq = int(np.asarray(geo["nq"]))
    del geo
    stream = torch.cuda.ExternalStream(core.stream_ptr())

    # pinned host buffers in the reference layout (marshal-in / marshal-out)
    h_prg = torch.from_numpy(prg).pin_memory()
    h_pl = torch.from_numpy(prg_pl).pin_memory()
    o_prg = torch.empty_like(h_prg).pin_memory()
    o_pl = torch.empty_like(h_pl).pin_memory()
    for c in cores.values():
        c.upload_ptr(h_prg.data_ptr(), h_pl.data_ptr())

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        for c in cores.values():
            c.sync()
        torch.cuda.synchronize()

    # warm-up (graph capture happens on the first step)
    for c in cores.values():
        c.step(args.warmup)
    barrier()

    vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
    clocks = Clocks(vis.split(",")[local] if vis else local)
    clocks.start()
    launches0 = core.kernel_launches()
    mass0 = core.mass_sums()
    ms = time_steps(core, stream, args.steps, world, barrier)
    gpu_launches = core.kernel_launches() - launches0
    other = {}
    for f in forms[1:]:
        c = cores[f]
        other[f] = time_steps(c, torch.cuda.ExternalStream(c.stream_ptr()), args.steps, world, barrier)
    clk = clocks.stop()
    mass1 = core.mass_sums()
    drift = [float(abs(b - a) / abs(a)) if a != 0 else 0.0 for a, b in zip(mass0, mass1)]
    value = replica_throughput(n_cl, args.steps, world, ms)

    # error of the mixed form against float64 after the same warm-up + timed steps
    errors = None
    if len(forms) == 2:
        sm = cores["mixed"].download()
        sd = cores["float64"].download()
        errors = {"steps": args.warmup + args.steps, "rel_l2": dg.state_errors(sfc, sm, sd)}
        for c in cores.values():
            c.upload_ptr(h_prg.data_ptr(), h_pl.data_ptr())
            c.step(1)
        errors["rel_l2_after_1_step"] = dg.state_errors(sfc, cores["mixed"].download(), cores["float64"].download())
        if args.accuracy_steps > 0:
            for c in cores.values():
                c.upload_ptr(h_prg.data_ptr(), h_pl.data_ptr())
                c.step(args.accuracy_steps)
            errors["rel_l2_after_%d_steps" % args.accuracy_steps] = dg.state_errors(
                sfc, cores["mixed"].download(), cores["float64"].download())
        del sm, sd

    # end to end: pinned host state -> device -> one step -> pinned host, per step
    e2e_steps = args.steps
    core.upload_ptr(h_prg.data_ptr(), h_pl.data_ptr())
    core.step(1)
    core.download_ptr(o_prg.data_ptr(), o_pl.data_ptr())
    barrier()
    t0 = torch.cuda.Event(enable_timing=True)
    t1 = torch.cuda.Event(enable_timing=True)
    t0.record(stream)
    for _ in range(e2e_steps):
        # each step: its input state host -> device, the step, its result device -> host;
        # the copies run on the library's copy streams and overlap the neighbouring steps
        core.upload_ptr(h_prg.data_ptr(), h_pl.data_ptr())
        core.step(1)
        core.download_ptr_async(o_prg.data_ptr(), o_pl.data_ptr())
    core.join_copies()
    t1.record(stream)
    barrier()
    e2e_ms = t0.elapsed_time(t1) / e2e_steps
    e2e_ms = max_over_ranks(e2e_ms, world, "cuda")
    io_bytes = int(h_prg.numel() + h_pl.numel()) * 8
    finite = bool(np.isfinite(o_prg.numpy()).all())
    core.check_finite()
    mass = core.mass_sums()

    # per-kernel device times of eager profiled steps; rooflines
    G = int(core.shape[0])
    npt = G * G * core.shape[2] * core.shape[3]
    npt2 = G * G * core.shape[3]
    peak, peak_kind = peaks()
    roof, step_roof, kern = profile_step(core, head, npt, npt2, halo_points, ms / args.steps, peak, peak_kind,
                                         args.profile_steps, sstep, nq)
    fp64 = None
    if "float64" in other:
        r64, s64, k64 = profile_step(cores["float64"], "float64", npt, npt2, halo_points, other["float64"] / args.steps,
                                     peak, peak_kind, args.profile_steps, sstep, nq)
        v64 = replica_throughput(n_cl, args.steps, world, other["float64"])
        fp64 = {"value": v64, "unit": UNIT, "ms_per_step": other["float64"] / args.steps,
                "vs_baseline": (v64 / PUBLISHED_F64 if args.glevel == 8 else None),
                "roofline": r64, "roofline_step": s64, "kernels": k64}
    for c in cores.values():
        c.close()

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline()

    if rank == 0:
        published = PUBLISHED_F32 if head == "mixed" else PUBLISHED_F64
        line = {"metric": METRIC + (": mixed-FP32 vs FP64" if len(forms) == 2 else ""), "value": value, "unit": UNIT,
                "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
                "scaling": "weak", "vs_baseline": (value / published if args.glevel == 8 else None),
                "dtype": "f32+f64" if head == "mixed" else "f64", "precision": head,
                "data": "synthetic (analytic JW initial state on a generated gl08 grid)",
                "config": {"workload": f"JW baroclinic wave gl0{args.glevel} z40 rl01 (40 regions of "
                                       f"{G - 2}x{G - 2} + halo), dtl {info['dtl']} s, RK3 HEVI [2,3,6], "
                                       f"DIRECT lap-2 hyperdiffusion/divdamp {info['gamma']:.2e}, "
                                       "MIURA2004 tracer nq=1",
                           "glevel": args.glevel, "vlayer": 40, "cell_levels": n_cl, "parallelism": f"replicas x{world}",
                           "forms": list(forms),
                           "l2": "inputs larger than L2 (114 MB float32 / 227 MB float64 per 3-D field at gl08)",
                           "cuda_graph": True, "setup_s": round(info["setup_s"], 1),
                           "spring_iterations": info["spring_iterations"],
                           "vs_baseline_ref": ("reference float32 stack, 0.100 s/step on 4x GH200" if head == "mixed"
                                               else "reference float64 stack, 0.190 s/step on 4x GH200")},
                "e2e": {"value": replica_throughput(n_cl, 1, world, e2e_ms), "unit": UNIT, "h2d_bytes_per_step": io_bytes,
                        "d2h_bytes_per_step": io_bytes},
                "roofline": roof, "roofline_step": step_roof, "cpu_baseline": cpu, "clocks": clk,
                "gpu_launches": gpu_launches, "finite_after_steps": finite, "air_mass": float(mass[0]),
                "mass_drift": {"steps": args.steps, "dry_air": drift[0], "tracers": drift[1:]}}
        if fp64 is not None:
            line["fp64"] = fp64
            line["mixed_over_fp64"] = fp64["ms_per_step"] / (ms / args.steps)
        if errors is not None:
            line["error_vs_fp64"] = errors
        line["kernels"] = kern
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
