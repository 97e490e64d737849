"""Project-written autotuner of the step's launch shapes.

The column and point kernels of the step take their threads per block at run
time (``nc_set_block``); the right size depends on the grid (columns per
region, regions and ensemble members), on the precision form (registers per
thread) and on the device.  ``tune`` picks each kernel's block size by
measurement: coordinate-wise, one kernel at a time, it times one eager
profiled step per candidate size (``nc_profile`` events, the kernel's own
time) and keeps the fastest, then writes the choice to a JSON cache keyed by
the device name, the state shape, the precision and the ensemble members, so
a later handle of the same case applies it without measuring.  The key also
holds a number that is raised when a tuned kernel changes its form, so a table
measured on other kernels is measured again.

The tiled stencil kernels keep their compile-time tile shapes (32 x 8 cells of
one region, 16 x 16 for regions of at most 16 cells a side, chosen by
measurement on B200) and their resident-block targets (``NC_F32_*`` / launch
bounds): those are template constants of the kernels, not launch parameters.
``vi_solve`` and ``vi_energy`` are accepted, but have no effect (their column
kernel has a fixed block): they keep their default and are not measured.

Tuning advances the handle's state by the profiled steps: upload the state
again afterwards (the ensemble driver does).
"""
from __future__ import annotations

import json
import os

# the largest block a launch uses (nc_set_block accepts 1024 for the tracer kernels too)
TUNABLE = {"diag": 128, "vi_solve": 128, "vi_energy": 128, "vp0_c": 256, "gtend": 1024, "hdiff1": 1024,
           "post": 1024, "split_init": 1024, "trc_vflux": 1024, "trc_vadv": 256, "trc_remap": 512,
           "trc_qout": 512, "trc_apply": 512, "trc_rhog": 1024}
FIXED = ("vi_solve", "vi_energy")
CANDIDATES = (64, 128, 256, 512)
KERNELS = 2   # 1: a thread per column; 2: a thread per point, batches of tracers


def _device_name() -> str:
    try:
        import torch
        return torch.cuda.get_device_name(torch.cuda.current_device())
    except Exception:
        return "cuda"


def cache_key(core, members: int = 1) -> str:
    return "|".join([_device_name(), "x".join(str(x) for x in core.shape), core.precision, f"members={members}",
                     f"kernels={KERNELS}"])


def tune(core, members: int = 1, candidates=CANDIDATES, cache: str | None = None, repeats: int = 1) -> dict:
    """Choose the block size of every tunable kernel on ``core`` (a
    NicamCuda with a state uploaded); returns {kernel: threads}.  With
    ``cache`` (a JSON file), a stored choice for the same key is applied
    without measuring, and a new one is stored."""
    key = cache_key(core, members)
    table = {}
    if cache and os.path.exists(cache):
        with open(cache) as f:
            table = json.load(f)
        if key in table:
            for k, t in table[key].items():
                core.set_block(k, t)
            return dict(table[key])

    def kernel_ms(name: str) -> float:
        core.profile(True)
        core.step(repeats)
        st = core.kernel_stats()
        core.profile(False)
        return st.get(name, (float("inf"), 0))[0] / repeats

    choice = {}
    for name, top in TUNABLE.items():
        sizes = [c for c in candidates if c <= top and name not in FIXED]
        timing = {}
        for c in sizes:
            core.set_block(name, c)
            timing[c] = kernel_ms(name)
        if not timing or min(timing.values()) == float("inf"):
            core.set_block(name, min(top, 128))   # fixed, or not launched in this configuration
            choice[name] = min(top, 128)
            continue
        best = min(timing, key=timing.get)
        core.set_block(name, best)
        choice[name] = best
    if cache:
        table[key] = choice
        os.makedirs(os.path.dirname(os.path.abspath(cache)), exist_ok=True)
        with open(cache, "w") as f:
            json.dump(table, f, indent=1, sort_keys=True)
    return choice
