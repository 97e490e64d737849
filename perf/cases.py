"""The work that programs have this package do, as cases that can be timed and checked.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call (a handle of
the grid, the state on the device), ``run`` makes one pass through the public entry points, ``work``
says what the pass cannot do without, ``tolerance`` how far two correct implementations of the same
precision may differ, ``exact`` what plain torch gives in 64 bits where that is quick.

The grids, time steps and coefficients are those of bench.py (grid levels 3 to 8, the balanced jet
of ``icogrid.Grid.jw_state``), the tracer-transport case of tests/test_gpu_tracer_transport.py and the
adjoint configurations of tests/test_gpu_dynstep.py and tests/test_gpu_adjoint.py.  A seed gives the
temperature perturbation (0.5 K, 500 km, as the ensemble's members have it), the moisture or tracers,
and the cotangents.  A handle is kept from one preparation to the next, as a program keeps its own:
every pass begins by putting its state on the handle.
"""
from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

_P = "pynicam-dc_b200"
pkg = importlib.import_module(_P)
icogrid = importlib.import_module(_P + ".icogrid")
ensemble = importlib.import_module(_P + ".ensemble")
adjoint = importlib.import_module(_P + ".adjoint")
dynstep = importlib.import_module(_P + ".dynstep")
halo = importlib.import_module(_P + ".halo")

A_EARTH = 6371220.0
DTL = {3: 1200.0, 4: 900.0, 5: 600.0, 6: 300.0, 7: 200.0, 8: 150.0}
GAMMA = {3: 7.68e17, 4: 9.6e16, 5: 1.2e16, 6: 1.5e15, 7: 2.0e14, 8: 2.5e13}
NAMES = ("RHOG", "RHOGVX", "RHOGVY", "RHOGVZ", "RHOGW", "RHOGE")


def listed():
    return [
        # the smallest grid of the test fixtures: launches and latency are all there is
        dict(name="step gl03 z10 f64", kind="step", glevel=3, vlayer=10, precision="float64", members=1, steps=4),
        # the reference's own day run (gl05 z40, 600 s), in chunks of four steps between outputs
        dict(name="step gl05 z40 f64", kind="step", glevel=5, vlayer=40, precision="float64", members=1, steps=4),
        # a run at moderate resolution in the fast form
        dict(name="step gl06 z40 mixed", kind="step", glevel=6, vlayer=40, precision="mixed", members=1, steps=2),
        # the form that reproduces the reference's numbers, at a size that fills the card
        dict(name="step gl07 z40 f64", kind="step", glevel=7, vlayer=40, precision="float64", members=1, steps=1),
        # the benchmark's workload
        dict(name="step gl08 z40 mixed", kind="step", glevel=8, vlayer=40, precision="mixed", members=1, steps=1),
        # an ensemble of perturbed members in one handle
        dict(name="ensemble gl05x12 z40 mixed", kind="step", glevel=5, vlayer=40, precision="mixed", members=12, steps=1),
        # a climate run: each step followed by the Held-Suarez relaxation; an odd number of layers
        dict(name="held-suarez gl06 z25 f64", kind="hs", glevel=6, vlayer=25, precision="float64", members=1, steps=1),
        # offline transport of 16 tracers (and the vapour slot) by the DCMIP 1-1 winds
        dict(name="tracers gl07 z60 x17 f64", kind="trcadv", glevel=7, vlayer=60, precision="float64", tracers=17, steps=1),
        # sensitivity of transported tracers to their initial fields
        dict(name="tracer gradient gl06 z60", kind="trcgrad", glevel=6, vlayer=60, tracers=4, steps=2),
        # sensitivity of the surface pressure in a box to the state a step earlier
        dict(name="dynamics gradient gl06 z40", kind="dyngrad", glevel=6, vlayer=40, steps=1),
        # a differentiable filter or loss term built from the stencil operators
        dict(name="gradient operator gl06 z40", kind="operator", op="gradient", glevel=6, vlayer=40),
        # the implicit vertical solve and its matrix cotangents
        dict(name="vertical solve gl06 z40", kind="vsolve", glevel=6, vlayer=40),
    ]


def draw(rng):
    """one more case of the same ranges: grid level, layers, form and kind at random"""
    kind = rng.choice(["step"] * 5 + ["hs", "trcadv", "trcgrad", "dyngrad", "operator", "operator", "vsolve"])
    prec = rng.choice(["float64", "mixed"])
    z = int(round(math.exp(rng.uniform(math.log(10.0), math.log(80.0)))))
    if kind == "step":
        gl = rng.choice([3, 4, 5, 6, 7])
        members = rng.choice([1, 1, rng.randint(2, 6)]) if gl <= 5 else 1
        return dict(kind="step", glevel=gl, vlayer=z, precision=prec, members=members, steps=rng.randint(1, 3))
    if kind == "hs":
        return dict(kind="hs", glevel=rng.choice([4, 5, 6]), vlayer=z, precision="float64", members=1,
                    steps=rng.randint(1, 2))
    if kind == "trcadv":
        return dict(kind="trcadv", glevel=rng.choice([4, 5, 6]), vlayer=z, precision=prec, tracers=rng.randint(1, 17),
                    steps=1)
    z = min(z, 62)     # the differentiable operators' limit
    if kind == "trcgrad":
        return dict(kind="trcgrad", glevel=rng.choice([4, 5, 6]), vlayer=z, tracers=rng.randint(1, 5), steps=1)
    if kind == "dyngrad":
        return dict(kind="dyngrad", glevel=rng.choice([4, 5]), vlayer=z, steps=1)
    gl = rng.choice([3, 4, 5, 6])
    if kind == "vsolve":
        return dict(kind="vsolve", glevel=gl, vlayer=z)
    return dict(kind="operator", op=rng.choice(["laplacian", "gradient", "divergence"]), glevel=gl, vlayer=z)


# ---------------------------------------------------------------------------
# grids, handles and unperturbed states
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=24)
def _case_of(glevel, vlayer, offline, nq):
    """the setup dict of a grid and its unperturbed state (reference layout, on the device)"""
    if offline:
        g = icogrid.Grid(glevel, vlayer=vlayer, ztop=12000.0, device="cuda", layer="EVEN", topo="NONE")
        geo = g.setup(dtl=300.0, gamma=GAMMA[glevel], nq=nq, trcadv=True)
        s, sp = g.trcadv_state(lambda lon, lat, z: np.zeros(z.shape + (1,)))
    else:
        g = icogrid.Grid(glevel, vlayer=vlayer, ztop=30000.0, device="cuda")
        geo = g.setup(dtl=DTL[glevel], gamma=GAMMA[glevel], nq=nq)
        geo["lat"] = np.ascontiguousarray(np.moveaxis(g.lat, 0, 2))
        s, sp = g.jw_state(nq=1)
    return geo, torch.from_numpy(s).cuda(), torch.from_numpy(sp).cuda()


@functools.lru_cache(maxsize=1)
def _handle(glevel, vlayer, offline, nq, precision, members, hs):
    geo, _, _ = _case_of(glevel, vlayer, offline, nq)
    g = dict(geo)
    lat = g.pop("lat", None)
    if hs:
        g["GRD_LAT"] = lat
    if members > 1:
        g = ensemble.stack_setup(g, members)
    return pkg.NicamCuda(g, graph=True, precision=precision)


def _case(case):
    kind = case["kind"]
    offline = kind in ("trcadv", "trcgrad")
    nq = case.get("tracers", 1)
    key = (case["glevel"], case["vlayer"], offline, nq)
    return key, key + (case.get("precision", "float64"), case.get("members", 1), kind == "hs")


def _bumps(x, gen, width, n=48):
    """sum of n seeded Gaussian bumps of the given width (radians) at the unit vectors x (..., 3)"""
    c = torch.randn(n, 3, generator=gen, dtype=torch.float64)
    c = (c / c.norm(dim=1, keepdim=True)).cuda()
    a = torch.randn(n, generator=gen, dtype=torch.float64).cuda()
    out = []
    for xx in x:
        o = torch.zeros(xx.shape[:-1], dtype=torch.float64, device="cuda")
        for m in range(n):
            o += a[m] * torch.exp(((xx * c[m]).sum(-1) - 1.0) / width ** 2)
        out.append(o)
    return out


def _moist_jet(case, seed):
    """the balanced jet with a smooth temperature perturbation and a vapour field with sharp edges,
    one perturbation per member"""
    key, _ = _case(case)
    geo, base, base_pl = _case_of(*key)
    gen = torch.Generator().manual_seed(seed)
    r = float(geo["rscale"])
    x = torch.from_numpy(geo["GRD_x"][:, :, 0]).cuda() / r                # (i, j, l, 3)
    x_pl = torch.from_numpy(geo["GRD_x_pl"][:, 0]).cuda() / r             # (g, l, 3)
    K = base.shape[2]
    cv = float(geo["CVdry"])
    prof = 0.012 * torch.exp(-torch.from_numpy(np.asarray(geo["GRD_gz"], np.float64)).clamp(min=0.0) / 2500.0).cuda()
    regs, pls = [], []
    for _ in range(case.get("members", 1)):
        t, t_pl = _bumps((x, x_pl), gen, 500e3 / A_EARTH)
        sc = 0.5 / float(t.std())
        b, b_pl = _bumps((x, x_pl), gen, 0.25, 12)
        for s0, tt, bb, out in ((base, t, b, regs), (base_pl, t_pl, b_pl, pls)):
            s = s0.clone()
            ax = 2 if s.dim() == 5 else 1
            pert = (tt * sc).unsqueeze(ax)
            wet = (0.3 + 0.6 * (bb > 0.2).double() + 0.1 * torch.tanh(bb)).unsqueeze(ax)
            s[..., 5] += s[..., 0] * cv * pert
            shape = [1] * (s.dim() - 1)
            shape[ax] = K
            s[..., 6] = s[..., 0] * (prof.view(shape) * wet)
            out.append(s)
    if len(regs) == 1:
        return regs[0], pls[0]
    return torch.cat(regs, 3).contiguous(), torch.cat(pls, 2).contiguous()


def _tracer_state(case, seed):
    """the offline-advection state with its tracers: a vapour slot of zeros, then Gaussian hills, cosine
    bells and slotted cylinders in turn at seeded centres"""
    key, _ = _case(case)
    geo, base, base_pl = _case_of(*key)
    rng = np.random.default_rng(seed)
    nq = case["tracers"]
    out = []
    lons, lats, zs = rng.uniform(0, 2 * np.pi, nq), rng.uniform(-1.0, 1.0, nq), rng.uniform(3000.0, 9000.0, nq)
    for s0, sfx in ((base, ""), (base_pl, "_pl")):
        ax = 2 if not sfx else 1
        lon = torch.from_numpy(np.nan_to_num(geo["GRD_LON" + sfx])).cuda().unsqueeze(ax)
        lat = torch.from_numpy(np.nan_to_num(geo["GRD_LAT" + sfx])).cuda().unsqueeze(ax)
        z = torch.from_numpy(geo["GRD_Z" + sfx]).cuda()
        s = torch.empty(s0.shape[:-1] + (6 + nq,), dtype=torch.float64, device="cuda")
        s[..., :6] = s0[..., :6]
        s[..., 6] = 0.0
        for n in range(1, nq):
            cosr = torch.sin(lat) * math.sin(lats[n]) + torch.cos(lat) * math.cos(lats[n]) * torch.cos(lon - lons[n])
            rr = torch.arccos(cosr.clamp(-1.0, 1.0))
            dz = (z - zs[n]) / 1000.0
            d = (rr / 0.5) ** 2 + dz ** 2
            if n % 4 in (1, 2):
                q = torch.exp(-(rr / 0.25) ** 2 - dz ** 2)
            elif n % 4 == 3:
                q = torch.where(d < 1.0, 0.1 + 0.45 * (1.0 + torch.cos(math.pi * d.clamp(max=1.0))), 0.1)
            else:
                slot = (torch.sin(lon - lons[n]).abs() < 0.1) & (lat < lats[n] + 0.25)
                q = torch.where((d < 1.0) & ~slot, 1.0, 0.1)
            s[..., 6 + n] = s[..., 0] * q
        out.append(s)
    return out[0], out[1]


def _device_layout(prg, prg_pl, v0, v1):
    """variables v0..v1 of a state as (nv, l, k, j, i) and (nv, g, k, l)"""
    return prg[..., v0:v1].permute(4, 3, 2, 1, 0).contiguous(), prg_pl[..., v0:v1].permute(3, 0, 1, 2).contiguous()


def _random(shape, gen):
    return torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    _, hkey = _case(case)
    core = _handle(*hkey)
    geo = _case_of(*_case(case)[0])[0]
    st = dict(kind=kind, core=core, steps=case.get("steps", 1))
    if kind in ("step", "hs"):
        st["prg"], st["prg_pl"] = _moist_jet(case, seed)
    elif kind == "trcadv":
        st["prg"], st["prg_pl"] = _tracer_state(case, seed)
    elif kind == "trcgrad":
        s, sp = _tracer_state(case, seed)
        st["model"] = adjoint.TracerTransport(core, s, sp, checkpoint_every=1)
        x, x_pl = st["model"].initial_tracers()
        gen = torch.Generator(device="cuda").manual_seed(seed)
        st["x"], st["x_pl"] = x.requires_grad_(True), x_pl.requires_grad_(True)
        st["g"], st["g_pl"] = _random(x.shape, gen), _random(x_pl.shape, gen)
    elif kind == "dyngrad":
        s, sp = _moist_jet(case, seed)
        x, x_pl = _device_layout(s, sp, 0, 6)
        st["x"], st["x_pl"] = x.requires_grad_(True), x_pl.requires_grad_(True)
        q, q_pl = _device_layout(s, sp, 6, 7)
        st["q"], st["q_pl"] = torch.zeros_like(q), torch.zeros_like(q_pl)
        st["stepper"] = _stepper(case["glevel"], case["vlayer"])
        L, K, G = core.field_shape[0], core.field_shape[1], core.field_shape[2]
        z = float(geo["GRD_gz"][1])
        st["zk"] = torch.full((L, 1, G, G), z, dtype=torch.float64, device="cuda")
        st["zk_pl"] = torch.full((6, 1, 2), z, dtype=torch.float64, device="cuda")
        lat = torch.from_numpy(geo["lat"]).permute(2, 1, 0).unsqueeze(1).cuda()
        st["box"] = ((lat - math.radians(40.0)).abs() < math.radians(10.0)).double()
        st["ps0"] = st["stepper"].surface_pressure(x.detach(), x_pl.detach(), st["zk"], st["zk_pl"])[0]
    elif kind == "operator":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        ni, no = _components(case["op"])
        shp = lambda n, f: ((n,) if n > 1 else ()) + tuple(f)
        st["op"] = getattr(adjoint, case["op"])
        for k, n in (("x", ni), ("g", no)):
            st[k], st[k + "_pl"] = (_random(shp(n, f), gen) for f in (core.field_shape, core.field_shape_pl))
        st["x"] = (280.0 + 30.0 * st["x"]).requires_grad_(True)
        st["x_pl"] = (280.0 + 30.0 * st["x_pl"]).requires_grad_(True)
    elif kind == "vsolve":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        f = core.field_shape
        st["M"] = tuple(t.requires_grad_(True) for t in (
            3.0 + 0.3 * _random(f, gen), -1.0 + 0.1 * _random(f, gen), -1.0 + 0.1 * _random(f, gen), _random(f, gen)))
        st["g"] = _random(f, gen)
    return st


@functools.lru_cache(maxsize=1)
def _stepper(glevel, vlayer):
    key = (glevel, vlayer, False, 1)
    return dynstep.DynamicsStep(_handle(*key, "float64", 1, False), _case_of(*key)[0])


def _components(op):
    return {"laplacian": (1, 1), "gradient": (1, 3), "divergence": (3, 1)}[op]


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    kind, core = st["kind"], st["core"]
    if kind in ("step", "hs", "trcadv"):
        if kind == "trcadv":
            core.set_time(0.0)
        core.upload_tensor(st["prg"], st["prg_pl"])
        if kind == "hs":
            for _ in range(st["steps"]):
                core.step(1)
                core.forcing_step()
        else:
            core.step(st["steps"])
        s, sp = core.download_tensor()
        out = {}
        for v in range(s.shape[-1]):
            name = NAMES[v] if v < 6 else "RHOGQ%d" % (v - 5)
            out[name], out[name + "_pl"] = s[..., v], sp[..., v]
        return out
    if kind == "trcgrad":
        y, y_pl = st["model"].run(st["x"], st["x_pl"], st["steps"])
        g, g_pl = torch.autograd.grad((y, y_pl), (st["x"], st["x_pl"]), (st["g"], st["g_pl"]))
        return {"y": y.detach(), "y_pl": y_pl.detach(), "g": g, "g_pl": g_pl}
    if kind == "dyngrad":
        m = st["stepper"]
        y, y_pl = m.run(st["x"], st["x_pl"], st["steps"], checkpoint=True, tracers=st["q"], tracers_pl=st["q_pl"])
        ps, _ = m.surface_pressure(y, y_pl, st["zk"], st["zk_pl"])
        loss = ((ps - st["ps0"]) ** 2 * st["box"]).sum()
        g, g_pl = torch.autograd.grad(loss, (st["x"], st["x_pl"]))
        return {"loss": loss.detach(), "y": y.detach(), "y_pl": y_pl.detach(),
                "g": [g[v] for v in range(6)], "g_pl": [g_pl[v] for v in range(6)]}
    if kind == "operator":
        y, y_pl = st["op"](core, st["x"], st["x_pl"])
        g, g_pl = torch.autograd.grad((y, y_pl), (st["x"], st["x_pl"]), (st["g"], st["g_pl"]))
        return {"y": y.detach(), "y_pl": y_pl.detach(), "g": g, "g_pl": g_pl}
    x = adjoint.vertical_solve(core, *st["M"])
    g = torch.autograd.grad(x, st["M"], st["g"])
    return {"x": x.detach(), "gMc": g[0], "gMu": g[1], "gMl": g[2], "gb": g[3]}


# ---------------------------------------------------------------------------
# what a pass needs, and how far two correct results may be apart
# ---------------------------------------------------------------------------
def work(case):
    """bytes: the inputs read once and the outputs written once, and for the steps the metrics (22 3-D arrays
    and 108 coefficient planes) read once; flops: counted by hand from the expressions of the step
    (about 11 x 320 for the acoustic steps, 3 x 1000 for the rest, 700 for each tracer, per point and step)"""
    kind = case["kind"]
    L, G, K = 40 * case.get("members", 1), 2 ** (case["glevel"] - 1) + 2, case["vlayer"] + 2
    n = L * G * G * K
    e = 4 if case.get("precision") == "mixed" else 8
    steps = case.get("steps", 1)
    if kind in ("step", "hs"):
        return {"bytes": 2 * 7 * 8 * n + e * (22 * n + 108 * n // K), "flops": steps * 7200 * n}
    if kind == "trcadv":
        nv = 6 + case["tracers"]
        return {"bytes": 2 * nv * 8 * n + e * (15 * n + 46 * n // K), "flops": steps * (300 + 700 * case["tracers"]) * n}
    if kind == "trcgrad":
        nq = case["tracers"]
        return {"bytes": 8 * n * (6 + 4 * nq + 15), "flops": steps * 3 * 700 * nq * n}
    if kind == "dyngrad":
        return {"bytes": 8 * n * (6 * 3 + 22), "flops": steps * 4 * 6500 * n}
    if kind == "operator":
        ni, no = _components(case["op"])
        planes = 7 * ni * no
        return {"bytes": 8 * (2 * (ni + no) * n + planes * n // K), "flops": 4 * planes * n}
    return {"bytes": 8 * 10 * n, "flops": 22 * n}


def tolerance(case):
    """About four times the largest difference measured on a B200 over the outputs of a case:
    float64 steps: the same step from a state changed by one rounding, 4.2e-13 (the momentum and RHOGW, which
    are small against the terms they are formed from);
    mixed steps: against the float64 form, up to 3.3e-4 (RHOGW and the pole momentum; RHOG and RHOGE 6e-8);
    offline tracers: 1.7e-16 and, mixed, 1.2e-6;
    gradients of a step: 1.5e-13 from a state changed by one rounding; of the tracers: 2e-16 between two runs
    (sums in another order; the limiter's branches must be the same, since a changed branch changes the
    gradient by its own size);
    single operators: 8e-16 against ``exact``"""
    kind, mixed = case["kind"], case.get("precision") == "mixed"
    if kind in ("step", "hs"):
        return {"rel": 1.5e-3 if mixed else 2e-12}
    if kind == "trcadv":
        return {"rel": 5e-6 if mixed else 1e-14}
    return {"rel": {"dyngrad": 6e-13, "trcgrad": 1e-14, "operator": 4e-15, "vsolve": 2e-15}[kind]}


# ---------------------------------------------------------------------------
# plain torch in 64 bits
# ---------------------------------------------------------------------------
def _exchange(plan, x, x_pl):
    """halo values of x (..., l, k, j, i) and the pole neighbours of x_pl (..., g, k, l) from their sources"""
    r_dst, r_src, p_dst, p_src = (torch.from_numpy(a).cuda() for a in plan)
    K, G, LP = x.shape[-3], x.shape[-1], x_pl.shape[-1]
    flat = lambda t: t.movedim(-3, -1).reshape(t.shape[:-4] + (-1, K))        # (..., l j i, k)
    flat_pl = lambda t: t.movedim(-2, -1).reshape(t.shape[:-3] + (-1, K))     # (..., g l, k)
    f, fp = flat(x), flat_pl(x_pl)
    both = torch.cat([f, fp], -2)
    n = f.shape[-2]
    src = torch.where(r_src >= 0, r_src, n + (-r_src - 1))
    y = f.index_copy(-2, r_dst, both.index_select(-2, src))
    y_pl = fp.index_copy(-2, p_dst, f.index_select(-2, p_src))
    back = y.reshape(x.shape[:-4] + (x.shape[-4], G, G, K)).movedim(-1, -3)
    back_pl = y_pl.reshape(x_pl.shape[:-3] + (x_pl.shape[-3], LP, K)).movedim(-1, -2)
    return back, back_pl


def _stencil(c, x):
    """sum over the hexagon of c (7, l, 1, j, i) times x (l, k, j, i), interior cells"""
    n = x.shape[-1]
    off = ((1, 1), (1, 2), (2, 2), (2, 1), (1, 0), (0, 0), (0, 1))            # (j, i) of the seven cells
    out = sum(c[m][..., 1:-1, 1:-1] * x[..., oj:n - 2 + oj, oi:n - 2 + oi] for m, (oj, oi) in enumerate(off))
    return torch.nn.functional.pad(out, (1, 1, 1, 1))


def exact(case, seed):
    if case["kind"] == "operator":
        return _exact_operator(case, seed)
    if case["kind"] == "vsolve":
        return _exact_vsolve(case, seed)
    return None      # a whole step in plain numpy takes from half a minute (gl05) to a quarter of an hour (gl08)


def _exact_operator(case, seed):
    st = prepare(case, seed)
    geo = _case_of(*_case(case)[0])[0]
    plan = halo.compose(geo["copy_r2r"], geo["copy_p2r"], geo["copy_r2p"], geo["copy_sgp"], int(geo["gall_1d"]),
                        int(geo["lall"]))
    name = {"laplacian": "lap", "gradient": "grad", "divergence": "div"}[case["op"]]
    c = torch.from_numpy(geo["OPRT_coef_" + name][:, :, 0]).cuda()            # (i, j, l[, d], m)
    c_pl = torch.from_numpy(geo["OPRT_coef_" + name + "_pl"][:, 0]).cuda()    # (g, l[, d])
    if case["op"] == "laplacian":
        c, c_pl = c.unsqueeze(-2), c_pl.unsqueeze(-1)
    c = c.permute(3, 4, 2, 1, 0).unsqueeze(3)                                 # (d, m, l, 1, j, i)
    c_pl = c_pl.permute(2, 0, 1).unsqueeze(2)                                 # (d, g, 1, l)
    x, x_pl = _exchange(plan, st["x"], st["x_pl"])
    row = lambda d, v: torch.nn.functional.pad((c_pl[d] * v).sum(0, keepdim=True), (0, 0, 0, 0, 0, 5))
    if case["op"] == "laplacian":
        y, y_pl = _stencil(c[0], x), row(0, x_pl)
    elif case["op"] == "gradient":
        y, y_pl = torch.stack([_stencil(c[d], x) for d in range(3)]), torch.stack([row(d, x_pl) for d in range(3)])
    else:
        y, y_pl = sum(_stencil(c[d], x[d]) for d in range(3)), sum(row(d, x_pl[d]) for d in range(3))
    g, g_pl = torch.autograd.grad((y, y_pl), (st["x"], st["x_pl"]), (st["g"], st["g_pl"]))
    return {"y": y.detach(), "y_pl": y_pl.detach(), "g": g, "g_pl": g_pl}


def _exact_vsolve(case, seed):
    st = prepare(case, seed)
    core = st["core"]
    k0, k1 = core.kmin + 1, core.kmax + 1
    Mc, Mu, Ml, b = (t.detach()[:, k0:k1] for t in st["M"])

    def solve(Mc, Mu, Ml, b):
        """cyclic elimination from both ends: rows downward, then the back substitution"""
        n = b.shape[1]
        d, r = [None] * n, [None] * n
        d[n - 1], r[n - 1] = Mc[:, n - 1], b[:, n - 1]
        for k in range(n - 2, -1, -1):
            w = Mu[:, k] / d[k + 1]
            d[k], r[k] = Mc[:, k] - w * Ml[:, k + 1], b[:, k] - w * r[k + 1]
        x = [r[0] / d[0]]
        for k in range(1, n):
            x.append((r[k] - Ml[:, k] * x[-1]) / d[k])
        return torch.stack(x, 1)
    x = solve(Mc, Mu, Ml, b)
    shift = lambda t, s: torch.roll(t, s, 1)
    lam = solve(Mc, shift(Ml, -1), shift(Mu, 1), st["g"].detach()[:, k0:k1])
    gMc, gMu, gMl = -lam * x, -lam * shift(x, -1), -lam * shift(x, 1)
    gMu[:, -1], gMl[:, 0] = 0.0, 0.0
    K = st["M"][0].shape[1]
    full = lambda t: torch.nn.functional.pad(t, (0, 0, 0, 0, k0, K - k1))
    return {"x": full(x), "gMc": full(gMc), "gMu": full(gMu), "gMl": full(gMl), "gb": full(lam)}
