"""What a handle accepts as an exchange plan: every plan of the model's grids;
no entry outside the state (set-up and the kernels use them as indices) and no
source that the same pass writes.  A plan that writes interior cells as well
works in every operator (on the GPU)."""
import glob
import importlib
import os

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def plan(pkg, golden):
    geo, _ = golden
    G, L = int(geo["gall_1d"]), int(geo["lall"])
    return pkg.halo.compose(geo["copy_r2r"], geo["copy_p2r"], geo["copy_r2p"], geo["copy_sgp"], G, L), G, L


def test_model_plans_accepted(pkg, golden, plan):
    from make_golden import load
    ens = importlib.import_module("pynicam-dc_b200.ensemble")
    check = pkg.runtime.check_halo_plan
    check(*plan)
    empty = np.zeros(0, np.int64)
    check((empty,) * 4, 6, 40)
    for m in (2, 5):
        check(ens._stacked_plan(golden[0], m), plan[1], plan[2] * m, 2 * m)
    for f in sorted(glob.glob(os.path.join(HERE, "golden", "*.npz"))):
        geo = dict(load(f)[0])
        if "copy_r2r" in geo:
            G, L = int(geo["gall_1d"]), int(geo["lall"])
            check(pkg.halo.compose(geo["copy_r2r"], geo["copy_p2r"], geo["copy_r2p"], geo["copy_sgp"], G, L), G, L)
    z = np.load(os.path.join(os.path.dirname(pkg.__file__), "data", "halo_rl01.npz"))
    for gl in range(3, 9):
        G = 2 ** (gl - 1) + 2
        check(pkg.halo.compose(*(z[f"gl{gl:02d}_{n}"].astype(np.int64) for n in ("r2r", "p2r", "r2p", "sgp")), G, 40), G, 40)


def _bad_plans(plan):
    (rd, rs, pd, ps), G, L = plan
    n = L * G * G
    put = lambda a, at, v: np.concatenate([a[:at], [v], a[at + 1:]]).astype(np.int64)
    pole = int(np.flatnonzero(rs < 0)[0])
    return {"r_dst negative": (put(rd, 3, -1), rs, pd, ps), "r_dst beyond": (put(rd, 3, n), rs, pd, ps),
            "r_dst far": (put(rd, 3, 2 ** 40), rs, pd, ps), "r_src beyond": (rd, put(rs, 0, n), pd, ps),
            "r_src pole beyond": (rd, put(rs, pole, -13), pd, ps), "r_src far": (rd, put(rs, 1, -2 ** 40), pd, ps),
            "p_dst negative": (rd, rs, put(pd, 2, -1), ps), "p_dst beyond": (rd, rs, put(pd, 2, 12), ps),
            "p_src negative": (rd, rs, pd, put(ps, 0, -1)), "p_src beyond": (rd, rs, pd, put(ps, 0, n)),
            "regional chain": (rd, put(rs, 5, int(rd[9])), pd, ps), "pole chain": (rd, rs, pd, put(ps, 4, int(rd[0]))),
            "pole source written": (rd, put(rs, pole, -1 - int(pd[0])), pd, ps), "itself": (rd, put(rs, 7, int(rd[7])), pd, ps)}


def test_refused_plans(pkg, plan):
    for what, p in _bad_plans(plan).items():
        with pytest.raises(pkg.NicamError, match="halo plan") as ei:
            pkg.runtime.check_halo_plan(p, *plan[1:])
        assert ei.value.status == pkg.runtime.NC_ERR_ARG, what
    with pytest.raises(pkg.NicamError):       # the plan of a larger grid
        pkg.runtime.check_halo_plan(plan[0], plan[1] - 1, plan[2])
    with pytest.raises(pkg.NicamError):       # of two members, for one
        ens = importlib.import_module("pynicam-dc_b200.ensemble")
        from make_golden import load
        geo, _ = load(os.path.join(HERE, "golden", "gl03_z10_trc.npz"))
        pkg.runtime.check_halo_plan(ens._stacked_plan(geo, 2), *plan[1:])
    with pytest.raises(pkg.NicamError, match="bad argument"):    # more cells than a handle can index
        pkg.runtime.check_halo_plan(plan[0], 2 ** 30, 2 ** 30)


@pytest.mark.gpu
def test_create_refuses(pkg, golden, plan):
    for what, p in _bad_plans(plan).items():
        with pytest.raises(pkg.NicamError, match="halo plan"):
            pkg.NicamCuda(dict(golden[0], halo_plan=p), graph=False).close()


@pytest.mark.gpu
@pytest.mark.parametrize("op, ni, no", [("laplacian", 1, 1), ("divergence", 3, 1), ("gradient", 1, 3)])
def test_operators_on_a_plan_that_writes_interior_cells(pkg, golden, plan, op, ni, no):
    import torch
    (rd, rs, pd, ps), G, L = plan
    src = set(rs.tolist()) | set(ps.tolist())
    cells = [(7 * G + j) * G + i for j in range(1, G - 1) for i in range(1, G - 1)]
    free = [c for c in cells if c not in src]
    give = [c for c in ((11 * G + 2) * G + 2, (3 * G + 1) * G + 3) if c not in rd]
    extra = list(zip(free[:2], give))
    assert len(extra) == 2
    p = (np.concatenate([rd, [d for d, _ in extra]]), np.concatenate([rs, [s for _, s in extra]]), pd, ps)
    plain, more = pkg.NicamCuda(golden[0], graph=False), pkg.NicamCuda(dict(golden[0], halo_plan=p), graph=False)
    try:
        gen = torch.Generator(device="cuda").manual_seed(8)
        rand = lambda n, f: torch.randn((() if n == 1 else (n,)) + tuple(f), generator=gen, dtype=torch.float64, device="cuda")
        F, P = plain.field_shape, plain.field_shape_pl
        x, x_pl, y, y_pl = rand(ni, F), rand(ni, P), rand(no, F), rand(no, P)
        g, g_pl = rand(no, F), rand(no, P)
        getattr(more, op)(x, x_pl, y, y_pl)
        # the exchange in place, then the operator of the ordinary plan
        e, e_pl, w, w_pl = x.clone(), x_pl.clone(), torch.empty_like(y), torch.empty_like(y_pl)
        more.exchange(e, e_pl)
        assert not torch.equal(e, x)
        getattr(plain, op)(e, e_pl, w, w_pl)
        assert torch.equal(y, w) and torch.equal(y_pl, w_pl)
        gx, gx_pl = torch.empty_like(x), torch.empty_like(x_pl)
        a = (gx, gx_pl, g, g_pl) if op != "laplacian" else (g, g_pl, gx, gx_pl)
        getattr(more, op)(*a, transpose=True)
        lhs = float((y * g).sum() + (y_pl * g_pl).sum())
        rhs = float((x * gx).sum() + (x_pl * gx_pl).sum())
        size = float((y * g).abs().sum() + (y_pl * g_pl).abs().sum())
        assert abs(lhs - rhs) <= 1e-13 * size     # sums of 2e4 products in another order
    finally:
        plain.close()
        more.close()
