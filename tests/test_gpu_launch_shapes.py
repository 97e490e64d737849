"""The step on both sides of each size rule of its launches, and at the
remainders of its splits (B200).

* Numbers of layers that do not divide by the warps of the vi_main column
  kernel, the levels per block of path 1 and the level chunks: one step at
  gl03 equals the oracle bit for bit.
* One gl05 grid alone (its tiles and columns do not fill the SMs: level chunks)
  against 17 of them stacked in one handle (whole marches): each member bit for
  bit, in both forms.
* Tracers in batches: every tracer of 6 (batches of 4 and 2, a thread of the
  vertical sweep for each) and of 7 (batches of 4 and 3, two tracers a thread,
  the last alone) equals the same tracer carried alone, bit for bit.
* The linear operators on an input that overlaps the output.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ig():
    return importlib.import_module("pynicam-dc_b200.icogrid")


def _perturbed(geo, s, sp, seed):
    ens = importlib.import_module("pynicam-dc_b200.ensemble")
    return ens.perturbed_members(geo, s, sp, 1, seed=seed, sigma=0.5, length=1500e3)[0]


@pytest.mark.parametrize("vlayer", [5, 7, 23, 41])
def test_odd_layers_equal_oracle(pkg, vlayer):
    from oracle import nicam_step as O
    g = _ig().Grid(3, vlayer=vlayer, ztop=30000.0, device="cuda")
    geo = g.setup(dtl=600.0, gamma=7.68e17, nq=1)
    s, sp = _perturbed(geo, *g.jw_state(nq=1), seed=3)
    s[..., 6], sp[..., 6] = 0.01 * s[..., 0], 0.01 * sp[..., 0]
    want, want_pl = O.dynamics_step(O.Geo(geo), s, sp)
    c = pkg.NicamCuda(geo, graph=True)
    try:
        c.upload(s, sp)
        c.step(1)
        got, got_pl = c.download()
    finally:
        c.close()
    assert np.array_equal(got, want) and np.array_equal(got_pl, want_pl)


@pytest.mark.parametrize("prec", ["float64", "mixed"])
def test_one_grid_equals_its_stack(pkg, prec):
    ens = importlib.import_module("pynicam-dc_b200.ensemble")
    g = _ig().Grid(5, vlayer=9, ztop=30000.0, device="cuda")
    geo = g.setup(dtl=300.0, gamma=1.2e16, nq=1)
    m, mp = _perturbed(geo, *g.jw_state(nq=1), seed=5)
    m[..., 6], mp[..., 6] = 0.01 * m[..., 0], 0.01 * mp[..., 0]

    def run(geo, s, sp):
        c = pkg.NicamCuda(geo, graph=True, precision=prec)
        try:
            c.upload(s, sp)
            c.step(2)
            return c.download()
        finally:
            c.close()
    lone, lone_pl = run(geo, m, mp)
    n = 17
    got = ens.unstack_states(*run(ens.stack_setup(geo, n), *ens.stack_states([(m, mp)] * n)), n)
    for x, xp in (got[0], got[n // 2], got[-1]):
        assert np.array_equal(x, lone) and np.array_equal(xp, lone_pl)


@pytest.mark.parametrize("glevel, lone", [(4, 5), (5, 6)])
@pytest.mark.parametrize("prec", ["float64", "mixed"])
def test_tracer_batches_equal_lone_tracers(pkg, prec, glevel, lone):
    g = _ig().Grid(glevel, vlayer=11, ztop=12000.0, device="cuda", layer="EVEN", topo="NONE")
    rng = np.random.default_rng(8)
    amp, lon0 = rng.uniform(0.2, 1.0, 6), rng.uniform(0.0, 6.0, 6)

    def fields(which):
        def f(lon, lat, z):
            lo, la = lon[..., None], lat[..., None]
            q = [np.zeros(z.shape)]
            for n in which:
                r = np.arccos(np.clip(np.cos(la) * np.cos(lo - lon0[n]), -1.0, 1.0))
                q.append(np.where(r < 0.6, amp[n], 0.1) * (1.0 + 0.1 * np.sin(z / 3000.0)))
            return np.stack(q, axis=-1)
        return f

    def run(which):
        geo = g.setup(dtl=600.0, gamma={4: 9.6e16, 5: 1.2e16}[glevel], nq=1 + len(which), trcadv=True)
        s, sp = g.trcadv_state(fields(which))
        c = pkg.NicamCuda(geo, graph=True, precision=prec)
        try:
            c.upload(s, sp)
            c.step(2)
            return c.download()
        finally:
            c.close()
    s, sp = run(range(lone))       # with the vapour slot one more
    for n in range(lone):
        a, ap = run([n])
        assert np.array_equal(s[..., 7 + n], a[..., 7]) and np.array_equal(sp[..., 7 + n], ap[..., 7]), n


def test_linear_operators_in_place(pkg):
    import torch
    g = _ig().Grid(4, vlayer=5, ztop=30000.0, device="cuda")
    geo = g.setup(dtl=600.0, gamma=9.6e16, nq=1)
    c = pkg.NicamCuda(geo, graph=False)
    try:
        gen = torch.Generator(device="cuda").manual_seed(4)
        F, P = c.field_shape, c.field_shape_pl
        rand = lambda n, f: torch.randn((n,) + tuple(f), generator=gen, dtype=torch.float64, device="cuda")
        for op, ni, no in ((c.gradient, 1, 3), (c.divergence, 3, 1)):
            for transpose in (False, True):
                x, x_pl, y, y_pl = rand(ni, F), rand(ni, P), rand(no, F), rand(no, P)
                one = lambda t: t[0] if t.shape[0] == 1 else t
                want = [t.clone() for t in (x, x_pl, y, y_pl)]
                op(*[one(t) for t in want], transpose=transpose)
                out = want[:2] if transpose else want[2:]
                # the single component shares its memory with the first of the three
                big, big_pl = (y, y_pl) if no == 3 else (x, x_pl)
                small, small_pl = (x, x_pl) if no == 3 else (y, y_pl)
                three_in = (no == 3) == transpose
                if not three_in:
                    big[0].copy_(small[0])
                    big_pl[0].copy_(small_pl[0])
                args = ((big[0], big_pl[0], big, big_pl) if no == 3 else (big, big_pl, big[0], big_pl[0]))
                op(*args, transpose=transpose)
                got = (big[:1], big_pl[:1]) if three_in else (big, big_pl)
                for a, b in zip(got, out):
                    assert float((a - b).abs().max()) <= 1e-15 * float(b.abs().max()) + 0.0, (op.__name__, transpose)
    finally:
        c.close()


@pytest.mark.parametrize("prec", ["float64", "mixed"])
def test_largest_blocks(pkg, prec):
    """a step with every tunable kernel at the largest block nc_set_block accepts equals the default's"""
    g = _ig().Grid(4, vlayer=9, ztop=30000.0, device="cuda")
    geo = g.setup(dtl=600.0, gamma=9.6e16, nq=3)
    s, sp = g.jw_state(nq=3)
    for q in range(3):
        s[..., 6 + q], sp[..., 6 + q] = 0.01 * s[..., 0] / (q + 1), 0.01 * sp[..., 0] / (q + 1)
    names = ("diag", "vi_solve", "vi_energy", "vp0_c", "gtend", "hdiff1", "post", "split_init", "trc_vflux", "trc_vadv",
             "trc_remap", "trc_qout", "trc_apply", "trc_rhog")

    def run(top):
        c = pkg.NicamCuda(geo, graph=not top, precision=prec)
        try:
            for n in names if top else ():
                with pytest.raises(pkg.NicamError):
                    c.set_block(n, 1056)
                for t in (1024, 256, 128):
                    try:
                        c.set_block(n, t)
                        break
                    except pkg.NicamError:
                        continue
                assert c.get_block(n) == t
            c.upload(s, sp)
            c.step(1)
            return c.download()
        finally:
            c.close()
    (a, ap), (b, bp) = run(False), run(True)
    assert np.array_equal(a, b) and np.array_equal(ap, bp)


def _column_case(pkg, vlayer, geo_edit=None):
    """a gl03 handle and random column fields: tracer mass, density, vertical flux, two directions"""
    import torch
    g = _ig().Grid(3, vlayer=vlayer, ztop=30000.0, device="cuda")
    geo = g.setup(dtl=600.0, gamma=7.68e17, nq=1)
    if geo_edit:
        geo_edit(geo)
    c = pkg.NicamCuda(geo, graph=False)
    gen = torch.Generator(device="cuda").manual_seed(vlayer)
    f = lambda lo, hi: lo + (hi - lo) * torch.rand(tuple(c.field_shape), generator=gen, dtype=torch.float64, device="cuda")
    den = f(0.5, 1.0)
    flx = f(-40.0, 40.0) * (30000.0 / vlayer / 500.0)      # Courant numbers below 0.2
    flx[:, :c.kmin + 1] = 0.0
    flx[:, c.kmax + 1:] = 0.0
    return c, den * f(0.5, 1.0), den, flx, torch.zeros_like(den), f(-1.0, 1.0), f(-1.0, 1.0)


@pytest.mark.parametrize("vlayer", [2, 3, 29, 62])
def test_column_operators_smallest_and_tallest(pkg, vlayer):
    """the linearised vertical step and the tridiagonal solve from the fewest layers to the most:
    the adjoint against the tangent-linear and the transpose against the solve (dot products)"""
    import torch
    c, rq, den, flx, fr, x, y = _column_case(pkg, vlayer)
    try:
        tl, ad = torch.empty_like(x), torch.empty_like(x)
        c.vadv_lin(1, rq, den, flx, fr, x, tl, 300.0, 0.0, True)
        c.vadv_lin(2, rq, den, flx, fr, y, ad, 300.0, 0.0, True)
        size = float((tl * y).abs().sum())
        assert size > 0 and abs(float((tl * y).sum() - (x * ad).sum())) <= 1e-13 * size
        Mc, Mu, Ml = 3.0 + 0.3 * x, -1.0 + 0.1 * y, -1.0 + 0.1 * rq
        c.vsolve(Mc, Mu, Ml, x, tl)
        c.vsolve(Mc, Mu, Ml, y, ad, transpose=True)
        k = slice(c.kmin + 1, c.kmax + 1)              # the rows of the solve
        size = float((tl * y)[:, k].abs().sum())
        assert size > 0 and abs(float((tl * y)[:, k].sum() - (x * ad)[:, k].sum())) <= 1e-13 * size
    finally:
        c.close()


def test_vertical_adjoint_reads_the_faces_factors_only(pkg):
    """the half-level factors below the lowest layer have no face: nothing of them enters the adjoint"""
    import torch

    def spoil(geo):
        for n in ("GRD_afact", "GRD_bfact"):
            geo[n] = np.array(geo[n], np.float64)
            geo[n][0] = np.nan
    out = []
    for edit in (None, spoil):
        c, rq, den, flx, fr, _, y = _column_case(pkg, 9, edit)
        try:
            o = torch.empty_like(y)
            c.vadv_lin(2, rq, den, flx, fr, y, o, 300.0, 0.0, True)
            out.append(o.clone())
        finally:
            c.close()
    assert bool(torch.isfinite(out[0]).all()) and torch.equal(out[0], out[1])


@pytest.mark.parametrize("vlayer", [62, 63, 100, 126])
def test_tall_columns_equal_oracle(pkg, vlayer):
    test_odd_layers_equal_oracle(pkg, vlayer)


@pytest.mark.parametrize("vlayer", [41, 42, 61, 126])
def test_tall_mixed_step_near_float64(pkg, vlayer):
    """the mixed step of tall columns against the float64 step (measured at 61 and 126 layers:
    RHOG and RHOGE 5e-8, RHOGVX and RHOGVY 1.6e-7, RHOGVZ 1.2e-4, RHOGW 5e-6; pole momentum 9e-6)"""
    g = _ig().Grid(4, vlayer=vlayer, ztop=30000.0, device="cuda")
    geo = g.setup(dtl=300.0, gamma=9.6e16, nq=1)
    s, sp = _perturbed(geo, *g.jw_state(nq=1), seed=7)
    out = []
    for prec in ("float64", "mixed"):
        c = pkg.NicamCuda(geo, graph=True, precision=prec)
        try:
            c.upload(s, sp)
            c.step(1)
            out.append(c.download())
        finally:
            c.close()
    (a, ap), (b, bp) = out
    for v, tol in enumerate((1e-6, 1e-5, 1e-5, 1e-3, 1e-4, 1e-6)):
        assert np.linalg.norm(b[..., v] - a[..., v]) <= tol * np.linalg.norm(a[..., v]), v
    # the pole points: horizontal momentum as one vector, then density, vertical momentum, energy
    assert np.linalg.norm((bp - ap)[..., 1:4]) <= 1e-4 * np.linalg.norm(ap[..., 1:4])
    for v, tol in ((0, 1e-6), (4, 1e-4), (5, 1e-6)):
        assert np.linalg.norm(bp[..., v] - ap[..., v]) <= tol * np.linalg.norm(ap[..., v]), v
