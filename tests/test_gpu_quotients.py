"""Quotients outside the range in which the kernels' reciprocal form is exact:
infinite and NaN operands, zero and subnormal divisors, subnormal quotients
(B200).  The bits are those of the IEEE division, as in numpy.

* The shared-divisor division of the tracer kernels on pairs of special values.
* One offline tracer step of tracers with subnormal masses equals the oracle
  bit for bit (the step's winds move them; every quotient by the density is
  subnormal).
* The pole velocities of subnormal momenta.
"""
import random

import numpy as np
import pytest

from test_divide_known import _div_by, _recip_runtime

pytestmark = pytest.mark.gpu


def _same(a, b):
    return (a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b))


def test_shared_divisor_any_operands(pkg):
    rng = np.random.default_rng(2)
    edge = [0.0, np.inf, np.nan, 5e-324, 1e-310, np.finfo(float).tiny, np.finfo(float).max]
    edge += [2.0 ** e * f for e in (100, 101, 699, 700, 701, 1000) for s in (1, -1) for e in (s * e,)
             for f in (1.0, 1.5, 1.0 + 2.0 ** -52)]
    edge = np.array(edge + [1.0, 3.0, 0.7])
    edge = np.concatenate([edge, -edge])
    x, y = (a.ravel() for a in np.meshgrid(edge, edge))
    n = 400_000
    sub = rng.uniform(1.0, 2.0, n) * 10.0 ** rng.uniform(-323.0, -300.0, n)
    den = rng.uniform(1.0, 2.0, n) * np.exp2(rng.integers(-12, 3, n))
    xs, ys = np.concatenate([x, sub]), np.concatenate([y, den])
    with np.errstate(all="ignore"):
        want = xs / ys
    got = pkg.runtime.divide_known(xs, ys)
    bad = np.flatnonzero(~_same(got, want))
    assert bad.size == 0, (xs[bad[:5]], ys[bad[:5]], got[bad[:5]], want[bad[:5]])


def test_subnormal_tracers_equal_oracle(pkg, golden_trcadv):
    from oracle import nicam_step as O
    geo, st = golden_trcadv
    rng = np.random.default_rng(4)
    s, sp = st["state0"].copy(), st["state0_pl"].copy()
    for a in (s, sp):
        for q in range(6, a.shape[-1]):
            a[..., q] = rng.uniform(0.2, 1.0, a.shape[:-1]) * a[..., 0] * 10.0 ** rng.uniform(-323.0, -306.0, a.shape[:-1])
    want, want_pl = s.copy(), sp.copy()
    g = O.Geo(geo)
    O.tracer_advection(g, want[..., 6:], want_pl[..., 6:], s[..., 0].copy(), sp[..., 0].copy(), s[..., :5].copy(),
                       sp[..., :5].copy(), np.zeros(s.shape[:-1]), np.zeros(sp.shape[:-1]), g.dtl)
    O.comm(g, want, want_pl)
    c = pkg.NicamCuda(geo, graph=False)
    try:
        c.upload(s, sp)
        c.step(1)
        got, got_pl = c.download()
    finally:
        c.close()
    assert np.array_equal(got[..., 6:], want[..., 6:]) and np.array_equal(got_pl[..., 6:], want_pl[..., 6:])


def test_subnormal_pole_velocity(pkg, golden):
    geo, st = golden
    kmin, kmax = int(geo["kmin"]), int(geo["kmax"])
    s, sp = st["state0"].copy(), st["state0_pl"].copy()
    rnd = random.Random(6)
    for k in range(kmin, kmax + 1):
        for lp in range(2):
            b = float(sp[0, k, lp, 0])
            h, lo = _recip_runtime(b)
            while True:      # a momentum whose quotient the reciprocal form rounds twice
                x = rnd.uniform(0.2, 1.0) * 10.0 ** rnd.uniform(-310.0, -307.7)
                if _div_by(x, b, h, lo) != x / b:
                    break
            sp[0, k, lp, 1] = x
    c = pkg.NicamCuda(geo, graph=False)
    try:
        c.upload(s, sp)
        c.run_phases(1)
        vx = c.field("vx")[1]
    finally:
        c.close()
    rows = slice(kmin, kmax + 1)
    assert np.array_equal(vx[0, rows], sp[0, rows, :, 1] / sp[0, rows, :, 0])
