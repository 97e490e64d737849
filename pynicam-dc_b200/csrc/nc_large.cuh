// Large-step kernels of one RK stage: diagnostics + boundary conditions,
// momentum advection, hyperdiffusion and the large-step tendency.
#pragma once
#include "nc_ops.cuh"

namespace nc {

// Field bundles (device pointers, one array per variable)
template <class R>
struct Prog { R* v[6]; };   // RHOG, RHOGVX, RHOGVY, RHOGVZ, RHOGW, RHOGE

// ---------------------------------------------------------------------------
// Pre_Post: diagnostics (kernels/diag.py:53-143), BNDCND_all
// (share/mod_bndcnd.py:182-264 with kernels/bndcnd.py), th/eth and the
// deviations (mod_dynamics.py:1043-1057), then the merged velocity of the
// momentum advection (kernels/advconvmom.py:54-78), regional and pole points
// alike.
// ---------------------------------------------------------------------------
template <class R>
struct DiagArgs {
  Prog<R> P;            // in/out (ghost rows written)
  const R* Pqw[NC_MAXQW];   // the water tracers (0: vapour)
  R *pre, *tem, *vx, *vy, *vz, *w, *rho, *ein, *eth;
  double *pregd, *rhogd;   // float64 in both forms
  R *vvx, *vvy, *vvz;
};

template <class R, bool POLE>
__device__ void diag_point(const Col c, const MetT<R> m, const DiagArgs<R>& a, int k, double gx, double gy, double gz) {
  const int kmin = cD.kmin, kmax = cD.kmax;
  if (k == kmin - 1 || k == kmax + 1) return;   // written with the row next to them
  R* const* P = a.P.v;
  struct D {
    double rhog, rho, vx, vy, vz, ein, tem, pre;
  };
  auto diag = [&](int kk) -> D {
    const int p = c.at(kk);
    D d;
    d.rhog = P[0][p];
    d.rho = d.rhog / m.GSGAM2[p];
    // the quotients by RHOG: through one reciprocal for the regional points, by
    // dividing for the few pole points (the same but for subnormal quotients)
    const auto rr = recip_of(d.rhog);
    auto by = [&](double x) -> double { return POLE ? x / d.rhog : div_by(x, rr); };
    d.vx = by(P[1][p]);
    d.vy = by(P[2][p]);
    d.vz = by(P[3][p]);
    d.ein = by(P[5][p]);
    const double q0 = by(a.Pqw[0][p]);
    double qd, cv;
    moist_qd_cv([&](int n) { return by(a.Pqw[n][p]); }, q0, qd, cv);
    d.tem = d.ein / cv;
    d.pre = d.rho * d.tem * (qd * cC.Rdry + q0 * cC.Rvap);
    return d;
  };
  auto put = [&](int p, double tem, double pre, double rho, double ein) {
    a.tem[p] = tem;
    a.pre[p] = pre;
    a.rho[p] = rho;
    a.ein[p] = ein;
  };
  auto w_at = [&](int kk) -> double {   // kmin+1..kmax
    const int p = c.at(kk);
    return P[4][p] / (mc(m.C2W, c, 0, 2, kk) * (double)P[0][p] + mc(m.C2W, c, 1, 2, kk) * (double)P[0][c.at(kk - 1)]);
  };
  auto finish = [&](int kk, int p, double pre, double rho, double ein, double vx, double vy, double vz, double wk,
                    double wk1) {
    a.eth[p] = ein + pre / rho;
    a.pregd[p] = (pre - m.pre_bs[p]) * m.GSGAM2[p];
    a.rhogd[p] = (rho - m.rho_bs[p]) * m.GSGAM2[p];
    if (kk >= kmin && kk <= kmax) {
      const double wc = cC.cfact[kk] * wk1 + cC.dfact[kk] * wk;
      a.vvx[p] = vx + div_r(wc * gx);
      a.vvy[p] = vy + div_r(wc * gy);
      a.vvz[p] = vz + div_r(wc * gz);
    } else {
      a.vvx[p] = 0.0; a.vvy[p] = 0.0; a.vvz[p] = 0.0;
    }
  };
  const int p = c.at(k);
  const D d = diag(k);
  if (k < kmin || k > kmax) {   // beyond the boundary rows
    a.vx[p] = d.vx; a.vy[p] = d.vy; a.vz[p] = d.vz;
    put(p, d.tem, d.pre, d.rho, d.ein);
    return;
  }
  if (k > kmin && k < kmax) {
    const double wk = w_at(k), wk1 = w_at(k + 1);
    // the pole points form the second pass from the stored (rounded) values
    auto Q = [](double x) -> double { return POLE ? (double)R(x) : x; };
    finish(k, p, Q(d.pre), Q(d.rho), Q(d.ein), Q(d.vx), Q(d.vy), Q(d.vz), Q(wk), Q(wk1));
    a.vx[p] = d.vx; a.vy[p] = d.vy; a.vz[p] = d.vz;
    put(p, d.tem, d.pre, d.rho, d.ein);
    a.w[p] = wk;
    return;
  }
  // ---- the rows at a boundary, from the stored (rounded) values: TEM top and
  // bottom, FREE top, RIGID bottom
  const bool top = k == kmax;
  const int kb = top ? kmax + 1 : kmin - 1, ki = top ? kmax - 1 : kmin + 1;
  const int pb = c.at(kb), pi = c.at(ki);
  const R tem = d.tem, rho = d.rho, pre = d.pre, ein = d.ein, vx = d.vx, vy = d.vy, vz = d.vz;
  const R pre_i = diag(ki).pre;
  const double tem_b = tem;
  const double pre_b = pre_i - rho * (m.PHI[pb] - m.PHI[pi]);
  const double rho_b = pre_b / (cC.Rdry * tem_b);
  const double rg = P[0][p], rgb = rho_b * m.GSGAM2[pb], ein_b = cC.CVdry * tem_b;
  const R Pp[3] = {P[1][p], P[2][p], P[3][p]};
  double vb[3];
#pragma unroll
  for (int n = 0; n < 3; ++n) vb[n] = (top ? 1.0 : -1.0) * (Pp[n] / rg) * rgb;
  const R rgbR = rgb;
  R wR, wbR;      // w at the half levels k and k+1 of the row inside (top), at kmin and kmin+1 (bottom)
  if (top) {
    const double rwT = -(mc(m.C2WGz, c, 0, 6, kb) * vb[0] + mc(m.C2WGz, c, 1, 6, kb) * Pp[0] +
                         mc(m.C2WGz, c, 2, 6, kb) * vb[1] + mc(m.C2WGz, c, 3, 6, kb) * Pp[1] +
                         mc(m.C2WGz, c, 4, 6, kb) * vb[2] + mc(m.C2WGz, c, 5, 6, kb) * Pp[2]);
    wR = w_at(k);
    wbR = rwT / (mc(m.C2W, c, 0, 2, kb) * rgb + mc(m.C2W, c, 1, 2, kb) * rg);
    a.w[p] = wR;
    a.w[pb] = wbR;
    P[4][pb] = rwT;
  } else {
    wbR = w_at(kmin + 1);
    wR = R(0.0) / (mc(m.C2W, c, 0, 2, kmin) * rg + mc(m.C2W, c, 1, 2, kmin) * rgb);
    a.w[p] = wR;
    a.w[pb] = 0.0;
    P[4][p] = 0.0;
    P[4][pb] = 0.0;
  }
  finish(k, p, pre, rho, ein, vx, vy, vz, wR, wbR);
  a.vx[p] = vx; a.vy[p] = vy; a.vz[p] = vz;
  put(p, tem, pre, rho, ein);
  // the boundary row
  finish(kb, pb, R(pre_b), R(rho_b), R(ein_b), 0.0, 0.0, 0.0, 0.0, 0.0);
  put(pb, tem_b, pre_b, rho_b, ein_b);
  P[0][pb] = rgb;
  P[5][pb] = rgb * ein_b;
  R* dv[3] = {a.vx, a.vy, a.vz};
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    P[1 + n][pb] = vb[n];
    dv[n][pb] = R(vb[n]) / rgbR;
  }
}

// A thread per point (a column per thread was bound by the chain of a level's
// loads, stores and divisions: 4 us a level at any grid level); w at the
// half levels k and k+1 is formed by both neighbours.  Eight and nine blocks of 128
// an SM although they spill (72 and 80 bytes stored a thread): a step at gl07 z40
// float64 0.96 ms, six blocks without spills 1.10, five 1.25; mixed nine 0.75,
// eight 0.81, six 1.00.
template <class R>
__global__ void __launch_bounds__(128, NC_MINB(R, 8, NC_F32_DIAG)) k_diag(const __grid_constant__ DiagArgs<R> a, const __grid_constant__ DiagArgs<R> ap, int npb) {
  Pt q;
  if ((int)blockIdx.x < npb) {
    if (!pole_point((int)(blockIdx.x * blockDim.x + threadIdx.x), q)) return;
    const R* X = CG.GRD_x_pl + (q.g * cD.LP + q.lp) * 3;
    diag_point<R, true>(col_pl(q.g, q.lp), met_of<R>(true), ap, q.k, (double)X[0], (double)X[1], (double)X[2]);
  } else {
    if (!reg_point((int)((blockIdx.x - npb) * blockDim.x + threadIdx.x), q)) return;
    diag_point<R, false>(col_reg(q.i, q.j, q.l), met_of<R>(false), a, q.k, (double)P2(CG.GRD_x, 0, q.i, q.j, q.l),
               (double)P2(CG.GRD_x, 1, q.i, q.j, q.l), (double)P2(CG.GRD_x, 2, q.i, q.j, q.l));
  }
}

// ---------------------------------------------------------------------------
// Momentum advection convergence + Coriolis + horizontalize
// (mod_src.py:96-497, kernels/advconv.py:42-108, fluxconv.py:111-208,
// advconvmom.py:111-194).  Outputs grhogv{x,y,z}, grhogw.
// ---------------------------------------------------------------------------
template <class R>
struct AdvMomArgs {
  const R *rg, *rvx, *rvy, *rvz, *rw;    // PROG (post BNDCND)
  const R *vvx, *vvy, *vvz;              // merged velocity
  R *gvx, *gvy, *gvz, *gw;               // out
};

// Tiled momentum advection for interior cells: one block per tile of a
// region, marching upward over kmin..kmax (the vertical-momentum tendency at k
// needs the projection at k-1, and the half-level flux at k is reused from the
// level below).  Per level the products of rhogv, the merged velocity and
// RGAM on the haloed tile are staged in shared memory for the 7-point divergences.  Halo
// cells and boundary levels are not written (their values are never read:
// the large-step tendencies derived from them are replaced by the exchanges).
// Arithmetic and association order are those of the reference's expressions
// (kernels/advconv.py, kernels/advconvmom.py), as in the pole kernel.
// The levels are split into gridDim.y chunks of nk where the tiles alone leave
// SMs idle (see tile_chunks); a chunk walks two levels below its first
// without storing them, for the projection and the flux that its first needs.
// (SPLIT; the unsplit instance keeps the registers of the chunk's bounds)
// Bound by shared-memory reads and, on small grids, by the latency of a level's
// staging.  So the nine products rhogv_d * vv_s * RGAM of a point are formed once
// where it is staged (each was formed for seven cells, from three reads), each
// coefficient is read once for the three velocities, and the next level's loads
// are in flight while this level is worked on (two levels in shared memory, one
// barrier a level).  At z40, before and now: gl05 float64 92 -> 59 us, gl06 mixed
// 153 -> 91 us, gl07 float64 611 -> 561 us, gl08 mixed 989 -> 820 us.
template <class R, class T, bool SPLIT>
__global__ void __launch_bounds__(TILE_THREADS, NC_MINB(R, 2, NC_F32_ADVMOM)) k_advmom_t(AdvMomArgs<R> a, int nk) {
  constexpr int TXD = T::X, TYD = T::Y;
  constexpr int PX = TXD + 2, PY = TYD + 2, NP = PX * PY, PT = (NP + TILE_THREADS - 1) / TILE_THREADS;
  __shared__ R s_p[2][9][NP];   // (rhogv_d * vv_s) * RGAM at [d * 3 + s], two levels
  const int ntx = (cD.G - 2 + TXD - 1) / TXD;
  const int l = (int)blockIdx.z;
  const int i0 = 1 + ((int)blockIdx.x % ntx) * TXD, j0 = 1 + ((int)blockIdx.x / ntx) * TYD;
  const int G = cD.G, gmax = cD.G - 2, kmin = cD.kmin, kmax = cD.kmax;
  const int tid = threadIdx.x, tx = tid % TXD, ty = tid / TXD;
  const int i = i0 + tx, j = j0 + ty;
  const bool own = (i <= gmax) && (j <= gmax);
  const R* rv[3] = {a.rvx, a.rvy, a.rvz};
  const R* vv[3] = {a.vvx, a.vvy, a.vvz};
  const R* cz = CG.C2WGz;
  const int n = cD.npti;
  R f[PT][7];   // a level's staged points of the thread on their way to shared memory
  auto fetch = [&](int k) {
#pragma unroll
    for (int e = 0; e < PT; ++e) {
      const int p = tid + e * TILE_THREADS;
      const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
      const bool ok = p < NP && ii < G && jj < G;
      const int q = ok ? ix(ii, jj, k, l) : 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        f[e][d] = ok ? __ldg(rv[d] + q) : R(0.0);
        f[e][3 + d] = ok ? __ldg(vv[d] + q) : R(0.0);
      }
      f[e][6] = ok ? gam_at(CG.RGAM, q) : R(0.0);
    }
  };
  auto put = [&](int b) {
#pragma unroll
    for (int e = 0; e < PT; ++e) {
      const int p = tid + e * TILE_THREADS;
      if (p < NP) {
#pragma unroll
        for (int m = 0; m < 9; ++m) s_p[b][m][p] = (f[e][m / 3] * f[e][3 + m % 3]) * f[e][6];
      }
    }
  };
  const int ka = SPLIT ? kmin + (int)blockIdx.y * nk : kmin, kb = SPLIT ? min(ka + nk - 1, kmax) : kmax;
  const int k0 = SPLIT ? max(ka - 2, kmin) : kmin;
  R gx = R(0.0), gy = R(0.0), gz = R(0.0);
  int q0 = 0;
  R r0[3] = {R(0.0), R(0.0), R(0.0)}, v0[3] = {R(0.0), R(0.0), R(0.0)};   // the own column's rhogv and vv at level k
  if (own) {
    gx = div_r(P2(CG.GRD_x, 0, i, j, l));
    gy = div_r(P2(CG.GRD_x, 1, i, j, l));
    gz = div_r(P2(CG.GRD_x, 2, i, j, l));
    q0 = ix(i, j, 0, l);
#pragma unroll
    for (int d = 0; d < 3; ++d) { r0[d] = __ldg(rv[d] + q0 + k0 * cD.planei); v0[d] = __ldg(vv[d] + q0 + k0 * cD.planei); }
  }
  R vmh_lo[3] = {R(0.0), R(0.0), R(0.0)};
  R gwc_prev = R(0.0);
  int b = 0;
  fetch(k0);
  put(0);
  __syncthreads();
  for (int k = k0; k <= kb; ++k, b ^= 1) {
    if (k < kb) fetch(k + 1);
    if (own) {
      const int c0 = (ty + 1) * PX + (tx + 1);
      const int nb[7] = {c0, c0 + 1, c0 + PX + 1, c0 + PX, c0 - 1, c0 - PX - 1, c0 - PX};
      const int p = q0 + k * cD.planei;
      const int kk = k + 1;
      const bool hv = (kk > kmin && kk <= kmax);
      const int qh = p + cD.planei;   // level k+1 of the own column
      R div[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        R sm[3];
#pragma unroll
        for (int m = 0; m < 7; ++m) {
          const R cf = P2(CG.coef_div, d * 7 + m, i, j, l);
#pragma unroll
          for (int s = 0; s < 3; ++s) {
            const R v = s_p[b][d * 3 + s][nb[m]];
            sm[s] = (m == 0) ? cf * v : mad(cf, v, sm[s]);
          }
        }
#pragma unroll
        for (int s = 0; s < 3; ++s) div[s] = (d == 0) ? sm[s] : div[s] + sm[s];
      }
      R vmh[3] = {R(0.0), R(0.0), R(0.0)}, r1[3] = {R(0.0), R(0.0), R(0.0)}, v1[3] = {R(0.0), R(0.0), R(0.0)};
      if (hv) {
#pragma unroll
        for (int d = 0; d < 3; ++d) { r1[d] = __ldg(rv[d] + qh); v1[d] = __ldg(vv[d] + qh); }
        R z[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) z[m] = cz[m * n + qh];
        const R rw = a.rw[qh], gh = gam_at(CG.RGAMH, qh), rgs = CG.RGSQRTH[qh];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          const R sh = v1[s], sl = v0[s];
          const R h = z[0] * (r1[0] * sh) + z[1] * (r0[0] * sl) + z[2] * (r1[1] * sh) + z[3] * (r0[1] * sl) +
                      z[4] * (r1[2] * sh) + z[5] * (r0[2] * sl);
          const R sw = rw * (CC.afact[kk] * sh + CC.bfact[kk] * sl);
          vmh[s] = h * gh + R(1.0) * sw * rgs;
        }
      }
      R dv[3];
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        dv[s] = -div[s] - (vmh[s] - vmh_lo[s]) * CC.rdgz[k];
        vmh_lo[s] = vmh[s];
      }
      const R rh = a.rg[p];
      const R dvx = dv[0] - (-R(2.0) * rh * (CC.OHM * v0[1]));
      const R dvy = dv[1] - (R(2.0) * rh * (CC.OHM * v0[0]));
      const R dvz = dv[2];
      const R prd = dvx * gx + dvy * gy + dvz * gz;
      const R gwc = prd * CC.alpha;
      if (!SPLIT || k >= ka) {
        a.gvx[p] = dvx - prd * gx;
        a.gvy[p] = dvy - prd * gy;
        a.gvz[p] = dvz - prd * gz;
        a.gw[p] = (k >= kmin + 1) ? (CG.C2W[p] * gwc + CG.C2W[n + p] * gwc_prev) : R(0.0);
      }
      gwc_prev = gwc;
#pragma unroll
      for (int d = 0; d < 3; ++d) { r0[d] = r1[d]; v0[d] = v1[d]; }
    }
    if (k < kb) put(b ^ 1);
    __syncthreads();
  }
}

// pole part of the momentum advection (one thread per pole column (g, lp))
template <class R>
__device__ R advconv_pl_at(int g, int lp, int k, const Col& c, const MetT<R>& m, const R* rvx,
                                const R* rvy, const R* rvz, const R* rw, const R* scl) {
  R div = R(0.0);
  if (g == 0) {
    const R* cd = CG.coef_div_pl;
    R row = R(0.0);
    for (int v = 0; v < 6; ++v) {
      int q = ipl(v, k, lp);
      R vx = (rvx[q] * scl[q]) * gam_at(CG.RGAM_pl, q);
      R vy = (rvy[q] * scl[q]) * gam_at(CG.RGAM_pl, q);
      R vz = (rvz[q] * scl[q]) * gam_at(CG.RGAM_pl, q);
      R pv = cd[(v * cD.LP + lp) * 3 + 0] * vx + cd[(v * cD.LP + lp) * 3 + 1] * vy +
                  cd[(v * cD.LP + lp) * 3 + 2] * vz;
      row = (v == 0) ? pv : row + pv;
    }
    div = row;
  }
  auto vmh = [&](int kk) -> R {
    if (kk <= cD.kmin || kk > cD.kmax) return R(0.0);
    R h = vmh_horiz(c, m, kk, [&](int k2, int d) -> R {
      int q = c.at(k2);
      const R* rv = (d == 0) ? rvx : ((d == 1) ? rvy : rvz);
      return rv[q] * scl[q];
    });
    int q = c.at(kk);
    R sw = rw[q] * (CC.afact[kk] * scl[q] + CC.bfact[kk] * scl[c.at(kk - 1)]);
    return h + R(1.0) * sw * m.RGSQRTH[q];
  };
  return -div - (vmh(k + 1) - vmh(k)) * CC.rdgz[k];
}

template <class R>
__global__ void k_advmom_pl(const __grid_constant__ AdvMomArgs<R> a) {
  Pt q_;
  if (!pole_point((int)(blockIdx.x * blockDim.x + threadIdx.x), q_)) return;
  const int g = q_.g, lp = q_.lp, k = q_.k;
  const Col c = col_pl(g, lp);
  const int p = c.at(k);
  if (k < cD.kmin || k > cD.kmax) {
    a.gvx[p] = R(0.0); a.gvy[p] = R(0.0); a.gvz[p] = R(0.0); a.gw[p] = R(0.0);
    return;
  }
  const MetT<R> m = met_of<R>(true);
  const R* X = CG.GRD_x_pl + (g * cD.LP + lp) * 3;
  const R gx = div_r(X[0]), gy = div_r(X[1]), gz = div_r(X[2]);
  auto conv = [&](int kk, R dv[3]) -> R {   // the tendency at kk and its vertical component
    const int q = c.at(kk);
    dv[0] = advconv_pl_at(g, lp, kk, c, m, a.rvx, a.rvy, a.rvz, a.rw, a.vvx);
    dv[1] = advconv_pl_at(g, lp, kk, c, m, a.rvx, a.rvy, a.rvz, a.rw, a.vvy);
    dv[2] = advconv_pl_at(g, lp, kk, c, m, a.rvx, a.rvy, a.rvz, a.rw, a.vvz);
    const R rh = a.rg[q];
    dv[0] = dv[0] - (-R(2.0) * rh * (CC.OHM * a.vvy[q]));
    dv[1] = dv[1] - (R(2.0) * rh * (CC.OHM * a.vvx[q]));
    return dv[0] * gx + dv[1] * gy + dv[2] * gz;
  };
  R dv[3], below[3];
  const R prd = conv(k, dv);
  a.gvx[p] = dv[0] - prd * gx;
  a.gvy[p] = dv[1] - prd * gy;
  a.gvz[p] = dv[2] - prd * gz;
  a.gw[p] = (k >= cD.kmin + 1) ? (mc(m.C2W, c, 0, 2, k) * (prd * CC.alpha) +
                                  mc(m.C2W, c, 1, 2, k) * (conv(k - 1, below) * CC.alpha))
                               : R(0.0);
}

// ---------------------------------------------------------------------------
// Hyperdiffusion (mod_numfilter.py:845-1469, lap_order 2, DIRECT).
// Pass 1: vt = -lap(src), src = (vx, vy, vz, w, tem - tem_bs, rho - rho_bs).
// Pass 2: vt2 = -(lap of comps 0..3, kh-weighted diffusion of comps 4, 5).
// ---------------------------------------------------------------------------
template <class R>
struct Six { const R* f[6]; };
template <class R>
struct SixOut { R* f[6]; };

template <class R>
__global__ void k_hdiff1_pl(const __grid_constant__ Six<R> src, const __grid_constant__ SixOut<R> out) {
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= cD.KA * cD.LP) return;
  int k = t / cD.LP, lp = t % cD.LP;
  for (int n = 0; n < 6; ++n) {
    R row = R(0.0);
    for (int v = 0; v < 6; ++v) {
      int q = ipl(v, k, lp);
      R s = src.f[n][q];
      if (n == 4) s = s - CG.tem_bs_pl[q];
      if (n == 5) s = s - CG.rho_bs_pl[q];
      R tv = CG.coef_lap_pl[v * cD.LP + lp] * s;
      row = (v == 0) ? tv : row + tv;
    }
    out.f[n][ipl(0, k, lp)] = -row;
    for (int g = 1; g < 6; ++g) out.f[n][ipl(g, k, lp)] = -R(0.0);
  }
}

// A thread per point: with a column per thread the stores of one field held
// back the loads of the next (5.4 us a level at every grid level).
template <class R>
__global__ void k_hdiff1(Six<R> src, SixOut<R> out) {
  Pt c;
  const int p = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (!reg_point(p, c)) return;
  if (!interior(c.i, c.j)) {
#pragma unroll
    for (int n = 0; n < 6; ++n) out.f[n][p] = -R(0.0);
    return;
  }
  const int G = cD.G;
  const int nb[7] = {p, p + 1, p + 1 + G, p + G, p - 1, p - 1 - G, p - G};
  R cl[7], v[6];
#pragma unroll
  for (int m = 0; m < 7; ++m) cl[m] = P2c(CG.coef_lap, m, c.i, c.j, c.l);
#pragma unroll
  for (int n = 0; n < 6; ++n) {
    const R* s = src.f[n];
    const R* bs = (n == 4) ? CG.tem_bs : CG.rho_bs;
    // lap7 (kernels/oprtlaplacian.py:41-55) with the reference-state
    // deviation for TEM and RHO
    auto scl = [&](int m) { return (n >= 4) ? __ldg(s + nb[m]) - __ldg(bs + nb[m]) : __ldg(s + nb[m]); };
    v[n] = cl[0] * scl(0);
#pragma unroll
    for (int m = 1; m < 7; ++m) v[n] = mad(cl[m], scl(m), v[n]);
  }
#pragma unroll
  for (int n = 0; n < 6; ++n) out.f[n][p] = -v[n];
}

// The three vertex weights of each triangle of the Kh-weighted diffusion,
// formed once from the interpolation coefficients with the reference's
// expressions (kernels/oprtdiffusion.py:59-90): for direction d and triangle
// t (i or j), 2*c1 - c2 - c3, -c1 + 2*c2 - c3 and -c1 - c2 + 2*c3 of
// coef_intp[d][0..2][t].  Planes [((d*3+m)*2+t)][l][j][i].
__global__ void k_intp_weights(const double* ci, double* w, int npt2) {
  const int q = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (q >= npt2) return;
  for (int d = 0; d < 3; ++d)
    for (int t = 0; t < 2; ++t) {
      const double c1 = ci[((d * 3 + 0) * 2 + t) * npt2 + q], c2 = ci[((d * 3 + 1) * 2 + t) * npt2 + q];
      const double c3 = ci[((d * 3 + 2) * 2 + t) * npt2 + q];
      w[((d * 3 + 0) * 2 + t) * npt2 + q] = 2.0 * c1 - c2 - c3;
      w[((d * 3 + 1) * 2 + t) * npt2 + q] = -c1 + 2.0 * c2 - c3;
      w[((d * 3 + 2) * 2 + t) * npt2 + q] = -c1 - c2 + 2.0 * c3;
    }
}


// Kh of the hyperdiffusion at level k: the uniform DIRECT coefficient, or for
// NONLINEAR1 (mod_numfilter.py:1153-1184) the coefficient from the
// temperature-deviation Laplacian lapT of the first pass,
// clip(2 AREA^2 / dtl * (|lapT| / 300 * AREA), Kh_coef_minlim, kh_max(k))
template <class R>
__device__ __forceinline__ R hdiff_kh(R lapT, int k) {
  if (!CC.hdiff_nl) return CC.Kh;
  const R c = CC.nl_c1 * (fabs(lapT) / R(300.0) * CC.nl_area);
  return fmin(fmax(c, CC.nl_min), CC.nl_khmax[k]);
}

// Second hyperdiffusion pass, one block per (HD_NK levels, tile)
// of interior cells: the haloed tile of the six Laplacians and of rhog is
// staged in shared memory per level, the triangle gradients of the
// temperature and density Laplacians are formed once (with the singular-point
// fix at the (0,0) vertex), then each thread writes its cell's four
// Laplacians and two Kh-weighted diffusions (kernels/oprtlaplacian.py:41-55,
// kernels/oprtdiffusion.py).  Halo cells are left to the exchange that
// follows.  The tile's k-independent triangle weights (intp_w, 18 planes) are
// staged in shared memory and the cell's Laplacian and diffusion coefficients
// (coef_lap 7, coef_diff 18) held in registers once for all of the block's
// levels, instead of re-read from L2 at every level.  Dynamic shared memory:
// hdiff2_m_smem<R, T>() bytes (46 KB float, 93 KB double).  rhog * Kh of the two
// diffusions, from hdiff_kh (the first pass's temperature Laplacian is the staged
// field 4), is formed where a point is staged; a cell formed the fourteen values
// that it reads.  gl08 mixed 889 -> 844 us, gl06 mixed 69 -> 65 us, gl07 float64
// 495 -> 490 us (constant Kh, z40; the nonlinear Kh costs a division besides).
#ifndef HD_NK
#define HD_NK 6
#endif
template <class R, class T>
constexpr int hdiff2_m_smem() {
  return ((18 + 12) * (T::X + 1) * (T::Y + 1) + 8 * (T::X + 2) * (T::Y + 2)) * (int)sizeof(R);
}
template <class R>
__global__ void k_hdiff2_pl(const __grid_constant__ Six<R> vt, const R* rhog, const __grid_constant__ SixOut<R> out) {
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= cD.KA * cD.LP) return;
  int k = t / cD.LP, lp = t % cD.LP;
  for (int n = 0; n < 6; ++n) {
    const R* s = vt.f[n];
    R row = R(0.0);
    if (n < 4) {
      for (int v = 0; v < 6; ++v) {
        R tv = CG.coef_lap_pl[v * cD.LP + lp] * s[ipl(v, k, lp)];
        row = (v == 0) ? tv : row + tv;
      }
    } else {
      // kernels/oprtdiffusion.py:137-177
      const R fac = (n == 4) ? CC.CVdry : CC.hdiff_fact_rho;
      R sn = s[ipl(0, k, lp)];
      R vt_[5][3];
      for (int v = 1; v <= 5; ++v) {
        int vp1 = (v == 5) ? 1 : v + 1;
        R sij = s[ipl(v, k, lp)], sp1 = s[ipl(vp1, k, lp)];
        for (int d = 0; d < 3; ++d) {
          const R* cI = CG.coef_intp_pl + ((v * cD.LP + lp) * 3 + d) * 3;
          R c0 = cI[0], c1 = cI[1], c2 = cI[2];
          vt_[v - 1][d] = div3((R(2.0) * c0 - c1 - c2) * sn + (-c0 + R(2.0) * c1 - c2) * sij + (-c0 - c1 + R(2.0) * c2) * sp1);
        }
      }
      R khn = rhog[ipl(0, k, lp)] * fac * hdiff_kh<R>(vt.f[4][ipl(0, k, lp)], k);
      for (int v = 1; v <= 5; ++v) {
        int vm1 = (v == 1) ? 5 : v - 1;
        R khv = rhog[ipl(v, k, lp)] * fac * hdiff_kh<R>(vt.f[4][ipl(v, k, lp)], k);
        R kavg = R(0.5) * (khn + khv);
        R sd = R(0.0);
        for (int d = 0; d < 3; ++d) {
          R cdv = CG.coef_diff_pl[(v * cD.LP + lp) * 3 + d];
          R tv = cdv * (vt_[vm1 - 1][d] + vt_[v - 1][d]);
          sd = (d == 0) ? tv : sd + tv;
        }
        R contrib = kavg * sd;
        row = (v == 1) ? contrib : row + contrib;
      }
    }
    out.f[n][ipl(0, k, lp)] = -row;
    for (int g = 1; g < 6; ++g) out.f[n][ipl(g, k, lp)] = -R(0.0);
  }
}

template <class R, class T>
__global__ void __launch_bounds__(TILE_THREADS, NC_MINB(R, 2, 4)) k_hdiff2_m(Six<R> vt, const R* rhog,
                                                                            SixOut<R> out) {
  constexpr int PX = T::X + 2, PY = T::Y + 2, NP = PX * PY, TX = T::X + 1, TY = T::Y + 1, NT = TX * TY;
  extern __shared__ __align__(16) unsigned char hd_smem[];
  R* s_w = reinterpret_cast<R*>(hd_smem);   // [18][NT] triangle weights
  R* s_f = s_w + 18 * NT;                     // [6][NP] the six Laplacians
  R* s_k = s_f + 6 * NP;                      // [2][NP] rhog * factor * Kh of fields 4 and 5
  R* s_t = s_k + 2 * NP;                      // [2][6][NT] triangle values of fields 4 and 5
  const int l = (int)blockIdx.z;
  const int ntx = (cD.G - 2 + T::X - 1) / T::X;
  const int i0 = 1 + ((int)blockIdx.y % ntx) * T::X, j0 = 1 + ((int)blockIdx.y / ntx) * T::Y;
  const int k0 = (int)blockIdx.x * HD_NK, k1 = min(k0 + HD_NK, cD.KA);
  const int G = cD.G, gmax = cD.G - 2;
  const int tid = threadIdx.x, tx = tid % T::X, ty = tid / T::X;
  const int i = i0 + tx, j = j0 + ty;
  const bool own = (i <= gmax) && (j <= gmax);
  const R kfac[2] = {CC.CVdry, CC.hdiff_fact_rho};
  for (int p = tid; p < NT; p += blockDim.x) {
    const int ii = i0 - 1 + p % TX, jj = j0 - 1 + p / TX;
    const bool ok = ii <= G - 2 && jj <= G - 2;
#pragma unroll
    for (int m = 0; m < 18; ++m) s_w[m * NT + p] = ok ? P2(CG.intp_w, m, ii, jj, l) : R(0.0);
  }
  R cl[7], cd[18];
  if (own) {
#pragma unroll
    for (int m = 0; m < 7; ++m) cl[m] = P2(CG.coef_lap, m, i, j, l);
#pragma unroll
    for (int m = 0; m < 18; ++m) cd[m] = P2(CG.coef_diff, m, i, j, l);
  }
  for (int k = k0; k < k1; ++k) {
    for (int p = tid; p < NP; p += blockDim.x) {
      const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
      const bool ok = ii < G && jj < G;
      const int q = ok ? ix(ii, jj, k, l) : 0;
#pragma unroll
      for (int n = 0; n < 6; ++n) s_f[n * NP + p] = ok ? vt.f[n][q] : R(0.0);
      const R rg = ok ? rhog[q] : R(0.0), kh = hdiff_kh<R>(s_f[4 * NP + p], k);
      s_k[p] = rg * kfac[0] * kh;
      s_k[NP + p] = rg * kfac[1] * kh;
    }
    __syncthreads();
    for (int p = tid; p < NT; p += blockDim.x) {
      const int px = p % TX, py = p / TX;
      const int ii = i0 - 1 + px, jj = j0 - 1 + py;
      const bool ok = ii <= G - 2 && jj <= G - 2;
      const int ia = py * PX + px, ib = ia + 1, ic = ia + PX + 1, id = ia + PX;
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const R* sf = s_f + (4 + f) * NP;
        const R s0 = sf[ia], sip = sf[ib], sd = sf[ic], sjp = sf[id];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          R ti = R(0.0), tj = R(0.0);
          if (ok) {
            // weights 2c1-c2-c3, -c1+2c2-c3, -c1-c2+2c3 of the i and j triangles (k_intp_weights)
            const R w1i = s_w[((d * 3 + 0) * 2 + 0) * NT + p], w2i = s_w[((d * 3 + 1) * 2 + 0) * NT + p];
            const R w3i = s_w[((d * 3 + 2) * 2 + 0) * NT + p], w1j = s_w[((d * 3 + 0) * 2 + 1) * NT + p];
            const R w2j = s_w[((d * 3 + 1) * 2 + 1) * NT + p], w3j = s_w[((d * 3 + 2) * 2 + 1) * NT + p];
            ti = div3(mad(w3i, sd, mad(w2i, sip, w1i * s0)));
            tj = div3(mad(w3j, sjp, mad(w2j, sd, w1j * s0)));
          }
          s_t[(f * 6 + d) * NT + p] = ti;
          s_t[(f * 6 + 3 + d) * NT + p] = tj;
        }
      }
    }
    __syncthreads();
    if (i0 == 1 && j0 == 1) {   // singular-point fix of the (0,0) triangle, fields 4 and 5 (block-uniform branch)
      if (tid < 6) {
        const int f = tid / 3, d = tid % 3;
        const R m0 = (R)CG.pntmask[l * 2 + 0], m1 = (R)CG.pntmask[l * 2 + 1];
        s_t[(f * 6 + d) * NT] = s_t[(f * 6 + d) * NT] * m0 + s_t[(f * 6 + 3 + d) * NT + 1] * m1;
      }
      __syncthreads();
    }
    if (own) {
      const int q = ix(i, j, k, l);
      const int c0 = (ty + 1) * PX + (tx + 1);
      const int nb[7] = {c0, c0 + 1, c0 + PX + 1, c0 + PX, c0 - 1, c0 - PX - 1, c0 - PX};
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const R* sf = s_f + n * NP;
        R v = cl[0] * sf[nb[0]];
#pragma unroll
        for (int m = 1; m < 7; ++m) v = mad(cl[m], sf[nb[m]], v);
        out.f[n][q] = -v;
      }
      const int ta = (ty + 1) * TX + (tx + 1), tb = ta - 1, tc = ta - TX - 1, td = ta - TX;
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        auto kh = [&](int pt) { return s_k[f * NP + pt]; };
        const R kh0 = kh(nb[0]);
        const R kf1 = R(0.5) * (kh0 + kh(nb[2])), kf2 = R(0.5) * (kh0 + kh(nb[3])), kf3 = R(0.5) * (kh0 + kh(nb[4]));
        const R kf4 = R(0.5) * (kh0 + kh(nb[5])), kf5 = R(0.5) * (kh0 + kh(nb[6])), kf6 = R(0.5) * (kh0 + kh(nb[1]));
        R inner = R(0.0);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const R* ti = s_t + (f * 6 + d) * NT;
          const R* tj = s_t + (f * 6 + 3 + d) * NT;
          const R aTI = ti[ta], aTJ = tj[ta], bTI = ti[tb];
          const R cTI = ti[tc], cTJ = tj[tc], dTJ = tj[td];
          R blk = kf1 * cd[d * 6 + 0] * (aTI + aTJ);
          blk = mad(kf2 * cd[d * 6 + 1], aTJ + bTI, blk);
          blk = mad(kf3 * cd[d * 6 + 2], bTI + cTJ, blk);
          blk = mad(kf4 * cd[d * 6 + 3], cTJ + cTI, blk);
          blk = mad(kf5 * cd[d * 6 + 4], cTI + dTJ, blk);
          blk = mad(kf6 * cd[d * 6 + 5], dTJ + aTI, blk);
          inner = (d == 0) ? blk : inner + blk;
        }
        out.f[4 + f][q] = -inner;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Large-step tendency: hyperdiffusion tendency (mod_numfilter.py:1519-1578)
// + horizontalize (mod_numfilter.py:1364-1369) + g_TEND = adv + f
// (mod_dynamics.py:1340-1464).  All columns; projection on interior points.
// ---------------------------------------------------------------------------
template <class R>
struct GtendArgs {
  Six<R> vt2;                       // post-COMM hyperdiffusion Laplacians
  const R* lapT;                    // the first pass's temperature Laplacian (NONLINEAR1 Kh)
  const R *vx, *vy, *vz, *w;        // diagnosed velocities (Rayleigh sponge)
  const R *rhog, *gvx, *gvy, *gvz, *gw;
  R* gT0[6];
  R* frhog;                 // f_TEND[RHOG] (tracer input)
};

template <class R>
__device__ void gtend_point(const Col c, const MetT<R> m, const GtendArgs<R>& a, int i, int j, int k, int l, int g,
                            int lp) {
  {
    const int p = c.at(k);
    R rg = a.rhog[p];
    R rgh = R(0.0);
    if (k >= cD.kmin) rgh = mc(m.C2W, c, 0, 2, k) * rg + mc(m.C2W, c, 1, 2, k) * a.rhog[c.at(k - 1)];
    const R Kh = hdiff_kh<R>(CC.hdiff_nl ? a.lapT[p] : R(0.0), k);
    // the coefficient of w: Kh itself (DIRECT), or for NONLINEAR1 the average of
    // levels k and k-1 on kmin+1..kmax and zero elsewhere (mod_numfilter.py:1186-1206)
    R Khh = Kh;
    if (CC.hdiff_nl)
      Khh = (k > cD.kmin && k <= cD.kmax) ? R(0.5) * (Kh + hdiff_kh<R>(a.lapT[c.at(k - 1)], k - 1)) : R(0.0);
    R fx = -(a.vt2.f[0][p] * Kh + R(0.0)) * rg;
    R fy = -(a.vt2.f[1][p] * Kh + R(0.0)) * rg;
    R fz = -(a.vt2.f[2][p] * Kh + R(0.0)) * rg;
    R fw = -(a.vt2.f[3][p] * Khh + R(0.0)) * rgh;
    R fe = -(a.vt2.f[4][p] + R(0.0));
    R fr = -(a.vt2.f[5][p] + R(0.0));
    if (!c.pole) {
      if (interior(i, j)) horiz_reg(i, j, l, fx, fy, fz);
    } else {
      horiz_pl(g, lp, fx, fy, fz);
    }
    if (CC.rayleigh) {   // the sponge on the hyperdiffusion tendency (mod_numfilter.py:240-271)
      if (!CC.rayleigh_only_w) {
        const R coef = CC.ray_c[k] * rg;
        fx = fx - coef * a.vx[p];
        fy = fy - coef * a.vy[p];
        fz = fz - coef * a.vz[p];
      }
      const R rgm1 = k > 0 ? a.rhog[c.at(k - 1)] : R(0.0);
      fw = fw - CC.ray_ch[k] * a.w[p] * (mc(m.C2W, c, 0, 2, k) * rg + mc(m.C2W, c, 1, 2, k) * rgm1);
    }
    a.gT0[0][p] = R(0.0) + fr;
    a.gT0[1][p] = a.gvx[p] + fx;
    a.gT0[2][p] = a.gvy[p] + fy;
    a.gT0[3][p] = a.gvz[p] + fz;
    a.gT0[4][p] = a.gw[p] + fw;
    a.gT0[5][p] = R(0.0) + fe;
    a.frhog[p] = fr;
  }
}

template <class R>
__global__ void k_gtend(const __grid_constant__ GtendArgs<R> a, const __grid_constant__ GtendArgs<R> ap, int npb) {
  Pt q;
  if ((int)blockIdx.x < npb) {
    if (pole_point((int)(blockIdx.x * blockDim.x + threadIdx.x), q))
      gtend_point(col_pl(q.g, q.lp), met_of<R>(true), ap, 0, 0, q.k, 0, q.g, q.lp);
  } else if (reg_point((int)((blockIdx.x - npb) * blockDim.x + threadIdx.x), q)) {
    gtend_point(col_reg(q.i, q.j, q.l), met_of<R>(false), a, q.i, q.j, q.k, q.l, 0, 0);
  }
}

}  // namespace nc
