// Tracer advection of the last RK stage: MIURA2004 horizontal scheme with
// the Thuburn horizontal and vertical flux limiters, Strang-split V/H/V
// (pynicamdc/nhm/dynamics/mod_src_tracer.py:83-1228).
#pragma once
#include "nc_small.cuh"

namespace nc {

// ---------------------------------------------------------------------------
// tracer-independent part of the first vertical step (kernels/tracervertflux.py)
// flx_v and the updated density rhog_t, on every column.
// ---------------------------------------------------------------------------
template <class R>
struct TrcFluxArgs {
  const R *rvx, *rvy, *rvz, *rw;    // time-mean momentum (PROG_mean)
  const R* rhog_in;                 // density at the start of the step
  const R* frhog;
  R *flx_v, *rhog_t;
  R dt;
};

// flx_v at level k and the density, one thread per point (the flux above is formed again)
template <class R>
__device__ __forceinline__ void trc_vflux_point(const Col c, const MetT<R> m, const TrcFluxArgs<R>& a, int k) {
  const int kmin = cD.kmin, kmax = cD.kmax;
  auto flux = [&](int kk) -> R {
    if (kk < kmin + 1 || kk > kmax) return R(0.0);
    const int p = c.at(kk), pm = c.at(kk - 1);
    const R horiz = (mc(m.C2WGz, c, 0, 6, kk) * a.rvx[p] + mc(m.C2WGz, c, 1, 6, kk) * a.rvx[pm] +
                     mc(m.C2WGz, c, 2, 6, kk) * a.rvy[p] + mc(m.C2WGz, c, 3, 6, kk) * a.rvy[pm] +
                     mc(m.C2WGz, c, 4, 6, kk) * a.rvz[p] + mc(m.C2WGz, c, 5, 6, kk) * a.rvz[pm]) *
                    gam_at(m.RGAMH, p);
    const R vert = a.rw[p] * m.RGSQRTH[p];
    return (horiz + vert) * R(0.5) * a.dt;
  };
  const int p = c.at(k);
  const R f = flux(k);
  R r = R(0.0);
  if (k >= kmin && k <= kmax) r = a.rhog_in[p] - (flux(k + 1) - f) * CC.rdgz[k] + R(0.0) * a.frhog[p] * a.dt;
  else if (k == kmin - 1) r = a.rhog_in[c.at(kmin)];
  else if (k == kmax + 1) r = a.rhog_in[c.at(kmax)];
  a.flx_v[p] = f;
  a.rhog_t[p] = r;
}

template <class R>
__global__ void k_trc_vflux(const __grid_constant__ TrcFluxArgs<R> a, const __grid_constant__ TrcFluxArgs<R> ap, int npb) {
  Pt q;
  if ((int)blockIdx.x < npb) {
    if (pole_point((int)(blockIdx.x * blockDim.x + threadIdx.x), q))
      trc_vflux_point(col_pl(q.g, q.lp), met_of<R>(true), ap, q.k);
  } else if (reg_point((int)((blockIdx.x - npb) * blockDim.x + threadIdx.x), q)) {
    trc_vflux_point(col_reg(q.i, q.j, q.l), met_of<R>(false), a, q.k);
  }
}

// ---------------------------------------------------------------------------
// one vertical fractional step of one tracer with the vertical Thuburn
// limiter (mod_src_tracer.py:389-533 and 1036-1204, limiter :1909-2074)
// ---------------------------------------------------------------------------
template <class R>
struct TrcVadvArgs {
  R* rhogq_of[NC_MAXNQ];   // the tracers of the launch (blockIdx.y)
  const R *den, *flx_v, *frhog;
  R dt, bcoef;      // d = bcoef*frhog/den*dt
  int clamp;             // second step: zero tiny negatives, then add dt*0
  R dtl;
};

// One upward sweep with the values of levels k-1, k, k+1 in registers: at
// level k the cell's outflow bounds are formed, the face value qh[k] is
// limited with the bounds of cells k-1 and k, and cell k-1, whose two faces
// are then final, is updated.  The same expressions as the three-pass form
// of the reference (q, qh and ck on every level, the limiter, the update),
// in the same order, so the same results.  NT tracers of the column (the nt
// first of rq) at once: the Courant numbers, the upwind masks and the
// reciprocals of a level are formed once for all of them.
template <class R, int NT>
__device__ __forceinline__ void trc_vadv_column(const Col c, const TrcVadvArgs<R>& a, R* const* rhogq, int nt) {
  const int KA = cD.KA, kmin = cD.kmin, kmax = cD.kmax;
  const R BIG = CC.HUGE_, EPS = CC.EPS;
  auto finish = [&](int m, int k, R x) {   // clamp and store of one updated level
    if (a.clamp && x > -R(1.0e-10) && x < R(0.0)) x = R(0.0);
    if (a.clamp) x = x + a.dtl * R(0.0);
    if (m < nt) rhogq[m][c.at(k)] = x;
  };
  R* rp[NT];
#pragma unroll
  for (int m = 0; m < NT; ++m) rp[m] = rhogq[min(m, nt - 1)];   // a surplus tracer repeats the last and stores nothing
  // q at kmin-1 and kmin, den and flx_v at kmin (read before the ghost levels are zeroed)
  const int p = c.at(kmin);
  using Div = typename DivOf<R>::type;
  Div by_k(__ldg(&a.den[p]));       // the divisions by a level's density share its reciprocal
  const R den_m = __ldg(&a.den[c.at(kmin - 1)]);
  R rq_k[NT], q_m[NT], q_k[NT], rq_n[NT], qmin_prev[NT], qmax_prev[NT], qh_prev[NT], rq_prev[NT];
#pragma unroll
  for (int m = 0; m < NT; ++m) {
    q_m[m] = rp[m][c.at(kmin - 1)] / den_m;
    rq_k[m] = rp[m][p];
    rq_n[m] = rp[m][c.at(kmin + 1)];
  }
#pragma unroll
  for (int m = 0; m < NT; ++m) {
    q_k[m] = by_k(rq_k[m]);
    qmin_prev[m] = qmax_prev[m] = qh_prev[m] = rq_prev[m] = R(0.0);
  }
  R flx_k = __ldg(&a.flx_v[p]);
  R ck0 = by_k(-flx_k) * CC.rdgz[kmin];
  R flx_prev = R(0.0);
  // the loads of level k+2 are issued before level k is worked on
  R den_n = __ldg(&a.den[c.at(kmin + 1)]), flx_n = __ldg(&a.flx_v[c.at(kmin + 1)]);
  R fr_n = __ldg(&a.frhog[p]);
  for (int k = kmin; k <= kmax; ++k) {
    const R den_p = den_n, flx_p = flx_n, fr_k = fr_n;
    R rq_p[NT];
#pragma unroll
    for (int m = 0; m < NT; ++m) rq_p[m] = rq_n[m];
    if (k < kmax) {
      const int p2 = c.at(k + 2);
#pragma unroll
      for (int m = 0; m < NT; ++m) rq_n[m] = rp[m][p2];
      den_n = __ldg(&a.den[p2]);
      flx_n = __ldg(&a.flx_v[p2]);
      fr_n = __ldg(&a.frhog[c.at(k + 1)]);
    }
    const Div by_p(den_p);
    // the level's quotients by its densities: one tracer a thread is bound by its
    // chain and tests them together, several test each (see DivD)
    R q_one = R(0.0), c1k, c0p, dk;
    if (NT == 1) {
      bool bad = false;
      c1k = by_k.fast(flx_p, bad); c0p = by_p.fast(-flx_p, bad); dk = by_k.fast(a.bcoef * fr_k, bad);
      q_one = by_p.fast(rq_p[0], bad);
      if (bad) {
        c1k = by_k.slow(flx_p); c0p = by_p.slow(-flx_p); dk = by_k.slow(a.bcoef * fr_k);
        q_one = by_p.slow(rq_p[0]);
      }
    } else {
      c1k = by_k(flx_p); c0p = by_p(-flx_p); dk = by_k(a.bcoef * fr_k);
    }
    const R ck1 = c1k * CC.rdgz[k];
    const R ck0_p = (k + 1 <= kmax) ? c0p * CC.rdgz[k + 1] : R(0.0);
    dk = dk * a.dt;
    const R inL = R(0.5) - copysign(R(0.5), ck0);
    const R inU = R(0.5) + copysign(R(0.5), ck0_p);
    const R c1 = ck0, c2 = ck1;
    const R Cin = inL * c1 + inU * c2;
    const R Cout = (R(1.0) - inL) * c1 + (R(1.0) - inU) * c2;
    const R zsw = R(0.5) - copysign(R(0.5), fabs(Cout) - EPS);
    const Div by_o(Cout + zsw);
#pragma unroll
    for (int m = 0; m < NT; ++m) {
      const R q_p = NT == 1 ? q_one : by_p(rq_p[m]);
      const R qh_raw = CC.afact[k] * q_k[m] + CC.bfact[k] * q_m[m];
      const R qc = q_k[m], qb = q_m[m], qa = q_p;
      const R QminL = (inL == R(1.0)) ? npmin(qc, qb) : BIG;
      const R QminU = (inU == R(1.0)) ? npmin(qc, qa) : BIG;
      const R QmaxL = (inL == R(1.0)) ? npmax(qc, qb) : -BIG;
      const R QmaxU = (inU == R(1.0)) ? npmax(qc, qa) : -BIG;
      const R qnmin = npmin(npmin(QminL, QminU), qc);
      const R qnmax = npmax(npmax(QmaxL, QmaxU), qc);
      const R CQmin = inL * c1 * QminL + inU * c2 * QminU;
      const R CQmax = inL * c1 * QmaxL + inU * c2 * QmaxU;
      const R nmin = (qc - qnmax) + qnmax * (Cin + Cout - dk) - CQmax;
      const R nmax = (qc - qnmin) + qnmin * (Cin + Cout - dk) - CQmin;
      R omin, omax;
      if (NT == 1) by_o.two(nmin, nmax, omin, omax);
      else { omin = by_o(nmin); omax = by_o(nmax); }
      const R qomin = omin * (R(1.0) - zsw) + qc * zsw;
      const R qomax = omax * (R(1.0) - zsw) + qc * zsw;
      R qh = R(0.0);   // the face at kmin stays zero
      if (k > kmin) {
        qh = inL * npmin(npmax(qh_raw, qmin_prev[m]), qmax_prev[m]) + (R(1.0) - inL) * npmin(npmax(qh_raw, qomin), qomax);
        finish(m, k - 1, rq_prev[m] - (flx_k * qh - flx_prev * qh_prev[m]) * CC.rdgz[k - 1]);
      }
      qmin_prev[m] = qomin;
      qmax_prev[m] = qomax;
      qh_prev[m] = qh;
      rq_prev[m] = rq_k[m];
      q_m[m] = q_k[m]; q_k[m] = q_p; rq_k[m] = rq_p[m];
    }
    flx_prev = flx_k;
    by_k = by_p; flx_k = flx_p;
    ck0 = ck0_p;
  }
  // cell kmax: its upper face (kmax+1) is zero
#pragma unroll
  for (int m = 0; m < NT; ++m) {
    finish(m, kmax, rq_prev[m] - (flx_k * R(0.0) - flx_prev * qh_prev[m]) * CC.rdgz[kmax]);
    for (int k = 0; k < kmin; ++k) finish(m, k, R(0.0));
    for (int k = kmax + 1; k < KA; ++k) finish(m, k, R(0.0));
  }
}

// Every tracer of the step in one launch: the sweep is a serial chain per
// column, so one tracer's columns alone leave the SMs waiting (263 us a tracer
// at gl07 z60 float64).  A thread takes NT tracers of its column: bound by
// memory (density, fluxes and tendency re-read for each tracer) and by the
// divisions, whose quotients are exact for all operands (DivD; without the test of
// their range two tracers a thread took 1.54 ms and gave the quotients below 1e-308
// another rounding, dividing throughout 2.39).  A launch of 17 tracers at gl07 z60
// float64: one a thread 2.16 ms, two 1.78, three 1.86; 6 at gl06 z40 153, 129,
// 146 us; 6 at gl05 z40 60, 58, 67 us.  Two, where the columns of all
// tracers are at least 256 for each SM; fewer are bound by the
// chain and take a tracer a thread.
#define TV_THREADS 256
#define TV_NT 2
template <class R, int NT>
__global__ void __launch_bounds__(TV_THREADS) k_trc_vadv(const __grid_constant__ TrcVadvArgs<R> a, int pole, int nx) {
  int t = (int)blockIdx.x * blockDim.x + threadIdx.x;
  int i, j, l, g, lp;
  if (!map_col(pole, t, i, j, l, g, lp)) return;
  const int first = (int)blockIdx.y * NT;
  trc_vadv_column<R, NT>(pole ? col_pl(g, lp) : col_reg(i, j, l), a, a.rhogq_of + first, min(NT, nx - first));
}

// ---------------------------------------------------------------------------
// horizontal mass flux through the six hexagon edges and the upwind mass
// centroids (mod_src_tracer.py:1376-1484), Courant numbers and the upwind
// mask (mod_src_tracer.py:716-718)
// ---------------------------------------------------------------------------
template <class R>
struct TrcHfluxArgs {
  const R *rho, *rvx, *rvy, *rvz;   // PROG_mean rhog and momentum (times RGAM on the fly)
  const R* rhog_t;
  R* flx[6];
  R* xc[9];                          // face*3 + dir (AI, AIJ, AJ)
  R* ch[6];
  R* cm[6];
  R dt;
};

// flux and centroid of face f of cell (ii,jj) given the summed vertex values
template <class R>
__device__ __forceinline__ R trc_face(const TrcHfluxArgs<R>& a, int ii, int jj, int l, int f, const R s[4],
                                           R xc[3]) {
  R rr2 = R(1.0) / npmax(s[0], CC.EPS);
  R flux = R(0.5) * (s[1] * P2c(CG.GMTR_a, f * 3 + 0, ii, jj, l) + s[2] * P2c(CG.GMTR_a, f * 3 + 1, ii, jj, l) +
                       s[3] * P2c(CG.GMTR_a, f * 3 + 2, ii, jj, l));
  for (int d = 0; d < 3; ++d) xc[d] = P2c(CG.GRD_xr, f * 3 + d, ii, jj, l) - s[1 + d] * rr2 * a.dt * R(0.5);
  return flux;
}

// One block per level and 32 x 8 tile of cells, the halo ring included (every
// cell gets its six faces; a face the reference leaves out is zero): rho and
// rho*v*RGAM of the haloed tile staged in shared memory, the triangle values
// TI/TJ of every vertex the tile's faces use formed once
// (mod_src_tracer.py:1390-1412, the singular-point fix at the (0,0) vertex
// after them), then each cell's faces 0..2 and its neighbours' faces 0..2
// (its faces 3..5, opposite sign) from those, with the face coefficients of
// the face's owner cell (mod_src_tracer.py:1414-1484).
#define TH_DX 32
#define TH_DY 8
template <class R>
__global__ void __launch_bounds__(TH_DX * TH_DY) k_trc_hflux_t(TrcHfluxArgs<R> a) {
  constexpr int PX = TH_DX + 2, PY = TH_DY + 2, TX = TH_DX + 1, TY = TH_DY + 1;
  __shared__ R s_f[4][PY * PX];
  __shared__ R s_ti[4][TY * TX], s_tj[4][TY * TX];
  const int G = cD.G, k = (int)blockIdx.x, l = (int)blockIdx.z;
  const int ntx = (G + TH_DX - 1) / TH_DX;
  const int i0 = ((int)blockIdx.y % ntx) * TH_DX, j0 = ((int)blockIdx.y / ntx) * TH_DY;
  const int tid = threadIdx.x;
  for (int p = tid; p < PX * PY; p += blockDim.x) {
    const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
    R f0 = R(0.0), f1 = R(0.0), f2 = R(0.0), f3 = R(0.0);
    if (ii >= 0 && jj >= 0 && ii < G && jj < G) {
      const int q = ix(ii, jj, k, l);
      const R rg = CG.RGAM[q];
      f0 = a.rho[q];
      f1 = a.rvx[q] * rg;
      f2 = a.rvy[q] * rg;
      f3 = a.rvz[q] * rg;
    }
    s_f[0][p] = f0; s_f[1][p] = f1; s_f[2][p] = f2; s_f[3][p] = f3;
  }
  __syncthreads();
  for (int p = tid; p < TX * TY; p += blockDim.x) {   // vertex values of (i0-1.., j0-1..)
    const int px = p % TX, py = p / TX;
    const int vi = i0 - 1 + px, vj = j0 - 1 + py;
    const bool ok = vi >= 0 && vj >= 0 && vi <= G - 2 && vj <= G - 2;
    R w1i = R(0.0), w2i = R(0.0), w3i = R(0.0), w1j = R(0.0), w2j = R(0.0), w3j = R(0.0);
    if (ok) {
      w1i = P2c(CG.GMTR_t, 0, vi, vj, l); w2i = P2c(CG.GMTR_t, 1, vi, vj, l); w3i = P2c(CG.GMTR_t, 2, vi, vj, l);
      w1j = P2c(CG.GMTR_t, 3, vi, vj, l); w2j = P2c(CG.GMTR_t, 4, vi, vj, l); w3j = P2c(CG.GMTR_t, 5, vi, vj, l);
    }
    const int ia = py * PX + px, ib = ia + 1, ic = ia + PX + 1, id = ia + PX;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      R ti = R(0.0), tj = R(0.0);
      if (ok) {
        const R f0 = s_f[n][ia], fi = s_f[n][ib], fd = s_f[n][ic], fj = s_f[n][id];
        ti = f0 * w1i + fi * w2i;
        ti = ti + fd * w3i;
        tj = f0 * w1j;
        tj = tj + (fd * w2j + fj * w3j);
      }
      s_ti[n][p] = ti;
      s_tj[n][p] = tj;
    }
  }
  __syncthreads();
  if (i0 == 0 && j0 == 0 && tid < 4) {   // singular-point fix of vertex (0,0) (mod_src_tracer.py:1409-1412)
    const int v00 = 1 * TX + 1, v10 = 1 * TX + 2;
    const R m0 = (R)CG.pntmask[l * 2 + 0], m1 = (R)CG.pntmask[l * 2 + 1];
    s_ti[tid][v00] = s_ti[tid][v00] * m0 + s_tj[tid][v10] * m1;
  }
  __syncthreads();
  const int i = i0 + tid % TH_DX, j = j0 + tid / TH_DX;
  if (i >= G || j >= G) return;
  const int p = ix(i, j, k, l);
  const R dt = a.dt;
  const R PR = P2c(CG.GMTR_p, 0, i, j, l);
  const int vc = (j - j0 + 1) * TX + (i - i0 + 1);   // vertex (i, j); (i-1, j) is vc-1, (i, j-1) vc-TX
  // face f of the cell (ci, cj) from the vertex sums TA + TB (mod_src_tracer.py:1414-1484)
  auto face = [&](int ci, int cj, int f, int va, bool a_is_j, int vb, bool b_is_j, R xc[3]) {
    R sv[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const R A = a_is_j ? s_tj[n][va] : s_ti[n][va];
      const R B = b_is_j ? s_tj[n][vb] : s_ti[n][vb];
      sv[n] = A + B;
    }
    return trc_face(a, ci, cj, l, f, sv, xc);
  };
  R fl[6], xc[3];
  // face 0: TJ(i, j-1) + TI(i, j)
  if (i >= 0 && i <= G - 2 && j >= 1 && j <= G - 2) {
    fl[0] = face(i, j, 0, vc - TX, true, vc, false, xc) * PR * dt;
  } else {
    fl[0] = R(0.0); xc[0] = xc[1] = xc[2] = R(0.0);
  }
  for (int d = 0; d < 3; ++d) a.xc[0 * 3 + d][p] = xc[d];
  // face 1: TI(i, j) + TJ(i, j)
  if (i >= 0 && i <= G - 2 && j >= 0 && j <= G - 2) {
    fl[1] = face(i, j, 1, vc, false, vc, true, xc) * PR * dt;
  } else {
    fl[1] = R(0.0); xc[0] = xc[1] = xc[2] = R(0.0);
  }
  for (int d = 0; d < 3; ++d) a.xc[1 * 3 + d][p] = xc[d];
  // face 2: TJ(i, j) + TI(i-1, j)
  if (i >= 1 && i <= G - 2 && j >= 0 && j <= G - 2) {
    fl[2] = face(i, j, 2, vc, true, vc - 1, false, xc) * PR * dt;
  } else {
    fl[2] = R(0.0); xc[0] = xc[1] = xc[2] = R(0.0);
  }
  for (int d = 0; d < 3; ++d) a.xc[2 * 3 + d][p] = xc[d];
  // faces 3..5: the neighbours' faces 0..2, opposite sign
  R xcn[3];
  fl[3] = (i - 1 >= 0 && i - 1 <= G - 2 && j >= 1 && j <= G - 2)
              ? -face(i - 1, j, 0, vc - 1 - TX, true, vc - 1, false, xcn) * PR * dt : R(0.0);
  fl[4] = (i - 1 >= 0 && i - 1 <= G - 2 && j - 1 >= 0 && j - 1 <= G - 2)
              ? -face(i - 1, j - 1, 1, vc - 1 - TX, false, vc - 1 - TX, true, xcn) * PR * dt : R(0.0);
  fl[5] = (i >= 1 && i <= G - 2 && j - 1 >= 0 && j - 1 <= G - 2)
              ? -face(i, j - 1, 2, vc - TX, true, vc - TX - 1, false, xcn) * PR * dt : R(0.0);
  if (i == 1 && j == 1) fl[5] *= (R)CG.pntmask[l * 2 + 0];
  const auto rg = recip_of(a.rhog_t[p]);   // six quotients by rhog_t
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    a.flx[f][p] = fl[f];
    const R chv = div_by(fl[f], rg);
    a.ch[f][p] = chv;
    a.cm[f][p] = R(0.5) - copysign(R(0.5), chv - CC.EPS);
  }
}

// The same with a march over nk levels in each block, the float form: the vertex
// weights GMTR_t in shared memory, the coefficients of the cell's own faces and
// of its neighbours' in registers once for the block's levels.  Bound by
// instructions, of which the 33 reads of coefficients a cell and level were the
// largest part; three blocks an SM (80 registers; four spill: 1.33 ms).
// gl08 z40 1.56 -> 1.20 ms, gl06 z40 164 -> 131 us, 12 x gl05 z40 518 -> 449 us.
// The double form stays with a block per level: the coefficients take 56 more
// registers (two blocks an SM: gl07 z40 0.62 -> 0.70 ms; read per level in the
// march instead: 0.79 ms).
// The next level's staging writes s_f, read before this level's last barrier,
// and its vertex pass writes s_ti / s_tj after the next barrier, which every
// thread reaches after its faces: two barriers a level.
template <class R>
__global__ void __launch_bounds__(TH_DX * TH_DY, 3) k_trc_hflux_m(const __grid_constant__ TrcHfluxArgs<R> a, int nk) {
  constexpr int PX = TH_DX + 2, PY = TH_DY + 2, TX = TH_DX + 1, TY = TH_DY + 1, NT = TX * TY;
  __shared__ R s_f[4][PY * PX];
  __shared__ R s_w[6][NT];
  __shared__ R s_ti[4][NT], s_tj[4][NT];
  const int G = cD.G, l = (int)blockIdx.z;
  const int ntx = (G + TH_DX - 1) / TH_DX;
  const int i0 = ((int)blockIdx.y % ntx) * TH_DX, j0 = ((int)blockIdx.y / ntx) * TH_DY;
  const int ka = (int)blockIdx.x * nk, kb = min(ka + nk, cD.KA);
  const int tid = threadIdx.x;
  for (int p = tid; p < NT; p += blockDim.x) {   // weights of the vertices (i0-1.., j0-1..)
    const int vi = i0 - 1 + p % TX, vj = j0 - 1 + p / TX;
    const bool ok = vi >= 0 && vj >= 0 && vi <= G - 2 && vj <= G - 2;
#pragma unroll
    for (int m = 0; m < 6; ++m) s_w[m][p] = ok ? P2c(CG.GMTR_t, m, vi, vj, l) : R(0.0);
  }
  const int i = i0 + tid % TH_DX, j = j0 + tid / TH_DX;
  const bool own = i < G && j < G;
  const bool hi = i <= G - 2, hj = j <= G - 2;
  // which of the cell's faces exist, and the owner cell of each
  const bool on[6] = {own && hi && hj && j >= 1, own && hi && hj, own && hi && hj && i >= 1,
                      own && i >= 1 && hj && j >= 1, own && i >= 1 && j >= 1, own && i >= 1 && hi && j >= 1};
  R ga[6][3], xr[9];
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const int ci = (f == 3 || f == 4) ? i - 1 : i, cj = f >= 4 ? j - 1 : j;
#pragma unroll
    for (int d = 0; d < 3; ++d) ga[f][d] = on[f] ? P2c(CG.GMTR_a, (f % 3) * 3 + d, ci, cj, l) : R(0.0);
  }
#pragma unroll
  for (int m = 0; m < 9; ++m) xr[m] = on[m / 3] ? P2c(CG.GRD_xr, m, i, j, l) : R(0.0);
  const R PR = own ? P2c(CG.GMTR_p, 0, i, j, l) : R(0.0);
  const R m0 = (R)CG.pntmask[l * 2 + 0], m1 = (R)CG.pntmask[l * 2 + 1];
  const R dt = a.dt;
  const bool corner = i == 1 && j == 1;
  // vertices (i, j), (i-1, j), (i, j-1) and (i-1, j-1)
  const int vc = (j - j0 + 1) * TX + (i - i0 + 1), vw = vc - 1, vs = vc - TX, vsw = vc - TX - 1;
  for (int k = ka; k < kb; ++k) {
    for (int p = tid; p < PX * PY; p += blockDim.x) {
      const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
      R f0 = R(0.0), f1 = R(0.0), f2 = R(0.0), f3 = R(0.0);
      if (ii >= 0 && jj >= 0 && ii < G && jj < G) {
        const int q = ix(ii, jj, k, l);
        const R rg = CG.RGAM[q];
        f0 = a.rho[q];
        f1 = a.rvx[q] * rg;
        f2 = a.rvy[q] * rg;
        f3 = a.rvz[q] * rg;
      }
      s_f[0][p] = f0; s_f[1][p] = f1; s_f[2][p] = f2; s_f[3][p] = f3;
    }
    const int p = own ? ix(i, j, k, l) : 0;
    const R rgt = a.rhog_t[p];
    __syncthreads();
    for (int v = tid; v < NT; v += blockDim.x) {
      const int ia = (v / TX) * PX + v % TX, ib = ia + 1, ic = ia + PX + 1, id = ia + PX;
      const int vi = i0 - 1 + v % TX, vj = j0 - 1 + v / TX;
      const bool ok = vi >= 0 && vj >= 0 && vi <= G - 2 && vj <= G - 2;
      R w[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) w[m] = s_w[m][v];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const R f0 = s_f[n][ia], fi = s_f[n][ib], fd = s_f[n][ic], fj = s_f[n][id];
        const R ti = mad(fd, w[2], mad(fi, w[1], f0 * w[0]));
        const R tj = mad(f0, w[3], mad(fj, w[5], fd * w[4]));
        s_ti[n][v] = ok ? ti : R(0.0);
        s_tj[n][v] = ok ? tj : R(0.0);
      }
    }
    __syncthreads();
    if (i0 == 0 && j0 == 0) {   // singular-point fix of vertex (0,0) (mod_src_tracer.py:1409-1412)
      const int v00 = 1 * TX + 1, v10 = 1 * TX + 2;
      if (tid < 4) s_ti[tid][v00] = s_ti[tid][v00] * m0 + s_tj[tid][v10] * m1;
      __syncthreads();
    }
    if (!own) continue;
    // sum n of the two vertex values of face f (mod_src_tracer.py:1414-1484)
    auto S = [&](int f, int n) -> R {
      switch (f) {
        case 0: return s_tj[n][vs] + s_ti[n][vc];     // TJ(i, j-1) + TI(i, j)
        case 1: return s_ti[n][vc] + s_tj[n][vc];     // TI(i, j) + TJ(i, j)
        case 2: return s_tj[n][vc] + s_ti[n][vw];     // TJ(i, j) + TI(i-1, j)
        case 3: return s_tj[n][vsw] + s_ti[n][vw];    // face 0 of (i-1, j)
        case 4: return s_ti[n][vsw] + s_tj[n][vsw];   // face 1 of (i-1, j-1)
        default: return s_tj[n][vs] + s_ti[n][vsw];   // face 2 of (i, j-1)
      }
    };
    const auto rg = recip_of(rgt);   // six quotients by rhog_t
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const R s1 = S(f, 1), s2 = S(f, 2), s3 = S(f, 3);
      const R flux = R(0.5) * mad(s3, ga[f][2], mad(s2, ga[f][1], s1 * ga[f][0]));
      R fl = (f < 3 ? flux : -flux) * PR * dt;
      fl = on[f] ? fl : R(0.0);
      if (f == 5 && corner) fl *= m0;
      a.flx[f][p] = fl;
      const R chv = div_by(fl, rg);
      a.ch[f][p] = chv;
      a.cm[f][p] = R(0.5) - copysign(R(0.5), chv - CC.EPS);
      if (f < 3) {
        const R rr2 = R(1.0) / npmax(S(f, 0), CC.EPS);
        const R sd[3] = {s1, s2, s3};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const R x = xr[f * 3 + d] - sd[d] * rr2 * dt * R(0.5);
          a.xc[f * 3 + d][p] = on[f] ? x : R(0.0);
        }
      }
    }
  }
}

// pole edges (mod_src_tracer.py:1487-1531) and Courant numbers
template <class R>
struct TrcHfluxPlArgs {
  const R *rho, *rvx, *rvy, *rvz, *rhog_t;
  R *flx, *xc, *ch, *cm;   // flx/ch/cm (g,k,l); xc (g,k,l,3)
  R dt;
};

template <class R>
__global__ void k_trc_hflux_pl(TrcHfluxPlArgs<R> a) {
  int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= cD.KA * cD.LP) return;
  int k = t / cD.LP, lp = t % cD.LP;
  const R* gt = CG.GMTR_t_pl;
  const R* ga = CG.GMTR_a_pl;
  const R* gp = CG.GMTR_p_pl;
  R tv[6][4];
  auto F = [&](int n, int q) -> R {
    if (n == 0) return a.rho[q];
    const R* r = (n == 1) ? a.rvx : ((n == 2) ? a.rvy : a.rvz);
    return r[q] * gam_at(CG.RGAM_pl, q);
  };
  for (int v = 1; v <= 5; ++v) {
    int vp1 = (v + 1 == 6) ? 1 : v + 1;
    const R* g5 = gt + (v * cD.LP + lp) * 5;
    for (int n = 0; n < 4; ++n)
      tv[v][n] = F(n, ipl(0, k, lp)) * g5[2] + F(n, ipl(v, k, lp)) * g5[3] + F(n, ipl(vp1, k, lp)) * g5[4];
  }
  R rc = a.rhog_t[ipl(0, k, lp)];
  for (int v = 1; v <= 5; ++v) {
    int vm1 = (v - 1 == 0) ? 5 : v - 1;
    R rr2 = R(1.0) / npmax(tv[vm1][0] + tv[v][0], CC.EPS);
    R v2[3];
    for (int n = 0; n < 3; ++n) v2[n] = tv[vm1][n + 1] + tv[v][n + 1];
    const R* g18 = ga + (v * cD.LP + lp) * 18;
    R flux = R(0.5) * (v2[0] * g18[0] + v2[1] * g18[1] + v2[2] * g18[2]);
    int q = ipl(v, k, lp);
    R fl = flux * gp[(0 * cD.LP + lp) * 8 + 1] * a.dt;
    a.flx[q] = fl;
    for (int d = 0; d < 3; ++d) a.xc[q * 3 + d] = CG.GRD_xr_pl[(v * cD.LP + lp) * 3 + d] - v2[d] * rr2 * a.dt * R(0.5);
    R chv = fl / rc;
    a.ch[q] = chv;
    a.cm[q] = R(0.5) - copysign(R(0.5), chv - CC.EPS);
  }
}

// ---------------------------------------------------------------------------
// per tracer: q and its gradient (mod_src_tracer.py:758-771, 1634-1640)
// ---------------------------------------------------------------------------
// One block per (level, tile of interior cells): q of the haloed tile
// is formed once into shared memory (one division per cell instead of one per
// stencil use), then each cell's gradient is read from there.  The region's
// halo cells get q and a zero gradient from the tile that holds their nearest
// interior cell, so every cell is written exactly once.
// The tracers of a batch (up to TRC_NB) share the block: each gradient
// coefficient and each cell's density is read once for all of them.
#define TRC_NB 4
template <class R>
struct TrcGradArgs {
  const R* rhogq[TRC_NB];
  const R* rhog_t;
  R *q[TRC_NB], *gq[TRC_NB][3];
  int nb;
};
template <class R, class T>
__global__ void __launch_bounds__(TILE_THREADS) k_trc_grad_t(const __grid_constant__ TrcGradArgs<R> a) {
  constexpr int PX = T::X + 2, PY = T::Y + 2, NP = PX * PY;
  __shared__ R s_q[TRC_NB][NP];
  const TileLv tl = tile_level<T>(0);
  const int k = tl.k, l = tl.l, i0 = tl.i0, j0 = tl.j0;
  const int G = cD.G, gmax = cD.G - 2;
  const int tid = threadIdx.x;
  for (int p = tid; p < NP; p += blockDim.x) {
    const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
    const bool ok = ii < G && jj < G;
    const int qq = ok ? ix(ii, jj, k, l) : 0;
    bool mine = false;   // a halo cell of the region that this tile writes
    if (ok && !interior(ii, jj)) {
      const int ci = min(max(ii, 1), gmax), cj = min(max(jj, 1), gmax);
      mine = ci >= i0 && ci < i0 + T::X && cj >= j0 && cj < j0 + T::Y;
    }
    const R den = ok ? __ldg(a.rhog_t + qq) : R(1.0);
#pragma unroll
    for (int n = 0; n < TRC_NB; ++n) {
      if (n >= a.nb) break;
      const R v = ok ? __ldg(a.rhogq[n] + qq) / den : R(0.0);
      s_q[n][p] = v;
      if (mine) {
        a.q[n][qq] = v;
        a.gq[n][0][qq] = R(0.0);
        a.gq[n][1][qq] = R(0.0);
        a.gq[n][2][qq] = R(0.0);
      }
    }
  }
  __syncthreads();
  const int tx = tid % T::X, ty = tid / T::X;
  const int i = i0 + tx, j = j0 + ty;
  if (i > gmax || j > gmax) return;
  const int qq = ix(i, j, k, l);
  const int c0 = (ty + 1) * PX + (tx + 1);
  const int nb[7] = {c0, c0 + 1, c0 + PX + 1, c0 + PX, c0 - 1, c0 - PX - 1, c0 - PX};
#pragma unroll
  for (int d = 0; d < 3; ++d) {   // grad7 (kernels/oprtgradient.py:45-70)
    R cg[7];
#pragma unroll
    for (int m = 0; m < 7; ++m) cg[m] = P2c(CG.coef_grad, d * 7 + m, i, j, l);
#pragma unroll
    for (int n = 0; n < TRC_NB; ++n) {
      if (n >= a.nb) break;
      R g = cg[0] * s_q[n][c0];
#pragma unroll
      for (int m = 1; m < 7; ++m) g = mad(cg[m], s_q[n][nb[m]], g);
      a.gq[n][d][qq] = g;
      if (d == 0) a.q[n][qq] = s_q[n][c0];
    }
  }
}

template <class R>
__global__ void k_trc_grad_pl(const __grid_constant__ TrcGradArgs<R> a) {
  int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= cD.KA * cD.LP) return;
  int k = t / cD.LP, lp = t % cD.LP;
  const int n = (int)blockIdx.y;
  R qv[6];
  for (int v = 0; v < 6; ++v) {
    int p = ipl(v, k, lp);
    qv[v] = a.rhogq[n][p] / a.rhog_t[p];
    a.q[n][p] = qv[v];
  }
  for (int d = 0; d < 3; ++d) {
    R row = R(0.0);
    for (int v = 0; v < 6; ++v) {
      R tv = CG.coef_grad_pl[(v * cD.LP + lp) * 3 + d] * qv[v];
      row = (v == 0) ? tv : row + tv;
    }
    a.gq[n][d][ipl(0, k, lp)] = row;
    for (int v = 1; v < 6; ++v) a.gq[n][d][ipl(v, k, lp)] = R(0.0);
  }
}

// ---------------------------------------------------------------------------
// MIURA2004 face values of edges 0..2 (mod_src_tracer.py:1696-1787)
// ---------------------------------------------------------------------------
// One thread per point: the offsets of the face centroids from the two cells
// of each face are formed once for the tracers of the batch.
template <class R>
struct TrcRemapArgs {
  const R *q[TRC_NB], *gq[TRC_NB][3];
  const R* xc[9];
  const R* cm[6];
  R* qa[TRC_NB][3];
  int nb;
};

// The largest block of the three kernels of a batch (80, 80 and 125 registers a
// thread in the float64 form; 1024 threads leave 64).  The float64 remap and
// outflow bounds are compiled for 768, which holds them to 80 registers, six
// blocks of 128 an SM: 17 tracers at gl07 z60, a step: remap 3.13 ms (for 512
// threads 3.70), outflow bounds 3.43 (unbounded 3.84).
#define TRC_BATCH_THREADS 512
template <class R>
__global__ void __launch_bounds__(NC_MINB(R, 768, TRC_BATCH_THREADS)) k_trc_remap(const __grid_constant__ TrcRemapArgs<R> a) {
  Pt c;
  const int p = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (!reg_point(p, c)) return;
  const int G = cD.G;
  if (c.i > G - 2 || c.j > G - 2) {
    for (int n = 0; n < a.nb; ++n) a.qa[n][0][p] = a.qa[n][1][p] = a.qa[n][2][p] = R(0.0);
    return;
  }
  const int mi[3] = {1, 1, 0}, mj[3] = {0, 1, 1};
  const int pn[3] = {p + 1, p + G + 1, p + G};
  R op[3][3], on[3][3], cf[3];   // offsets from the cell and from the face's other cell
#pragma unroll
  for (int f = 0; f < 3; ++f) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const R x = __ldg(a.xc[f * 3 + d] + p);
      op[f][d] = x - P2c(CG.GRD_x, d, c.i, c.j, c.l);
      on[f][d] = x - P2c(CG.GRD_x, d, c.i + mi[f], c.j + mj[f], c.l);
    }
    cf[f] = __ldg(a.cm[f] + p);
  }
  for (int n = 0; n < a.nb; ++n) {
    R v[3];
    const R q0 = __ldg(a.q[n] + p), g0 = __ldg(a.gq[n][0] + p), g1 = __ldg(a.gq[n][1] + p), g2 = __ldg(a.gq[n][2] + p);
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const int m = pn[f];
      R ap = q0, am = __ldg(a.q[n] + m);
      ap = ap + g0 * op[f][0];
      ap = ap + g1 * op[f][1];
      ap = ap + g2 * op[f][2];
      am = am + __ldg(a.gq[n][0] + m) * on[f][0];
      am = am + __ldg(a.gq[n][1] + m) * on[f][1];
      am = am + __ldg(a.gq[n][2] + m) * on[f][2];
      v[f] = cf[f] * am + (R(1.0) - cf[f]) * ap;
    }
#pragma unroll
    for (int f = 0; f < 3; ++f) a.qa[n][f][p] = v[f];
  }
}

template <class R>
struct TrcRemapPlArgs {
  const R *q[TRC_NB], *gq[TRC_NB][3], *xc, *cm;
  R* qa[TRC_NB];
};

template <class R>
__global__ void k_trc_remap_pl(const __grid_constant__ TrcRemapPlArgs<R> a) {
  int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= cD.KA * cD.LP) return;
  int k = t / cD.LP, lp = t % cD.LP;
  const int n = (int)blockIdx.y;
  const R* X = CG.GRD_x_pl;
  int p0 = ipl(0, k, lp);
  for (int v = 1; v <= 5; ++v) {
    int pv = ipl(v, k, lp);
    R ap = a.q[n][p0];
    for (int d = 0; d < 3; ++d) ap = ap + a.gq[n][d][p0] * (a.xc[pv * 3 + d] - X[(0 * cD.LP + lp) * 3 + d]);
    R am = a.q[n][pv];
    for (int d = 0; d < 3; ++d) am = am + a.gq[n][d][pv] * (a.xc[pv * 3 + d] - X[(v * cD.LP + lp) * 3 + d]);
    R c = a.cm[pv];
    a.qa[n][pv] = c * am + (R(1.0) - c) * ap;
  }
}

// ---------------------------------------------------------------------------
// horizontal Thuburn limiter (mod_src_tracer.py:2190-2605, numpy branch)
// ---------------------------------------------------------------------------
template <class R>
struct TrcLimArgs {
  const R *q[TRC_NB], *rhog_t, *frhog;
  const R* ch[6];
  const R* cm[6];
  const R* qa[TRC_NB][3];
  R *Qmin[TRC_NB], *Qmax[TRC_NB];   // Qout
  const R* flx[6];
  R* rhogq[TRC_NB];
  R dt;
  int nb;
};

// The six faces of a cell (slots 0..2: its own faces 0..2; slots 3..5: faces
// 0..2 of the cells behind it) touch the seven cells of its hexagon only,
// numbered as the stencils' offsets (kNbI, kNbJ).  For each slot: the four cells
// whose smallest and largest q bound the face, in the reference's order
// (mod_src_tracer.py:2191-2217), the cell that owns the face and the other one.
struct FaceCells {
  int c[4], own, other;
};
__device__ __forceinline__ constexpr FaceCells face_cells(int m) {
  return m == 0   ? FaceCells{{0, 6, 1, 2}, 0, 1}
         : m == 1 ? FaceCells{{0, 1, 2, 3}, 0, 2}
         : m == 2 ? FaceCells{{0, 2, 3, 4}, 0, 3}
         : m == 3 ? FaceCells{{4, 5, 0, 3}, 4, 0}
         : m == 4 ? FaceCells{{5, 6, 0, 4}, 5, 0}
                  : FaceCells{{6, 1, 0, 5}, 6, 0};
}
// Smallest and largest q of face slot m.  sgp: the face at a singular point,
// slot 4 of cell (1,1): np.min over [q(0,0), q(1,1), q(2,1), q(0,1)] (:2298-2323)
template <class R>
__device__ __forceinline__ void trc_face_minmax(const R q[7], int m, bool sgp, R& qn, R& qx) {
  const FaceCells f = face_cells(m);
  const R q0 = q[f.c[0]];
  R v1 = q[f.c[1]], v2 = q[f.c[2]], v3 = q[f.c[3]];
  if (m == 4 && sgp) { v1 = q[0]; v2 = q[1]; }
  qn = npmin(npmin(npmin(q0, v1), v2), v3);
  qx = npmax(npmax(npmax(q0, v1), v2), v3);
}
// The bounds that a face with the upwind mask c gives the cell it belongs to
// (slots 0..2) and the cell behind it (slots 3..5) (mod_src_tracer.py:2220-2234)
template <class R>
__device__ __forceinline__ void trc_qin(R c, bool sgp, R qn, R qx, bool behind, R& qin_min, R& qin_max) {
  const R BIG = CC.HUGE_;
  if (!behind) {
    qin_min = sgp ? ((c == R(1.0)) ? qn : BIG) : c * qn + (R(1.0) - c) * BIG;
    qin_max = sgp ? ((c == R(1.0)) ? qx : -BIG) : c * qx + (R(1.0) - c) * (-BIG);
  } else {
    qin_min = sgp ? ((c == R(1.0)) ? BIG : qn) : c * BIG + (R(1.0) - c) * qn;
    qin_max = sgp ? ((c == R(1.0)) ? -BIG : qx) : c * (-BIG) + (R(1.0) - c) * qx;
  }
}
// offset of cell n of the hexagon, and the owner of face slot m
__device__ __forceinline__ int hex_off(int n) { return kNbI[n] + kNbJ[n] * cD.G; }

// Outflow bounds, one thread per point; the Courant numbers and masks are read
// once for the tracers of the batch.
template <class R>
__global__ void __launch_bounds__(NC_MINB(R, 768, TRC_BATCH_THREADS)) k_trc_qout(const __grid_constant__ TrcLimArgs<R> a) {
  Pt t;
  const int p = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (!reg_point(p, t)) return;
  if (!interior(t.i, t.j)) {
    for (int n = 0; n < a.nb; ++n) a.Qmin[n][p] = a.Qmax[n][p] = a.q[n][p];
    return;
  }
  const R EPS = CC.EPS;
  R ch[6], cm[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    ch[m] = __ldg(a.ch[m] + p);
    cm[m] = __ldg(a.cm[m % 3] + p + hex_off(face_cells(m).own));
  }
  const bool sgp = CG.have_sgp[t.l] && t.i == 1 && t.j == 1;
  const R d = R(1.0) * __ldg(a.frhog + p) / __ldg(a.rhog_t + p) * a.dt;
  for (int n = 0; n < a.nb; ++n) {
    R q[7];
#pragma unroll
    for (int m = 0; m < 7; ++m) q[m] = __ldg(a.q[n] + p + hex_off(m));
    const R qc = q[0];
    R qnmin = qc, qnmax = qc;
    R Cin = R(0.0), Cout = R(0.0), CQmin = R(0.0), CQmax = R(0.0);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      R qn, qx, qi, qxi;
      const bool s = m == 4 && sgp;
      trc_face_minmax(q, m, s, qn, qx);
      trc_qin(cm[m], s, qn, qx, m >= 3, qi, qxi);
      qnmin = npmin(qnmin, qi);
      qnmax = npmax(qnmax, qxi);
      const R chm = npmin(ch[m], R(0.0));
      if (m == 0) {
        Cin = chm; Cout = ch[m] - chm; CQmin = chm * qi; CQmax = chm * qxi;
      } else {
        Cin = Cin + chm; Cout = Cout + (ch[m] - chm); CQmin = CQmin + chm * qi; CQmax = CQmax + chm * qxi;
      }
    }
    const R zsw = R(0.5) - copysign(R(0.5), fabs(Cout) - EPS);
    const typename DivOf<R>::type den(Cout + zsw);
    R omin, omax;
    den.two(qc - CQmax - qnmax * (R(1.0) - Cin - Cout + d), qc - CQmin - qnmin * (R(1.0) - Cin - Cout + d), omin, omax);
    a.Qmin[n][p] = omin * (R(1.0) - zsw) + qc * zsw;
    a.Qmax[n][p] = omax * (R(1.0) - zsw) + qc * zsw;
  }
}

// Limited face values (mod_src_tracer.py:2545-2605) and the flux update, one
// thread per point: the cell limits its six faces from the q and outflow bounds
// of its hexagon, each face's extremes formed once for both cells' bounds.
// (A tile that shares the faces through shared memory was slower for one tracer,
// 0.94 against 0.62 ms at gl08 mixed: two barriers and 22 KB a block.)
template <class R>
__global__ void __launch_bounds__(TRC_BATCH_THREADS) k_trc_apply(const __grid_constant__ TrcLimArgs<R> a) {
  Pt t;
  const int p = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (!reg_point(p, t) || !interior(t.i, t.j)) return;
  const bool sgp = CG.have_sgp[t.l] && t.i == 1 && t.j == 1;
  R fl[6], cm[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    fl[m] = __ldg(a.flx[m] + p);
    cm[m] = __ldg(a.cm[m % 3] + p + hex_off(face_cells(m).own));
  }
  for (int n = 0; n < a.nb; ++n) {
    R q[7], lo[7], hi[7], v[6];
#pragma unroll
    for (int m = 0; m < 7; ++m) {
      q[m] = __ldg(a.q[n] + p + hex_off(m));
      lo[m] = __ldg(a.Qmin[n] + p + hex_off(m));
      hi[m] = __ldg(a.Qmax[n] + p + hex_off(m));
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) v[m] = __ldg(a.qa[n][m % 3] + p + hex_off(face_cells(m).own));
    R upd = R(0.0);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const FaceCells f = face_cells(m);
      const bool s = m == 4 && sgp;
      R qn, qx, i0n, i0x, i1n, i1x;
      trc_face_minmax(q, m, s, qn, qx);
      const R c = cm[m];
      trc_qin(c, s, qn, qx, false, i0n, i0x);
      trc_qin(c, s, qn, qx, true, i1n, i1x);
      R x = c * npmin(npmax(v[m], i0n), i0x) + (R(1.0) - c) * npmin(npmax(v[m], i1n), i1x);
      x = c * npmax(npmin(x, hi[f.other]), lo[f.other]) + (R(1.0) - c) * npmax(npmin(x, hi[f.own]), lo[f.own]);
      upd = m ? upd + fl[m] * x : fl[m] * x;
    }
    a.rhogq[n][p] = a.rhogq[n][p] - upd;
  }
}

// pole Qout (mod_src_tracer.py:2437-2495) at g = 0
template <class R>
struct TrcLimPlArgs {
  const R *q_of[TRC_NB], *ch, *cm, *rhog_t, *frhog, *qa[TRC_NB], *flx;
  R *Qmin[TRC_NB], *Qmax[TRC_NB];
  R* rhogq[TRC_NB];
  R dt;
};

template <class R>
__device__ void trc_qin_pl(const TrcLimPlArgs<R>& a, const R* q, int v, int k, int lp, R& in0n, R& in1n, R& in0x,
                           R& in1x) {
  const R BIG = CC.HUGE_;
  int vp1 = (v + 1 > 5) ? 1 : v + 1, vm1 = (v - 1 < 1) ? 5 : v - 1;
  R q0 = q[ipl(0, k, lp)], qv = q[ipl(v, k, lp)], qm = q[ipl(vm1, k, lp)], qp = q[ipl(vp1, k, lp)];
  R qn = pymin(pymin(pymin(q0, qv), qm), qp);
  R qx = pymax(pymax(pymax(q0, qv), qm), qp);
  R c = a.cm[ipl(v, k, lp)];
  in0n = (c == R(1.0)) ? qn : BIG;
  in1n = (c == R(1.0)) ? BIG : qn;
  in0x = (c == R(1.0)) ? qx : -BIG;
  in1x = (c == R(1.0)) ? -BIG : qx;
}

template <class R>
__global__ void k_trc_qout_pl(const __grid_constant__ TrcLimPlArgs<R> a) {
  int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= cD.KA * cD.LP) return;
  int k = t / cD.LP, lp = t % cD.LP;
  int p0 = ipl(0, k, lp);
  const int n = (int)blockIdx.y;   // the tracer of the batch
  const R* q = a.q_of[n];
  R qnm = q[p0], qnx = q[p0];
  R in0n[6], in0x[6], d1, d2;
  for (int v = 1; v <= 5; ++v) {
    trc_qin_pl(a, q, v, k, lp, in0n[v], d1, in0x[v], d2);
    qnm = pymin(qnm, in0n[v]);
    qnx = pymax(qnx, in0x[v]);
  }
  R Ci = R(0.0), Co = R(0.0), CQn = R(0.0), CQx = R(0.0);
  for (int v = 1; v <= 5; ++v) {
    int pv = ipl(v, k, lp);
    R chm = a.cm[pv] * a.ch[pv];
    Ci = Ci + chm;
    Co = Co + (a.ch[pv] - chm);
    CQn = CQn + chm * in0n[v];
    CQx = CQx + chm * in0x[v];
  }
  R zs = R(0.5) - copysign(R(0.5), fabs(Co) - CC.EPS);
  R den = Co + zs;
  R fac = R(1.0) - zs;
  R q0 = q[p0];
  R dv = R(1.0) * a.frhog[p0] / a.rhog_t[p0] * a.dt;
  a.Qmin[n][p0] = (q0 - CQx - qnx * (R(1.0) - Ci - Co + dv)) / den * fac + q0 * zs;
  a.Qmax[n][p0] = (q0 - CQn - qnm * (R(1.0) - Ci - Co + dv)) / den * fac + q0 * zs;
}

template <class R>
__global__ void k_trc_apply_pl(const __grid_constant__ TrcLimPlArgs<R> a) {
  int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= cD.KA * cD.LP) return;
  int k = t / cD.LP, lp = t % cD.LP;
  int p0 = ipl(0, k, lp);
  const int n = (int)blockIdx.y;   // the tracer of the batch
  const R* q = a.q_of[n];
  R acc = a.rhogq[n][p0];
  for (int v = 1; v <= 5; ++v) {
    int pv = ipl(v, k, lp);
    R in0n, in1n, in0x, in1x;
    trc_qin_pl(a, q, v, k, lp, in0n, in1n, in0x, in1x);
    R c = a.cm[pv];
    R x = a.qa[n][pv];
    R a0 = npmin(npmax(x, in0n), in0x);
    R a1 = npmin(npmax(x, in1n), in1x);
    x = c * a0 + (R(1.0) - c) * a1;
    R a2 = npmax(npmin(x, a.Qmax[n][pv]), a.Qmin[n][pv]);
    R a3 = npmax(npmin(x, a.Qmax[n][p0]), a.Qmin[n][p0]);
    x = c * a2 + (R(1.0) - c) * a3;
    acc = acc - a.flx[pv] * x;
  }
  a.rhogq[n][p0] = acc;
}

// density after the horizontal step (mod_src_tracer.py:890-916)
template <class R>
__global__ void k_trc_rhog(R* rhog_t, const R* f0, const R* f1, const R* f2, const R* f3,
                           const R* f4, const R* f5, const R* frhog, R dt, const R* flx_pl,
                           R* rhog_t_pl, const R* frhog_pl) {
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  Pt q;
  if (reg_point(t, q)) {
    if (!interior(q.i, q.j)) return;
    const R s = __ldg(f0 + t) + __ldg(f1 + t) + __ldg(f2 + t) + __ldg(f3 + t) + __ldg(f4 + t) + __ldg(f5 + t);
    rhog_t[t] = rhog_t[t] - (s - (R(1.0) * __ldg(frhog + t) * dt));
  } else {
    int tp = t - cD.npti;
    if (tp < cD.KA * cD.LP) {
      int k = (int)(tp / cD.LP), lp = (int)(tp % cD.LP);
      int p0 = ipl(0, k, lp);
      R r = rhog_t_pl[p0];
      for (int v = 1; v <= 5; ++v) r = r - flx_pl[ipl(v, k, lp)];
      r = r + R(1.0) * frhog_pl[p0] * dt;
      rhog_t_pl[p0] = r;
    }
  }
}

}  // namespace nc
