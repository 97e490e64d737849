// HEVI small-step kernels: 3-D/2-D divergence damping, pressure gradient,
// vp0 source terms + tridiagonal matrix, the acoustic-loop path1 update and
// vi_main (flux convergences + Thomas solve + energy update).
#pragma once
#include "nc_large.cuh"

namespace nc {

// ---------------------------------------------------------------------------
// 3-D divergence damping operator (kernels/oprt3ddivdamp.py:85-173)
// ---------------------------------------------------------------------------
template <class R>
struct Four { const R* f[4]; };   // rhogvx, rhogvy, rhogvz, rhogw
template <class R>
struct Three { R* f[3]; };
template <class R>
struct CThree { const R* f[3]; };

// Tiled 3-D divergence damping: one block per T::X x T::Y tile of output
// cells of one region, marching upward in k.  Per level the block stages the
// haloed tile of RGAM-scaled momentum and the vertical mass flux rwv(k+1) in
// shared memory (rwv(k) is kept from the level below), evaluates every
// triangle value once, applies the singular-point fix, then each thread forms
// its cell's three components.  Per triangle: the RGAM-weighted momenta at
// its three vertices against coef_intp plus the vertical flux difference
// ((rwv(k+1) summed over the vertices) - (rwv(k) summed)) / 3 * rdgz(k)
// (kernels/oprt3ddivdamp.py:50-173); the rwv sums and coefficient products
// are added left to right in the reference's order.
// The tile's k-invariant coefficients are read once per block instead of
// once per level: the triangle weights coef_intp (18 planes) staged in shared
// memory, the cell's coef_diff (18) held in registers.  Dynamic shared memory
// dd3d_m_smem<R, T>().
template <class R, class T>
constexpr int dd3d_m_smem() {
  return (18 * (T::X + 1) * (T::Y + 1) + 9 * (T::X + 2) * (T::Y + 2) + 4 * (T::X + 1) * (T::Y + 1)) * (int)sizeof(R);
}
// The march takes two levels at a time: a triangle's coefficients are read once
// for both, and a pair of levels costs two barriers.  Bound by shared-memory
// reads and barriers: gl08 mixed 636 -> 509 us, gl06 mixed 66 -> 58 us, gl07
// float64 385 -> 362 us, gl05 float64 42 -> 41 us against one level at a time
// (z40); with three float blocks an SM instead of four 546 us at gl08.
// The next pair's staging writes s_vm and the rwv buffers of this pair's lower
// half levels, which only this pair's triangle pass reads (done before its
// second barrier), and the next triangle pass writes s_ti / s_tj only after the
// next first barrier, which every thread reaches after its cell pass: no barrier
// is needed at the end of a pair, and the corner tile alone waits for its
// singular-point fix.

// pole 3-D divergence damping (kernels/oprt3ddivdamp.py:176-237): eight lanes
// per (level, pole), a lane for each pole point's momenta and half-level fluxes
// and for each triangle between them (one thread formed every flux up to six
// times over: 22 us a call, longer than the regional kernel on small grids)
template <class R>
__global__ void k_dd3d_pl(const __grid_constant__ Four<R> v, const __grid_constant__ Three<R> out) {
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int g = t % 8, np = cD.KA * cD.LP;
  const bool live = t / 8 < np;
  const int e = live ? t / 8 : np - 1;
  const int k = e / cD.LP, lp = e % cD.LP;
  const bool in = k >= cD.kmin && k <= cD.kmax;
  R r0 = R(0.0), r1 = R(0.0), vm[3] = {R(0.0), R(0.0), R(0.0)};
  if (g < 6 && in) {
    auto rw = [&](int kk) -> R {
      if (kk <= cD.kmin || kk > cD.kmax) return R(0.0);
      const int q = ipl(g, kk, lp), qm = ipl(g, kk - 1, lp);
      const R* cz = CG.C2WGz_pl;
      const R h = cz[q * 6 + 0] * v.f[0][q] + cz[q * 6 + 1] * v.f[0][qm] + cz[q * 6 + 2] * v.f[1][q] +
                  cz[q * 6 + 3] * v.f[1][qm] + cz[q * 6 + 4] * v.f[2][q] + cz[q * 6 + 5] * v.f[2][qm];
      return h * gam_at(CG.RGAMH_pl, q) + v.f[3][q] * CG.RGSQRTH_pl[q];
    };
    r0 = rw(k);
    r1 = rw(k + 1);
    const int q = ipl(g, k, lp);
#pragma unroll
    for (int d = 0; d < 3; ++d) vm[d] = v.f[d][q] * gam_at(CG.RGAM_pl, q);
  }
  // lane g = 1..5: the triangle of the pole, point g and the next point
  const int gn = (g >= 5) ? 1 : g + 1;
  auto of = [&](R x, int lane) { return __shfl_sync(0xffffffffu, x, lane, 8); };
  const R u0 = of(r1, 0), un = of(r1, gn), d0 = of(r0, 0), dn = of(r0, gn);
  R a[3], n[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    a[d] = of(vm[d], 0);
    n[d] = of(vm[d], gn);
  }
  R sclt = R(0.0);
  if (g >= 1 && g <= 5 && in) {
    const R sw = div3((u0 + r1 + un) - (d0 + r0 + dn)) * CC.rdgz[k];
    const R* cI = CG.coef_intp_pl + (g * cD.LP + lp) * 9;
    sclt = cI[0] * a[0] + cI[1] * vm[0] + cI[2] * n[0] + cI[3] * a[1] + cI[4] * vm[1] + cI[5] * n[1] + cI[6] * a[2] +
           cI[7] * vm[2] + cI[8] * n[2] + sw;
  }
  R s[6];
#pragma unroll
  for (int m = 1; m <= 5; ++m) s[m] = of(sclt, m);
  // lane g = 0..2: component g of the pole row; the other rows are zero
  R row = R(0.0);
  if (g < 3 && in) {
#pragma unroll
    for (int m = 1; m <= 5; ++m) {
      const R tv = CG.coef_diff_pl[(m * cD.LP + lp) * 3 + g] * (s[m == 1 ? 5 : m - 1] + s[m]);
      row = (m == 1) ? tv : row + tv;
    }
  }
  if (live && g < 3) {
    R* o = out.f[g];
    o[ipl(0, k, lp)] = row;
#pragma unroll
    for (int m = 1; m <= 5; ++m) o[ipl(m, k, lp)] = R(0.0);
  }
}

// The levels are split into chunks of nk where the tiles alone leave SMs idle
// (see tile_chunks); blockIdx.z counts (region, chunk).
template <class R, class T>
__global__ void __launch_bounds__(TILE_THREADS, NC_MINB(R, 2, 4)) k_dd3d_m(Four<R> v, Three<R> out,
                                                                                           int nk) {
  constexpr int PX = T::X + 2, PY = T::Y + 2, NP = PX * PY;
  constexpr int TX = T::X + 1, TY = T::Y + 1, NT = TX * TY;
  extern __shared__ __align__(16) unsigned char dd_smem[];
  R* s_ci = reinterpret_cast<R*>(dd_smem);   // [18][NT] coef_intp of each triangle
  R* s_vm = s_ci + 18 * NT;                    // [2][3][NP] of the pair's levels
  R* s_rw = s_vm + 6 * NP;                     // [3][NP] half levels k, k+1, k+2
  R* s_ti = s_rw + 3 * NP;                     // [2][NT]
  R* s_tj = s_ti + 2 * NT;                     // [2][NT]
  const int l = (int)blockIdx.z % cD.L;
  const int ka = cD.kmin + (int)blockIdx.z / cD.L * nk, kb = min(ka + nk - 1, cD.kmax);
  const int i0 = 1 + blockIdx.x * T::X, j0 = 1 + blockIdx.y * T::Y;
  const int G = cD.G, gmax = cD.G - 2, kmax = cD.kmax;
  const int tid = threadIdx.x, tx = tid % T::X, ty = tid / T::X;
  const int i = i0 + tx, j = j0 + ty;
  const bool own = (i <= gmax) && (j <= gmax);
  const int n = cD.npti;
  const R* cz = CG.C2WGz;
  for (int p = tid; p < NT; p += blockDim.x) {
    const int ii = i0 - 1 + p % TX, jj = j0 - 1 + p / TX;
    const bool ok = ii <= G - 2 && jj <= G - 2;
#pragma unroll
    for (int m = 0; m < 18; ++m) s_ci[m * NT + p] = ok ? P2c(CG.coef_intp, m, ii, jj, l) : R(0.0);
  }
  R cd[18];
  if (own) {
#pragma unroll
    for (int m = 0; m < 18; ++m) cd[m] = P2c(CG.coef_diff, m, i, j, l);
  }
  // vertical mass flux at the half level of q from the momenta at q (u) and below (d)
  auto rwv = [&](int q, const R* u, const R* d, R w) -> R {
    const R h = mad(cz[5 * n + q], d[2], mad(cz[4 * n + q], u[2], mad(cz[3 * n + q], d[1],
                mad(cz[2 * n + q], u[1], mad(cz[n + q], d[0], cz[q] * u[0])))));
    return h * gam_at(CG.RGAMH, q) + w * CG.RGSQRTH[q];
  };
  for (int p = tid; p < NP; p += blockDim.x) {   // at the chunk's first level (zero at kmin)
    const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
    R r = R(0.0);
    if (ka > cD.kmin && ii < G && jj < G) {
      const int q = ix(ii, jj, ka, l), qm = q - cD.planei;
      const R u[3] = {v.f[0][q], v.f[1][q], v.f[2][q]}, d[3] = {v.f[0][qm], v.f[1][qm], v.f[2][qm]};
      r = rwv(q, u, d, v.f[3][q]);
    }
    s_rw[p] = r;
  }
  int c0 = 0;   // slot of half level k
  for (int k = ka; k <= kb; k += 2) {
    const int c1 = (c0 + 1) % 3, c2 = (c0 + 2) % 3;
    for (int p = tid; p < NP; p += blockDim.x) {
      const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
      R f[3][3], r1 = R(0.0), r2 = R(0.0), rg0 = R(0.0), rg1 = R(0.0);
#pragma unroll
      for (int m = 0; m < 9; ++m) f[m / 3][m % 3] = R(0.0);
      if (ii < G && jj < G) {
        const int q = ix(ii, jj, k, l);
#pragma unroll
        for (int d = 0; d < 3; ++d) f[0][d] = v.f[d][q];
        rg0 = gam_at(CG.RGAM, q);
        if (k + 1 <= kmax) {          // rwv is zero above kmax
          const int q1 = q + cD.planei;
#pragma unroll
          for (int d = 0; d < 3; ++d) f[1][d] = v.f[d][q1];
          rg1 = gam_at(CG.RGAM, q1);
          r1 = rwv(q1, f[1], f[0], v.f[3][q1]);
          if (k + 2 <= kmax) {
            const int q2 = q1 + cD.planei;
#pragma unroll
            for (int d = 0; d < 3; ++d) f[2][d] = v.f[d][q2];
            r2 = rwv(q2, f[2], f[1], v.f[3][q2]);
          }
        }
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        s_vm[d * NP + p] = f[0][d] * rg0;
        s_vm[(3 + d) * NP + p] = f[1][d] * rg1;
      }
      s_rw[c1 * NP + p] = r1;
      s_rw[c2 * NP + p] = r2;
    }
    __syncthreads();
    const R* rw[3] = {s_rw + c0 * NP, s_rw + c1 * NP, s_rw + c2 * NP};
    for (int p = tid; p < NT; p += blockDim.x) {
      const int px = p % TX, py = p / TX;
      const int a = py * PX + px, b = a + 1, c = a + PX + 1, d = a + PX;
      const int vI[3] = {a, b, c}, vJ[3] = {a, c, d};
      R sI[2], sJ[2];
#pragma unroll
      for (int m = 0; m < 9; ++m) {   // direction m / 3, vertex m % 3, left to right
        const R cI = s_ci[(m * 2) * NT + p], cJ = s_ci[(m * 2 + 1) * NT + p];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const R* x = s_vm + (3 * e + m / 3) * NP;
          sI[e] = m ? mad(cI, x[vI[m % 3]], sI[e]) : cI * x[vI[0]];
          sJ[e] = m ? mad(cJ, x[vJ[m % 3]], sJ[e]) : cJ * x[vJ[0]];
        }
      }
      const int ii = i0 - 1 + px, jj = j0 - 1 + py;
      const bool ok = ii <= G - 2 && jj <= G - 2;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const R* rU = rw[e + 1];
        const R* rD = rw[e];
        const R rdz = CC.rdgz[k + e];
        const R wI = div3((rU[a] + rU[b] + rU[c]) - (rD[a] + rD[b] + rD[c])) * rdz;
        const R wJ = div3((rU[a] + rU[c] + rU[d]) - (rD[a] + rD[c] + rD[d])) * rdz;
        s_ti[e * NT + p] = ok ? sI[e] + wI : R(0.0);
        s_tj[e * NT + p] = ok ? sJ[e] + wJ : R(0.0);
      }
    }
    __syncthreads();
    if (i0 == 1 && j0 == 1) {   // singular-point fix at the (0,0) triangle (block-uniform branch)
      if (tid < 2)
        s_ti[tid * NT] = s_ti[tid * NT] * (R)CG.pntmask[l * 2 + 0] + s_tj[tid * NT + 1] * (R)CG.pntmask[l * 2 + 1];
      __syncthreads();
    }
    if (own) {
      const int ta = (ty + 1) * TX + (tx + 1);   // triangle (i, j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (k + e > kb) break;
        const R* I = s_ti + e * NT;
        const R* J = s_tj + e * NT;
        const R aTI = I[ta], aTJ = J[ta];
        const R bTI = I[ta - 1];                                // (i-1, j)
        const R cTI = I[ta - TX - 1], cTJ = J[ta - TX - 1];     // (i-1, j-1)
        const R dTJ = J[ta - TX];                               // (i, j-1)
        const int q = ix(i, j, k + e, l);
#pragma unroll
        for (int d = 0; d < 3; ++d)
          out.f[d][q] = mad(cd[d * 6 + 5], dTJ + aTI, mad(cd[d * 6 + 4], cTI + dTJ, mad(cd[d * 6 + 3], cTJ + cTI,
                        mad(cd[d * 6 + 2], bTI + cTJ, mad(cd[d * 6 + 1], aTJ + bTI, cd[d * 6 + 0] * (aTI + aTJ))))));
      }
    }
    c0 = c2;
  }
}

// Block -> (level, tile, region) of the per-level tiled kernels: the level
// is the fastest block index so that blocks sharing a tile's haloed data at
// neighbouring levels run together and meet in L2.
struct TileLv {
  int k, l, i0, j0;
};
template <class T>
__device__ __forceinline__ TileLv tile_level(int kbase) {
  constexpr int TDX = T::X, TDY = T::Y;
  const int ntx = (cD.G - 2 + TDX - 1) / TDX;
  TileLv t;
  t.k = kbase + (int)blockIdx.x;
  t.l = (int)blockIdx.z;
  t.i0 = 1 + ((int)blockIdx.y % ntx) * TDX;
  t.j0 = 1 + ((int)blockIdx.y / ntx) * TDY;
  return t;
}

// ---------------------------------------------------------------------------
// post-COMM 2-D divergence damping (kernels/divdamppostcomm.py:29-81):
// gd = coef * OPRT_divdamp(-vtmp2), then horizontalize.
// ---------------------------------------------------------------------------
// pole 2-D divergence damping of -vtmp2 at (g,k,lp) (kernels/oprtdivdamp.py:125-173
// then horizontalize over all g)
template <class R>
__device__ void divdamp2d_pl_at(const CThree<R>& vt, int g, int k, int lp, R gd[3]) {
  R o[3] = {R(0.0), R(0.0), R(0.0)};
  if (g == 0) {
    R vv[6][3];
    for (int q = 0; q < 6; ++q)
      for (int d = 0; d < 3; ++d) vv[q][d] = -vt.f[d][ipl(q, k, lp)];
    R sclt[5];
    for (int v_ = 1; v_ <= 5; ++v_) {
      int vp1 = (v_ == 5) ? 1 : v_ + 1;
      const R* cI = CG.coef_intp_pl + (v_ * cD.LP + lp) * 9;
      sclt[v_ - 1] = cI[0] * vv[0][0] + cI[1] * vv[v_][0] + cI[2] * vv[vp1][0] + cI[3] * vv[0][1] +
                     cI[4] * vv[v_][1] + cI[5] * vv[vp1][1] + cI[6] * vv[0][2] + cI[7] * vv[v_][2] +
                     cI[8] * vv[vp1][2];
    }
    for (int d = 0; d < 3; ++d) {
      R row = R(0.0);
      for (int v_ = 1; v_ <= 5; ++v_) {
        int vm1 = (v_ == 1) ? 5 : v_ - 1;
        R tv = CG.coef_diff_pl[(v_ * cD.LP + lp) * 3 + d] * (sclt[vm1 - 1] + sclt[v_ - 1]);
        row = (v_ == 1) ? tv : row + tv;
      }
      o[d] = row;
    }
  }
  for (int d = 0; d < 3; ++d) o[d] = CC.divdamp_coef * o[d];
  horiz_pl(g, lp, o[0], o[1], o[2]);
  gd[0] = o[0]; gd[1] = o[1]; gd[2] = o[2];
}

// ---------------------------------------------------------------------------
// pressure gradient (kernels/presgrad.py:126-265): horizontal part at level
// k with the first-layer remedy and the tangent-plane projection.
// P(ii,jj,kk) gives the pressure; returns Pgrad (3 comps).
// ---------------------------------------------------------------------------
template <class R, class PF>
__device__ void presgrad_pl(int g, int k, int lp, const Col& c, const MetT<R>& m, PF P, R out[3]) {
  const int kmin = cD.kmin, kmax = cD.kmax;
  out[0] = out[1] = out[2] = R(0.0);
  if (k >= kmin && k <= kmax) {
    const int kk = (k == kmin) ? kmin + 1 : k;
    R gh[3] = {R(0.0), R(0.0), R(0.0)};
    if (g == 0) {
      for (int d = 0; d < 3; ++d) {
        R row = R(0.0);
        for (int v_ = 0; v_ < 6; ++v_) {
          R pvm = P(v_, kk) * gam_at(CG.RGAM_pl, ipl(v_, kk, lp)) * R(1.0);
          R tv = CG.coef_grad_pl[(v_ * cD.LP + lp) * 3 + d] * pvm;
          row = (v_ == 0) ? tv : row + tv;
        }
        gh[d] = row;
      }
    }
    auto pvmh = [&](int k2, int d) {
      return (mc(m.C2WGz, c, 2 * d, 6, k2) * P(g, k2) + mc(m.C2WGz, c, 2 * d + 1, 6, k2) * P(g, k2 - 1)) *
             gam_at(m.RGAMH, c.at(k2));
    };
    for (int d = 0; d < 3; ++d) out[d] = gh[d] + (pvmh(kk + 1, d) - pvmh(kk, d)) * CC.rdgz[kk];
  }
  horiz_pl(g, lp, out[0], out[1], out[2]);
}

// flux convergence at level k of a regional or pole column given the
// horizontal divergence value (zero on the halo) and the flux accessors
// (kernels/fluxconv.py:111-208, vflag 1 or 0)
template <class R, class FH, class FW>
__device__ __forceinline__ R fluxconv_col(const Col& c, const MetT<R>& m, int k, typename Id<R>::type div,
                                          typename Id<R>::type vflag, FH fh, FW fw) {
  if (k < cD.kmin || k > cD.kmax) return R(0.0);
  auto vmh = [&](int kk) -> R {
    if (kk <= cD.kmin || kk > cD.kmax) return R(0.0);
    R h = vmh_horiz(c, m, kk, fh);
    return h + vflag * fw(kk) * m.RGSQRTH[c.at(kk)];
  };
  return -div - (vmh(k + 1) - vmh(k)) * CC.rdgz[k];
}

// pole divergence row of (fx,fy,fz)*RGAM at level k (kernels/fluxconv.py:81-108)
template <class R, class F>
__device__ __forceinline__ R div_pl(int lp, int k, F f) {
  R row = R(0.0);
  for (int v_ = 0; v_ < 6; ++v_) {
    int q = ipl(v_, k, lp);
    R rg = gam_at(CG.RGAM_pl, q);
    R vx = f(q, 0) * rg, vy = f(q, 1) * rg, vz = f(q, 2) * rg;
    const R* cd = CG.coef_div_pl + (v_ * cD.LP + lp) * 3;
    R pv = cd[0] * vx + cd[1] * vy + cd[2] * vz;
    row = (v_ == 0) ? pv : row + pv;
  }
  return row;
}

// ---------------------------------------------------------------------------
// vp0: small-step source terms, g_TEND of the small step, the vertical
// implicit matrix and ethtot0 (mod_vi.py:295-878 numpy path,
// kernels/vimatrix.py:67-136, kernels/vimain.py:195-239)
// ---------------------------------------------------------------------------
template <class R>
struct Vp0Args {
  Prog<R> P;                    // PROG (post BNDCND)
  const R *vx, *vy, *vz, *eth;
  const double *pregd, *rhogd;  // float64 in both forms
  CThree<R> vt;                 // post-COMM 3-D divdamp of PROG
  const R* gT0[6];              // large-step tendency
  R* gT[6];                     // out: small-step tendency
  double *Mc, *Mu, *Ml;         // float64 in both forms
  R* ethtot0;
  double dt;                    // small-step dt
};

// One pole point of vp0.  In the mixed form the horizontal operators run in
// float32 (R) and the vertical part -- buoyancy and vertical pressure gradient
// of the float64 deviations, gz, the implicit matrix and the vertical-momentum
// tendency -- in float64, as in the regional column kernel k_vp0_cr.
template <class R>
__global__ void k_vp0_pl(const __grid_constant__ Vp0Args<R> a) {
  Pt q_;
  if (!pole_point((int)(blockIdx.x * blockDim.x + threadIdx.x), q_)) return;
  const int g = q_.g, lp = q_.lp, k = q_.k;
  const Col c = col_pl(g, lp);
  const MetT<R> m = met_of<R>(true);
  const int kmin = cD.kmin, kmax = cD.kmax;
  const R* const* P = a.P.v;
  const double dt = a.dt;
  // column-local half-level values (float64)
  auto rhog_h = [&](int k) -> double {
    int kk = (k < kmin) ? kmin : k;
    return (double)mc(m.C2W, c, 0, 2, kk) * (double)P[0][c.at(kk)] +
           (double)mc(m.C2W, c, 1, 2, kk) * (double)P[0][c.at(kk - 1)];
  };
  auto eth_h = [&](int k) -> double {
    int kk = (k < kmin) ? kmin : k;
    return cC.afact[kk] * (double)a.eth[c.at(kk)] + cC.bfact[kk] * (double)a.eth[c.at(kk - 1)];
  };
  auto dbuo = [&](int k) -> double {
    if (k < kmin + 1 || k > kmax) return 0.0;
    return -cC.GRAV * ((double)mc(m.C2W, c, 0, 2, k) * a.rhogd[c.at(k)] +
                       (double)mc(m.C2W, c, 1, 2, k) * a.rhogd[c.at(k - 1)]);
  };
  auto dpgw = [&](int k) -> double {
    if (k < kmin + 1 || k > kmax) return 0.0;
    const int p = c.at(k), pm = c.at(k - 1);
    return (double)gam_at(m.GAM2H, p) *
           (a.pregd[p] * (double)m.RGSGAM2[p] - a.pregd[pm] * (double)m.RGSGAM2[pm]) * cC.rdgzh[k];
  };
  auto gz = [&](int k) -> double { return cC.GRAV - (dpgw(k) - dbuo(k)) / rhog_h(k); };
  auto pwh = [&](int k) -> R { return R(-gz(k) * (double)P[4][c.at(k)]); };
  auto PF = [&](int k, int d) -> R { return P[1 + d][c.at(k)]; };
  auto PEF = [&](int k, int d) -> R { return P[1 + d][c.at(k)] * a.eth[c.at(k)]; };
  {
    const int p = c.at(k);
    // horizontal divergences
    R div1 = R(0.0), div2 = R(0.0);
    if (g == 0) {
      div1 = div_pl<R>(lp, k, [&](int q, int d) { return P[1 + d][q]; });
      div2 = div_pl<R>(lp, k, [&](int q, int d) { return P[1 + d][q] * a.eth[q]; });
    }
    R drhog = fluxconv_col(c, m, k, div1, R(1.0), PF, [&](int kk) { return P[4][c.at(kk)]; });
    R drhoge = fluxconv_col(c, m, k, div2, R(1.0), PEF, [&](int kk) {
      int q = c.at(kk);
      return P[4][q] * (CC.afact[kk] * a.eth[q] + CC.bfact[kk] * a.eth[c.at(kk - 1)]);
    });
    R dd[3], dpg[3];
    divdamp2d_pl_at(a.vt, g, k, lp, dd);
    presgrad_pl(g, k, lp, c, m, [&](int gg, int kk) { return R(a.pregd[ipl(gg, kk, lp)]); }, dpg);
    R pw = R(0.0);
    if (k >= kmin && k <= kmax)
      pw = a.vx[p] * dpg[0] + a.vy[p] * dpg[1] + a.vz[p] * dpg[2] + mc(m.W2C, c, 0, 2, k) * pwh(k + 1) +
           mc(m.W2C, c, 1, 2, k) * pwh(k);
    a.gT[0][p] = a.gT0[0][p] + drhog;
    a.gT[1][p] = a.gT0[1][p] - dpg[0] + dd[0] + R(0.0);
    a.gT[2][p] = a.gT0[2][p] - dpg[1] + dd[1] + R(0.0);
    a.gT[3][p] = a.gT0[3][p] - dpg[2] + dd[2] + R(0.0);
    a.gT[4][p] = R((double)a.gT0[4][p] + 0.0 * cC.alpha - dpgw(k) + dbuo(k));
    a.gT[5][p] = a.gT0[5][p] + drhoge + pw;
    // vertical implicit matrix on k = kmin+1..kmax (float64)
    if (k >= kmin + 1 && k <= kmax) {
      const double GCVovR = cC.GRAV * cC.CVdry / cC.Rdry;
      const double ACVovRt2 = cC.alpha * cC.CVdry / cC.Rdry / (dt * dt);
      int pm = c.at(k - 1), pp = c.at(k + 1);
      double rg = cC.rdgz[k], rgm = cC.rdgz[k - 1];
      double Ca = ((double)m.RGSGAM2[p] * rg + (double)m.RGSGAM2[pm] * rgm) * (double)gam_at(m.GAM2H, p);
      double Cb = cC.dfact[k] - cC.cfact[k - 1];
      double Cu1 = (double)m.RGSGAM2[p] * rg * (double)gam_at(m.GAM2H, pp);
      double rgh2 = (double)gam_at(m.RGAMH, p) * (double)gam_at(m.RGAMH, p);
      double Cu2 = (double)gam_at(m.GAM2H, pp) * rgh2 * GCVovR;
      double Cl1 = (double)m.RGSGAM2[p] * rg * (double)gam_at(m.GAM2H, pm);
      double Cl2 = (double)gam_at(m.GAM2H, pm) * rgh2 * GCVovR;
      double rgh = cC.rdgzh[k];
      a.Mc[p] = ACVovRt2 / (double)m.RGSQRTH[p] + rgh * (Ca * eth_h(k) - Cb * (gz(k) + GCVovR));
      a.Mu[p] = -rgh * (Cu1 * eth_h(k + 1) + cC.cfact[k] * (gz(k + 1) + Cu2));
      a.Ml[p] = -rgh * (Cl1 * eth_h(k - 1) - cC.dfact[k - 1] * (gz(k - 1) + Cl2));
    }
    // total energy at the start of the small steps
    R kin0 = rhogkin_at(c, m, k, [&](int kk, int comp) { return P[comp][c.at(kk)]; });
    a.ethtot0[p] = a.eth[p] + kin0 / P[0][p] + m.PHI[p];
  }
}

// Horizontal terms of vp0, tiled like k_path1_l: for interior cells and
// levels kmin..kmax, the divergences of RGAM*rhogv and RGAM*rhogv*eth
// (div1, div2), the 2-D divergence damping of -vtmp2 (dd) and the pressure
// gradient of pregd (dpg), written to eight work fields for the column kernel.
template <class R>
struct Vp0H {
  R* out[8];               // div1, div2, dd x/y/z, dpg x/y/z
};

// vp0 horizontal terms, one block per (NK levels, tile): like k_path1_l, each of
// the 78 coefficients is loaded once and applied to the block's NK levels (the
// float32 instance; two float64 levels do not leave room for four blocks of
// shared memory).
template <class R> constexpr int VP_NK = sizeof(R) == 8 ? 1 : 2;
template <class R, class T, int NK>
__global__ void __launch_bounds__(TILE_THREADS, NC_MINB(R, 4, NC_F32_VP0H)) k_vp0_hl(Vp0Args<R> a, Vp0H<R> h) {
  constexpr int PX = T::X + 2, PY = T::Y + 2, TX = T::X + 1, TY = T::Y + 1, NP = PX * PY, NT = TX * TY;
  __shared__ R s_m[NK][3][NP];    // RGAM * rhogv
  __shared__ R s_e[NK][3][NP];    // RGAM * rhogv * eth
  __shared__ R s_v[NK][3][NP];    // -vtmp2
  __shared__ R s_p[NK][NP];       // RGAM * pregd at the gradient level
  __shared__ R s_ti[NK][NT], s_tj[NK][NT];
  const TileLv tl = tile_level<T>(0);
  const int l = tl.l, i0 = tl.i0, j0 = tl.j0;
  const int G = cD.G, gmax = cD.G - 2, kmin = cD.kmin, kmax = cD.kmax;
  const int ka = kmin + tl.k * NK;
  const int tid = threadIdx.x, tx = tid % T::X, ty = tid / T::X;
  const R* cz = CG.C2WGz;
  const R* const* P = a.P.v;
  for (int p = tid; p < NP; p += blockDim.x) {
    const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
    const bool ok = ii < G && jj < G;
    const int q0 = ok ? ix(ii, jj, 0, l) : 0;
#pragma unroll
    for (int n = 0; n < NK; ++n) {
      const int k = min(ka + n, kmax), kk = (k == kmin) ? kmin + 1 : k;   // a level past kmax repeats it
      R mv[3] = {R(0.0), R(0.0), R(0.0)}, ev[3] = {R(0.0), R(0.0), R(0.0)}, vv[3] = {R(0.0), R(0.0), R(0.0)}, pp = R(0.0);
      if (ok) {
        const int q = q0 + k * cD.planei, qk = q0 + kk * cD.planei;
        const R rg = CG.RGAM[q], e = a.eth[q];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const R pv = P[1 + d][q];
          mv[d] = pv * rg;
          ev[d] = (pv * e) * rg;
          vv[d] = -a.vt.f[d][q];
        }
        pp = a.pregd[qk] * CG.RGAM[qk];
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        s_m[n][d][p] = mv[d];
        s_e[n][d][p] = ev[d];
        s_v[n][d][p] = vv[d];
      }
      s_p[n][p] = pp;
    }
  }
  __syncthreads();
  for (int p = tid; p < NT; p += blockDim.x) {
    const int px = p % TX, py = p / TX;
    const int ii = i0 - 1 + px, jj = j0 - 1 + py;
    R sI[NK], sJ[NK];
#pragma unroll
    for (int n = 0; n < NK; ++n) sI[n] = sJ[n] = R(0.0);
    if (ii <= G - 2 && jj <= G - 2) {
      const int ia = py * PX + px;
      const int vI[3] = {ia, ia + 1, ia + PX + 1}, vJ[3] = {ia, ia + PX + 1, ia + PX};
#pragma unroll
      for (int m = 0; m < 9; ++m) {   // direction m / 3, vertex m % 3, left to right
        const R cI = P2(CG.coef_intp, m * 2, ii, jj, l), cJ = P2(CG.coef_intp, m * 2 + 1, ii, jj, l);
#pragma unroll
        for (int n = 0; n < NK; ++n) {
          const R xI = s_v[n][m / 3][vI[m % 3]], xJ = s_v[n][m / 3][vJ[m % 3]];
          sI[n] = m ? mad(cI, xI, sI[n]) : cI * xI;
          sJ[n] = m ? mad(cJ, xJ, sJ[n]) : cJ * xJ;
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NK; ++n) {
      s_ti[n][p] = sI[n];
      s_tj[n][p] = sJ[n];
    }
  }
  __syncthreads();
  const int i = i0 + tx, j = j0 + ty;
  if (i > gmax || j > gmax) return;
  const R ddc = CC.divdamp_coef;
  const int npt = cD.npti;
  const R gx = P2(CG.GRD_x, 0, i, j, l), gy = P2(CG.GRD_x, 1, i, j, l), gz = P2(CG.GRD_x, 2, i, j, l);
  const int q0 = ix(i, j, 0, l);
  const int ta = (ty + 1) * TX + (tx + 1), c0 = (ty + 1) * PX + (tx + 1);
  const int nb[7] = {c0, c0 + 1, c0 + PX + 1, c0 + PX, c0 - 1, c0 - PX - 1, c0 - PX};
  {
    // divergences (div7: per direction left to right, then x + y + z)
    R d1[NK], d2[NK];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      R s1[NK], s2[NK];
#pragma unroll
      for (int m = 0; m < 7; ++m) {
        const R cf = P2(CG.coef_div, d * 7 + m, i, j, l);
#pragma unroll
        for (int n = 0; n < NK; ++n) {
          s1[n] = m ? mad(cf, s_m[n][d][nb[m]], s1[n]) : cf * s_m[n][d][nb[m]];
          s2[n] = m ? mad(cf, s_e[n][d][nb[m]], s2[n]) : cf * s_e[n][d][nb[m]];
        }
      }
#pragma unroll
      for (int n = 0; n < NK; ++n) {
        d1[n] = d ? d1[n] + s1[n] : s1[n];
        d2[n] = d ? d2[n] + s2[n] : s2[n];
      }
    }
#pragma unroll
    for (int n = 0; n < NK; ++n)
      if (ka + n <= kmax) {
        h.out[0][q0 + (ka + n) * cD.planei] = d1[n];
        h.out[1][q0 + (ka + n) * cD.planei] = d2[n];
      }
  }
  auto flat = [&](R* x) {   // tangent-plane projection
    const R prd = div_r(x[0] * gx + x[1] * gy + x[2] * gz);
    x[0] = x[0] - div_r(prd * gx);
    x[1] = x[1] - div_r(prd * gy);
    x[2] = x[2] - div_r(prd * gz);
  };
  R x[NK][3];
  // 2-D divergence damping
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      const R cf = P2(CG.coef_diff, d * 6 + e, i, j, l);
#pragma unroll
      for (int n = 0; n < NK; ++n) {
        const R* I = s_ti[n];
        const R* J = s_tj[n];
        const R t = e == 0 ? I[ta] + J[ta] : e == 1 ? J[ta] + I[ta - 1] : e == 2 ? I[ta - 1] + J[ta - TX - 1]
                  : e == 3 ? J[ta - TX - 1] + I[ta - TX - 1] : e == 4 ? I[ta - TX - 1] + J[ta - TX] : J[ta - TX] + I[ta];
        x[n][d] = e ? mad(cf, t, x[n][d]) : cf * t;
      }
    }
  }
#pragma unroll
  for (int n = 0; n < NK; ++n) {
    if (ka + n > kmax) break;
    const int q = q0 + (ka + n) * cD.planei;
#pragma unroll
    for (int d = 0; d < 3; ++d) x[n][d] = ddc * x[n][d];
    flat(x[n]);
#pragma unroll
    for (int d = 0; d < 3; ++d) h.out[2 + d][q] = x[n][d];
  }
  // pressure gradient of pregd
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int m = 0; m < 7; ++m) {
      const R cf = P2(CG.coef_grad, d * 7 + m, i, j, l);
#pragma unroll
      for (int n = 0; n < NK; ++n) x[n][d] = m ? mad(cf, s_p[n][nb[m]], x[n][d]) : cf * s_p[n][nb[m]];
    }
  }
#pragma unroll
  for (int n = 0; n < NK; ++n) {
    const int k = ka + n, kk = (k == kmin) ? kmin + 1 : k;
    if (k > kmax) break;
    const int q = q0 + k * cD.planei, qkk = q0 + kk * cD.planei, qk1 = qkk + cD.planei, qkm = qkk - cD.planei;
    const R P_k1 = a.pregd[qk1], P_k = a.pregd[qkk], P_km = a.pregd[qkm];
    const R rgh1 = CG.RGAMH[qk1], rgh0 = CG.RGAMH[qkk];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const R up = (cz[(2 * d) * npt + qk1] * P_k1 + cz[(2 * d + 1) * npt + qk1] * P_k) * rgh1;
      const R dn = (cz[(2 * d) * npt + qkk] * P_k + cz[(2 * d + 1) * npt + qkk] * P_km) * rgh0;
      x[n][d] = x[n][d] + (up - dn) * CC.rdgz[kk];
    }
    flat(x[n]);
#pragma unroll
    for (int d = 0; d < 3; ++d) h.out[5 + d][q] = x[n][d];
  }
}

// Column part of vp0 for every regional column: vertical flux convergences,
// small-step tendencies, the implicit matrix and ethtot0, with the horizontal
// terms read from k_vp0_hl (zero on halo columns and outside kmin..kmax, where
// the values that depend on them are replaced by the halo exchanges or the
// boundary rows before they are read).  The column marches upward with every
// half-level quantity evaluated once: at level k the values at k+1 (vertical
// mass and energy fluxes, buoyancy, vertical pressure gradient, gz, pwh,
// half-level eth, the vertical kinetic-energy term) are formed and the ones at
// k and k-1 are carried in registers.  Each value is the expression of
// k_vp0_pl (the pole form), so regional and pole columns round alike.
// 256-thread blocks, three an SM (80 registers).  blockIdx.y takes a chunk of nk
// levels: a whole column per thread walked 42 levels at 9 us each, however few the
// columns; a chunk forms the half-level values of its first two levels again (see
// column_chunks).
#define NC_VP0C_BLOCK 256
template <class R>
__global__ void __launch_bounds__(NC_VP0C_BLOCK, NC_MINB(R, 3, NC_F32_VP0C)) k_vp0_cr(Vp0Args<R> a, Vp0H<R> h,
                                                                                   int nk) {
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  int i, j, l;
  if (!col_of(t, i, j, l)) return;
  const Col c = col_reg(i, j, l);
  const int KA = cD.KA, kmin = cD.kmin, kmax = cD.kmax;
  const int ka = (int)blockIdx.y * nk, kb = min(ka + nk, KA);
  const int n = cD.npti;
  const bool in = interior(i, j);
  const R* const* P = a.P.v;
  const double dt = a.dt;
  const double GRAV = cC.GRAV;
  const R* cz = CG.C2WGz;
  const R* c2w = CG.C2W;
  const R* w2c = CG.W2C;
  const double GCVovR = cC.GRAV * cC.CVdry / cC.Rdry;
  const double ACVovRt2 = cC.alpha * cC.CVdry / cC.Rdry / (dt * dt);
  // half-level values; those at level k (h0) and k-1 (hm) are carried upward
  struct Half {
    double vA, vE, gz, eh, pwh, dpgw, dbuo, vint;   // vertical fluxes of rhog / rhoge, gz, eth, ...
  };
  auto half = [&](int kn) -> Half {
    Half r{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (kn < kmin || kn > kmax + 1) return r;
    const int q = c.at(kn), qm = c.at(kn - 1);
    const double e = __ldg(a.eth + q), em = __ldg(a.eth + qm), w = __ldg(P[4] + q);
    const double c0 = __ldg(c2w + q), c1 = __ldg(c2w + n + q);
    const double r0 = __ldg(P[0] + q), r1 = __ldg(P[0] + qm);
    const double rh = c0 * r0 + c1 * r1;
    if (kn > kmin && kn <= kmax) {
      const double rgh = gam_at(CG.RGAMH, q), rsq = __ldg(CG.RGSQRTH + q);
      const double z0 = __ldg(cz + q), z1 = __ldg(cz + n + q), z2 = __ldg(cz + 2 * n + q), z3 = __ldg(cz + 3 * n + q),
                   z4 = __ldg(cz + 4 * n + q), z5 = __ldg(cz + 5 * n + q);
      const double px = __ldg(P[1] + q), pxm = __ldg(P[1] + qm), py = __ldg(P[2] + q), pym = __ldg(P[2] + qm),
                   pz = __ldg(P[3] + q), pzm = __ldg(P[3] + qm);
      const double hA = z0 * px + z1 * pxm + z2 * py + z3 * pym + z4 * pz + z5 * pzm;
      r.vA = hA * rgh + 1.0 * w * rsq;
      const double hE = z0 * (px * e) + z1 * (pxm * em) + z2 * (py * e) + z3 * (pym * em) + z4 * (pz * e) +
                        z5 * (pzm * em);
      r.vE = hE * rgh + 1.0 * (w * (cC.afact[kn] * e + cC.bfact[kn] * em)) * rsq;
      // vertical kinetic-energy term of rhogkin
      r.vint = 0.5 * (w * w) / rh;
      // buoyancy and vertical pressure gradient
      r.dbuo = -GRAV * (c0 * __ldg(a.rhogd + q) + c1 * __ldg(a.rhogd + qm));
      r.dpgw = gam_at(CG.GAM2H, q) * (__ldg(a.pregd + q) * __ldg(CG.RGSGAM2 + q) - __ldg(a.pregd + qm) * __ldg(CG.RGSGAM2 + qm)) *
               cC.rdgzh[kn];
    }
    r.gz = GRAV - (r.dpgw - r.dbuo) / rh;
    r.pwh = -r.gz * w;
    r.eh = cC.afact[kn] * e + cC.bfact[kn] * em;
    return r;
  };
  double gzm = 0.0, ehm = 0.0;
  if (ka > 0) {
    const Half x = half(ka - 1);
    gzm = x.gz;
    ehm = x.eh;
  }
  Half h0 = half(ka);
  for (int k = ka; k < kb; ++k) {
    const int p = c.at(k);
    const Half h1 = half(k + 1);   // zero at KA
    // ---- level k
    const bool hk = in && k >= kmin && k <= kmax;
    const bool kin = k >= kmin && k <= kmax;
    // every load of the level before its stores
    double hv[8], g[6];
#pragma unroll
    for (int d = 0; d < 8; ++d) hv[d] = hk ? __ldg(h.out[d] + p) : R(0.0);
#pragma unroll
    for (int d = 0; d < 6; ++d) g[d] = __ldg(a.gT0[d] + p);
    const double rg0 = __ldg(P[0] + p), eth = __ldg(a.eth + p), phi = __ldg(CG.PHI + p);
    const double* dd = hv + 2;
    const double* dpg = hv + 5;
    double pw = 0.0, drhog = 0.0, drhoge = 0.0, kin0 = 0.0;
    if (kin) {
      drhog = -hv[0] - (h1.vA - h0.vA) * cC.rdgz[k];
      drhoge = -hv[1] - (h1.vE - h0.vE) * cC.rdgz[k];
      const double w0 = __ldg(w2c + p), w1 = __ldg(w2c + n + p);
      pw = __ldg(a.vx + p) * dpg[0] + __ldg(a.vy + p) * dpg[1] + __ldg(a.vz + p) * dpg[2] + w0 * h1.pwh + w1 * h0.pwh;
      const double vx = __ldg(P[1] + p), vy = __ldg(P[2] + p), vz = __ldg(P[3] + p);
      const double kh = 0.5 * (vx * vx + vy * vy + vz * vz) / rg0;
      kin0 = kh + w0 * h1.vint + w1 * h0.vint;
    }
    if (k >= kmin + 1 && k <= kmax) {
      const int pm = c.at(k - 1), pp = c.at(k + 1);
      const double rg = cC.rdgz[k], rgm = cC.rdgz[k - 1];
      const double rs = __ldg(CG.RGSGAM2 + p);
      const double Ca = (rs * rg + __ldg(CG.RGSGAM2 + pm) * rgm) * gam_at(CG.GAM2H, p);
      const double Cb = cC.dfact[k] - cC.cfact[k - 1];
      const double Cu1 = rs * rg * gam_at(CG.GAM2H, pp);
      const double rgh2 = gam_at(CG.RGAMH, p) * gam_at(CG.RGAMH, p);
      const double Cu2 = gam_at(CG.GAM2H, pp) * rgh2 * GCVovR;
      const double Cl1 = rs * rg * gam_at(CG.GAM2H, pm);
      const double Cl2 = gam_at(CG.GAM2H, pm) * rgh2 * GCVovR;
      const double rgh = cC.rdgzh[k];
      a.Mc[p] = ACVovRt2 / __ldg(CG.RGSQRTH + p) + rgh * (Ca * h0.eh - Cb * (h0.gz + GCVovR));
      a.Mu[p] = -rgh * (Cu1 * h1.eh + cC.cfact[k] * (h1.gz + Cu2));
      a.Ml[p] = -rgh * (Cl1 * ehm - cC.dfact[k - 1] * (gzm + Cl2));
    }
    a.gT[0][p] = g[0] + drhog;
    a.gT[1][p] = g[1] - dpg[0] + dd[0] + 0.0;
    a.gT[2][p] = g[2] - dpg[1] + dd[1] + 0.0;
    a.gT[3][p] = g[3] - dpg[2] + dd[2] + 0.0;
    a.gT[4][p] = g[4] + 0.0 * cC.alpha - h0.dpgw + h0.dbuo;
    a.gT[5][p] = g[5] + drhoge + pw;
    a.ethtot0[p] = eth + kin0 / rg0 + phi;
    gzm = h0.gz;
    ehm = h0.eh;
    h0 = h1;
  }
}

// ---------------------------------------------------------------------------
// acoustic loop, path1 (kernels/vipath1.py:68-160): diff_vh with BNDCND and
// the running mean of the horizontal momentum.
// ---------------------------------------------------------------------------
template <class R>
struct Path1Args {
  const R* PS[6];     // PROG_split (RHOGE boundary rows read clamped)
  const R* rhog;      // PROG rhog
  const R* gT[6];
  CThree<R> vt;               // post-COMM 3-D divdamp of PROG_split
  R* dvh[3];          // out
  R* PM[5];           // running mean (in/out)
  R dt, rweight, RovCV;
};

// One pole point; the points at kmin and kmax also write the boundary rows
// kmin-1 and kmax+1 from their values.
template <class R>
__global__ void k_path1_pl(const __grid_constant__ Path1Args<R> a) {
  Pt q_;
  if (!pole_point((int)(blockIdx.x * blockDim.x + threadIdx.x), q_)) return;
  const int g = q_.g, lp = q_.lp, k = q_.k;
  const Col c = col_pl(g, lp);
  const MetT<R> m = met_of<R>(true);
  const int kmin = cD.kmin, kmax = cD.kmax;
  if (k == kmin - 1 || k == kmax + 1) return;
  auto pregs = [&](int gg, int kk) -> R {  // preg_prim_split with clamped boundary rows
    const int k2 = kk < kmin ? kmin : (kk > kmax ? kmax : kk);
    return a.PS[5][ipl(gg, k2, lp)] * a.RovCV;
  };
  const int p = c.at(k);
  R dd[3], pg[3];
  divdamp2d_pl_at(a.vt, g, k, lp, dd);
  presgrad_pl(g, k, lp, c, m, pregs, pg);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const R drv = a.gT[1 + d][p] - pg[d] + dd[d] + R(0.0);
    const R v = a.PS[1 + d][p] + drv * a.dt;
    a.dvh[d][p] = v;
    a.PM[1 + d][p] = a.PM[1 + d][p] + v * a.rweight;
    if (k == kmin) {
      const int pB = c.at(kmin - 1);
      const R vB = -R(1.0) * (v / a.rhog[p]) * a.rhog[pB];
      a.dvh[d][pB] = vB;
      a.PM[1 + d][pB] = a.PM[1 + d][pB] + vB * a.rweight;
    }
    if (k == kmax) {
      const int pT = c.at(kmax + 1);
      const R vT = R(1.0) * (v / a.rhog[p]) * a.rhog[pT];
      a.dvh[d][pT] = vT;
      a.PM[1 + d][pT] = a.PM[1 + d][pT] + vT * a.rweight;
    }
  }
}

// Regional path 1, one block per (NK levels, tile): same stencils and
// arithmetic as k_path1_pl.  The kernel is bound by the instructions it issues
// (920 a point for one level per block, a third of them the addresses and
// loads of the 60 coefficient planes), so each coefficient is loaded once and
// applied to the block's NK levels, whose sums run side by side.  The levels
// kmin and kmax also write the boundary rows kmin-1 and kmax+1 from the values
// they computed.
#ifndef P1_NK_F32
#define P1_NK_F32 4
#define P1_MINB_F32 3
#endif
#ifndef P1_NK_F64
#define P1_NK_F64 2
#define P1_MINB_F64 4
#endif
template <class R> constexpr int P1_NK = sizeof(R) == 8 ? P1_NK_F64 : P1_NK_F32;
template <class R> constexpr int P1_MINB = sizeof(R) == 8 ? P1_MINB_F64 : P1_MINB_F32;
template <class R, class T, int NK, int MINB>
__global__ void __launch_bounds__(TILE_THREADS, MINB) k_path1_l(Path1Args<R> a) {
  constexpr int PX = T::X + 2, PY = T::Y + 2, TX = T::X + 1, TY = T::Y + 1, NP = PX * PY, NT = TX * TY;
  __shared__ R s_v[NK][3][NP];
  __shared__ R s_p[NK][NP];
  __shared__ R s_ti[NK][NT], s_tj[NK][NT];
  const TileLv tl = tile_level<T>(0);
  const int l = tl.l, i0 = tl.i0, j0 = tl.j0;
  const int G = cD.G, gmax = cD.G - 2, kmin = cD.kmin, kmax = cD.kmax;
  const int ka = kmin + tl.k * NK;
  const int tid = threadIdx.x, tx = tid % T::X, ty = tid / T::X;
  const R RovCV = a.RovCV;
  for (int p = tid; p < NP; p += blockDim.x) {
    const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
    const bool ok = ii < G && jj < G;
    const int q0 = ok ? ix(ii, jj, 0, l) : 0;
#pragma unroll
    for (int n = 0; n < NK; ++n) {
      const int k = min(ka + n, kmax), kk = (k == kmin) ? kmin + 1 : k;   // a level past kmax repeats it
      const int q = q0 + k * cD.planei, qk = q0 + kk * cD.planei;
      s_v[n][0][p] = ok ? -__ldg(&a.vt.f[0][q]) : R(0.0);
      s_v[n][1][p] = ok ? -__ldg(&a.vt.f[1][q]) : R(0.0);
      s_v[n][2][p] = ok ? -__ldg(&a.vt.f[2][q]) : R(0.0);
      s_p[n][p] = ok ? __ldg(&a.PS[5][qk]) * RovCV * __ldg(&CG.RGAM[qk]) : R(0.0);
    }
  }
  __syncthreads();
  for (int p = tid; p < NT; p += blockDim.x) {
    const int px = p % TX, py = p / TX;
    const int ii = i0 - 1 + px, jj = j0 - 1 + py;
    R sI[NK], sJ[NK];
#pragma unroll
    for (int n = 0; n < NK; ++n) sI[n] = sJ[n] = R(0.0);
    if (ii <= G - 2 && jj <= G - 2) {
      const int ia = py * PX + px;
      const int vI[3] = {ia, ia + 1, ia + PX + 1}, vJ[3] = {ia, ia + PX + 1, ia + PX};
#pragma unroll
      for (int m = 0; m < 9; ++m) {   // direction m / 3, vertex m % 3, left to right
        const R cI = P2c(CG.coef_intp, m * 2, ii, jj, l), cJ = P2c(CG.coef_intp, m * 2 + 1, ii, jj, l);
#pragma unroll
        for (int n = 0; n < NK; ++n) {
          const R xI = s_v[n][m / 3][vI[m % 3]], xJ = s_v[n][m / 3][vJ[m % 3]];
          sI[n] = m ? mad(cI, xI, sI[n]) : cI * xI;
          sJ[n] = m ? mad(cJ, xJ, sJ[n]) : cJ * xJ;
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NK; ++n) {
      s_ti[n][p] = sI[n];
      s_tj[n][p] = sJ[n];
    }
  }
  __syncthreads();
  const int i = i0 + tx, j = j0 + ty;
  if (i > gmax || j > gmax) return;
  const R ddc = CC.divdamp_coef, dt = a.dt, rweight = a.rweight;
  const int npt = cD.npti;
  const R* cz = CG.C2WGz;
  const R gx = P2c(CG.GRD_x, 0, i, j, l), gy = P2c(CG.GRD_x, 1, i, j, l), gz = P2c(CG.GRD_x, 2, i, j, l);
  const int q0 = ix(i, j, 0, l);
  const int ta = (ty + 1) * TX + (tx + 1), c0 = (ty + 1) * PX + (tx + 1);
  R dd[NK][3], pg[NK][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      const R cf = P2c(CG.coef_diff, d * 6 + e, i, j, l);
#pragma unroll
      for (int n = 0; n < NK; ++n) {
        const R* I = s_ti[n];
        const R* J = s_tj[n];
        const R x = e == 0 ? I[ta] + J[ta] : e == 1 ? J[ta] + I[ta - 1] : e == 2 ? I[ta - 1] + J[ta - TX - 1]
                  : e == 3 ? J[ta - TX - 1] + I[ta - TX - 1] : e == 4 ? I[ta - TX - 1] + J[ta - TX] : J[ta - TX] + I[ta];
        dd[n][d] = e ? mad(cf, x, dd[n][d]) : cf * x;
      }
    }
  }
  const int nb[7] = {c0, c0 + 1, c0 + PX + 1, c0 + PX, c0 - 1, c0 - PX - 1, c0 - PX};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int m = 0; m < 7; ++m) {
      const R cf = P2c(CG.coef_grad, d * 7 + m, i, j, l);
#pragma unroll
      for (int n = 0; n < NK; ++n) pg[n][d] = m ? mad(cf, s_p[n][nb[m]], pg[n][d]) : cf * s_p[n][nb[m]];
    }
  }
  auto flat = [&](R* x) {   // tangent-plane projection
    const R prd = div_r(x[0] * gx + x[1] * gy + x[2] * gz);
    x[0] = x[0] - div_r(prd * gx);
    x[1] = x[1] - div_r(prd * gy);
    x[2] = x[2] - div_r(prd * gz);
  };
  auto Pown = [&](int k2) {
    const int kc = k2 < kmin ? kmin : (k2 > kmax ? kmax : k2);
    return __ldg(&a.PS[5][q0 + kc * cD.planei]) * RovCV;
  };
#pragma unroll
  for (int n = 0; n < NK; ++n) {
    const int k = ka + n, kk = (k == kmin) ? kmin + 1 : k;
    if (k > kmax) return;
    const int qkk = q0 + kk * cD.planei, qk1 = qkk + cD.planei;
    const R P_k1 = Pown(kk + 1), P_k = Pown(kk), P_km = Pown(kk - 1);
    const R rgh1 = __ldg(&CG.RGAMH[qk1]), rgh0 = __ldg(&CG.RGAMH[qkk]);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      dd[n][d] = ddc * dd[n][d];
      const R up = mad(__ldg(&cz[(2 * d + 1) * npt + qk1]), P_k, __ldg(&cz[(2 * d) * npt + qk1]) * P_k1) * rgh1;
      const R dn = mad(__ldg(&cz[(2 * d + 1) * npt + qkk]), P_km, __ldg(&cz[(2 * d) * npt + qkk]) * P_k) * rgh0;
      pg[n][d] = pg[n][d] + (up - dn) * CC.rdgz[kk];
    }
    flat(dd[n]);
    flat(pg[n]);
    const int q = q0 + k * cD.planei;
    R v[3], pm[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const R drv = __ldg(&a.gT[1 + d][q]) - pg[n][d] + dd[n][d] + R(0.0);
      v[d] = __ldg(&a.PS[1 + d][q]) + drv * dt;
      pm[d] = a.PM[1 + d][q];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a.dvh[d][q] = v[d];
      a.PM[1 + d][q] = pm[d] + v[d] * rweight;
    }
    if (k == kmin) {
      const int pB = q - cD.planei;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const R vB = -R(1.0) * (v[d] / __ldg(&a.rhog[q])) * __ldg(&a.rhog[pB]);
        a.dvh[d][pB] = vB;
        a.PM[1 + d][pB] = a.PM[1 + d][pB] + vB * rweight;
      }
    }
    if (k == kmax) {
      const int pT = q + cD.planei;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const R vT = R(1.0) * (v[d] / __ldg(&a.rhog[q])) * __ldg(&a.rhog[pT]);
        a.dvh[d][pT] = vT;
        a.PM[1 + d][pT] = a.PM[1 + d][pT] + vT * rweight;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// vi_main (kernels/vimain.py:127-262): horizontal divergences (kernel A),
// then per column the flux convergences, the tridiagonal Thomas solve
// (kernels/virhowsolver.py:42-120), kinetic energies and the energy update.
// ---------------------------------------------------------------------------
template <class R>
struct VimainArgs {
  const R* PS[6];
  const R* P[6];          // PROG
  const R *eth, *ethtot0;
  const R* gT[6];         // small-step tendency
  const R* gT0e;          // large-step tendency of RHOGE (grhogetot)
  const double *Mc, *Mu, *Ml;  // float64 in both forms
  CThree<R> dvh;                  // post-COMM diff_vh
  R* hdiv[3];             // kernel A output
  R* dwe[3];              // out: rhog_s1, rhogw_s1, rhoge_s1
  R* PM0;                 // running mean of RHOG (in/out)
  R* PM4;                 // running mean of RHOGW (in/out)
  double dt, rweight, RovCV;
};

template <class R>
__global__ void k_vimain_a_pl(const __grid_constant__ VimainArgs<R> a) {
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t < cD.KA * cD.LP) {
    const int k = t / cD.LP, lp = t % cD.LP;
    for (int g = 0; g < 6; ++g) {
      const int p = ipl(g, k, lp);
      R h1 = R(0.0), h2 = R(0.0), h3 = R(0.0);
      if (g == 0 && k >= cD.kmin && k <= cD.kmax) {
        h1 = div_pl<R>(lp, k, [&](int q, int d) { return a.dvh.f[d][q]; });
        h2 = div_pl<R>(lp, k, [&](int q, int d) { return a.dvh.f[d][q] * a.eth[q]; });
        h3 = div_pl<R>(lp, k, [&](int q, int d) { return (a.P[1 + d][q] + a.dvh.f[d][q]) * a.ethtot0[q]; });
      }
      a.hdiv[0][p] = h1; a.hdiv[1][p] = h2; a.hdiv[2][p] = h3;
    }
  }
}

// vi_main kernel A, one block per (level, tile): the horizontal divergences
// of RGAM*diff_vh, RGAM*diff_vh*eth and RGAM*(rhogv + diff_vh)*ethtot0 (the
// double form; the float form marches, see k_vimain_a_m).
template <class R, class T>
__global__ void __launch_bounds__(TILE_THREADS, 6) k_vimain_a_l(VimainArgs<R> a) {
  constexpr int PX = T::X + 2, PY = T::Y + 2;
  __shared__ R s_h[3][3][PY * PX];
  const TileLv tl = tile_level<T>(cD.kmin);
  const int l = tl.l, i0 = tl.i0, j0 = tl.j0;
  const int G = cD.G, gmax = cD.G - 2;
  const int tid = threadIdx.x, tx = tid % T::X, ty = tid / T::X;
  const int i = i0 + tx, j = j0 + ty;
  const bool own = (i <= gmax) && (j <= gmax);
  {
    const int k = tl.k;
    for (int p = tid; p < PX * PY; p += blockDim.x) {
      const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
      if (ii < G && jj < G) {
        const int q = ix(ii, jj, k, l);
        const R rg = gam_at_ldg(CG.RGAM, q), e = __ldg(&a.eth[q]), et = __ldg(&a.ethtot0[q]);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const R dv = __ldg(&a.dvh.f[d][q]);
          s_h[0][d][p] = dv * rg;
          s_h[1][d][p] = (dv * e) * rg;
          s_h[2][d][p] = ((__ldg(&a.P[1 + d][q]) + dv) * et) * rg;
        }
      } else {
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
          for (int d = 0; d < 3; ++d) s_h[f][d][p] = R(0.0);
      }
    }
    __syncthreads();
    if (own) {
      const int c0 = (ty + 1) * PX + (tx + 1);
      const int nb[7] = {c0, c0 + 1, c0 + PX + 1, c0 + PX, c0 - 1, c0 - PX - 1, c0 - PX};
      const int q = ix(i, j, k, l);
      R acc[3][3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        R s[3] = {R(0.0), R(0.0), R(0.0)};
#pragma unroll
        for (int m = 0; m < 7; ++m) {
          const R cdv = P2c(CG.coef_div, d * 7 + m, i, j, l);
#pragma unroll
          for (int f = 0; f < 3; ++f) {
            const R t = cdv * s_h[f][d][nb[m]];
            s[f] = (m == 0) ? t : s[f] + t;
          }
        }
#pragma unroll
        for (int f = 0; f < 3; ++f) acc[f][d] = s[f];
      }
#pragma unroll
      for (int f = 0; f < 3; ++f) a.hdiv[f][q] = acc[f][0] + acc[f][1] + acc[f][2];
    }
    __syncthreads();
  }
}

// vi_main A with VA_NK levels per block, the float form: the cell's divergence
// coefficients (coef_div, 21 planes) are held in registers once for the block's
// levels, and the next level's loads are in flight while this level is worked on
// (two levels of products in shared memory, one barrier a level).  Same
// expressions in the same order as k_vimain_a_l.
// Bound by the latency of a level's staging: gl08 z40 489 -> 387 us, gl06 z40
// 41 -> 33 us, 12 x gl05 129 -> 109 us against the march that staged a level
// between two barriers.  Ten levels a block: 400 us at gl08, 37 at gl06; five
// blocks an SM instead of four (spills): 460 us.  The double form stays on
// k_vimain_a_l: 224 against 221 us at gl07 z40, 25 against 23 at gl05.
#define VA_NK 5
template <class R, class T>
__global__ void __launch_bounds__(TILE_THREADS, 4) k_vimain_a_m(const __grid_constant__ VimainArgs<R> a) {
  constexpr int PX = T::X + 2, PY = T::Y + 2, NP = PX * PY, PT = (NP + TILE_THREADS - 1) / TILE_THREADS;
  __shared__ R s_h[2][9][NP];   // [field * 3 + direction], two levels
  const int ntx = (cD.G - 2 + T::X - 1) / T::X;
  const int l = (int)blockIdx.z;
  const int i0 = 1 + ((int)blockIdx.y % ntx) * T::X, j0 = 1 + ((int)blockIdx.y / ntx) * T::Y;
  const int ka = cD.kmin + (int)blockIdx.x * VA_NK, kb = min(ka + VA_NK - 1, cD.kmax);
  const int G = cD.G, gmax = cD.G - 2;
  const int tid = threadIdx.x, tx = tid % T::X, ty = tid / T::X;
  const int i = i0 + tx, j = j0 + ty;
  const bool own = (i <= gmax) && (j <= gmax);
  R w[PT][9];   // a level's staged points of the thread on their way to shared memory
  auto fetch = [&](int k) {
#pragma unroll
    for (int e = 0; e < PT; ++e) {
      const int p = tid + e * TILE_THREADS;
      const int ii = i0 - 1 + p % PX, jj = j0 - 1 + p / PX;
      const bool ok = p < NP && ii < G && jj < G;
      const int q = ok ? ix(ii, jj, k, l) : 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        w[e][d] = ok ? __ldg(&a.dvh.f[d][q]) : R(0.0);
        w[e][3 + d] = ok ? __ldg(&a.P[1 + d][q]) : R(0.0);
      }
      w[e][6] = ok ? __ldg(&a.eth[q]) : R(0.0);
      w[e][7] = ok ? __ldg(&a.ethtot0[q]) : R(0.0);
      w[e][8] = ok ? gam_at_ldg(CG.RGAM, q) : R(0.0);
    }
  };
  auto put = [&](int b) {
#pragma unroll
    for (int e = 0; e < PT; ++e) {
      const int p = tid + e * TILE_THREADS;
      if (p < NP) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const R dv = w[e][d], rg = w[e][8];
          s_h[b][d][p] = dv * rg;
          s_h[b][3 + d][p] = (dv * w[e][6]) * rg;
          s_h[b][6 + d][p] = ((w[e][3 + d] + dv) * w[e][7]) * rg;
        }
      }
    }
  };
  R cdv[21];
  if (own) {
#pragma unroll
    for (int m = 0; m < 21; ++m) cdv[m] = P2c(CG.coef_div, m, i, j, l);
  }
  int b = 0;
  fetch(ka);
  put(0);
  __syncthreads();
  for (int k = ka; k <= kb; ++k, b ^= 1) {
    if (k < kb) fetch(k + 1);
    if (own) {
      const int c0 = (ty + 1) * PX + (tx + 1);
      const int nb[7] = {c0, c0 + 1, c0 + PX + 1, c0 + PX, c0 - 1, c0 - PX - 1, c0 - PX};
      const int q = ix(i, j, k, l);
      R acc[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        R sv[3];
#pragma unroll
        for (int m = 0; m < 7; ++m) {
#pragma unroll
          for (int f = 0; f < 3; ++f) {
            const R x = s_h[b][f * 3 + d][nb[m]];
            sv[f] = (m == 0) ? cdv[d * 7 + m] * x : mad(cdv[d * 7 + m], x, sv[f]);
          }
        }
#pragma unroll
        for (int f = 0; f < 3; ++f) acc[f] = (d == 0) ? sv[f] : acc[f] + sv[f];
      }
#pragma unroll
      for (int f = 0; f < 3; ++f) a.hdiv[f][q] = acc[f];
    }
    if (k < kb) put(b ^ 1);
    __syncthreads();
  }
}

// vi_main, column part: flux convergences of diff_vh, the Thomas solve
// (kernels/virhowsolver.py:42-120), rhog_split1, the kinetic energies and the
// energy update, for the interior regional columns (the halo columns of the
// outputs are replaced by the exchange that follows) and the pole columns.
//
// One block takes VC_COLS columns (a lane each) and splits the levels over its
// warps: each warp assembles the right-hand side of its levels marching upward,
// warp 0 walks the two sweeps of the elimination on operands in shared memory
// (five doubles per level and column: 54 KB at 42 levels), then each warp
// finishes its levels, again marching upward; a part of the column repeats one
// level (assembly) or two (finish) of its neighbour instead of exchanging them.
// Bound by memory latency: a warp waits for each level's loads, and a column per
// thread (a kernel for the solve and a point kernel for the energies) was bound
// by its chain of loads and divisions besides (6 us a level on small grids) and
// kept the sweep's factors in local memory.  So every level's loads stand before
// its arithmetic, under no condition and as read-only loads, which the stores of
// the level below cannot hold up; the finish finds what both parts read in L2.
// Launch bounds: two blocks an SM in double (128 registers; three: spills, 1.12
// against 0.71 ms at gl07 z40), three in float (two: 1.87, four: 2.89 against
// 1.63 ms at gl08 z40).
// One layer of 40 levels, solve and energies, two kernels -> this one: gl05
// float64 287 -> 83 us, gl06 mixed 307 -> 125 us, gl07 float64 1049 -> 705 us,
// gl08 mixed 2065 -> 1627 us.
// Slots, by level (kmin..kmax+1) and lane:
//   0 horizontal part of the half-level mass flux
//   1 the right-hand side, then the solution
//   2 Mu, then the sweep's gamma      3 Ml      4 Mc
// DEEP, for tall columns: the first three slots alone (98 KB at 128 levels).  The
// sweep then reads the matrix from memory, VC_PF levels ahead of the ones it works
// on (eight instead of four spill in float: gl07 z80 0.91 -> 1.22 ms).  Five slots a
// level take a block of 82 levels to 105 KB: fewer blocks an SM, or hardly any L1
// beside them.  A step's eleven launches at gl07, the two kernels before / five
// slots / three: float64 82 levels 23.1 / 24.7 / 15.8 ms, 128 levels 36.9 / 33.4 /
// 24.6 (five: one block); mixed 82 levels 16.0 / 15.3 / 10.0, 128 levels 25.1 /
// 29.8 / 18.4.
#define VC_COLS 32
#define VC_MAXW 8
#define VC_PF 4
static inline size_t vi_col_smem(int KA, bool deep) { return (size_t)(deep ? 3 : 5) * KA * VC_COLS * sizeof(double); }

// the contiguous part [lo, hi) of the levels first..last that a warp takes
__device__ __forceinline__ void warp_levels(int first, int last, int& lo, int& hi) {
  const int nw = (int)(blockDim.x / 32), w = (int)(threadIdx.x / 32);
  const int per = (last - first + nw) / nw;
  lo = first + w * per;
  hi = min(lo + per, last + 1);
}

template <class R, bool GU, bool POLE, bool DEEP>
__device__ __forceinline__ void vi_col(const VimainArgs<R>& a, int blk, double* sm) {
  const int KA = cD.KA, kmin = cD.kmin, kmax = cD.kmax, kT = kmax + 1;
  const int lane = (int)(threadIdx.x % 32);
  const int ni = cD.G - 2;
  const int ncol = POLE ? 6 * cD.LP : cD.L * ni * ni;
  const int t0 = blk * VC_COLS + lane;
  const bool act = t0 < ncol;              // surplus lanes repeat the last column and store nothing
  const int t = act ? t0 : ncol - 1;
  const Col c = POLE ? col_pl(t / cD.LP, t % cD.LP) : col_reg(1 + t % ni, 1 + (t / ni) % ni, t / (ni * ni));
  const MetT<R> m = met_of<R>(POLE);
  const double dt = a.dt, Rdry = cC.Rdry, CVdry = cC.CVdry, RovCV = a.RovCV;
  const R* const* DV = a.dvh.f;
  // the pole columns form fluxes, rhog_split1 and the running means in R, the
  // regional ones in double
  using F = typename std::conditional<POLE, R, double>::type;
  const F rweight = F(a.rweight);
  auto rdgz = [](int k) -> F { return POLE ? F(CC.rdgz[k]) : F(cC.rdgz[k]); };
  double* s0 = sm + lane;
  double* s1 = s0 + KA * VC_COLS;
  double* s2 = s1 + KA * VC_COLS;
  double* s3 = s2 + KA * VC_COLS;   // not there with DEEP
  double* s4 = s3 + KA * VC_COLS;
  auto S = [](double* s, int k) -> double& { return s[k * VC_COLS]; };
  auto cz = [&](int comp, int q) -> R { return __ldg(POLE ? m.C2WGz + q * 6 + comp : m.C2WGz + comp * cD.npti + q); };
  auto two = [&](const R* w, int comp, int q) -> R { return __ldg(POLE ? w + q * 2 + comp : w + comp * cD.npti + q); };
  int lo, hi;
  // ---- right-hand side on kmin+1..kmax.  Every level's loads stand before its
  // arithmetic and under no condition (indices clamped to the column), so that
  // a level waits for memory once.
  warp_levels(kmin + 1, kmax, lo, hi);
  if (lo < hi) {
    const double CVovRt2 = CVdry / Rdry / (dt * dt);
    R m0, m1, m2, me;                     // diff_vh and eth one level below
    R f0, f1, f2, fe, z0, z1, z2, z3, z4, z5, gh;
    auto load = [&](int k) {
      const int q = c.at(k);
      f0 = __ldg(DV[0] + q); f1 = __ldg(DV[1] + q); f2 = __ldg(DV[2] + q); fe = __ldg(a.eth + q);
      z0 = cz(0, q); z1 = cz(1, q); z2 = cz(2, q); z3 = cz(3, q); z4 = cz(4, q); z5 = cz(5, q);
      gh = GU ? R(1.0) : __ldg(m.RGAMH + q);
    };
    auto flux = [&](F& hd, F& he) {   // half-level fluxes at the loaded level
      const F a0 = f0, a1 = f1, a2 = f2, e = fe, b0 = m0, b1 = m1, b2 = m2, em = me;
      hd = (z0 * a0 + z1 * b0 + z2 * a1 + z3 * b1 + z4 * a2 + z5 * b2) * (F)gh;
      he = (z0 * (a0 * e) + z1 * (b0 * em) + z2 * (a1 * e) + z3 * (b1 * em) + z4 * (a2 * e) + z5 * (b2 * em)) * (F)gh;
    };
    {
      const int q = c.at(lo - 2);
      m0 = __ldg(DV[0] + q); m1 = __ldg(DV[1] + q); m2 = __ldg(DV[2] + q); me = __ldg(a.eth + q);
    }
    load(lo - 1);
    F hD, hE;
    flux(hD, hE);
    if (lo - 1 == kmin) hD = hE = F(0.0);    // zero at kmin and at kmax+1
    m0 = f0; m1 = f1; m2 = f2; me = fe;
    double T1m = 0.0, T2m = 0.0;
    for (int k = lo - 1; k < hi; ++k) {
      const int p = c.at(k);
      load(k + 1);
      const R hd0 = __ldg(a.hdiv[0] + p), hd1 = __ldg(a.hdiv[1] + p), g0 = __ldg(a.gT[0] + p), g5 = __ldg(a.gT[5] + p);
      const R ps5 = __ldg(a.PS[5] + p), ps0 = __ldg(a.PS[0] + p), rs2 = __ldg(m.RGSGAM2 + p);
      const R g4 = __ldg(a.gT[4] + p), ps4 = __ldg(a.PS[4] + p);
      const double mu = !DEEP || k == kmax ? __ldg(a.Mu + p) : 0.0, ml = !DEEP || k == kmin + 1 ? __ldg(a.Ml + p) : 0.0;
      const double mcc = DEEP ? 0.0 : __ldg(a.Mc + p);
      const double rgm = GU ? 1.0 : (double)__ldg(m.RGAM + p), rgh = GU ? 1.0 : (double)__ldg(m.RGAMH + p);
      F hDn, hEn;
      flux(hDn, hEn);
      if (k == kmax) hDn = hEn = F(0.0);
      const double drhog = -hd0 - (hDn - hD) * rdgz(k);
      const double drhoge = -hd1 - (hEn - hE) * rdgz(k);
      const double g1 = g0 + drhog;
      const double gp = (g5 + drhoge) * Rdry / CVdry;
      const double T1 = (ps5 * RovCV + dt * gp) * rs2;
      const double T2 = (ps0 + dt * g1) * (rgm * rgm);
      if (k >= lo) {
        const double Sw = g4 + 0.0 * cC.alpha;
        double b = ((ps4 * cC.alpha + dt * Sw) * (rgh * rgh) - (T1 - T1m) * dt * cC.rdgzh[k] -
                    (T2 * cC.afact[k] + T2m * cC.bfact[k]) * dt * cC.GRAV) *
                   CVovRt2;
        if (k == kmin + 1) {
          const double rw_kmin = 0.0 * __ldg(m.RGSGAM2H + c.at(kmin));
          b = b - ml * rw_kmin;
          S(s1, kmin) = rw_kmin;
        }
        if (k == kmax) {   // the loaded level is kmax+1
          using W = typename std::conditional<POLE, double, R>::type;   // as the fluxes, the other way round
          const double top = -(W(z0) * f0 + W(z1) * m0 + W(z2) * f1 + W(z3) * m1 + W(z4) * f2 + W(z5) * m2);
          const double rw_top = top * __ldg(m.RGSGAM2H + c.at(kT));
          b = b - mu * rw_top;
          S(s1, kT) = rw_top;
        }
        S(s0, k) = hD;
        S(s1, k) = b;
        if (!DEEP) {
          S(s2, k) = mu;
          S(s3, k) = ml;
          S(s4, k) = mcc;
        }
      }
      T1m = T1; T2m = T2; hD = hDn; hE = hEn;
      m0 = f0; m1 = f1; m2 = f2; me = fe;
    }
  }
  __syncthreads();
  // ---- Thomas sweeps, one lane per column; the operands of the next level are
  // read before this level's are overwritten
  if (threadIdx.x < 32) {
    const int k0 = kmin + 1;
    double u;
    if constexpr (DEEP) {
      double mc_[VC_PF], mu_[VC_PF], ml_[VC_PF];
      auto fetch = [&](int k) {
#pragma unroll
        for (int e = 0; e < VC_PF; ++e) {
          const int p = c.at(min(k + e, kmax));
          mc_[e] = __ldg(a.Mc + p); mu_[e] = __ldg(a.Mu + p); ml_[e] = __ldg(a.Ml + p);
        }
      };
      double beta = __ldg(a.Mc + c.at(k0)), mu = __ldg(a.Mu + c.at(k0));
      fetch(k0 + 1);
      u = S(s1, k0) / beta;
      S(s1, k0) = u;
      for (int k = k0 + 1; k <= kmax; k += VC_PF) {
        double mc0[VC_PF], mu0[VC_PF], ml0[VC_PF];
#pragma unroll
        for (int e = 0; e < VC_PF; ++e) { mc0[e] = mc_[e]; mu0[e] = mu_[e]; ml0[e] = ml_[e]; }
        if (k + VC_PF <= kmax) fetch(k + VC_PF);
#pragma unroll
        for (int e = 0; e < VC_PF; ++e) {
          if (k + e > kmax) break;
          const double gg = mu / beta;
          beta = mc0[e] - ml0[e] * gg;
          u = (S(s1, k + e) - ml0[e] * u) / beta;
          S(s2, k + e - 1) = gg;      // gamma of level k + e
          S(s1, k + e) = u;
          mu = mu0[e];
        }
      }
    } else {
      double beta = S(s4, k0);
      u = S(s1, k0) / beta;
      double mu = S(s2, k0);
      double mc_ = S(s4, k0 + 1), ml = S(s3, k0 + 1), b = S(s1, k0 + 1), mu1 = S(s2, k0 + 1);   // k0+1 <= kT < KA
      S(s1, k0) = u;
      for (int k = k0 + 1; k <= kmax; ++k) {
        const int kn = min(k + 1, kmax);
        const double mcn = S(s4, kn), mln = S(s3, kn), bn = S(s1, kn), mun = S(s2, kn);
        const double gg = mu / beta;
        beta = mc_ - ml * gg;
        u = (b - ml * u) / beta;
        S(s2, k - 1) = gg;      // gamma of level k beside the level below, whose Mu is spent
        S(s1, k) = u;
        mu = mu1;
        mu1 = mun; mc_ = mcn; ml = mln; b = bn;
      }
    }
    double x = u, un = S(s1, kmax - 1), gn = S(s2, kmax - 1);
    for (int k = kmax - 1; k >= k0; --k) {
      const int kn = max(k - 1, k0);
      const double un1 = S(s1, kn), gn1 = S(s2, kn);
      x = un - gn * x;
      S(s1, k) = x;
      un = un1; gn = gn1;
    }
  }
  __syncthreads();
  // ---- rhogw_split1, rhog_split1, the kinetic energies before and after, the
  // total-energy advection and rhoge_split1 on every level: the march reads level
  // kk, forms its half-level terms with the level below and writes level kk-1
  warp_levels(0, KA - 1, lo, hi);
  if (lo >= hi) return;
  const R dtR = R(dt);
  const int kk0 = max(lo - 1, 0);
  R gs = __ldg(m.GSGAM2H + c.at(kk0)), rq = __ldg(m.RGSQRTH + c.at(kk0));
  // values of level kk-1 (d...) and its half-level terms (h...)
  R drg = R(0.0), dr0 = R(0.0), dr1 = R(0.0), dvx = R(0.0), dvy = R(0.0), dvz = R(0.0), dx = R(0.0), dy = R(0.0),
    dz = R(0.0), det = R(0.0), h10 = R(0.0), h11 = R(0.0), hfl = R(0.0);
  F drs = F(0.0), drw = F(0.0);
  for (int kk = kk0; kk <= hi; ++kk) {
    const int ke = min(kk, KA - 1), kn = min(kk + 1, KA - 1), ko = max(kk - 1, 0);
    const int p = c.at(ke), pn = c.at(kn), po = c.at(ko);
    const R gsn = __ldg(m.GSGAM2H + pn), rqn = __ldg(m.RGSQRTH + pn);
    const R rg = __ldg(a.P[0] + p), vx = __ldg(a.P[1] + p), vy = __ldg(a.P[2] + p), vz = __ldg(a.P[3] + p),
            w = __ldg(a.P[4] + p), r0 = __ldg(a.PS[0] + p), ps4 = __ldg(a.PS[4] + p), et = __ldg(a.ethtot0 + p),
            u0 = __ldg(DV[0] + p), u1 = __ldg(DV[1] + p), u2 = __ldg(DV[2] + p), hd0 = __ldg(a.hdiv[0] + p),
            g0 = __ldg(a.gT[0] + p), c0 = two(m.C2W, 0, p), c1 = two(m.C2W, 1, p), z0 = cz(0, p), z1 = cz(1, p),
            z2 = cz(2, p), z3 = cz(3, p), z4 = cz(4, p), z5 = cz(5, p);
    const R ps1 = __ldg(a.PS[1] + po), ps2 = __ldg(a.PS[2] + po), ps3 = __ldg(a.PS[3] + po), w2c0 = two(m.W2C, 0, po),
            w2c1 = two(m.W2C, 1, po), hd2 = __ldg(a.hdiv[2] + po), g0e = __ldg(a.gT0e + po), phi = __ldg(m.PHI + po),
            re0 = __ldg(a.PS[5] + c.at(min(max(ko, kmin), kmax))), pm0 = a.PM0[po], pm4 = a.PM4[po];
    const R ghh = GU && !POLE ? R(1.0) : gam_at(m.RGAMH, p);
    // rhogw_split1 and its mass flux at the half levels kk and kk+1
    auto rws_at = [&](int k, R g) -> F { return (k >= kmin && k <= kT) ? F(S(s1, k) * g) : F(0.0); };
    auto v2_at = [&](int k, F r, R q) -> F { return (k > kmin && k <= kmax) ? F(S(s0, k)) + F(1.0) * r * q : F(0.0); };
    const F rws = rws_at(ke, gs), rwn = rws_at(kn, gsn);
    const F v2 = v2_at(ke, rws, rq), v2n = v2_at(kn, rwn, rqn);
    const bool in = kk >= kmin && kk <= kmax;
    const F drhog2 = in ? -hd0 - (v2n - v2) * rdgz(ke) : F(0.0);
    const F rs = r0 + (g0 + drhog2) * F(dt);
    const R r1 = R(rs);
    const R x1 = vx + u0, y1 = vy + u1, z1v = vz + u2;
    // between the levels kk and kk-1
    R k10 = R(0.0), k11 = R(0.0), fl = R(0.0);
    if (kk > kmin && kk <= kmax) {
      const R w0 = w + ps4, w1 = w + R(rws);
      k10 = R(0.5) * (w0 * w0) / (c0 * (rg + r0) + c1 * (drg + dr0));
      k11 = R(0.5) * (w1 * w1) / (c0 * (rg + r1) + c1 * (drg + dr1));
      const R f = z0 * (x1 * et) + z1 * (dx * det) + z2 * (y1 * et) + z3 * (dy * det) + z4 * (z1v * et) + z5 * (dz * det);
      fl = f * ghh + R(1.0) * (w1 * (CC.afact[ke] * et + CC.bfact[ke] * det)) * rq;
    }
    if (kk > lo) {   // level kk-1
      R kin10 = R(0.0), kin11 = R(0.0), adv = R(0.0);
      if (ko >= kmin && ko <= kmax) {
        const R x0 = dvx + ps1, y0 = dvy + ps2, z0v = dvz + ps3;
        kin10 = R(0.5) * (x0 * x0 + y0 * y0 + z0v * z0v) / (drg + dr0) + w2c0 * k10 + w2c1 * h10;
        kin11 = R(0.5) * (dx * dx + dy * dy + dz * dz) / (drg + dr1) + w2c0 * k11 + w2c1 * h11;
        adv = -hd2 - (fl - hfl) * CC.rdgz[ko];
      }
      const R re = re0 + (g0e + adv) * dtR + (kin10 - kin11) + (dr0 - dr1) * phi;
      if (act) {
        a.dwe[0][po] = dr1;
        a.dwe[1][po] = R(drw);
        a.dwe[2][po] = re;
        a.PM0[po] = pm0 + drs * rweight;
        a.PM4[po] = pm4 + drw * rweight;
      }
    }
    drg = rg; dr0 = r0; dr1 = r1; dvx = vx; dvy = vy; dvz = vz; dx = x1; dy = y1; dz = z1v; det = et;
    h10 = k10; h11 = k11; hfl = fl;
    drs = rs; drw = rws;
    gs = gsn; rq = rqn;
  }
}

// GU: the gamma factors are all 1 and are not loaded
template <class R, bool GU, bool POLE, bool DEEP>
__global__ void __launch_bounds__(32 * VC_MAXW, NC_MINB(R, 2, 3)) k_vi_col(const __grid_constant__ VimainArgs<R> a) {
  extern __shared__ __align__(16) double vi_sm[];
  vi_col<R, GU, POLE, DEEP>(a, (int)blockIdx.x, vi_sm);
}
// Three slots above 64 levels in float64 and 43 in float, where the five no
// longer fit in 164 KB for the blocks an SM that the registers allow (two and
// three).  A step at gl07, five and three slots: float64 42 levels 7.87 and 8.19 ms,
// 62 11.7 and 12.2, 68 14.0 and 13.3; mixed 42 levels 4.73 and 4.77 ms, 46 5.49
// and 5.23, 52 8.88 and 5.93; gl05 mixed 52 levels 0.89 and 0.57.
#define VI_DEEP_F64 64
#define VI_DEEP_F32 43
static inline bool vi_deep(int KA, bool mixed) { return KA > (mixed ? VI_DEEP_F32 : VI_DEEP_F64); }

// ---------------------------------------------------------------------------
// elementwise helpers of the small step
// ---------------------------------------------------------------------------
// PROG_split = 0 (first stage) or PROG0 - PROG; PROG_mean = PROG[0:5]
template <class R>
struct SplitArgs {
  const R *P0[6], *P[6];
  R *PS[6], *PM[5];
};
template <class R>
__global__ void k_split_init(const __grid_constant__ SplitArgs<R> a, int n, const __grid_constant__ SplitArgs<R> ap, int np, int npb, int first) {
  const bool pole = (int)blockIdx.x < npb;
  const int t = (int)((pole ? blockIdx.x : blockIdx.x - npb) * blockDim.x + threadIdx.x);
  if (t >= (pole ? np : n)) return;
  const SplitArgs<R>& s = pole ? ap : a;
  R v[6], v0[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    v[m] = s.P[m][t];
    v0[m] = first ? R(0.0) : s.P0[m][t];
  }
#pragma unroll
  for (int m = 0; m < 6; ++m) s.PS[m][t] = first ? R(0.0) : (v0[m] - v[m]);
#pragma unroll
  for (int m = 0; m < 5; ++m) s.PM[m][t] = v[m];
}

// PROG += PROG_split, then horizontalize the momentum (mod_vi.py:1572-1583)
template <class R>
struct PostArgs {
  R* P[6];
  const R* PS[6];
};
template <class R>
__device__ __forceinline__ void post_point(const PostArgs<R>& a, int p, const Pt& q, bool pole) {
  R v[6];
#pragma unroll
  for (int n = 0; n < 6; ++n) v[n] = a.P[n][p] + a.PS[n][p];
  if (pole) horiz_pl(q.g, q.lp, v[1], v[2], v[3]);
  else if (interior(q.i, q.j)) horiz_reg(q.i, q.j, q.l, v[1], v[2], v[3]);
#pragma unroll
  for (int n = 0; n < 6; ++n) a.P[n][p] = v[n];
}
template <class R>
__global__ void k_post(const __grid_constant__ PostArgs<R> a, const __grid_constant__ PostArgs<R> ap, int npb) {
  Pt q;
  if ((int)blockIdx.x < npb) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (pole_point(t, q)) post_point(ap, t, q, true);   // the pole layout is (g, k, lp), as the threads'
  } else {
    const int t = (int)((blockIdx.x - npb) * blockDim.x + threadIdx.x);
    if (reg_point(t, q)) post_point(a, t, q, false);
  }
}

}  // namespace nc
