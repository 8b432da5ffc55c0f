// EGLIB precision-1 mixture transport and the viscous flux that uses it:
// viscflux_eg_xyz with egvars (module_eg_lib.f90:106-310, 2140-2676).
//
// Per point, the kernel evaluates the EGlib 3.4 routines that egvars calls
// with eglib_precision = 1 (A. Ern and V. Giovangigli, devel-izem/src/eglib/
// EGSlib.f): EGSPAR/LSPAR with IFLAG = 7 (pure viscosities, reciprocal binary
// diffusion coefficients, collision-integral ratios A*, B*, C*, internal heat
// capacities and Parker's rotational relaxation), EGSE2 (shear viscosity, one
// conjugate-gradient step on the matrix H with the 1000 K A*), EGSLCT2
// (conductivity and rescaled thermal diffusion ratios, a direct
// factorisation of Lambda_[e]) and EGSDR1 (rho times the flux diffusion
// matrix, two stationary steps on L_[00] and the mass-conservation
// projection).  The formulas are the reference's, the order of operations is
// not: what depends on the temperature alone comes from a table (eg_table.cuh),
// and rho D is applied to the driving forces and never formed (EgPoint).  EGSL2
// and EGSK2, also called there, only produce values that the reference discards
// (the conductivity is recomputed by EGSLCT2 and the volume viscosity is set to
// zero, module_eg_lib.f90:288).
//
// The species gradients keep the fitted-transport layout of fd
// (12 + 3 l + d) so that k_visc_div is shared; the pressure gradients of
// the EGLIB flux (fd 13-15 in the reference) sit after them (12 + 3 NRV + d).
#pragma once
#include <cmath>
#include "common.cuh"
#include "kernels_visc.cuh"

struct DevEg {
  int ns;
  int lin[IZEM_NSMAX];
  double wt[IZEM_NSMAX], eps[IZEM_NSMAX], dip[IZEM_NSMAX], zrot[IZEM_NSMAX];
  double cofe[IZEM_NSMAX][4];
  double cofd[IZEM_NSMAX][IZEM_NSMAX][4];
  double ctaij[IZEM_NSMAX][IZEM_NSMAX];              // A*_ij at 1000 K
  double fita[IZEM_NSMAX][IZEM_NSMAX][7];            // A*, B*, C* in powers of ln T
  double fitb[IZEM_NSMAX][IZEM_NSMAX][7];
  double fitc[IZEM_NSMAX][IZEM_NSMAX][7];
  // egvars scalings (module_eg_lib.f90:140-145)
  double cp_cgs, eta_adim, lbda_adim, rd_adim;
  // species and pair constants of the device evaluation (molar masses,
  // Parker's reference factor, EGLIB's fixed coefficients folded together)
  double wtru[IZEM_NSMAX];        // W_k / RU
  double cx[IZEM_NSMAX];          // CROT / (AAAA max(1, ZROT) pi): cxi = cx * BBBB
  double bdiag[IZEM_NSMAX];       // 5 PATMOS W / (6 RU): D_int,kk = bdiag / (T A*_kk eta_k)
  double lfac[IZEM_NSMAX];        // 5 PATMOS W / (3 RU): FAC of Lambda_[e] = lfac / (T eta_k)
  double wsinv[IZEM_NSMAX][IZEM_NSMAX];                    // 1 / (W_i + W_j)
  // the shear matrix's pair constants over W_i + W_j: A*(1000) - 5/3, A* W_j/W_i + 5/3, A* W_i/W_j + 5/3
  double hoff[IZEM_NSMAX][IZEM_NSMAX];
  double hdi[IZEM_NSMAX][IZEM_NSMAX], hdj[IZEM_NSMAX][IZEM_NSMAX];
  double cr[2][IZEM_NSMAX][5];    // internal heat capacity c_int in powers of the code-unit temperature
  double p1[IZEM_NSMAX][IZEM_NSMAX];                       // wwi wwj
  double tti[IZEM_NSMAX][IZEM_NSMAX], ttj[IZEM_NSMAX][IZEM_NSMAX];   // 4/3 wioj, 4/3 wjoi
  double c1j[IZEM_NSMAX][IZEM_NSMAX], c2j[IZEM_NSMAX][IZEM_NSMAX], c3j[IZEM_NSMAX][IZEM_NSMAX];
  double c1i[IZEM_NSMAX][IZEM_NSMAX], c2i[IZEM_NSMAX][IZEM_NSMAX], c3i[IZEM_NSMAX][IZEM_NSMAX];
  double c4[IZEM_NSMAX][IZEM_NSMAX];
};

static __constant__ DevEg c_eg;

// Host: EGINI's set-up (EGini.f:58-301) from the linking data -- pair well
// depths with the polar correction (LEVEPS), A* at 1000 K, and the A*, B*,
// C* fits re-expanded in ln T for every pair (EGABC).  The fit constants are
// EGLIB's published collision-integral ratio fits.
inline void eg_prepare(const izem_eglib& L, const izem_thd& t, const izem_adi& a, DevEg& E) {
  static const double fa0[7] = {.1106910525e+01, -.7065517161e-02, -.1671975393e-01, .1188708609e-01,
                                .7569367323e-03, -.1313998345e-02, .1720853282e-03};
  static const double fb0[7] = {.1199673577e+01, -.1140928763e+00, -.2147636665e-02, .2512965407e-01,
                                -.3030372973e-02, -.1445009039e-02, .2492954809e-03};
  static const double fc0[7] = {.8386993788e+00, .4748325276e-01, .3250097527e-01, -.1625859588e-01,
                                -.2260153363e-02, .1844922811e-02, -.2115417788e-03};
  const int n = L.ns;
  E = DevEg{};
  E.ns = n;
  for (int k = 0; k < n; ++k) {
    E.lin[k] = L.lin[k];
    E.wt[k] = L.wt[k];
    E.eps[k] = L.eps[k];
    E.dip[k] = L.dip[k];
    E.zrot[k] = L.zrot[k];
    for (int q = 0; q < 4; ++q) E.cofe[k][q] = L.cofe[k][q];
    for (int l = 0; l < n; ++l)
      for (int q = 0; q < 4; ++q) E.cofd[k][l][q] = L.cofd[k][l][q];
  }
  double lneps[IZEM_NSMAX][IZEM_NSMAX];
  const double fac = 1.0e-12, dipmin = 1.0e-20, boltz = 1.38056e-16;
  auto cube = [](double s) { return s * s * s; };
  for (int j = 0; j < n; ++j)
    for (int k = 0; k <= j; ++k) {
      double e = std::sqrt(L.eps[j] * L.eps[k]);
      int polar = -1, nonpolar = -1;
      if (L.dip[j] < dipmin && L.dip[k] > dipmin) { polar = k; nonpolar = j; }
      else if (L.dip[j] > dipmin && L.dip[k] < dipmin) { polar = j; nonpolar = k; }
      if (polar >= 0) {
        const double xi = 1.0 + 0.25 * (L.pol[nonpolar] / cube(L.sig[nonpolar])) * (fac / boltz) *
                                    (L.dip[polar] * L.dip[polar] / (L.eps[polar] * cube(L.sig[polar]))) *
                                    std::sqrt(L.eps[polar] / L.eps[nonpolar]);
        e = e * (xi * xi);
      }
      lneps[k][j] = lneps[j][k] = std::log(e);
    }
  const double l1000 = std::log(1.0e3);
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < n; ++i) {
      const double t1 = l1000 - lneps[i][j];
      const double t2 = t1 * t1, t3 = t1 * t2, t4 = t1 * t3, t5 = t1 * t4, t6 = t1 * t5;
      E.ctaij[i][j] = fa0[0] + fa0[1] * t1 + fa0[2] * t2 + fa0[3] * t3 + fa0[4] * t4 + fa0[5] * t5 + fa0[6] * t6;
    }
  for (int j = 0; j < n; ++j)
    for (int i = j; i < n; ++i)
      for (int m = 0; m < 7; ++m) {
        double sa = 0.0, sb = 0.0, sc = 0.0;
        for (int k = m; k <= 6; ++k) {
          double prod = 1.0;
          for (int l = 1; l <= k - m; ++l) prod = prod * (-lneps[i][j]) * double(m + l) / double(l);
          sa = sa + fa0[k] * prod;
          sb = sb + fb0[k] * prod;
          sc = sc + fc0[k] * prod;
        }
        E.fita[i][j][m] = E.fita[j][i][m] = sa;
        E.fitb[i][j][m] = E.fitb[j][i][m] = sb;
        E.fitc[i][j][m] = E.fitc[j][i][m] = sc;
      }
  const double ru = 8.314e7, patmos = 1.01325e6, pi = 3.1415926535;
  for (int k = 0; k < n; ++k) {
    const double crot = L.lin[k] == 1 ? 1.0 : (L.lin[k] == 2 ? 1.5 : 0.0);
    const double dr = L.eps[k] / 298.0, sqdr = std::sqrt(dr);
    const double aaaa = 1.0 + 2.7842 * sqdr + 4.4674 * dr + 5.5683 * (sqdr * dr);
    E.wtru[k] = L.wt[k] / ru;
    E.cx[k] = crot / (aaaa * std::max(1.0, L.zrot[k]) * pi);
    E.bdiag[k] = 5.0 * patmos * L.wt[k] / (6.0 * ru);
    E.lfac[k] = 5.0 * patmos * L.wt[k] / (3.0 * ru);
  }
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      const double wi = L.wt[i], wj = L.wt[j];
      const double wwi = wi / (wi + wj), wwj = wj / (wi + wj);
      const double wioj = 3.0 * wi / wj - 2.0, wjoi = 3.0 * wj / wi - 2.0;
      const double A = E.ctaij[i][j];
      E.wsinv[i][j] = 1.0 / (wi + wj);
      E.hoff[i][j] = (A - 5.0 / 3.0) / (wi + wj);
      E.hdi[i][j] = (A * wj / wi + 5.0 / 3.0) / (wi + wj);
      E.hdj[i][j] = (A * wi / wj + 5.0 / 3.0) / (wi + wj);
      const double p1 = wwi * wwj;
      E.p1[i][j] = p1;
      E.tti[i][j] = 4.0 / 3.0 * wioj;
      E.ttj[i][j] = 4.0 / 3.0 * wjoi;
      E.c1j[i][j] = 7.5 * wwi * wwi;
      E.c2j[i][j] = wwj * wwj;
      E.c3j[i][j] = 4.0 / 15.0 * p1 * wioj * wioj;
      E.c1i[i][j] = 7.5 * wwj * wwj;
      E.c2i[i][j] = wwi * wwi;
      E.c3i[i][j] = 4.0 / 15.0 * p1 * wjoi * wjoi;
      E.c4[i][j] = 20.0 / 3.0 * p1;
    }
  E.cp_cgs = 1.0e4 * a.cp_ref;
  E.eta_adim = 1.0e-1 / t.muinf;
  E.lbda_adim = 1.0e-5 / t.laminf;
  E.rd_adim = 1.0e-1 / (a.rho_ref * t.dinf[0]);
  for (int k = 0; k < n; ++k)
    for (int r = 0; r < 2; ++r) {
      double tp = t.gam2 * t.Wc_i[k] * E.cp_cgs * E.wtru[k];
      for (int j = 0; j < 5; ++j) {
        E.cr[r][k][j] = L.lin[k] ? t.heatcap[k][r][j] * tp : 0.0;
        tp *= t.tinf;
      }
      if (L.lin[k]) E.cr[r][k][0] -= 2.5;
    }
}

#include "eg_table.cuh"

// Species cp of egvars (module_eg_lib.f90:170-240): NASA-7 with the linear
// extrapolation outside [Tpolymin, Tpolymax], in erg/g/K.
template <int N>
__device__ __noinline__ void eg_species_cp(double T, double* cpk) {
#pragma unroll
  for (int is = 0; is < N; ++is) {
    double t1 = T * c_thd.tinf, t2 = t1 * t1, t3 = t2 * t1, t4 = t3 * t1;
    const double* lo = c_thd.hc[is][0];
    const double* hi = c_thd.hc[is][1];
    double cpv;
    if (t1 < c_thd.tpolymin[is]) {
      t1 = c_thd.tpolymin[is]; t2 = t1 * t1; t3 = t2 * t1; t4 = t3 * t1;
      const double cp0 = lo[0] + lo[1] * t1 + lo[2] * t2 + lo[3] * t3 + lo[4] * t4;
      const double dcp0 = lo[1] + lo[2] * t1 * 2.0 + lo[3] * t2 * 3.0 + lo[4] * t3 * 4.0;
      cpv = c_thd.gam2 * c_thd.Wc_i[is] * (dcp0 * (T * c_thd.tinf - c_thd.tpolymin[is]) + cp0);
    } else if (t1 < c_thd.tpolylim[is]) {
      cpv = c_thd.gam2 * c_thd.Wc_i[is] * (lo[0] + lo[1] * t1 + lo[2] * t2 + lo[3] * t3 + lo[4] * t4);
    } else if (t1 < c_thd.tpolymax[is]) {
      cpv = c_thd.gam2 * c_thd.Wc_i[is] * (hi[0] + hi[1] * t1 + hi[2] * t2 + hi[3] * t3 + hi[4] * t4);
    } else {
      t1 = c_thd.tpolymax[is]; t2 = t1 * t1; t3 = t2 * t1; t4 = t3 * t1;
      const double cp0 = hi[0] + hi[1] * t1 + hi[2] * t2 + hi[3] * t3 + hi[4] * t4;
      const double dcp0 = hi[1] + hi[2] * t1 * 2.0 + hi[3] * t2 * 3.0 + hi[4] * t3 * 4.0;
      cpv = c_thd.gam2 * c_thd.Wc_i[is] * (dcp0 * (T * c_thd.tinf - c_thd.tpolymax[is]) + cp0);
    }
    cpk[is] = cpv * c_eg.cp_cgs;
  }
}

// c_int of every species: c_p / R - 5/2 (0 for an atom)
template <int N>
__device__ __forceinline__ void eg_cint(double T, double* cint) {
  const int r = th_range(T);
  if (r >= 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const double* a = c_eg.cr[r][k];
      cint[k] = fma(T, fma(T, fma(T, fma(T, a[4], a[3]), a[2]), a[1]), a[0]);
    }
    return;
  }
  double cpk[N];
  eg_species_cp<N>(T, cpk);
#pragma unroll
  for (int k = 0; k < N; ++k) cint[k] = c_eg.lin[k] ? cpk[k] * c_eg.wtru[k] - 2.5 : 0.0;
}

// What the fluxes of one point take from EGLIB: the viscosity, the
// conductivity, the thermal diffusion ratios, and the flux diffusion matrix
// rho D as an operator.  EGSDR1 forms D = P2 (y_i (dmi_i a_ij dmi_j + (1 +
// y_i) dmi_i delta_ij) - a_i) with the row averages a_i and the column
// projection P2; its product with a vector needs the symmetric a_ij and
// rank-one terms only, 99 FP64 operations a vector plus 43 for the
// projections, against 400 to build the projected 9 x 9 matrix and 81 a
// product.
template <int N>
struct EgPoint {
  double eta, tc;                         // [g/cm/s], [erg/cm/s/K]
  double chi[N];
  double a[N * (N - 1) / 2];              // x_i x_j / D_ij
  double dmi[N], yd[N], oney[N], sa[N], yr[N];
  double scale;                           // PATM / RU times W / T

  // rho D u over `scale`
  __device__ __forceinline__ void apply(const double* u, double* out) const {
    double e[N], U = 0.0, Q = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      e[i] = dmi[i] * u[i];
      out[i] = oney[i] * u[i];
      U = U + u[i];
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = i + 1; j < N; ++j) {
        const double aij = a[egp<N>(i, j)];
        out[i] = fma(aij, e[j], out[i]);
        out[j] = fma(aij, e[i], out[j]);
      }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      out[i] = fma(yd[i], out[i], -(sa[i] * U));
      Q = Q + out[i];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = fma(-yr[i], Q, out[i]);
  }
};

// One point: T [K], mole fractions X, c_int -> EgPoint.  The EGLIB formulas
// of the routines named above on the tabulated functions of T, in another
// order of operations: the same quantities up to rounding (against 80-bit
// arithmetic on random states: eta 8e-16 -> 2e-16, rho D 1.0e-15 -> 2.9e-16,
// the conductivity and the thermal diffusion ratios, which an ill-conditioned
// solve dominates, unchanged).
template <int N>
__device__ __forceinline__ void eg_point(double T, const double* X, const double* cint,
                                         const long long* __restrict__ tab, EgPoint<N>& o) {
  using I = EgIdx<N>;
  const double patmos = 1.01325e6, ru = 8.314e7;
  const EgRow row = eg_row<N>(tab, T);
  double tv[I::NF];   // functions of T of a point outside the table (local memory)
  if (!row.row) eg_direct<N>(T, tv);
  auto f = [&](int k) -> double { return row.row ? eg_eval<true>(row, k) : tv[k]; };
  auto fs = [&](int k) -> double { return row.row ? eg_eval<false>(row, k) : tv[k]; };   // of either sign
  // ---- EGSPAR: regularised mole and mass fractions
  double sum = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) sum = sum + X[i];
  const double xm = sum * (1.0 / double(N)), sss = 1.0e-16;
  double xtr[N], ytr[N], wwtr = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    xtr[i] = fma(sss, xm - X[i], X[i]);
    wwtr = fma(xtr[i], c_eg.wt[i], wwtr);
  }
  const double wwtr_i = fm_rcp(wwtr);
  double ysum = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    ytr[i] = xtr[i] * c_eg.wt[i] * wwtr_i;
    ysum = ysum + ytr[i];
  }
  double gd[N];
#pragma unroll
  for (int i = 0; i < N; ++i) gd[i] = 0.0;
  double g[I::NP], gdiag[N];
  // ---- EGSE2: matrix H over its common factor 6 RU T / (5 PATM), with the
  // 1000 K A*; one conjugate-gradient step.  The pairs' x_i x_j / D_ij and
  // their row sums serve the other routines too.
  {
#pragma unroll
    for (int i = 0; i < N; ++i) gdiag[i] = xtr[i] * xtr[i] * f(I::shear + i);
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = i + 1; j < N; ++j) {
        const double a = (xtr[i] * xtr[j]) * f(I::bin + egp<N>(i, j));
        o.a[egp<N>(i, j)] = a;
        gd[i] = gd[i] + a;
        gd[j] = gd[j] + a;
        g[egp<N>(i, j)] = a * c_eg.hoff[i][j];
        gdiag[i] = fma(a, c_eg.hdi[i][j], gdiag[i]);
        gdiag[j] = fma(a, c_eg.hdj[i][j], gdiag[j]);
      }
    // z = x / diag(H), (z.x)^2 / (z.H z); H z holds x from the diagonal
    double zn[N], zx = 0.0, zo = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      zn[i] = fm_div(xtr[i], gdiag[i]);
      zx = fma(zn[i], xtr[i], zx);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      double t = 0.0;
#pragma unroll
      for (int j = i + 1; j < N; ++j) t = fma(g[egp<N>(i, j)], zn[j], t);
      zo = fma(zn[i], t, zo);
    }
    o.eta = fm_div(zx * zx, fma(2.0, zo, zx) * ((6.0 * ru / (5.0 * patmos)) * T));
  }
  // ---- EGSLCT2: matrix Lambda_[e], factorisation (EGSDEC: L D L^T), solve
  {
    double an[N], beta[N], ri[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      beta[i] = (2.5 + cint[i]) * xtr[i];
      an[i] = beta[i];
      const double d = fma(cint[i], f(I::spec + 2 * i + 1), f(I::spec + 2 * i));
      gdiag[i] = fma(xtr[i] * xtr[i], d, cint[i] * gd[i]);
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = i + 1; j < N; ++j) {
        const int q = I::lam + 3 * egp<N>(i, j);
        const double xx = xtr[i] * xtr[j];
        g[egp<N>(i, j)] = -xx * f(q);
        gdiag[i] = fma(xx, f(q + 1), gdiag[i]);
        gdiag[j] = fma(xx, f(q + 2), gdiag[j]);
      }
    // row by row: the multipliers of column k replace its entries
#pragma unroll
    for (int k = 0; k < N; ++k) {
      double w[N];
#pragma unroll
      for (int j = 0; j < k; ++j) w[j] = gdiag[j] * g[egp<N>(j, k)];
#pragma unroll
      for (int j = 0; j < k; ++j) gdiag[k] = fma(-w[j], g[egp<N>(j, k)], gdiag[k]);
      ri[k] = fm_rcp(gdiag[k]);
#pragma unroll
      for (int i = k + 1; i < N; ++i) {
        double t = g[egp<N>(k, i)];
#pragma unroll
        for (int j = 0; j < k; ++j) t = fma(-g[egp<N>(j, i)], w[j], t);
        g[egp<N>(k, i)] = t * ri[k];
      }
    }
#pragma unroll
    for (int j = 0; j < N - 1; ++j)
#pragma unroll
      for (int k = j + 1; k < N; ++k) an[k] = fma(-g[egp<N>(j, k)], an[j], an[k]);
#pragma unroll
    for (int j = 0; j < N; ++j) an[j] = an[j] * ri[j];
#pragma unroll
    for (int j = N - 1; j >= 1; --j)
#pragma unroll
      for (int k = 0; k < j; ++k) an[k] = fma(-g[egp<N>(k, j)], an[j], an[k]);
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) s = fma(an[i], beta[i], s);
    const double Tinv = fm_rcp(T);
    o.tc = s * patmos * Tinv;
    o.scale = (patmos / ru) * wwtr * Tinv;
#pragma unroll
    for (int i = 0; i < N; ++i) o.chi[i] = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = i + 1; j < N; ++j) {
        const double term = fs(I::chi + egp<N>(i, j)) * (c_eg.wt[i] * an[j] - c_eg.wt[j] * an[i]);
        o.chi[i] = fma(xtr[j], term, o.chi[i]);
        o.chi[j] = fma(-xtr[i], term, o.chi[j]);
      }
  }
  // ---- EGSDR1: the operator's vectors (L_[00], two stationary steps, projection)
  {
    const double rsumy = fm_rcp(sum);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      o.dmi[i] = fm_div(ysum - ytr[i], gd[i]);
      o.yd[i] = ytr[i] * o.dmi[i];
      o.oney[i] = 1.0 + ytr[i];
      o.yr[i] = ytr[i] * rsumy;
    }
    double t[N], e[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      e[i] = o.dmi[i] * ytr[i];
      t[i] = o.oney[i] * ytr[i];
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = i + 1; j < N; ++j) {
        const double aij = o.a[egp<N>(i, j)];
        t[i] = fma(aij, e[j], t[i]);
        t[j] = fma(aij, e[i], t[j]);
      }
#pragma unroll
    for (int i = 0; i < N; ++i) o.sa[i] = o.yd[i] * t[i] * rsumy;
  }
}

// Pressure gradients of the EGLIB flux (fd slots 12 + 3 NRV + d) from the
// primitive pressure P = rho T W_i.
template <int NRV, int NG>
__global__ void k_grad_p(Geo g, Metrics mt, const double* __restrict__ prim, double* __restrict__ fd) {
  long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= g.nint) return;
  int c[3];
  c[0] = (int)(idx % g.n[0]) + 1;
  long long r = idx / g.n[0];
  c[1] = (int)(r % g.n[1]) + 1;
  c[2] = (int)(r / g.n[1]) + 1;
  const long long nc = g.ncell;
  const long long p = gid(g, c[0], c[1], c[2]);
  const long long strides[3] = {1LL, (long long)g.g[0], (long long)g.g[0] * g.g[1]};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    fd[(12 + 3 * NRV + d) * nc + p] =
        deriv_at<NG>(prim + PR_P * nc, p, deriv_row<NG>(strides[d], c[d], g.n[d], g.bnd[2 * d], g.bnd[2 * d + 1],
                                                        mt.dxi[d][c[d] - 1 + NG]));
  }
}

// The W_i gradients of viscflux_eg_LES_xyz (dx_fixed1 etc., module_eg_lib.f90:
// 2866-2871) and the criterion of shock_det_slv (module_tools.f90:1945-2085)
// at the interior points: 0 where, on the 2 ng-point stencil of the point's
// x or y face, the relative density jump and the relative pressure jump of
// some neighbour pair both exceed PERCENT_WEIGHT_SGS, else 1.  The
// reference's z pass writes with the y pass's final j_l and the final k, a
// ghost corner that no later step reads, so only the x and y passes shape
// the criterion.  3-D only.
// With ducros != 0 (LES with the fitted transport, viscflux_LES_xyz) the
// criterion is shock_det_ducros_slv's (module_tools.f90:2099-2181): 0 where
// (div u)^2 / ((div u)^2 + |curl u|^2 + 1e-30) > PERCENT_WEIGHT_SGS, else 1,
// from velocity gradients by uncontracted dx_fixed1 stencils (deriv_rn), so
// that the 0/1 decision is the host evaluation's.
// Bound by the FP64 pipe: two quotients for each of 12 neighbour pairs.  A
// density jump a hundredth below the threshold (positive densities, compared
// as bit patterns) settles a pair without them: 0.20 ms on 160 x 128 x 64,
// 1.18 with the quotients always.
template <int NG>
__global__ void k_les_prep(Geo g, Metrics mt, const double* __restrict__ v, const double* __restrict__ T,
                           const double* __restrict__ W_i, double pw, double* __restrict__ les,
                           const double* __restrict__ prim = nullptr, int ducros = 0) {
  long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= g.nint) return;
  int c[3];
  c[0] = (int)(idx % g.n[0]) + 1;
  long long r = idx / g.n[0];
  c[1] = (int)(r % g.n[1]) + 1;
  c[2] = (int)(r / g.n[1]) + 1;
  const long long nc = g.ncell;
  const long long p = gid(g, c[0], c[1], c[2]);
  const long long strides[3] = {1LL, (long long)g.g[0], (long long)g.g[0] * g.g[1]};
#pragma unroll
  for (int d = 0; d < 3; ++d)
    les[d * nc + p] = deriv_at<NG>(W_i, p, deriv_row<NG>(strides[d], c[d], g.n[d], g.bnd[2 * d], g.bnd[2 * d + 1],
                                                        mt.dxi[d][c[d] - 1 + NG]));
  double crit = 1.0;
  if (ducros) {
    double du[9];
    for (int a = 0; a < 3; ++a)
      for (int d = 0; d < 3; ++d)
        du[a * 3 + d] = deriv_rn(prim + (PR_U + a) * nc, p, strides[d], c[d], g.n[d], g.bnd[2 * d], g.bnd[2 * d + 1],
                                 mt.dxi[d][c[d] - 1 + g.ng], g.ng);
    double div = __dadd_rn(__dadd_rn(du[0], du[4]), du[8]);
    div = __dmul_rn(div, div);
    double wrk = __dsub_rn(du[7], du[5]);
    double vort = __dmul_rn(wrk, wrk);
    wrk = __dsub_rn(du[2], du[6]);
    vort = __dadd_rn(vort, __dmul_rn(wrk, wrk));
    wrk = __dsub_rn(du[3], du[1]);
    vort = __dadd_rn(vort, __dmul_rn(wrk, wrk));
    const double ratio = __ddiv_rn(div, __dadd_rn(__dadd_rn(div, vort), 1.0e-30));
    les[3 * nc + p] = ratio > pw ? 0.0 : 1.0;
    return;
  }
  const double pw_low = 0.99 * pw;
#pragma unroll
  for (int d = 0; d < 2; ++d)
#pragma unroll
    for (int st = 1; st <= 2 * NG; ++st) {
      const int s = c[d] + st - NG;             // i_s, from c - ng + 1 to c + ng
      const int sp = min(s + 1, g.n[d]);        // min(i_s + 1, ex)
      const long long pa = p + (long long)(s - c[d]) * strides[d];
      const long long pb = p + (long long)(sp - c[d]) * strides[d];
      const double ra = v[pa], rb = v[pb];
      const long long rm = min(__double_as_longlong(ra), __double_as_longlong(rb));
      if (rm > 0 && __double_as_longlong(fabs(rb - ra)) < __double_as_longlong(pw_low * __longlong_as_double(rm))) continue;
      const double drho = fabs(rb - ra) / fmin(rb, ra);
      const double pp = rb * T[pb] * W_i[pb];
      const double pm = ra * T[pa] * W_i[pa];
      const double dpres = fabs(pp - pm) / fmin(pp, pm);
      if (drho > pw && dpres > pw) crit = 0.0;
    }
  les[3 * nc + p] = crit;
}

// egvars + the stresses, rho Y_k V_k and heat flux of viscflux_eg_xyz at
// interior points and the ghost slabs of periodic faces.  Writes tau (6),
// q (3) and overwrites the species gradients of fd with rho Y_k V_k.  With
// LES the terms of viscflux_eg_LES_xyz (module_eg_lib.f90:3017-3239): the
// divergence gets the stresses scaled by 1 + mu_SGS / mu, the species
// fluxes the SGS diffusion and W_i-gradient terms, the heat flux the SGS
// conductivity mu_SGS cp / Pr_SGS; the work term keeps the molecular
// stresses.  The reference reuses its temperature-gradient scalar wrk1 for
// the SGS factor of each species, so the x thermal-diffusion term of species
// l >= 2 uses the SGS factor of species l - 1; that is reproduced.
// Bound by the FP64 pipe: 5154 -> 1893 instructions a point with nine species,
// 91.2 -> 35.7 ms on 256 x 256 x 128 (73 % of the pipe busy), 0.75 -> 0.25 ms
// on 33 x 40 x 21.  Two blocks of 256 threads an SM, i.e. 128 registers: the
// spills hit L1, and 16 warps hide the integer chains of the table better than
// 8 with 255 registers do (41.5 ms; 168: 39.5, 96: 38.4, 80: 40.2).
template <int NRV, bool LES = false>
__global__ void __launch_bounds__(256, 2) k_visc_point_eg(Geo g, const double* __restrict__ v,
                                                       const double* __restrict__ T, const double* __restrict__ W_i,
                                                       const double* __restrict__ ha, const double* __restrict__ Xa,
                                                       const double* __restrict__ prim, double* __restrict__ fd,
                                                       double* __restrict__ tau, double* __restrict__ qv,
                                                       const long long* __restrict__ tab, SgsArgs sa = SgsArgs{}) {
  long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int i, j, k, dom;
  if (!slab_point(g, idx, i, j, k, dom)) return;
  if (dom > 0 && g.bnd[dom - 1]) return;
  const long long nc = g.ncell;
  const long long p = gid(g, i, j, k);
  const double rho = v[p], Tp = T[p], Wi = W_i[p];
  const double rho_i = fm_rcp(rho);
  // ---- egvars
  EgPoint<NRV> eg;
  {
    double Xe[NRV], cint[NRV];
    const double wrk = rho_i * fm_rcp(Wi);
#pragma unroll
    for (int l = 0; l < NRV; ++l) Xe[l] = v[(IZEM_NIV + l) * nc + p] * wrk * c_thd.Wc_i[l];
    eg_cint<NRV>(Tp, cint);
    eg_point<NRV>(Tp * c_thd.tinf, Xe, cint, tab, eg);
  }
  const double mu = eg.eta * c_eg.eta_adim;
  const double ct = eg.tc * c_eg.lbda_adim;
  // ---- fluxes
  auto F = [&](int q1) -> double { return fd[(long long)(q1 - 1) * nc + p]; };
  const double rmu = -c_thd.sqgmr * mu;   // the volume viscosity is 0 (module_eg_lib.f90:288)
  const double twothirds = 2.0 / 3.0;
  const double sxx = twothirds * rmu * (F(1) + F(1) - (F(5) + F(9)));
  const double sxy = rmu * (F(4) + F(2));
  const double sxz = rmu * (F(7) + F(3));
  const double syy = twothirds * rmu * (F(5) + F(5) - (F(1) + F(9)));
  const double syz = rmu * (F(8) + F(6));
  const double szz = twothirds * rmu * (F(9) + F(9) - (F(1) + F(5)));
  double mu_sgs = 0.0;
  if constexpr (LES) {
    const double dxv = sa.dxi[0][i - 1 + g.ng], dyv = sa.dxi[1][j - 1 + g.ng], dzv = sa.dxi[2][k - 1 + g.ng];
    const double delta = fm_rcp(fm_root(dxv * dyv * dzv, 1.0 / 3.0));
    const double s11 = F(1), s12 = 0.5 * (F(2) + F(4)), s13 = 0.5 * (F(3) + F(7));
    const double s22 = F(5), s23 = 0.5 * (F(6) + F(8)), s33 = F(9);
    double sb = s11 * s11 + s12 * s12 + s13 * s13 + s12 * s12 + s22 * s22 + s23 * s23 + s13 * s13 + s23 * s23 +
                s33 * s33;
    sb = sqrt(sb + sb);
    mu_sgs = rho * sa.cs2 * (delta * delta) * sb * sa.les[3 * nc + p];
  }
  const double Ps = fm_rcp(prim[PR_P * nc + p]);
  const double Ts = fm_rcp(Tp);
  // the diffusion driving forces of the three directions, one by one
  double xt[NRV], hk[NRV];
#pragma unroll
  for (int l = 0; l < NRV; ++l) {
    xt[l] = Xa[l * nc + p] * eg.chi[l];
    hk[l] = fma(Tp * c_thd.Wc_i[l], eg.chi[l], ha[l * nc + p]);
  }
  const double jsc = -c_thd.rvd0 * eg.scale * c_eg.rd_adim;
  double sh[3];
  // LES: rho D of the thermal diffusion ratios on its own, since the x term
  // of species l takes the reference's reused scalar (wrk1)
  double jt[LES ? NRV : 1];
  if constexpr (LES) eg.apply(xt, jt);
  const double dm_sgs = mu_sgs * rho_i * sa.sc_sgs_i;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double wT = F(10 + d) * Ts, wP = fd[(12 + 3 * NRV + d) * nc + p] * Ps;
    double u[NRV], jd[NRV];
#pragma unroll
    for (int l = 0; l < NRV; ++l) {
      const double xy = fma(-v[(IZEM_NIV + l) * nc + p], rho_i, Xa[l * nc + p]);
      u[l] = fma(xy, wP, F(13 + 3 * l + d));
      if constexpr (!LES) u[l] = fma(xt[l], wT, u[l]);
    }
    eg.apply(u, jd);
    double s = 0.0;
#pragma unroll
    for (int l = 0; l < NRV; ++l) {
      double jl;
      if constexpr (LES) {
        const double wk = rho * dm_sgs * sa.sc * c_thd.Wc[l];
        const double fw = 1.0 + wk * Wi;
        const double wx = wk * Xa[l * nc + p];
        // wrk1 at species l: the temperature factor for the first, then the
        // SGS factor of the species before
        const double w1 = (d == 0 && l > 0) ? rho * dm_sgs * sa.sc * c_thd.Wc[l > 0 ? l - 1 : 0] : wT;
        const double jm = fma(w1, jt[LES ? l : 0], jd[l]) * (eg.scale * c_eg.rd_adim);
        jl = -c_thd.rvd0 * (jm * fw + wx * sa.les[d * nc + p]);
      } else {
        jl = jsc * jd[l];
      }
      fd[(long long)(12 + 3 * l + d) * nc + p] = jl;
      s = fma(jl, hk[l], s);
    }
    sh[d] = s;
  }
  const double uxs = v[nc + p] * rho_i, vys = v[2 * nc + p] * rho_i, wzs = v[3 * nc + p] * rho_i;
  double wl;
  if constexpr (LES) {
    const double ct_sgs = mu_sgs * sa.cp[p] * sa.pr_sgs_i;
    wl = -c_thd.rlam0 * (ct + ct_sgs);
    const double fs = 1.0 + fm_div(-c_thd.sqgmr * mu_sgs, rmu);
    tau[0 * nc + p] = sxx * fs; tau[1 * nc + p] = sxy * fs; tau[2 * nc + p] = sxz * fs;
    tau[3 * nc + p] = syy * fs; tau[4 * nc + p] = syz * fs; tau[5 * nc + p] = szz * fs;
  } else {
    wl = -c_thd.rlam0 * ct;
    tau[0 * nc + p] = sxx; tau[1 * nc + p] = sxy; tau[2 * nc + p] = sxz;
    tau[3 * nc + p] = syy; tau[4 * nc + p] = syz; tau[5 * nc + p] = szz;
  }
  qv[0 * nc + p] = sh[0] + wl * F(10) + uxs * sxx + vys * sxy + wzs * sxz;
  qv[1 * nc + p] = sh[1] + wl * F(11) + uxs * sxy + vys * syy + wzs * syz;
  qv[2 * nc + p] = sh[2] + wl * F(12) + uxs * sxz + vys * syz + wzs * szz;
}
