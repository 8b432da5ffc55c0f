// Convective part of the RHS: primitive pre-pass (K1), characteristic
// LLF-WENO face fluxes (K2), flux difference, Adams-Shariff sensor (K3).
//
// Reference: module_weno.f90 euler_LLF_x/_y/_z (:537-2125), wenorec_nw
// (:236-275), wenorec (:286-527); module_tools.f90 sensor (:2733-2814).
#pragma once
#include "common.cuh"
#include "thermo.cuh"
#include "fmath.cuh"

enum { PR_RHOI = 0, PR_U = 1, PR_V = 2, PR_W = 3, PR_P = 4, PR_CS = 5, PR_HT = 6, PR_ET = 7, PR_N = 8 };

// Maps a linear index over the interior + face-ghost slabs (the points the
// reference's pencil pre-passes touch) to (i,j,k).  Returns false past the end.
__device__ __forceinline__ bool slab_point(const Geo& g, long long idx, int& i, int& j, int& k, int& dom) {
  const long long nin = g.nint;
  if (idx < nin) {
    i = (int)(idx % g.n[0]) + 1;
    long long r = idx / g.n[0];
    j = (int)(r % g.n[1]) + 1;
    k = (int)(r / g.n[1]) + 1;
    dom = 0;
    return true;
  }
  idx -= nin;
  // face f: ng layers x the two interior extents of the other axes
  for (int f = 0; f < 6; ++f) {
    int d = f >> 1;
    int a1 = d == 0 ? 1 : 0, a2 = d == 2 ? 1 : 2;
    long long sz = (long long)g.ng * g.n[a1] * g.n[a2];
    if (idx < sz) {
      int c1 = (int)(idx % g.n[a1]) + 1;
      long long r = idx / g.n[a1];
      int c2 = (int)(r % g.n[a2]) + 1;
      int layer = (int)(r / g.n[a2]) + 1;     // 1..ng
      int s = (f & 1) ? g.n[d] + layer : 1 - layer;
      int c[3];
      c[d] = s; c[a1] = c1; c[a2] = c2;
      i = c[0]; j = c[1]; k = c[2];
      dom = 1 + f;
      return true;
    }
    idx -= sz;
  }
  return false;
}

__host__ __device__ inline long long slab_count(const Geo& g) {
  long long s = g.nint;
  for (int d = 0; d < 3; ++d) {
    int a1 = d == 0 ? 1 : 0, a2 = d == 2 ? 1 : 2;
    s += 2LL * g.ng * g.n[a1] * g.n[a2];
  }
  return s;
}

// K1: per-point primitives used by the sweeps (module_weno.f90:634-667 and
// the y/z copies): 1/rho, u, v, w, P = rho T W_i, c = sqrt(gam P / rho),
// h_t = sum h_k Y_k + |u|^2/2, e_t = rho e_t / rho.  Also the mole fractions
// of molefrac (module_thermodynamics.f90:1669-1697) for the viscous flux.
template <int NRV>
__global__ void k_prim(Geo g, const double* __restrict__ v, const double* __restrict__ T,
                       const double* __restrict__ W_i, const double* __restrict__ cp,
                       const double* __restrict__ ha, double* __restrict__ prim,
                       double* __restrict__ Xa, DevStatus* st) {
  long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int i, j, k, dom;
  if (!slab_point(g, idx, i, j, k, dom)) return;
  const long long nc = g.ncell;
  long long p = gid(g, i, j, k);
  double rho = v[p];
  double rho_i = fm_rcp(rho);
  double ux = v[nc + p] * rho_i, vy = v[2 * nc + p] * rho_i, wz = v[3 * nc + p] * rho_i;
  double Wi = W_i[p];
  const double TW = T[p] * Wi;
  double P = rho * TW;
  if (P <= 0.0) atomicExch(&st->neg_pressure, 1);
  // gamma = cp / (cp - gam2 W_i); one reciprocal for the mole fractions
  // instead of a quotient each (213 -> 82 FP64 instructions a point with nine
  // species, 2.83 -> 1.33 ms on 256 x 256 x 128)
  const double cpp = cp[p];
  double cs = sqrt(fm_div(cpp, cpp - c_thd.gam2 * Wi) * TW);
  double ht = 0.0;
  // the roundings of 1 / (rho W_i) carried along: second derivatives of the
  // mole fractions see their last bits
  const fm_pair rw_i = fm_rcp_prod(rho, Wi);
#pragma unroll
  for (int l = 0; l < NRV; ++l) {
    double rY = v[(IZEM_NIV + l) * nc + p];
    ht = fma(ha[l * nc + p], rY, ht);
    if (Xa) Xa[l * nc + p] = fm_over(rY * c_thd.Wc_i[l], rw_i);
  }
  ht = ht * rho_i;
  ht = ht + 0.5 * (ux * ux + vy * vy + wz * wz);
  prim[PR_RHOI * nc + p] = rho_i;
  prim[PR_U * nc + p] = ux;
  prim[PR_V * nc + p] = vy;
  prim[PR_W * nc + p] = wz;
  prim[PR_P * nc + p] = P;
  prim[PR_CS * nc + p] = cs;
  prim[PR_HT * nc + p] = ht;
  prim[PR_ET * nc + p] = v[4 * nc + p] * rho_i;
}

// d / e^2, the unnormalised weight of a sub-stencil
__device__ __forceinline__ double weno_alpha(double d, double e) {
  const double r = fm_rcp(e);
  return (d * r) * r;
}

// Nonlinear WENO5 reconstruction (wenorec, ng = 3) of one characteristic
// field; gp/gm hold the 2ng = 6 stencil values (index 0 = point il-2).
__device__ __forceinline__ double weno5_nl(const double* vp, const double* vm) {
  const double eps = 1.0e-10;
  const double z1 = 13.0 / 12.0, z2 = 1.0 / 4.0;
  // '-' state at i+1/2, centre vp[2]
  double a, b, b0, b1, b2;
  double q0 = (1.0 / 3.0) * vp[2] + (5.0 / 6.0) * vp[3] + (-1.0 / 6.0) * vp[4];
  double q1 = (-1.0 / 6.0) * vp[1] + (5.0 / 6.0) * vp[2] + (1.0 / 3.0) * vp[3];
  double q2 = (1.0 / 3.0) * vp[0] + (-7.0 / 6.0) * vp[1] + (11.0 / 6.0) * vp[2];
  a = vp[2] + -2.0 * vp[3] + vp[4]; b = 3.0 * vp[2] + -4.0 * vp[3] + vp[4];
  b0 = z1 * a * a + z2 * b * b;
  a = vp[1] + -2.0 * vp[2] + vp[3]; b = vp[1] + -1.0 * vp[3];
  b1 = z1 * a * a + z2 * b * b;
  a = vp[0] + -2.0 * vp[1] + vp[2]; b = vp[0] + -4.0 * vp[1] + 3.0 * vp[2];
  b2 = z1 * a * a + z2 * b * b;
  double al0 = weno_alpha((3.0 / 10.0), eps + b0);
  double al1 = weno_alpha((3.0 / 5.0), eps + b1);
  double al2 = weno_alpha((1.0 / 10.0), eps + b2);
  const double vminus = (al0 * q0 + al1 * q1 + al2 * q2) * fm_rcp(al0 + al1 + al2);
  // '+' state at i+1/2, centre vm[3]
  q0 = (11.0 / 6.0) * vm[3] + (-7.0 / 6.0) * vm[4] + (1.0 / 3.0) * vm[5];
  q1 = (1.0 / 3.0) * vm[2] + (5.0 / 6.0) * vm[3] + (-1.0 / 6.0) * vm[4];
  q2 = (-1.0 / 6.0) * vm[1] + (5.0 / 6.0) * vm[2] + (1.0 / 3.0) * vm[3];
  a = vm[3] + -2.0 * vm[4] + vm[5]; b = 3.0 * vm[3] + -4.0 * vm[4] + vm[5];
  b0 = z1 * a * a + z2 * b * b;
  a = vm[2] + -2.0 * vm[3] + vm[4]; b = vm[2] + -1.0 * vm[4];
  b1 = z1 * a * a + z2 * b * b;
  a = vm[1] + -2.0 * vm[2] + vm[3]; b = vm[1] + -4.0 * vm[2] + 3.0 * vm[3];
  b2 = z1 * a * a + z2 * b * b;
  al0 = weno_alpha((1.0 / 10.0), eps + b0);
  al1 = weno_alpha((3.0 / 5.0), eps + b1);
  al2 = weno_alpha((3.0 / 10.0), eps + b2);
  const double vplus = (al0 * q0 + al1 * q1 + al2 * q2) * fm_rcp(al0 + al1 + al2);
  return vminus + vplus;
}

// Nonlinear WENO7 reconstruction (wenorec, ng = 4, module_weno.f90:286-527):
// vp/vm hold the 2ng = 8 stencil values (index 0 = point il-3).
__device__ __forceinline__ double weno7_nl(const double* vp, const double* vm) {
  const double eps = 1.0e-10;
  const double za = 547.0, zb = -1854.0, zc = 4642.0, zd = -3882.0, ze = -17246.0, zf = 2107.0, zg = 7043.0,
               zh = -9402.0, zi = 11003.0, zl = 7042.0, zm = 3443.0, zn = -5966.0, zo = -2522.0, zp = 1602.0,
               zq = 2843.0, zr = 267.0, zs = 1922.0, zt = -494.0, zu = -1642.0;
  // cweno(r, j), r = -1..3
  const double cw[5][4] = {{25.0 / 12.0, -23.0 / 12.0, 13.0 / 12.0, -1.0 / 4.0},
                           {1.0 / 4.0, 13.0 / 12.0, -5.0 / 12.0, 1.0 / 12.0},
                           {-1.0 / 12.0, 7.0 / 12.0, 7.0 / 12.0, -1.0 / 12.0},
                           {1.0 / 12.0, -5.0 / 12.0, 13.0 / 12.0, 1.0 / 4.0},
                           {-1.0 / 4.0, 13.0 / 12.0, -23.0 / 12.0, 25.0 / 12.0}};
  const double dw[4] = {4.0 / 35.0, 18.0 / 35.0, 12.0 / 35.0, 1.0 / 35.0};
  auto betas = [&](const double* q, int i, double* be) {   // q 0-based, centre i
    be[0] = q[i] * (zf * q[i] + zh * q[i + 1] + zl * q[i + 2] + zb * q[i + 3]) +
            q[i + 1] * (zi * q[i + 1] + ze * q[i + 2] + zc * q[i + 3]) + q[i + 2] * (zg * q[i + 2] + zd * q[i + 3]) +
            q[i + 3] * (za * q[i + 3]);
    be[1] = q[i - 1] * (za * q[i - 1] + zo * q[i] + zs * q[i + 1] + zt * q[i + 2]) +
            q[i] * (zm * q[i] + zn * q[i + 1] + zp * q[i + 2]) + q[i + 1] * (zq * q[i + 1] + zu * q[i + 2]) +
            q[i + 2] * (zr * q[i + 2]);
    be[2] = q[i - 2] * (zr * q[i - 2] + zu * q[i - 1] + zp * q[i] + zt * q[i + 1]) +
            q[i - 1] * (zq * q[i - 1] + zn * q[i] + zs * q[i + 1]) + q[i] * (zm * q[i] + zo * q[i + 1]) +
            q[i + 1] * (za * q[i + 1]);
    be[3] = q[i - 3] * (za * q[i - 3] + zd * q[i - 2] + zc * q[i - 1] + zb * q[i]) +
            q[i - 2] * (zg * q[i - 2] + ze * q[i - 1] + zl * q[i]) + q[i - 1] * (zi * q[i - 1] + zh * q[i]) +
            q[i] * (zf * q[i]);
  };
  double be[4], al[4], s, vminus = 0.0, vplus = 0.0;
  // '-' state at i+1/2: centre vp[3], cweno(r, j) on vp[3 - r + j]
  betas(vp, 3, be);
  s = 0.0;
#pragma unroll
  for (int r = 0; r < 4; ++r) { al[r] = weno_alpha(dw[r], eps + be[r]); s = s + al[r]; }
  s = fm_rcp(s);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    double q = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) q = q + cw[r + 1][j] * vp[3 - r + j];
    vminus = vminus + (al[r] * s) * q;
  }
  // '+' state at i+1/2: centre vm[4], cweno(r-1, j) on vm[4 - r + j], weights reversed
  betas(vm, 4, be);
  s = 0.0;
#pragma unroll
  for (int r = 0; r < 4; ++r) { al[r] = weno_alpha(dw[3 - r], eps + be[r]); s = s + al[r]; }
  s = fm_rcp(s);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    double q = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) q = q + cw[r][j] * vm[4 - r + j];
    vplus = vplus + (al[r] * s) * q;
  }
  return vminus + vplus;
}

template <int NG>
__device__ __forceinline__ double weno_nl(const double* vp, const double* vm) {
  if constexpr (NG == 4) return weno7_nl(vp, vm);
  else return weno5_nl(vp, vm);
}

// The face-constant data of a sensed face, held by the thread that owns it.
template <int NRV>
struct FaceState {
  double uc[3], Yc[NRV], psi[NRV];
  double un, cs, cs_i, b2, xi, q, ht;
  double lm0, lm1, lm2;
  long long p0;   // first stencil point
};

// Nonlinear reconstruction (wenorec) of the sensed faces of one warp, GL lanes
// to a face: lane m holds variable m while the characteristic projections are
// formed (their species products are sums over the lanes), then reconstructs
// field m, and writes component m of R ghat.  A face a thread instead
// serialises 2 NG projections and NV reconstructions, some 1900 FP64 operations
// with nine species, for the few lanes that need them while the rest of the
// warp waits.  The sweeps of the 400 x 11 shock tube (WENO7, two
// species), all latency, took 98 us in x and in y and take 80 and 43; a sweep
// of 61 x 50 x 38 with nine species and 1 % of the points flagged 0.61 ms and
// 0.28.
template <int NRV, int D, int NG>
__device__ __forceinline__ void weno_face_lanes(unsigned sensed, const FaceState<NRV>& own, long long own_idx,
                                                long long nc, long long stride, const double* __restrict__ v,
                                                const double* __restrict__ prim, double* __restrict__ fhat,
                                                long long nfaces) {
  constexpr int NV = IZEM_NIV + NRV;
  constexpr int GL = NV <= 8 ? 8 : 16, PER = 32 / GL;
  constexpr int T1 = D == 0 ? 1 : 0;
  constexpr int T2 = D == 2 ? 1 : 2;
  static_assert(NV <= 16, "a variable a lane");
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, grp = lane / GL, m = lane % GL;
  while (sensed) {
    // the faces of this pass: group g takes the g-th set bit (the first
    // again when there are fewer; it does not store then)
    unsigned rest = sensed;
    for (int g = 0; g < grp && rest; ++g) rest &= rest - 1;
    const bool store = rest != 0;
    const int src = __ffs(store ? rest : sensed) - 1;
    for (int g = 0; g < PER; ++g) sensed &= sensed - 1;
    auto from = [&](double x) { return __shfl_sync(full, x, src); };
    const double uT1 = from(own.uc[T1]), uT2 = from(own.uc[T2]), un = from(own.un);
    const double u0 = D == 0 ? un : uT1, u1 = D == 1 ? un : (D == 0 ? uT1 : uT2), u2 = D == 2 ? un : uT2;
    const double cs = from(own.cs), cs_i = from(own.cs_i), b2 = from(own.b2), xi = from(own.xi), q = from(own.q);
    const double ht = from(own.ht), lm0 = from(own.lm0), lm1 = from(own.lm1), lm2 = from(own.lm2);
    const long long p0 = __shfl_sync(full, own.p0, src), idx = __shfl_sync(full, own_idx, src);
    double psi_v = 0.0, psi_r = 0.0, Y_v = 0.0, Y_r = 0.0, psi_n = 0.0;   // of variable m, of field m (species m - 6)
#pragma unroll
    for (int l = 0; l < NRV; ++l) {
      const double ps = from(own.psi[l]), y = from(own.Yc[l]);
      if (m == IZEM_NIV + l) { psi_v = ps; Y_v = y; }
      if (m == IZEM_NIV + 1 + l && l < NRV - 1) { psi_r = ps; Y_r = y; }
      if (l == NRV - 1) psi_n = ps;
    }
    // row m of L as coefficients of x_0, x_n, x_t1, x_t2, kappa, psi.x_s and x_{m-1}
    const double h = 0.5 * cs_i;
    double k0 = 0.0, kn = 0.0, kt1 = 0.0, kt2 = 0.0, kk = 0.0, ks = 0.0, kx = 0.0;
    if (m == 0) { k0 = un * h; kn = -h; kk = 0.5 * b2; }
    else if (m == 1) { k0 = 1.0; kk = -b2; }
    else if (m == 2) { k0 = -un * h; kn = h; kk = 0.5 * b2; }
    else if (m == 3) { k0 = -uT1; kt1 = 1.0; }
    else if (m == 4) { k0 = -uT2; kt2 = 1.0; }
    else if (m == 5) { kk = 1.0 + xi; ks = -1.0; }
    else { kk = -Y_r * b2; kx = 1.0; }
    const double lam = m == 0 ? lm0 : (m == 2 ? lm2 : lm1);
    auto project = [&](double x) {
      const double x0 = __shfl_sync(full, x, 0, GL), x1 = __shfl_sync(full, x, 1, GL);
      const double x2 = __shfl_sync(full, x, 2, GL), x3 = __shfl_sync(full, x, 3, GL);
      const double x4 = __shfl_sync(full, x, 4, GL), xp = __shfl_up_sync(full, x, 1, GL);
      double sw = psi_v * x;   // psi_v is 0 outside the species
#pragma unroll
      for (int o = GL / 2; o > 0; o >>= 1) sw = sw + __shfl_xor_sync(full, sw, o, GL);
      const double kappa = fma(q, x0, x4) - (u0 * x1 + u1 * x2 + u2 * x3) + sw;
      const double xn = D == 0 ? x1 : (D == 1 ? x2 : x3);
      const double xt1 = T1 == 0 ? x1 : x2, xt2 = T2 == 1 ? x2 : x3;
      double r = fma(kk, kappa, ks * sw);
      r = fma(k0, x0, r);
      r = fma(kn, xn, r);
      r = fma(kt1, xt1, r);
      r = fma(kt2, xt2, r);
      return fma(kx, xp, r);
    };
    double gpl[2 * NG], gmi[2 * NG];
#pragma unroll
    for (int st = 0; st < 2 * NG; ++st) {
      const long long ps = p0 + st * stride;
      const double w = m < NV ? v[m * nc + ps] : 0.0;
      const double u_s = prim[(PR_U + D) * nc + ps], P_s = prim[PR_P * nc + ps];
      const double wn = __shfl_sync(full, w, 1 + D, GL);
      double f = u_s * w;
      if (m == 0) f = wn;
      if (m == 1 + D) f = f + P_s;
      if (m == 4) f = u_s * (w + P_s);
      const double pw = project(w), pf = project(f);
      gpl[st] = 0.5 * (pf + lam * pw);
      gmi[st] = pf - gpl[st];
    }
    const double gh = weno_nl<NG>(gpl, gmi);
    // component m of R ghat (module_weno.f90:881-989)
    const double g0 = __shfl_sync(full, gh, 0, GL), g1 = __shfl_sync(full, gh, 1, GL);
    const double g2 = __shfl_sync(full, gh, 2, GL), g3 = __shfl_sync(full, gh, 3, GL);
    const double g4 = __shfl_sync(full, gh, 4, GL), g5 = __shfl_sync(full, gh, 5, GL);
    const double gd = __shfl_down_sync(full, gh, 1, GL);
    double sg = psi_r * gh;   // sum_s psi_s ghat_{6+s}
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) sg = sg + __shfl_xor_sync(full, sg, o, GL);
    const double s3 = g0 + g1 + g2, s2 = g0 + g2;
    double fh;
    if (m == 0) fh = s3;
    else if (m == 1 + D) fh = un * s3 + cs * (g2 - g0);
    else if (m == 1 + T1) fh = uT1 * s3 + g3;
    else if (m == 1 + T2) fh = uT2 * s3 + g4;
    else if (m == 4) fh = ht * s2 + un * cs * (g2 - g0) + q * g1 + uT1 * g3 + uT2 * g4 + g5;
    else if (m < NV - 1) fh = Y_v * s2 + gd;
    else fh = Y_v * s2 - fm_div(g5 + sg, psi_n);
    if (store && m < NV) fhat[m * nfaces + idx] = fh;
  }
}

// K2: one thread per cell face along axis D.  Linear (sensor-off) faces take
// the reconstruction of wenorec_nw without forming the characteristic
// variables.  The LLF speeds of a face are one number per field and L, R and
// the reconstruction are linear, so with the stencil sums
//   F = sum_s a_s f_s / 2,  W = sum_s b_s w_s / 2   (a = c- + c+, b = c- - c+)
// the flux is R L F + R Lambda L W, Lambda = diag(lam0, lam1, lam2, lam1, ...).
// For the eigenvectors of module_weno.f90:775-916, R L = I + delta e_N kappa^T:
// all rows but the last species' are exact inverses of each other, whatever
// the averages, and there
//   kappa(x) = q x_0 - u.x_m + x_4 + psi.x_s,
//   delta = -(1 + xi - b2 sum_l psi_l Y_l) / psi_N,
// so that R Lambda L W = lam1 (W + delta e_N kappa(W)) plus the two acoustic
// columns r0, r2 scaled by lam - lam1.  One pass over the stencil and two dot
// products per face replace four projections and R, and the sums weight w
// with a_s u_s, so that no point's flux is formed.  The FP64 pipe bounds the
// kernel (87 % busy): 1165 -> 496 FP64 instructions a face with nine species,
// 18.1 -> 7.5 ms a sweep of 256 x 256 x 128; 0.300 -> 0.144 ms a sweep of 64^3
// with two.  The result equals the reference's dense nv x nv products up to
// rounding (relative error against dense 64-bit products 7.6e-15 -> 6.2e-15).
// Sensed faces keep the 2NG projected values for the nonlinear weights: a warp
// with few of them takes them together (weno_face_lanes), one with many a face
// a thread.
// NG = 3 is WENO5, NG = 4 WENO7 (module_weno.f90, ng branches).
//
// Sensor blocks (x sweep only): with bx < n[0] the x direction is read as
// n[0] / bx blocks of bx points, as in a run decomposed into MPI blocks whose
// shock sensor is never exchanged (module_weno.f90:973 reads the block's own
// flags; its ghosts stay unflagged).  A face then sees only the flags of the
// block that uses it.  With edge = 0 the kernel writes every face as seen by
// its left cell's block; with edge = 1 it runs over the faces on block edges
// only (nfaces = (n[0]/bx - 1) n[1] n[2]) and writes them as seen by the
// right block into fhat.
template <int NRV, int D, int NG>
__global__ void __launch_bounds__(256) k_euler_face(Geo g, int weno_avg, int linfix,
                                                    const double* __restrict__ v,
                                                    const double* __restrict__ prim,
                                                    const uint8_t* __restrict__ sensor,
                                                    double* __restrict__ fhat, long long nfaces, int bx, int edge, int share) {
  constexpr int NV = IZEM_NIV + NRV;
  constexpr int T1 = D == 0 ? 1 : 0;
  constexpr int T2 = D == 2 ? 1 : 2;
  // 2^share lanes to a face, the first of which stores it; lanes past the end
  // repeat the last face: sensed faces are a warp's work
  long long idx = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> share;
  const bool valid = idx < nfaces && (threadIdx.x & ((1 << share) - 1)) == 0;
  if (idx >= nfaces) idx = nfaces - 1;
  int c[3];
  if (D == 0 && edge) {
    const int ne = g.n[0] / bx - 1;
    long long r = idx;
    c[0] = ((int)(r % ne) + 1) * bx;   // face between the last cell of a block and the next
    r /= ne;
    c[1] = (int)(r % g.n[1]) + 1;
    c[2] = (int)(r / g.n[1]) + 1;
  } else {
    long long r = idx;
    int e0 = D == 0 ? g.n[0] + 1 : g.n[0];
    int e1 = D == 1 ? g.n[1] + 1 : g.n[1];
    c[0] = (int)(r % e0); r /= e0;
    c[1] = (int)(r % e1); r /= e1;
    c[2] = (int)r;
    // faces run 0..n along D (face s between cells s and s+1); cells 1..n across
    if (D != 0) c[0] += 1;
    if (D != 1) c[1] += 1;
    if (D != 2) c[2] += 1;
  }
  const long long nc = g.ncell;
  const long long stride = D == 0 ? 1LL : (D == 1 ? (long long)g.g[0] : (long long)g.g[0] * g.g[1]);
  const long long pl = gid(g, c[0], c[1], c[2]);   // cell il
  const long long pr = pl + stride;                  // cell il+1
  const long long p0 = pl - (NG - 1) * stride;       // stencil point il-ng+1

  // ---- Roe average compatible with the EOS (module_weno.f90:726-761)
  const double rho_i_l = prim[PR_RHOI * nc + pl], rho_i_r = prim[PR_RHOI * nc + pr];
  const double r = sqrt(v[pr] * rho_i_l);
  const double al = fm_rcp(r + 1.0), ar = r * al;   // weights of the left and right cell
  double uc[3];
  uc[0] = fma(ar, prim[PR_U * nc + pr], al * prim[PR_U * nc + pl]);
  uc[1] = fma(ar, prim[PR_V * nc + pr], al * prim[PR_V * nc + pl]);
  uc[2] = fma(ar, prim[PR_W * nc + pr], al * prim[PR_W * nc + pl]);
  double Yc[NRV];
  double W_i_c = 0.0;
  {
    const double yl = al * rho_i_l, yr = ar * rho_i_r;
#pragma unroll
    for (int l = 0; l < NRV; ++l) {
      Yc[l] = fma(yr, v[(IZEM_NIV + l) * nc + pr], yl * v[(IZEM_NIV + l) * nc + pl]);
      W_i_c = fma(Yc[l], c_thd.Wc_i[l], W_i_c);
    }
  }
  const double ht_c = fma(ar, prim[PR_HT * nc + pr], al * prim[PR_HT * nc + pl]);
  const double et_c = fma(ar, prim[PR_ET * nc + pr], al * prim[PR_ET * nc + pl]);
  const double rt_c = ht_c - et_c;               // T W_i
  const double T_c = fm_div(rt_c, W_i_c);
  double psi[NRV];
  const double cp_c = th_cp_ha<NRV>(T_c, Yc, psi);   // psi <- h_k(T_c)
  // gamma = cp / (cp - gam2 W_i), gamma - 1 = gam2 W_i / (cp - gam2 W_i)
  const double gw = c_thd.gam2 * W_i_c;
  const double gd_i = fm_rcp(cp_c - gw);
  const double gm1 = gw * gd_i, gam_c = cp_c * gd_i;
  const double cs2 = gam_c * rt_c;
  const double cs_c = sqrt(cs2);
  {
    const double wrk = c_thd.gam2_i * cp_c * fm_div(T_c, W_i_c);   // gamma T / (gamma - 1)
#pragma unroll
    for (int l = 0; l < NRV; ++l) psi[l] = fma(wrk, c_thd.Wc_i[l], -psi[l]);
  }
  const double q = 0.5 * (uc[0] * uc[0] + uc[1] * uc[1] + uc[2] * uc[2]);
  const double cs2_i = fm_rcp(cs2);
  const double b2 = gm1 * cs2_i;
  const double cs_c_i = cs_c * cs2_i;
  const double b1 = b2 * q;
  const double xi = b1 - b2 * ht_c;
  const double un = uc[D];

  // ---- stencil eigenvalue maxima (LLF) and shock flag
  // maxima of |u - c|, |u|, |u + c| as bit patterns (ordered like the values)
  long long m0 = 0, m1 = 0, m2 = 0;
  double us[2 * NG];
  bool shk = false;
  // the block whose flags count (x sweep with sensor blocks only)
  const bool blocks = D == 0 && bx < g.n[0];
  auto xblock = [&](int s) { return (min(max(s, 1), g.n[0]) - 1) / bx; };
  const int view = blocks ? xblock(edge ? c[0] + 1 : c[0]) : 0;
#pragma unroll
  for (int st = 0; st < 2 * NG; ++st) {
    const long long ps = p0 + st * stride;
    const double u_s = prim[(PR_U + D) * nc + ps], c_s = prim[PR_CS * nc + ps];
    us[st] = u_s;
    m0 = max(m0, __double_as_longlong(fabs(u_s - c_s)));
    m1 = max(m1, __double_as_longlong(fabs(u_s)));
    m2 = max(m2, __double_as_longlong(fabs(u_s + c_s)));
    const bool counts = !blocks || xblock(c[0] - NG + 1 + st) == view;
    shk = shk || (counts && sensor[ps] != 0);
  }
  const double lm0 = __longlong_as_double(m0), lm1 = __longlong_as_double(m1), lm2 = __longlong_as_double(m2);
  shk = shk && (weno_avg != 0) && valid;
  // about where the two forms meet: 300 FP64 operations a round of 2 (4 with
  // two species) faces against some 1900 (800) for the whole warp.  The sweeps
  // of 61 x 50 x 38 with 1 % of the points flagged take 1.17 ms with a line of
  // 6, 1.09 of 12 and 1.13 with lanes always.
  constexpr int kLanesMost = 12;
  const unsigned sensed = __ballot_sync(0xffffffffu, shk);

  double fh[NV];
  if (!shk) {
    // Half the sum and half the difference of the two one-sided stencils,
    // divided by their denominators.  WENO5: c- = (-3, 27, 47, -13, 2) / 60
    // on points 0..4 and its mirror on 1..5 (the reference's coefficients),
    // or the textbook (2, -13, 47, 27, -3) / 60 (linfix); WENO7: c- = (-3, 25,
    // -101, 319, 214, -38, 4) / 420 on points 0..6.
    constexpr double ar5[6] = {-3.0 / 120, 29.0 / 120, 34.0 / 120, 34.0 / 120, 29.0 / 120, -3.0 / 120};
    constexpr double br5[6] = {-3.0 / 120, 25.0 / 120, 60.0 / 120, -60.0 / 120, -25.0 / 120, 3.0 / 120};
    constexpr double af5[6] = {2.0 / 120, -16.0 / 120, 74.0 / 120, 74.0 / 120, -16.0 / 120, 2.0 / 120};
    constexpr double bf5[6] = {2.0 / 120, -10.0 / 120, 20.0 / 120, -20.0 / 120, 10.0 / 120, -2.0 / 120};
    constexpr double a7[8] = {-3.0 / 840,  29.0 / 840,  -139.0 / 840, 533.0 / 840,
                              533.0 / 840, -139.0 / 840, 29.0 / 840,  -3.0 / 840};
    constexpr double b7[8] = {-3.0 / 840,   21.0 / 840, -63.0 / 840, 105.0 / 840,
                              -105.0 / 840, 63.0 / 840, -21.0 / 840, 3.0 / 840};
    double ca[2 * NG], cb[2 * NG], cau[2 * NG];
#pragma unroll
    for (int st = 0; st < 2 * NG; ++st) {
      ca[st] = NG == 4 ? a7[st] : (linfix ? af5[st % 6] : ar5[st % 6]);
      cb[st] = NG == 4 ? b7[st] : (linfix ? bf5[st % 6] : br5[st % 6]);
      cau[st] = ca[st] * us[st];
    }
    // F of the mass flux is the stencil sum of the normal momentum; the
    // pressure enters the normal momentum and the energy flux
    double sp = 0.0, sup = 0.0;
#pragma unroll
    for (int st = 0; st < 2 * NG; ++st) {
      const double P_s = prim[PR_P * nc + p0 + st * stride];
      sp = fma(ca[st], P_s, sp);
      sup = fma(cau[st], P_s, sup);
    }
    double kF = 0.0, kW = 0.0, W0 = 0.0, Wn = 0.0;
#pragma unroll
    for (int m = 0; m < NV; ++m) {
      double F = m == 1 + D ? sp : (m == 4 ? sup : 0.0), W = 0.0, F0 = 0.0;
#pragma unroll
      for (int st = 0; st < 2 * NG; ++st) {
        const double w = v[m * nc + p0 + st * stride];
        if (m != 0) F = fma(cau[st], w, F);
        if (m == 1 + D) F0 = fma(ca[st], w, F0);
        W = fma(cb[st], w, W);
      }
      // kappa: q x_0 - u.x_m + x_4 + psi.x_s
      const double kc = m == 0 ? q : (m < 4 ? -uc[(m + 2) % 3] : (m == 4 ? 1.0 : psi[m >= IZEM_NIV ? m - IZEM_NIV : 0]));
      if (m != 0) kF = m == 4 ? kF + F : fma(kc, F, kF);
      kW = m == 4 ? kW + W : fma(kc, W, kW);
      if (m == 0) W0 = W;
      if (m == 1 + D) {
        Wn = W;
        kF = fma(q, F0, kF);
        fh[0] = F0;
      }
      if (m != 0) fh[m] = fma(lm1, W, F);
    }
    fh[0] = fma(lm1, W0, fh[0]);
    double psiY = 0.0;
#pragma unroll
    for (int l = 0; l < NRV; ++l) psiY = fma(psi[l], Yc[l], psiY);
    const double delta = -fm_div(1.0 + xi - b2 * psiY, psi[NRV - 1]);
    const double g0 = 0.5 * (lm0 - lm1), g2 = 0.5 * (lm2 - lm1);
    const double kb = b2 * kW, ac = (un * W0 - Wn) * cs_c_i;
    const double A = g0 * (kb + ac), B = g2 * (kb - ac);
    const double S = A + B, Dm = (B - A) * cs_c;
    fh[0] = fh[0] + S;
    fh[1 + D] = fma(un, S, fh[1 + D]) + Dm;
    fh[1 + T1] = fma(uc[T1], S, fh[1 + T1]);
    fh[1 + T2] = fma(uc[T2], S, fh[1 + T2]);
    fh[4] = fma(ht_c, S, fma(un, Dm, fh[4]));
#pragma unroll
    for (int l = 0; l < NRV; ++l)
      fh[IZEM_NIV + l] = fma(Yc[l], S, fh[IZEM_NIV + l]);
    fh[NV - 1] = fma(delta, fma(lm1, kW, kF), fh[NV - 1]);
  } else if (__popc(sensed) > kLanesMost) {
    // nonlinear reconstruction (wenorec): keep the 2NG stencil values of every
    // field.  The three acoustic/entropy rows of L are dense over (rho, m, rho
    // e_t) plus a rank-one species term psi.w, the shear rows have two
    // entries, the species rows are Y_s (a.w) + w_s (module_weno.f90:775-874).
    const double A0 = 0.5 * (b1 + un * cs_c_i), An = -0.5 * (b2 * un + cs_c_i);
    const double C0 = 0.5 * (b1 - un * cs_c_i), Cn = -0.5 * (b2 * un - cs_c_i);
    const double At1 = -0.5 * (b2 * uc[T1]), At2 = -0.5 * (b2 * uc[T2]);
    const double hb2 = 0.5 * b2;
    const double B1 = b2 * uc[0], B2 = b2 * uc[1], B3 = b2 * uc[2];
    const double opx = 1.0 + xi;
    const double E0 = opx * q, E1 = -opx * uc[0], E2 = -opx * uc[1], E3 = -opx * uc[2];
    double gh[NV];
    double gpl[NV][2 * NG], gmi[NV][2 * NG];
#pragma unroll 1
    for (int st = 0; st < 2 * NG; ++st) {
      const long long ps = p0 + st * stride;
      double w[NV], f[NV];
#pragma unroll
      for (int m = 0; m < NV; ++m) w[m] = v[m * nc + ps];
      const double u_s = prim[(PR_U + D) * nc + ps], P_s = prim[PR_P * nc + ps];
      f[0] = w[1 + D];
      f[1] = w[1] * u_s; f[2] = w[2] * u_s; f[3] = w[3] * u_s;
      f[1 + D] = w[1 + D] * u_s + P_s;
      f[4] = u_s * (w[4] + P_s);
#pragma unroll
      for (int l = IZEM_NIV; l < NV; ++l) f[l] = w[l] * u_s;
      double sw = 0.0, sf = 0.0;
#pragma unroll
      for (int l = 0; l < NRV; ++l) { sw = sw + psi[l] * w[IZEM_NIV + l]; sf = sf + psi[l] * f[IZEM_NIV + l]; }
      const double Gw = -b1 * w[0] + B1 * w[1] + B2 * w[2] + B3 * w[3] - b2 * w[4] - b2 * sw;
      const double Gf = -b1 * f[0] + B1 * f[1] + B2 * f[2] + B3 * f[3] - b2 * f[4] - b2 * sf;
      double pw[NV], pf[NV];
      pw[0] = A0 * w[0] + An * w[1 + D] + At1 * w[1 + T1] + At2 * w[1 + T2] + hb2 * w[4] + hb2 * sw;
      pf[0] = A0 * f[0] + An * f[1 + D] + At1 * f[1 + T1] + At2 * f[1 + T2] + hb2 * f[4] + hb2 * sf;
      pw[1] = w[0] + Gw;
      pf[1] = f[0] + Gf;
      pw[2] = C0 * w[0] + Cn * w[1 + D] + At1 * w[1 + T1] + At2 * w[1 + T2] + hb2 * w[4] + hb2 * sw;
      pf[2] = C0 * f[0] + Cn * f[1 + D] + At1 * f[1 + T1] + At2 * f[1 + T2] + hb2 * f[4] + hb2 * sf;
      pw[3] = -uc[T1] * w[0] + w[1 + T1];
      pf[3] = -uc[T1] * f[0] + f[1 + T1];
      pw[4] = -uc[T2] * w[0] + w[1 + T2];
      pf[4] = -uc[T2] * f[0] + f[1 + T2];
      pw[5] = E0 * w[0] + E1 * w[1] + E2 * w[2] + E3 * w[3] + opx * w[4] + xi * sw;
      pf[5] = E0 * f[0] + E1 * f[1] + E2 * f[2] + E3 * f[3] + opx * f[4] + xi * sf;
#pragma unroll
      for (int s = 0; s < NRV - 1; ++s) {
        pw[6 + s] = Yc[s] * Gw + w[IZEM_NIV + s];
        pf[6 + s] = Yc[s] * Gf + f[IZEM_NIV + s];
      }
#pragma unroll
      for (int m = 0; m < NV; ++m) {
        const double lam = m == 0 ? lm0 : (m == 2 ? lm2 : lm1);
        const double gp = 0.5 * (pf[m] + lam * pw[m]);
        gpl[m][st] = gp;
        gmi[m][st] = pf[m] - gp;
      }
    }
#pragma unroll 1
    for (int m = 0; m < NV; ++m) gh[m] = weno_nl<NG>(gpl[m], gmi[m]);
    // fhat = R ghat (module_weno.f90:881-989)
    fh[0] = gh[0] + gh[1] + gh[2];
    fh[1 + D] = (un - cs_c) * gh[0] + un * gh[1] + (un + cs_c) * gh[2];
    fh[1 + T1] = uc[T1] * gh[0] + uc[T1] * gh[1] + uc[T1] * gh[2] + gh[3];
    fh[1 + T2] = uc[T2] * gh[0] + uc[T2] * gh[1] + uc[T2] * gh[2] + gh[4];
    fh[4] = (ht_c - un * cs_c) * gh[0] + q * gh[1] + (ht_c + un * cs_c) * gh[2] + uc[T1] * gh[3] + uc[T2] * gh[4] + gh[5];
#pragma unroll
    for (int s = 0; s < NRV - 1; ++s) fh[IZEM_NIV + s] = Yc[s] * gh[0] + Yc[s] * gh[2] + gh[6 + s];
    const double wrk = -1.0 / psi[NRV - 1];
    double acc = Yc[NRV - 1] * gh[0] + Yc[NRV - 1] * gh[2] + wrk * gh[5];
#pragma unroll
    for (int s = 0; s < NRV - 1; ++s) acc = acc + (wrk * psi[s]) * gh[6 + s];
    fh[NV - 1] = acc;
  }
  if (valid && (!shk || __popc(sensed) > kLanesMost)) {
#pragma unroll
    for (int m = 0; m < NV; ++m) fhat[m * nfaces + idx] = fh[m];
  }
  if (sensed && __popc(sensed) <= kLanesMost) {
    FaceState<NRV> own;
#pragma unroll
    for (int d = 0; d < 3; ++d) own.uc[d] = uc[d];
#pragma unroll
    for (int l = 0; l < NRV; ++l) { own.Yc[l] = Yc[l]; own.psi[l] = psi[l]; }
    own.un = un; own.cs = cs_c; own.cs_i = cs_c_i; own.b2 = b2; own.xi = xi; own.q = q; own.ht = ht_c;
    own.lm0 = lm0; own.lm1 = lm1; own.lm2 = lm2;
    own.p0 = p0;
    weno_face_lanes<NRV, D, NG>(sensed, own, idx, nc, stride, v, prim, fhat, nfaces);
  }
}

// fl(i) = (fhat(i) - fhat(i-1)) * dx_i(i); the x sweep overwrites, y and z
// accumulate (module_weno.f90:995-1020, 1534-1558).
// With sensor blocks (bx < n[0], x sweep) the first cell of every block but
// the first takes its left face from fhat_edge, the block-edge faces as seen
// by that block (k_euler_face with edge = 1).
template <int D>
__global__ void k_flux_diff(Geo g, int nv, const double* __restrict__ fhat, long long nfaces,
                            const double* __restrict__ dxi, double* __restrict__ fl, int accumulate, int bx,
                            const double* __restrict__ fhat_edge, long long nedge) {
  long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= g.nint) return;
  int i = (int)(idx % g.n[0]) + 1;
  long long r = idx / g.n[0];
  int j = (int)(r % g.n[1]) + 1;
  int k = (int)(r / g.n[1]) + 1;
  // face index of the right face (s) in the face grid of axis D
  long long fr, fl_;
  int s;
  if (D == 0) { s = i; fr = (long long)i + (long long)(g.n[0] + 1) * ((j - 1) + (long long)g.n[1] * (k - 1)); fl_ = fr - 1; }
  else if (D == 1) { s = j; fr = (long long)(i - 1) + (long long)g.n[0] * (j + (long long)(g.n[1] + 1) * (k - 1)); fl_ = fr - g.n[0]; }
  else { s = k; fr = (long long)(i - 1) + (long long)g.n[0] * ((j - 1) + (long long)g.n[1] * k); fl_ = fr - (long long)g.n[0] * g.n[1]; }
  const double* fleft = fhat;
  long long nleft = nfaces;
  if (D == 0 && bx < g.n[0] && i > 1 && (i - 1) % bx == 0) {
    const int ne = g.n[0] / bx - 1;
    fleft = fhat_edge;
    nleft = nedge;
    fl_ = (long long)((i - 1) / bx - 1) + (long long)ne * ((j - 1) + (long long)g.n[1] * (k - 1));
  }
  // fl_W / fl_E (and S, N, B, F): the boundary points of a non-reflecting
  // face take 0 times their flux difference (module_weno.f90:620-623, 1002,
  // 1018); bc_noreflectionweno supplies their normal term
  const bool drop = (s == 1 && g.bc[2 * D] == IZEM_BC_NOREFLECTION) ||
                    (s == g.n[D] && g.bc[2 * D + 1] == IZEM_BC_NOREFLECTION);
  const double di = drop ? 0.0 : dxi[s - 1 + g.ng];
  for (int m = 0; m < nv; ++m) {
    const double df = fhat[m * nfaces + fr] - fleft[m * nleft + fl_];
    long long o = (long long)m * g.nint + idx;
    fl[o] = accumulate ? fma(df, di, fl[o]) : df * di;
  }
}

// bc_noreflectionweno (module_weno.f90:2129-4498), one face per launch, one
// thread per boundary point.  At the point's own state: the characteristic
// vectors of the flux Jacobian along the face normal D (the structure of
// k_euler_face's projections), the eigenvalues of the waves leaving the
// domain (min(., 0) on the low face, max(., 0) on the high one), and the
// one-sided derivative of the conserved variables over 2NG-1 points with
// wenopar's cnr weights (:199-217; for NG = 3 the reference keeps the first
// five of the 7-point set).  fl += R diag(L_s) L dw * dx_i.
template <int NRV, int D, int NG>
__global__ void k_bc_nr(Geo g, int hi, const double* __restrict__ v, const double* __restrict__ T,
                        const double* __restrict__ W_i, const double* __restrict__ cp,
                        const double* __restrict__ ha, const double* __restrict__ dxi, double* __restrict__ fl) {
  constexpr int NV = IZEM_NIV + NRV;
  constexpr int T1 = D == 0 ? 1 : 0;
  constexpr int T2 = D == 2 ? 1 : 2;
  const int m1 = D == 0 ? g.n[1] : g.n[0], m2 = D == 2 ? g.n[1] : g.n[2];
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= (long long)m1 * m2) return;
  const int q1 = (int)(idx % m1) + 1, q2 = (int)(idx / m1) + 1;
  const int sc = hi ? g.n[D] : 1;
  int c[3];
  c[D] = sc;
  c[D == 0 ? 1 : 0] = q1;
  c[D == 2 ? 1 : 2] = q2;
  const long long nc = g.ncell;
  const long long stride = D == 0 ? 1LL : (D == 1 ? (long long)g.g[0] : (long long)g.g[0] * g.g[1]);
  const long long p = gid(g, c[0], c[1], c[2]);
  const double rho_i = 1.0 / v[p];
  double uc[3];
  uc[0] = v[nc + p] * rho_i;
  uc[1] = v[2 * nc + p] * rho_i;
  uc[2] = v[3 * nc + p] * rho_i;
  const double P = v[p] * T[p] * W_i[p];
  double gam_c = c_thd.gam2 * W_i[p] / cp[p];
  gam_c = 1.0 / (1.0 - gam_c);
  const double cs_c = sqrt(gam_c * P * rho_i);
  double Yc[NRV], psi[NRV];
  double ht_c = 0.0;
  {
    const double wrk = (gam_c / (gam_c - 1.0)) * T[p];
#pragma unroll
    for (int l = 0; l < NRV; ++l) {
      Yc[l] = v[(IZEM_NIV + l) * nc + p] * rho_i;
      const double h = ha[l * nc + p];
      ht_c = ht_c + h * Yc[l];
      psi[l] = -h + wrk * c_thd.Wc_i[l];
    }
  }
  const double cs_c_i = 1.0 / cs_c;
  const double q = 0.5 * (uc[0] * uc[0] + uc[1] * uc[1] + uc[2] * uc[2]);
  ht_c = ht_c + q;
  const double b2 = (gam_c - 1.0) / (cs_c * cs_c);
  const double b1 = b2 * q;
  const double xi = b1 - b2 * ht_c;
  const double un = uc[D];
  // one-sided derivative (times the spacing) into the domain
  const double cnr[7] = {-49.0 / 20.0, 6.0, -15.0 / 2.0, 20.0 / 3.0, -15.0 / 4.0, 6.0 / 5.0, -1.0 / 6.0};
  const double sgn = hi ? -1.0 : 1.0;
  double w[NV];
#pragma unroll
  for (int m = 0; m < NV; ++m) w[m] = 0.0;
#pragma unroll
  for (int st = 0; st < 2 * NG - 1; ++st) {
    const long long ps = hi ? p - st * stride : p + st * stride;
    const double cw = sgn * cnr[st];
#pragma unroll
    for (int m = 0; m < NV; ++m) w[m] = w[m] + cw * v[m * nc + ps];
  }
  // L w (module_weno.f90:2224-2332 and the other faces' copies)
  double sw = 0.0;
#pragma unroll
  for (int l = 0; l < NRV; ++l) sw = sw + psi[l] * w[IZEM_NIV + l];
  const double hb2 = 0.5 * b2;
  const double Gw = -b1 * w[0] + b2 * uc[0] * w[1] + b2 * uc[1] * w[2] + b2 * uc[2] * w[3] - b2 * w[4] - b2 * sw;
  double pw[NV];
  pw[0] = 0.5 * (b1 + un * cs_c_i) * w[0] - 0.5 * (b2 * un + cs_c_i) * w[1 + D] - 0.5 * (b2 * uc[T1]) * w[1 + T1] -
          0.5 * (b2 * uc[T2]) * w[1 + T2] + hb2 * w[4] + hb2 * sw;
  pw[1] = w[0] + Gw;
  pw[2] = 0.5 * (b1 - un * cs_c_i) * w[0] - 0.5 * (b2 * un - cs_c_i) * w[1 + D] - 0.5 * (b2 * uc[T1]) * w[1 + T1] -
          0.5 * (b2 * uc[T2]) * w[1 + T2] + hb2 * w[4] + hb2 * sw;
  pw[3] = -uc[T1] * w[0] + w[1 + T1];
  pw[4] = -uc[T2] * w[0] + w[1 + T2];
  {
    const double opx = 1.0 + xi;
    pw[5] = opx * q * w[0] - opx * uc[0] * w[1] - opx * uc[1] * w[2] - opx * uc[2] * w[3] + opx * w[4] + xi * sw;
  }
#pragma unroll
  for (int s = 0; s < NRV - 1; ++s) pw[6 + s] = Yc[s] * Gw + w[IZEM_NIV + s];
  // the waves leaving the domain
  auto side = [&](double x) { return hi ? fmax(x, 0.0) : fmin(x, 0.0); };
  double gh[NV];
  gh[0] = side(un - cs_c) * pw[0];
  gh[2] = side(un + cs_c) * pw[2];
#pragma unroll
  for (int m = 0; m < NV; ++m)
    if (m != 0 && m != 2) gh[m] = side(un) * pw[m];
  // R gh (module_weno.f90:2334-2418)
  double fh[NV];
  fh[0] = gh[0] + gh[1] + gh[2];
  fh[1 + D] = (un - cs_c) * gh[0] + un * gh[1] + (un + cs_c) * gh[2];
  fh[1 + T1] = uc[T1] * gh[0] + uc[T1] * gh[1] + uc[T1] * gh[2] + gh[3];
  fh[1 + T2] = uc[T2] * gh[0] + uc[T2] * gh[1] + uc[T2] * gh[2] + gh[4];
  fh[4] = (ht_c - un * cs_c) * gh[0] + q * gh[1] + (ht_c + un * cs_c) * gh[2] + uc[T1] * gh[3] + uc[T2] * gh[4] + gh[5];
#pragma unroll
  for (int s = 0; s < NRV - 1; ++s) fh[IZEM_NIV + s] = Yc[s] * gh[0] + Yc[s] * gh[2] + gh[6 + s];
  {
    const double wrk = -1.0 / psi[NRV - 1];
    double acc = Yc[NRV - 1] * gh[0] + Yc[NRV - 1] * gh[2] + wrk * gh[5];
#pragma unroll
    for (int s = 0; s < NRV - 1; ++s) acc = acc + (wrk * psi[s]) * gh[6 + s];
    fh[NV - 1] = acc;
  }
  const double di = dxi[sc - 1 + g.ng];
  const long long o = fidx(g, c[0], c[1], c[2]);
#pragma unroll
  for (int m = 0; m < NV; ++m) fl[(long long)m * g.nint + o] += fh[m] * di;
}

// K3: Adams-Shariff sensor, sticky (only ever sets).  Interior neighbour tests
// along +x, +y, +z (module_tools.f90:2756-2812).
// With x blocks of bx points (bx < n[0]) a block's last point is not
// compared with the next block's first (each MPI block loops to its own ex).
__global__ void k_sensor(Geo g, double mrw, const double* __restrict__ v, const double* __restrict__ T,
                         const double* __restrict__ W_i, uint8_t* __restrict__ sensor, int bx) {
  long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= g.nint) return;
  int c[3];
  c[0] = (int)(idx % g.n[0]) + 1;
  long long r = idx / g.n[0];
  c[1] = (int)(r % g.n[1]) + 1;
  c[2] = (int)(r / g.n[1]) + 1;
  const long long p = gid(g, c[0], c[1], c[2]);
  const double rho = v[p];
  const double P = rho * T[p] * W_i[p];
  bool set = false;
  const long long strides[3] = {1LL, (long long)g.g[0], (long long)g.g[0] * g.g[1]};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (c[d] <= g.n[d] - 1 && !(d == 0 && c[0] % bx == 0)) {
      const long long q = p + strides[d];
      const double rq = v[q];
      const double Pq = rq * T[q] * W_i[q];
      // a pressure jump a hundredth below the threshold settles most points
      // without the quotients (positive pressures, compared as bit patterns)
      const long long pm = min(__double_as_longlong(P), __double_as_longlong(Pq));
      const double lim = (0.99 * mrw) * __longlong_as_double(pm);
      if (pm > 0 && __double_as_longlong(fabs(Pq - P)) < __double_as_longlong(lim)) continue;
      const double drho = fabs(rq - rho) * fmin(1.0 / rho, 1.0 / rq);
      const double dpres = fabs(Pq - P) / fmin(P, Pq);
      if (drho > mrw && dpres > mrw) set = true;
    }
  }
  if (set) sensor[p] = 1;
}
