// EGLIB's temperature functions of one point from a table.
//
// All that EGSPAR/LSPAR, EGSE2, EGSLCT2 and EGSDR1 take from the temperature
// -- 36 binary diffusion fits, 117 collision-integral fits, 9 viscosities and
// Parker's relaxation, for nine species 45 exponentials and 1600 other FP64
// operations a point -- enters the mixture formulas through five functions of
// T a species pair and three a species.  They are smooth, and the FP64 pipe
// bounds the point kernel (two operations a clock and SM), so they are
// tabulated when the linking data are set: polynomials of degree 5 on 256
// intervals an octave of T, coefficients and Horner's rule in 64-bit fixed
// point on the integer pipes (about 50 instructions a function, no FP64
// operation).  Degree and width: for T^-p with p <= 5 the interpolation error
// is below 2^-55, half a rounding of the result; degree 4 would need four
// times the intervals.  The nodes' values are formed in double-double
// arithmetic, so that a tabulated value is closer to the exact one (3e-16)
// than the direct FP64 evaluation, whose exponents of size 30 lose 5e-15.
//
// One row of the table (NF functions x 48 bytes, 9.9 kB for nine species) is
// read per point; neighbouring points share it.  128 K <= T < 4096 K are
// tabulated (1280 rows, 12.7 MB, resident in L2); elsewhere a point evaluates
// the functions directly.
#pragma once
#include "common.cuh"
#include "fmath.cuh"

constexpr int kEgBits = 8;                     // 2^8 intervals an octave
constexpr int kEgOct0 = 7, kEgOct1 = 12;       // 2^7 K .. 2^12 K
constexpr int kEgRows = (kEgOct1 - kEgOct0) << kEgBits;
constexpr int kEgNodes = 6;

// function indices: f1 of every pair, the species' shear term, f2..f4 of every
// pair, the species' two conductivity terms, f5 of every pair (the order in
// which the point kernel reads them)
template <int N>
struct EgIdx {
  static constexpr int NP = N * (N - 1) / 2;
  static constexpr int bin = 0, shear = NP, lam = NP + N, spec = lam + 3 * NP, chi = spec + 2 * N, NF = chi + NP;
};
// pair index, i < j
template <int N>
__host__ __device__ constexpr int egp(int i, int j) { return i * N - i * (i + 1) / 2 + j - i - 1; }

// ---- double-double arithmetic (T. J. Dekker, Numer. Math. 18, 1971)
struct dd {
  double h, l;
  dd() = default;
  __device__ dd(double a, double b = 0.0) : h(a), l(b) {}
};
__device__ __forceinline__ dd dd_fast(double a, double b) {
  const double s = __dadd_rn(a, b);
  return dd(s, __dsub_rn(b, __dsub_rn(s, a)));
}
__device__ __forceinline__ dd operator+(dd a, dd b) {
  const double s = __dadd_rn(a.h, b.h), t = __dsub_rn(s, a.h);
  const double e = __dadd_rn(__dsub_rn(a.h, __dsub_rn(s, t)), __dsub_rn(b.h, t));
  return dd_fast(s, __dadd_rn(e, __dadd_rn(a.l, b.l)));
}
__device__ __forceinline__ dd operator-(dd a) { return dd(-a.h, -a.l); }
__device__ __forceinline__ dd operator-(dd a, dd b) { return a + (-b); }
__device__ __forceinline__ dd operator*(dd a, dd b) {
  const double p = __dmul_rn(a.h, b.h);
  return dd_fast(p, __fma_rn(a.h, b.h, -p) + (__dmul_rn(a.h, b.l) + __dmul_rn(a.l, b.h)));
}
__device__ __forceinline__ dd operator/(dd a, dd b) {
  const double q = a.h / b.h;
  const dd r = a - b * dd(q);
  return dd_fast(q, (r.h + r.l) / b.h);
}
__device__ inline dd eg_sqrt(dd a) {
  const double s = sqrt(a.h);
  const dd r = a - dd(s) * dd(s);
  return dd_fast(s, (r.h + r.l) / (2.0 * s));
}
// e^a: a = k ln 2 + 64 r, Taylor's series of e^r (|r| < 0.0055: the term after
// the last is below 1e-33), squared six times
__device__ __noinline__ dd eg_exp(dd a) {
  const double k = rint(a.h * 1.4426950408889634);
  const dd ln2(0.6931471805599453, 2.3190468138462996e-17);
  dd r = a - dd(k) * ln2;
  r.h *= 0.015625;
  r.l *= 0.015625;
  dd s(1.0);
#pragma unroll 1
  for (int n = 11; n >= 1; --n) {
    const double q = 1.0 / n;
    s = dd(1.0) + s * (r * dd(q, fma(-q, (double)n, 1.0) * q));
  }
#pragma unroll 1
  for (int n = 0; n < 6; ++n) s = s * s;
  return dd(ldexp(s.h, (int)k), ldexp(s.l, (int)k));
}
// ln a by one Newton step on e^y = a from the double value
__device__ inline dd eg_log(dd a) {
  const dd y(log(a.h));
  const dd d = a * eg_exp(-y) - dd(1.0);   // small
  return y + (d - dd(0.5) * d * d);
}
__device__ __forceinline__ double eg_sqrt(double a) { return sqrt(a); }
__device__ __forceinline__ double eg_exp(double a) { return fm_exp(a); }
__device__ __forceinline__ double eg_log(double a) { return fm_log(a); }

template <class R>
__device__ inline R eg_poly(const double* f, int deg, R x) {
  R s(f[deg]);
  for (int q = deg - 1; q >= 0; --q) s = s * x + R(f[q]);
  return s;
}
// Parker's rotational relaxation of species i (internal energy exchange)
template <class R>
__device__ inline R eg_cxi(int i, R Tinv) {
  const R d = R(c_eg.eps[i]) * Tinv, s = eg_sqrt(d);
  return R(c_eg.cx[i]) * (R(1.0) + R(2.7842) * s + R(4.4674) * d + R(5.5683) * (s * d));
}
// the five functions of a pair: the reciprocal diffusion coefficient b, and
// with EGLIB's A*, B*, C* minus the off-diagonal and the two diagonal terms of
// Lambda_[e] and the thermal-diffusion factor, each times b
template <class R>
__device__ inline void eg_pair_T(R T, R lnT, int i, int j, R* o) {
  const R Tinv = R(1.0) / T;
  const R b = eg_exp(-eg_poly<R>(c_eg.cofd[i][j], 3, lnT));
  const R A = eg_poly<R>(c_eg.fita[i][j], 6, lnT), B = eg_poly<R>(c_eg.fitb[i][j], 6, lnT);
  const R C = eg_poly<R>(c_eg.fitc[i][j], 6, lnT);
  const R xi = eg_cxi<R>(i, Tinv), xj = eg_cxi<R>(j, Tinv);
  const R b3 = R(6.25) - R(3.0) * B, a4 = R(4.0 * c_eg.p1[i][j]) * A;
  o[0] = b;
  o[1] = b * R(c_eg.p1[i][j]) * (R(13.75) - R(3.0) * B - R(4.0) * A + A * (R(c_eg.tti[i][j]) * xi + R(c_eg.ttj[i][j]) * xj));
  o[2] = b * (R(c_eg.c1j[i][j]) + b3 * R(c_eg.c2j[i][j]) + a4 + A * (R(c_eg.c3j[i][j]) * xi + R(c_eg.c4[i][j]) * xj));
  o[3] = b * (R(c_eg.c1i[i][j]) + b3 * R(c_eg.c2i[i][j]) + a4 + A * (R(c_eg.c3i[i][j]) * xj + R(c_eg.c4[i][j]) * xi));
  o[4] = R(0.5 * c_eg.wsinv[i][j]) * b * (R(6.0) * C - R(5.0));
}
// the three functions of a species: the diagonal term of the shear matrix
// (1 / eta over its common factor 6 RU T / (5 PATM)), and of Lambda_[e] the
// coefficients of x^2 and of x^2 c_int
template <class R>
__device__ inline void eg_spec_T(R T, R lnT, int i, R* o) {
  const R Tinv = R(1.0) / T;
  const R e = eg_exp(-eg_poly<R>(c_eg.cofe[i], 3, lnT)) * Tinv;
  o[0] = e * R(5.0 * 1.01325e6 / (6.0 * 8.314e7));
  o[1] = R(c_eg.lfac[i]) * e * (R(1.0) + R(8.0 / 15.0) * eg_cxi<R>(i, Tinv));
  R b = R(c_eg.bdiag[i]) * e / eg_poly<R>(c_eg.fita[i][i], 6, lnT);
  if (c_eg.dip[i] != 0.0) b = b * (R(1.0) + R(2.985e3) / (T * eg_sqrt(T)));
  o[2] = b;
}
// where function q of pair / species `item` sits
template <int N>
__device__ __forceinline__ int eg_slot(int item, int q) {
  using I = EgIdx<N>;
  if (item < I::NP) return q == 0 ? I::bin + item : (q == 4 ? I::chi + item : I::lam + 3 * item + q - 1);
  const int s = item - I::NP;
  return q == 0 ? I::shear + s : I::spec + 2 * s + q - 1;
}
template <int N>
__device__ inline void eg_pair_of(int item, int& i, int& j) {
  i = 0;
  while (item >= N - 1 - i) { item -= N - 1 - i; ++i; }
  j = i + 1 + item;
}

// ---- building the table
// Chebyshev nodes of [0, 1] in units of 2^-30 (the temperatures are exact)
// and the inverse of their Vandermonde matrix in units of 2^-52
static __constant__ int c_eg_node[kEgNodes] = {18293433, 157245850, 397918495, 675823329, 916495974, 1055448391};
static __constant__ long long c_eg_inv[kEgNodes][kEgNodes] = {
    {5701372584849615LL, -1812108583772799LL, 978200905028637LL, -575955601462573LL, 310908681141299LL, -98818358413683LL},
    {-75854022385758718LL, 118097964976368255LL, -67790890475839824LL, 40553729862146378LL, -22021172574861115LL, 7014390597945025LL},
    {336864669092674550LL, -715747841199520660LL, 638762054067681227LL, -419371308408396926LL, 235363879506084183LL, -75871453058522374LL},
    {-661285673062846605LL, 1607165095596133152LL, -1782238773372728254LL, 1397931603281546543LL, -838550757012274476LL, 276978504570169640LL},
    {593406864272332962LL, -1550884613749467969LL, 1952137893775462449LL, -1759984308729871593LL, 1166577444457538631LL, -401253280025994480LL},
    {-198932028859665488LL, 543492411641401320LL, -742424440501066808LL, 742424440501066808LL, -543492411641401320LL, 198932028859665488LL}};

// Coefficients of one function on one interval from its values at the nodes:
// c_n 2^n in units of 2^(E-62) (each step of the evaluation halves), the two
// last ones in units 64 times that, as 32-bit words.  2^E bounds the values;
// where a function changes its sign inside the interval (6 C* - 5 does) E
// grows until the coefficients fit.  False: not a finite function, or one
// that should be positive and is not.
__device__ inline bool eg_coef(const dd* v, int stride, bool positive, long long* __restrict__ o) {
  double mx = 0.0;
  for (int k = 0; k < kEgNodes; ++k) {
    const double x = v[k * stride].h;
    if (!(fabs(x) < 1e300) || (positive && !(x > 0.0))) return false;
    mx = fmax(mx, fabs(x));
  }
  int E = 0;
  if (mx > 0.0) frexp(mx, &E);   // mx < 2^E
  for (int tries = 0; tries < 48; ++tries, ++E) {
    long long F[kEgNodes], c[kEgNodes];
    for (int k = 0; k < kEgNodes; ++k)
      F[k] = llrint(ldexp(v[k * stride].h, 61 - E)) + llrint(ldexp(v[k * stride].l, 61 - E));
    bool fits = true;
    for (int n = 0; n < kEgNodes; ++n) {
      __int128 s = 0;
      for (int k = 0; k < kEgNodes; ++k) s += (__int128)c_eg_inv[n][k] * (F[k] - F[0]);
      s = (s + ((__int128)1 << 51)) >> 52;
      if (n == 0) s += F[0];
      s = s << n;
      if (s > (__int128)0x3fffffffffffffffLL || s < -(__int128)0x3fffffffffffffffLL) fits = false;
      c[n] = (long long)s;
    }
    const long long c4 = (c[4] + 32) >> 6, c5 = (c[5] + 32) >> 6;
    if (c4 > 0x3fffffffLL || c4 < -0x3fffffffLL || c5 > 0x3fffffffLL || c5 < -0x3fffffffLL) fits = false;
    if (!fits) continue;
    for (int n = 0; n < 4; ++n) o[n] = c[n];
    o[4] = (long long)((unsigned long long)c5 << 32 | (unsigned long long)(unsigned)c4);
    o[5] = E + 1;
    return true;
  }
  return false;
}

// One block per row; one thread per pair and species.
constexpr int kEgBuildThreads = 64;
template <int N>
__global__ void k_eg_table(long long* __restrict__ tab, int* bad) {
  using I = EgIdx<N>;
  static_assert(I::NP + N <= kEgBuildThreads, "one thread per pair and species");
  __shared__ dd s_T[kEgNodes], s_ln[kEgNodes];
  const int row = blockIdx.x, item = threadIdx.x;
  if (item < kEgNodes) {
    const double m = (double)((1 << kEgBits) + (row & ((1 << kEgBits) - 1))) + c_eg_node[item] * (1.0 / 1073741824.0);
    const dd T(ldexp(m, kEgOct0 + (row >> kEgBits) - kEgBits));
    s_T[item] = T;
    s_ln[item] = eg_log(T);
  }
  __syncthreads();
  if (item >= I::NP + N) return;
  dd v[kEgNodes * 5];
  int i = 0, j = 0;
  if (item < I::NP) eg_pair_of<N>(item, i, j);
#pragma unroll 1
  for (int k = 0; k < kEgNodes; ++k) {
    if (item < I::NP) eg_pair_T<dd>(s_T[k], s_ln[k], i, j, v + 5 * k);
    else eg_spec_T<dd>(s_T[k], s_ln[k], item - I::NP, v + 5 * k);
  }
#pragma unroll 1
  for (int q = 0; q < (item < I::NP ? 5 : 3); ++q) {
    const int f = eg_slot<N>(item, q);
    if (!eg_coef(v + q, 5, f < I::chi, tab + ((long long)row * I::NF + f) * 6)) *bad = 1;
  }
}

// ---- reading it
struct EgRow {
  const longlong2* row;   // null: outside the table
  int hi;                 // position in the interval, units of 2^-31 ...
  unsigned lo;            // ... and the bits below it
};
template <int N>
__device__ __forceinline__ EgRow eg_row(const long long* __restrict__ tab, double T) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(T);
  const unsigned q = (unsigned)(u >> (52 - kEgBits)) - ((1023u + kEgOct0) << kEgBits);
  EgRow r{nullptr, 0, 0};
  // negative T, NaN and infinity give a large q
  if (!tab || (u >> 63) || q >= (unsigned)kEgRows) return r;
  r.row = reinterpret_cast<const longlong2*>(tab + (long long)q * EgIdx<N>::NF * 6);
  const unsigned long long x = (u << (12 + kEgBits)) >> 1;
  r.hi = (int)(x >> 32);
  r.lo = (unsigned)x;
  return r;
}
// c + q x / 2 with x = hi:lo, two units short at most (the low product is left out)
__device__ __forceinline__ long long eg_step(long long c, long long q, const EgRow& r) {
  const int qh = (int)(q >> 32);
  const unsigned ql = (unsigned)q;
  c += (long long)qh * r.hi;
  c += ((long long)qh * (long long)r.lo) >> 32;
  c += ((long long)((unsigned long long)ql * (unsigned)r.hi)) >> 32;   // below 2^63
  return c;
}
// function f at the row's point; POS: a positive one
template <bool POS>
__device__ __forceinline__ double eg_eval(const EgRow& r, int f) {
  const longlong2 a = __ldg(r.row + 3 * f), b = __ldg(r.row + 3 * f + 1), c = __ldg(r.row + 3 * f + 2);
  const int q4 = (int)c.x + __mulhi((int)(c.x >> 32), r.hi);
  long long q = b.y + ((long long)__mulhi(q4, r.hi) << 6);
  q = eg_step(b.x, q, r);
  q = eg_step(a.y, q, r);
  q = eg_step(a.x, q, r);
  unsigned long long m = (unsigned long long)q, sign = 0;
  if (!POS) {
    sign = m & 0x8000000000000000ULL;
    if (sign) m = 0 - m;
    if (m == 0) return 0.0;
  }
  // the leading bit to bit 62, rounded to 53 bits
  const int z = POS ? __clz((int)(m >> 32)) : __clzll((long long)m);
  const unsigned long long s = ((m << (z - 1)) + 0x200) >> 10;
  return __longlong_as_double((long long)(sign | (((unsigned long long)(unsigned)((int)c.y + 1023 - z) << 52) + s)));
}
// every function of a point outside the table
template <int N>
__device__ __noinline__ void eg_direct(double T, double* tv) {
  using I = EgIdx<N>;
  const double lnT = fm_log(T);
  double o[5];
#pragma unroll 1
  for (int item = 0; item < I::NP + N; ++item) {
    int i, j;
    if (item < I::NP) {
      eg_pair_of<N>(item, i, j);
      eg_pair_T<double>(T, lnT, i, j, o);
    } else {
      eg_spec_T<double>(T, lnT, item - I::NP, o);
    }
    for (int q = 0; q < (item < I::NP ? 5 : 3); ++q) tv[eg_slot<N>(item, q)] = o[q];
  }
}
