// The FP64 mode's interlayer pair terms in double-float arithmetic (dfloat.cuh): what
// calc_FvdW and calc_FRep (pair_ilp_graphene_hbn.cpp:449-675) form per pair.
//
// With q = r^2, Tap and dTap of r, E0 = e^{-lambda (r - z0)}, E = e^{-d (r/seff - 1)},
// X = 1/(r^6 (1 + E)), G_n = e^{-rho_n^2/delta^2} of the two normals n, S = G_i + G_j:
//   f on i = crad del - tp n_i - tq n_j
//   crad = A + (C M + B) S, B = TE 2C/delta^2, tp = (n_i.del) B G_i, tq = (n_j.del) B G_j
//   A  = [C6 X (Tap (d/seff E r^6 X - 6/r) + dTap) + (lambda Tap - dTap) E0 eps] / r
//   TE = Tap E0,  M = (lambda Tap - dTap) E0 / r,  U = -C6 X Tap + eps TE
//   energies: vdW U - eps TE, repulsion V_ij + V_ji = TE (eps + C S)
// A, M, U and TE depend on q and the element pair alone, A = -2 dU/dq and M = -2 dTE/dq.
// They are tabulated per potential: 2^TAB_BITS intervals per factor of two in q; on each,
// A and M are polynomials of degree 4 in q about the interval's centre (Chebyshev
// interpolation of FP64 values, the interpolation error below 2e-14 of the function where
// it is steepest and 1e-15 over most of the range), U and TE their integrals from the FP64
// values at the centre.  A takes 26 FP32 instructions, where square root, taper, two
// exponentials and the divisions of it take about 290 in double-float arithmetic; two
// 16-byte loads bring its coefficients, since the gathers of the tables load the L1 pipe
// (degree 6 over half as many intervals, three loads: the pipe 76 % busy and the kernel
// no faster than the direct evaluation).
//
// The part the normals enter is left out for lanes whose pairs lie so far sideways
// (rho > 8 A for carbon) that G_n < 2^-64: S is then below a double's rounding of the rest.
#pragma once

#include "dfloat.cuh"

namespace lmff {
namespace df {

// per element pair constants, each as hi and lo
enum PairK {
  K_ND2 = 0,      // -log2(e) / delta^2
  K_C = 2,        // C
  K_EPS = 4,      // epsilon (both repulsion terms' halves together)
  K_C2D = 6,      // 2 C / delta^2
  K_N = 8
};

constexpr float Q_MIN = 0.25f;          // A^2: the tables' range, [Q_MIN, Q_MAX)
constexpr float Q_MAX = 1024.f;
constexpr int TAB_BITS = 9;             // mantissa bits of q that select an interval
constexpr int TAB_SHIFT = 23 - TAB_BITS;
constexpr int TAB_BASE = (127 - 2) << TAB_BITS;          // of Q_MIN = 2^-2
constexpr int TAB_N = 12 << TAB_BITS;                    // 12 octaves

// the parameters of one element pair, for the tables
struct TabP {
  double z0, lambda, eps, d, seff, C6, cut;
  int tap;
};
// A, M, U and TE at q in FP64
static __device__ inline void tab_functions(const TabP &p, double q, double &A, double &M, double &U, double &TE) {
  const double r = sqrt(q), ri = 1.0 / r;
  double Tap = 1.0, dTap = 0.0;
  if (p.tap) {
    const double x = r / p.cut, y = 1.0 - x, xy = x * y;
    Tap = (y * y) * (y * y) * (1.0 + x * (4.0 + x * (10.0 + x * 20.0)));
    dTap = -140.0 / p.cut * (xy * xy * xy);
  }
  const double E = exp(-p.d * (r / p.seff - 1.0)), E0 = exp(-p.lambda * (r - p.z0));
  const double c = p.C6 / (q * q * q * (1.0 + E));
  M = (p.lambda * Tap - dTap) * E0 * ri;
  A = ri * (c * (Tap * (p.d / p.seff * (E / (1.0 + E)) - 6.0 * ri) + dTap)) + M * p.eps;
  TE = Tap * E0;
  U = p.eps * TE - c * Tap;
}
// interval k's coefficients: of A and M c0, c1, c2 (hi, lo), c3, c4, and U and TE at the centre
static __device__ inline void tab_fill(const TabP &p, int k, float ca[8], float cm[8], float u[2], float te[2]) {
  const double lo = ldexp(1.0 + (k & ((1 << TAB_BITS) - 1)) / (double)(1 << TAB_BITS), (k >> TAB_BITS) - 2);
  const double half = 0.5 * ldexp(1.0, (k >> TAB_BITS) - 2 - TAB_BITS), mid = lo + half;
  double v[2][5], U, TE;
  for (int j = 0; j < 5; j++) tab_functions(p, mid + half * cos(M_PI * (2 * j + 1) / 10.0), v[0][j], v[1][j], U, TE);
  for (int f = 0; f < 2; f++) {
    double a[5];
    for (int m = 0; m < 5; m++) {
      double s = 0.0;
      for (int j = 0; j < 5; j++) s += v[f][j] * cos(M_PI * (m * (2 * j + 1)) / 10.0);
      a[m] = s * (m ? 0.4 : 0.2);
    }
    // Chebyshev to powers of (q - mid) / half, then of q - mid
    const double c[5] = {a[0] - a[2] + a[4], a[1] - 3.0 * a[3], 2.0 * a[2] - 8.0 * a[4], 4.0 * a[3], 8.0 * a[4]};
    float *o = f ? cm : ca;
    double w = 1.0;
    for (int m = 0; m < 5; m++, w /= half) {
      const float h = (float)(c[m] * w);
      if (m < 3) {
        o[2 * m] = h;
        o[2 * m + 1] = (float)(c[m] * w - (double)h);
      } else {
        o[3 + m] = h;
      }
    }
  }
  double a, m;
  tab_functions(p, mid, a, m, U, TE);
  u[0] = (float)U;
  u[1] = (float)(U - (double)u[0]);
  te[0] = (float)TE;
  te[1] = (float)(TE - (double)te[0]);
}

// The same functions in FP64 (the per-atom virial's near pairs): 2^TAB64_BITS intervals
// per factor of two, A and M of degree 6 and TE of degree 7 (M's integral), 8 doubles each
constexpr int TAB64_BITS = 7;
constexpr int TAB64_SHIFT = 23 - TAB64_BITS;
constexpr int TAB64_BASE = (127 - 2) << TAB64_BITS;
constexpr float Q64_MAX = 64.f;         // their range, [Q_MIN, Q64_MAX)
constexpr int TAB64_N = 8 << TAB64_BITS;
static __device__ inline void tab64_fill(const TabP &p, int k, double *ca, double *cm, double *ct) {
  const double lo = ldexp(1.0 + (k & ((1 << TAB64_BITS) - 1)) / (double)(1 << TAB64_BITS), (k >> TAB64_BITS) - 2);
  const double half = 0.5 * ldexp(1.0, (k >> TAB64_BITS) - 2 - TAB64_BITS), mid = lo + half;
  double v[2][7], U, TE;
  for (int j = 0; j < 7; j++) tab_functions(p, mid + half * cos(M_PI * (2 * j + 1) / 14.0), v[0][j], v[1][j], U, TE);
  for (int f = 0; f < 2; f++) {
    double a[7];
    for (int m = 0; m < 7; m++) {
      double s = 0.0;
      for (int j = 0; j < 7; j++) s += v[f][j] * cos(M_PI * (m * (2 * j + 1)) / 14.0);
      a[m] = s * (m ? 2.0 : 1.0) / 7.0;
    }
    const double c[7] = {a[0] - a[2] + a[4] - a[6], a[1] - 3.0 * a[3] + 5.0 * a[5], 2.0 * a[2] - 8.0 * a[4] + 18.0 * a[6],
                         4.0 * a[3] - 20.0 * a[5], 8.0 * a[4] - 48.0 * a[6], 16.0 * a[5], 32.0 * a[6]};
    double w = 1.0;
    for (int m = 0; m < 7; m++, w /= half) (f ? cm : ca)[m] = c[m] * w;
  }
  double a, m;
  tab_functions(p, mid, a, m, U, TE);
  ca[7] = cm[7] = 0.0;
  ct[0] = TE;
  for (int k2 = 0; k2 < 7; k2++) ct[k2 + 1] = -0.5 * cm[k2] / (k2 + 1);
}
// interval of q and q minus its centre.  The interval is the FP32 neighbour's, at most one
// rounding outside which its polynomial serves; the clamps are for a q whose FP32 sum is
// inside the range while q itself rounds to its end
static __device__ __forceinline__ int tab64_at(double q, double &t) {
  const int u = min(max(__float_as_int((float)q), TAB64_BASE << TAB64_SHIFT),
                    ((TAB64_BASE + TAB64_N) << TAB64_SHIFT) - 1);
  t = q - (double)__int_as_float((u & ~((1 << TAB64_SHIFT) - 1)) | (1 << (TAB64_SHIFT - 1)));
  return (u >> TAB64_SHIFT) - TAB64_BASE;
}
template <int N>
static __device__ __forceinline__ double tab64_poly(const double *c, double t) {
  double s = __ldg(c + N);
#pragma unroll
  for (int k = N - 1; k >= 0; k--) s = fma(s, t, __ldg(c + k));
  return s;
}

// interval of q.h (in [Q_MIN, Q_MAX)) and q.h minus its centre (exact)
static __device__ __forceinline__ int tab_at(float qh, float &t) {
  const int u = __float_as_int(qh);
  t = __fsub_rn(qh, __int_as_float((u & ~((1 << TAB_SHIFT) - 1)) | (1 << (TAB_SHIFT - 1))));
  return (u >> TAB_SHIFT) - TAB_BASE;
}
// one interval's coefficients
struct Coef {
  float c0h, c0l, c1h, c1l, c2h, c2l, c3, c4;
};
static __device__ __forceinline__ void coef_set(Coef &o, const float4 *a) {
  const float4 x = __ldg(a), y = __ldg(a + 1);
  o.c0h = x.x; o.c0l = x.y; o.c1h = x.z; o.c1l = x.w;
  o.c2h = y.x; o.c2l = y.y; o.c3 = y.z; o.c4 = y.w;
}
// the polynomial at t (normalised).  |t| is below 2^-TAB_BITS-1 of q, so the terms fall off
// by ~2^-7 each and FP32 serves from the third power on
static __device__ __forceinline__ D tab_poly(const Coef &c, D t) {
  D s = mul(mk(c.c2h, vfma(vfma(c.c4, t.h, c.c3), t.h, c.c2l)), t);
  const D s1 = two_sum(c.c1h, s.h);
  s = mul(mk(s1.h, vadd(s1.l, vadd(s.l, c.c1l))), t);
  const D s0 = two_sum(c.c0h, s.h);
  return mk(s0.h, vadd(s0.l, vadd(s.l, c.c0l)));
}
// f0 - 1/2 the integral of the polynomial from 0 to t
static __device__ __forceinline__ D tab_integral(const Coef &c, float f0h, float f0l, D t) {
  const float half = 0.5f;
  float u = vfma(vmul(c.c4, 0.2f), t.h, vmul(c.c3, 0.25f));
  u = vfma(u, t.h, vmul(c.c2h, 1.f / 3.f));
  D s = mul(mk(vmul(half, c.c1h), vfma(u, t.h, vmul(half, c.c1l))), t);
  const D s1 = two_sum(c.c0h, s.h);
  s = scale(mul(mk(s1.h, vadd(s1.l, vadd(s.l, c.c0l))), t), -0.5f);
  const D s0 = two_sum(f0h, s.h);
  return mk(s0.h, vadd(s0.l, vadd(s.l, f0l)));
}

// whether G_n of a pair can matter: log2 G_n above FAR_EXP for either normal, in FP32
constexpr float FAR_EXP = -64.f;
static __device__ __forceinline__ bool near_one(float nd2, float q, float p1, float p2) {
  return nd2 * (q - p1 * p1) > FAR_EXP || nd2 * (q - p2 * p2) > FAR_EXP;
}

// The parts the normals enter: crad += (C M + B) S, tp, tq, and S (weighted).  pn = n_i .
// del, qn = n_j . del; K(k): constant k; tab: the exp2 table.  W (subdomain mode): weights
// wi and wj of the repulsion terms with n_i and n_j.
template <bool W, class KF>
static __device__ __forceinline__ void pair_near(KF K, const float2 *tab, D q, D TE, D M, D pn, D qn, float wi,
                                                 float wj, D &crad, D &tp, D &tq, D &S) {
  auto KD = [&](int k) { return mk(K(k), K(k + 1)); };
  const D rho1 = add_ordered(q, neg(sqr(pn))), rho2 = add_ordered(q, neg(sqr(qn)));
  D G1 = exp2(mul(renorm(rho1), KD(K_ND2)), tab);
  D G2 = exp2(mul(renorm(rho2), KD(K_ND2)), tab);
  if constexpr (W) {
    G1 = scale(G1, wi);
    G2 = scale(G2, wj);
  }
  S = renorm(add(G1, G2));
  const D B = renorm(mul(TE, KD(K_C2D)));
  tp = mul(mul(pn, B), G1);
  tq = mul(mul(qn, B), G2);
  crad = add(crad, mul(S, renorm(add(mul(M, KD(K_C)), B))));
}

}  // namespace df
}  // namespace lmff
