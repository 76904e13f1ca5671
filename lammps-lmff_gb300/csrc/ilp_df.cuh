// The FP64 mode's interlayer pair terms in double-float arithmetic (dfloat.cuh): what
// calc_FvdW and calc_FRep (pair_ilp_graphene_hbn.cpp:449-675) form per pair, for two pairs
// at a time (V = float2) or one (V = float).
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
  K_LAM = 8,      // lambda
  K_LAM2 = 10,    // lambda log2(e)
  K_Z0 = 12,
  K_TSA = 14,     // (d / seff) log2(e)
  K_SEFF = 16,
  K_C6 = 18,
  K_DOS = 20,     // d / seff
  K_N = 22
};
// per potential constants
struct PairG {
  float irc_h, irc_l;        // 1 / r_cut
  float dt_h, dt_l;          // -140 / r_cut
  float cut_h, cut_l;        // r_cut^2
  int tap;
};

template <class V>
struct PairOut {
  D<V> crad;      // radial factor of the pair force: f = crad del - tp n_i - tq n_j
  D<V> tp, tq;    // Tap (n . del) fpair1 of the two repulsion terms
  D<V> evdw, erep;   // Tap V_vdw and Tap (V_ij + V_ji) (EV)
};

// del: x_i - x_j; q = |del|^2; pn = n_i . del, qn = n_j . del; on: 1 for a pair that counts
// (0 zeroes every output); K(k): constant k; tab: the exp2 table.  W (subdomain mode):
// weights wv of the vdW pair, wi and wj of the repulsion terms with n_i and n_j.
template <bool EV, bool W, class V, class KF>
static __device__ __forceinline__ void pair_terms(const PairG &g, KF K, const float2 *tab, D<V> q, D<V> pn, D<V> qn,
                                                  V on, V wv, V wi, V wj, PairOut<V> &o) {
  auto KD = [&](int k) { return mk<V>(K(k), K(k + 1)); };
  D<V> r, ri;
  sqrt_rsqrt(q, r, ri);
  // taper (pair_ilp_graphene_hbn.h:80-115) in y = 1 - x, x = r / r_cut: its degree-7
  // polynomial is y^4 (1 + 4x + 10x^2 + 20x^3), all terms positive, and
  // dTap/dr = -140 (x y)^3 / r_cut
  D<V> Tap = mk(on, vall<V>(0.f)), dTap = mk(vall<V>(0.f), vall<V>(0.f));
  if (g.tap) {
    const D<V> x = mul(r, mk(vall<V>(g.irc_h), vall<V>(g.irc_l)));
    const V one = vall<V>(1.f);
    const V s = vsub(one, x.h);
    const D<V> y = mk(s, vsub(vsub(vsub(one, s), x.h), x.l));
    const V c20 = vall<V>(20.f);
    const V u = vmul(c20, x.h);
    D<V> p = add1(mk(u, vfma(c20, x.l, vfma(c20, x.h, vneg(u)))), vall<V>(10.f));
    p = add1(mul(x, p), vall<V>(4.f));
    p = renorm(add1(mul(x, p), one));
    const D<V> y2 = sqr(y), xy = mul(x, y);
    Tap = renorm(mul(sqr(renorm(y2)), p));
    dTap = mul(renorm(mul(sqr(xy), xy)), mk(vall<V>(g.dt_h), vall<V>(g.dt_l)));
    Tap = mk(vmul(Tap.h, on), vmul(Tap.l, on));
    dTap = mk(vmul(dTap.h, on), vmul(dTap.l, on));
  }
  const D<V> DR = renorm(mul(dTap, ri));
  // ---- vdW: -C6 r^-6 / TS, TS = 1 + E, E = exp(-d (r / seff - 1)); 1 - 1/TS = E / TS
  const D<V> ri2 = sqr(ri);
  const D<V> rm = neg(r);
  const D<V> E = exp2(mul(add(KD(K_SEFF), rm), KD(K_TSA)), tab);
  const D<V> TSi = rcp(renorm(add1(E, vall<V>(1.f))));
  D<V> c6r6 = mul(renorm(mul(sqr(renorm(ri2)), ri2)), mul(TSi, KD(K_C6)));   // -V
  c6r6 = renorm(c6r6);
  if constexpr (W) c6r6 = mk(vmul(c6r6.h, wv), vmul(c6r6.l, wv));
  const D<V> G = add1(mul(renorm(mul(E, TSi)), mul(r, KD(K_DOS))), vall<V>(-6.f));
  // fpv Tap - V dTap / r = c6r6 (G Tap / r^2 + DR)
  const D<V> TR2 = mul(Tap, ri2);
  D<V> fv = mul(c6r6, renorm(add(mul(renorm(G), renorm(TR2)), DR)));
  // ---- repulsion of the terms with n_i and n_j: E0 (eps/2 + C e^{-rho^2/delta^2})
  const D<V> E0 = renorm(exp2(mul(add(KD(K_Z0), rm), KD(K_LAM2)), tab));
  const D<V> rho1 = renorm(add_ordered(q, neg(sqr(pn)))), rho2 = renorm(add_ordered(q, neg(sqr(qn))));
  D<V> F1 = mul(E0, exp2(mul(rho1, KD(K_ND2)), tab));
  D<V> F2 = mul(E0, exp2(mul(rho2, KD(K_ND2)), tab));
  D<V> Ee = mul(E0, KD(K_EPS));
  if constexpr (W) {
    F1 = mk(vmul(F1.h, wi), vmul(F1.l, wi));
    F2 = mk(vmul(F2.h, wj), vmul(F2.l, wj));
    const V wm = vmul(vall<V>(0.5f), vadd(wi, wj));
    Ee = mk(vmul(Ee.h, wm), vmul(Ee.l, wm));
  }
  const D<V> S = renorm(add(F1, F2));
  const D<V> VS = renorm(add(Ee, mul(S, KD(K_C))));
  const D<V> TC = renorm(mul(Tap, KD(K_C2D)));   // Tap 2 C / delta^2
  const D<V> LT = add(mul(mul(Tap, ri), KD(K_LAM)), neg(DR));
  o.crad = renorm(add(fv, add(mul(S, TC), mul(VS, renorm(LT)))));
  o.tp = renorm(mul(mul(pn, TC), F1));
  o.tq = renorm(mul(mul(qn, TC), F2));
  if constexpr (EV) {
    o.evdw = neg(mul(c6r6, Tap));
    o.erep = mul(VS, Tap);
  }
}

}  // namespace df
}  // namespace lmff
