// Double-float arithmetic: a value held as the unevaluated sum of two FP32 numbers, about
// 48 significand bits, in FP32 instructions only.  GB300 issues FP64 at 1/75 of its FP32
// rate (measured: 0.52 against 39 T lane operations per second), and a double-float
// product costs 4 FP32 instructions and a sum 8, so the FP64 mode's heavy arithmetic runs
// here several times faster than on the FP64 pipe.
//
// Everything is built from error-free transformations (T. J. Dekker, Numer. Math. 18, 1971;
// D. E. Knuth, TAOCP vol. 2): two_sum and the FMA product error.  (Two values at a time with
// the packed FP32x2 instructions took half the issue slots at the same arithmetic rate, and
// twice the registers: the pair kernel was 10 % slower.)
//
// Results are left unnormalised (|l| of a few ulp of h): products and sums accept that, and
// renorm is called where a chain would let it grow.
#pragma once

#include <cuda_runtime.h>

namespace lmff {
namespace df {

#define LMFF_DF static __device__ __forceinline__
LMFF_DF float vneg(float a) { return -a; }
LMFF_DF float vadd(float a, float b) { return __fadd_rn(a, b); }
LMFF_DF float vsub(float a, float b) { return __fsub_rn(a, b); }
LMFF_DF float vmul(float a, float b) { return __fmul_rn(a, b); }
LMFF_DF float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
struct D {
  float h, l;
};
LMFF_DF D mk(float h, float l) {
  D r;
  r.h = h;
  r.l = l;
  return r;
}
LMFF_DF D neg(D a) { return mk(vneg(a.h), vneg(a.l)); }

// s + e = a + b exactly
LMFF_DF D two_sum(float a, float b) {
  const float s = vadd(a, b), bb = vsub(s, a);
  return mk(s, vadd(vsub(a, vsub(s, bb)), vsub(b, bb)));
}
// the same for |a| >= |b| or a = 0
LMFF_DF D fast_two_sum(float a, float b) {
  const float s = vadd(a, b);
  return mk(s, vsub(b, vsub(s, a)));
}
LMFF_DF D renorm(D a) { return fast_two_sum(a.h, a.l); }

LMFF_DF D mul(D a, D b) {
  const float p = vmul(a.h, b.h);
  float e = vfma(a.h, b.h, vneg(p));
  e = vfma(a.h, b.l, e);
  return mk(p, vfma(a.l, b.h, e));
}
LMFF_DF D sqr(D a) {
  const float p = vmul(a.h, a.h);
  const float e = vfma(a.h, a.h, vneg(p));
  return mk(p, vfma(vadd(a.h, a.h), a.l, e));
}
LMFF_DF D add(D a, D b) {
  const D s = two_sum(a.h, b.h);
  return mk(s.h, vadd(s.l, vadd(a.l, b.l)));
}
// |a| >= |b|
LMFF_DF D add_ordered(D a, D b) {
  const D s = fast_two_sum(a.h, b.h);
  return mk(s.h, vadd(s.l, vadd(a.l, b.l)));
}
// a + b, b in single precision
LMFF_DF D add1(D a, float b) {
  const D s = two_sum(a.h, b);
  return mk(s.h, vadd(s.l, a.l));
}
LMFF_DF D scale(D a, float m) { return mk(vmul(a.h, m), vmul(a.l, m)); }   // m a power of two or zero
// running sum: acc += a
LMFF_DF void acc(D &s, D a) { s = add(s, a); }
// running sum of products: s += a b, s -= a b
LMFF_DF void acc_mul(D &s, D a, D b) { acc(s, mul(a, b)); }

// a . b of three-vectors
LMFF_DF D dot3(const D *a, const D *b) {
  const D x = mul(a[0], b[0]), y = mul(a[1], b[1]), z = mul(a[2], b[2]);
  const D s = two_sum(x.h, y.h), t = two_sum(s.h, z.h);
  const float lo = vadd(vadd(vadd(x.l, y.l), z.l), vadd(s.l, t.l));
  return fast_two_sum(t.h, lo);
}

// 2^a by Tang's table-driven method (P. T. P. Tang, ACM TOMS 15, 1989): a = k/64 + f,
// |f| <= 1/128, 2^a = 2^(k>>6) T[k & 63] e^g with g = f ln 2 as a double-float and
// e^g - 1 = g + g^2/2 + g^3 (1/6 + g/24 + g^2/120), the last bracket in FP32 (truncation
// below 2^-54).  tab holds T as double-floats (EXP2_TAB entries, filled by exp2_entry).
// For a <= 0 (a.h is clamped to [-125, 1]: results below 2^-125 come out as about 2^-125).
constexpr int EXP2_TAB = 64;
LMFF_DF float2 exp2_entry(int j) {
  const double t = exp2((double)j / EXP2_TAB);
  const float h = (float)t;
  return make_float2(h, (float)(t - (double)h));
}
LMFF_DF float clamp_exp(float x) { return fminf(fmaxf(x, -125.f), 1.f); }
LMFF_DF void exp2_parts(float t, const float2 *tab, float &th, float &tl, float &sc) {
  const int k = __float_as_int(t) - 0x4b400000;   // t = 1.5 2^23 + k
  const float2 T = tab[k & (EXP2_TAB - 1)];
  th = T.x;
  tl = T.y;
  sc = __int_as_float(((k >> 6) + 127) << 23);
}
LMFF_DF D exp2(D a, const float2 *tab) {
  const float magic = 12582912.f;   // 1.5 2^23
  const float ah = clamp_exp(a.h);
  const float t = vfma(ah, (float)EXP2_TAB, magic);
  const float k = vsub(t, magic);
  // ah - k/64 is exact and a multiple of ulp(ah), so zero or larger than a.l
  const D f = fast_two_sum(vfma(vneg(k), 1.f / EXP2_TAB, ah), a.l);
  const float L = 0.693147182464599609375f, Ll = -1.90465429995776804525e-9f;   // ln 2
  const float p = vmul(f.h, L);
  float e = vfma(f.h, L, vneg(p));
  e = vfma(f.h, Ll, e);
  e = vfma(f.l, L, e);
  const float c = vfma(vfma(p, 1.f / 60.f, 1.f / 12.f), p, 1.f / 3.f);
  const float hp = vmul(0.5f, p);
  const float q = vmul(hp, p);
  float qe = vfma(hp, p, vneg(q));
  qe = vfma(p, e, qe);
  qe = vfma(vmul(q, p), c, qe);
  const D s = fast_two_sum(p, q);
  const float sl = vadd(s.l, vadd(e, qe));
  float th, tl, sc;
  exp2_parts(t, tab, th, tl, sc);
  const float m = vmul(th, s.h);
  float me = vfma(th, s.h, vneg(m));
  me = vfma(th, sl, me);
  me = vfma(tl, s.h, me);
  const D r = fast_two_sum(th, m);
  return mk(vmul(r.h, sc), vmul(vadd(r.l, vadd(me, tl)), sc));
}
#undef LMFF_DF

}  // namespace df
}  // namespace lmff
