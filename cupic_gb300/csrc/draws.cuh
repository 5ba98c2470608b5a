// draws.cuh -- the initial plasma's draws without FP64 arithmetic.
//
// A particle of the initial plasma is a function of four 32-bit words, defined
// in FP64 (u01, dev_log, dev_sincos2pi, sqrt) and rounded once to FP32.  FP64
// runs at 2 operations a clock and SM on GB300 and a particle takes about 120
// of them, so 2.1e8 particles took 47 ms.  Here the same four numbers are
// evaluated in double-float arithmetic (a value as the unevaluated sum of
// two floats, about 2^-45 relative; T. J. Dekker 1971, and the error-free
// product by fused multiply-add) and rounded to FP32 where both ends of their
// error interval round to the same float -- the rounding test of A. Ziv
// (1991).  The FP64 value lies in that interval too, so its rounding is the
// same float; about one particle in 2000 fails the test and takes the FP64
// path.  47 -> 4 ms.
#pragma once

#include "cupic_internal.cuh"

namespace cupic {

struct df {
  float h, l;
};

__device__ __forceinline__ df two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
// |a| >= |b|
__device__ __forceinline__ df fast_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ df df_add(df a, df b) {
  const df s = two_sum(a.h, b.h);
  return fast_two_sum(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ df df_mul(df a, df b) {
  const float p = __fmul_rn(a.h, b.h);
  const float e = __fmaf_rn(a.h, b.h, -p);
  return fast_two_sum(p, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, e)));
}
__device__ __forceinline__ df df_neg(df a) { return {-a.h, -a.l}; }
__device__ __forceinline__ df df_scale(df a, float pow2) { return {__fmul_rn(a.h, pow2), __fmul_rn(a.l, pow2)}; }
// the double c (a compile-time constant, or a kernel argument) as a double-float
__device__ __forceinline__ df df_of(double c) {
  const float h = (float)c;
  return {h, (float)(c - (double)h)};
}
// an integer of at most 48 bits, exactly
__device__ __forceinline__ df df_int(unsigned long long n) {
  return fast_two_sum(__fmul_rn((float)(unsigned)(n >> 24), 16777216.0f), (float)(unsigned)(n & 0xffffffu));
}

// log((r + 1/2) 2^-32) by the atanh series of (m-1)/(m+1), m in [0.7, 1.42]
__device__ __forceinline__ df df_log_u01(uint32_t r) {
  const df n = df_int(2ull * r + 1ull);  // u = n 2^-33
  int k = (__float_as_int(n.h) >> 23) - 127;
  float sc = __int_as_float((127 - k) << 23);
  if (__fmul_rn(n.h, sc) > 1.41421356f) {
    sc *= 0.5f;
    ++k;
  }
  const df m = df_scale(n, sc);
  const df num = fast_two_sum(__fadd_rn(m.h, -1.0f), m.l);  // m.h - 1 is exact
  df den = two_sum(m.h, 1.0f);
  den = fast_two_sum(den.h, __fadd_rn(den.l, m.l));
  // s = num / den: a float quotient, and its remainder's quotient
  const float inv = __frcp_rn(den.h);
  const float q0 = __fmul_rn(num.h, inv);
  const df t = df_mul({q0, 0.0f}, den);
  const df rem = df_add(num, df_neg(t));
  const df s = fast_two_sum(q0, __fmul_rn(rem.h, inv));
  const df s2 = df_mul(s, s);
  // 2 s (1 + s2/3 + s2^2/5 + s2^3 (1/7 + ...)), s2 <= 0.03: the terms from
  // the fourth on are below 2^-17, so float is enough for them
  const float z = s2.h;
  float p = 1.0f / 17.0f;
  p = __fmaf_rn(p, z, 1.0f / 15.0f);
  p = __fmaf_rn(p, z, 1.0f / 13.0f);
  p = __fmaf_rn(p, z, 1.0f / 11.0f);
  p = __fmaf_rn(p, z, 1.0f / 9.0f);
  p = __fmaf_rn(p, z, 1.0f / 7.0f);
  p = __fmul_rn(p, z);
  df q = df_add(df_of(1.0 / 5.0), {p, 0.0f});
  q = df_add(df_of(1.0 / 3.0), df_mul(q, s2));
  q = df_add({1.0f, 0.0f}, df_mul(q, s2));
  q = df_mul(q, s);
  q = df_scale(q, 2.0f);
  const float e = (float)(k - 33);
  return df_add(df_mul({e, 0.0f}, df_of(0.69314718055994531)), q);
}

// sqrt(a), a > 0: a float root and one Newton step on the double-float rest
__device__ __forceinline__ df df_sqrt(df a) {
  const float y = __fsqrt_rn(a.h);
  const float p = __fmul_rn(y, y), e = __fmaf_rn(y, y, -p);
  const df d = df_add(a, {-p, -e});
  return fast_two_sum(y, __fdiv_rn(d.h, __fadd_rn(y, y)));
}

// sin and cos of 2 pi (r + 1/2) 2^-32 by octants, Taylor series on [0, pi/4]
__device__ __forceinline__ void df_sincos2pi_u01(uint32_t r, df *sn, df *cs) {
  const int o = (int)(r >> 29);
  unsigned long long f = 2ull * (r & 0x1fffffffu) + 1ull;  // f 2^-30 in (0, 1)
  if (o & 1) f = (1ull << 30) - f;
  const df th = df_mul(df_scale(df_int(f), 0x1p-30f), df_of(0.78539816339744831));
  const df t2 = df_mul(th, th);
  const float z = t2.h;
  // sin: th (1 + t2 (-1/6 + t2 (1/120 + t2 (-1/5040 + ...))))
  float p = 1.0f / 6227020800.0f;
  p = __fmaf_rn(p, z, -1.0f / 39916800.0f);
  p = __fmaf_rn(p, z, 1.0f / 362880.0f);
  p = __fmul_rn(p, z);
  df q = df_add(df_of(-1.0 / 5040.0), {p, 0.0f});
  q = df_add(df_of(1.0 / 120.0), df_mul(q, t2));
  q = df_add(df_of(-1.0 / 6.0), df_mul(q, t2));
  q = df_add({1.0f, 0.0f}, df_mul(q, t2));
  const df sa = df_mul(q, th);
  // cos: 1 + t2 (-1/2 + t2 (1/24 + t2 (-1/720 + t2 (1/40320 + ...))))
  p = -1.0f / 87178291200.0f;
  p = __fmaf_rn(p, z, 1.0f / 479001600.0f);
  p = __fmaf_rn(p, z, -1.0f / 3628800.0f);
  p = __fmul_rn(p, z);
  q = df_add(df_of(1.0 / 40320.0), {p, 0.0f});
  q = df_add(df_of(-1.0 / 720.0), df_mul(q, t2));
  q = df_add(df_of(1.0 / 24.0), df_mul(q, t2));
  q = df_add({-0.5f, 0.0f}, df_mul(q, t2));
  const df ca = df_add({1.0f, 0.0f}, df_mul(q, t2));
  // octant o: (s, c) swap where o is 1, 2, 5, 6; c < 0 in 2..5, s < 0 in 4..7
  const bool swap = ((o + 1) & 2) != 0;
  const df a = swap ? ca : sa, b = swap ? sa : ca;
  *sn = o >= 4 ? df_neg(a) : a;
  *cs = (o >= 2 && o <= 5) ? df_neg(b) : b;
}

// v rounded to float; clears ok when the FP64 value could round to another
// one.  kDrawEps bounds the relative distance of the two evaluations: the
// steps above lose a few units of 2^-45, the FP64 ones a few of 2^-52.
// (In normal floats: the products' low parts are 2^-48 of them and round off
// near 2^-149, so the constants that the callers multiply by are bounded,
// df_plain, and beyond those bounds FP64 decides.)
constexpr float kDrawEps = 0x1p-38f;
__device__ __forceinline__ bool df_plain(df c, float least, float most) { return c.h >= least && c.h <= most; }
__device__ __forceinline__ float df_round(df v, bool &ok) {
  const float e = __fmul_rn(fabsf(v.h), kDrawEps);
  const float a = __fadd_rn(v.h, __fadd_rn(v.l, e)), b = __fadd_rn(v.h, __fsub_rn(v.l, e));
  ok = ok && a == b;
  return a;
}

}  // namespace cupic
