// The Sturm counts of the bisection (steig.cu).  __host__ __device__: the kernel
// k_stebz calls them, and a host harness checks the counts themselves, where the
// eigenvalues that come out of the bisection hide single wrong counts.
#pragma once

#include <cmath>
#include <cstring>

#include "common.cuh"

// 1/q from the hardware approximation refined by two Newton-Raphson steps
// r <- r (2 - q r) (each roughly doubles the correct bits).
EXCFV_HD double recip_nr(double q) {
  double r;
#ifdef __CUDA_ARCH__
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(q));
#else
  r = 1.0 / q;
  if (fabs(r) < 0x1p-1022) r = copysign(0.0, r);
#endif
  r = fma(r, fma(-q, r, 1.0), r);
  r = fma(r, fma(-q, r, 1.0), r);
  return r;
}

// Sturm counts: the numbers of eigenvalues of T below the points x[0..NPT), from
// the signs of the pivots q_i = d_i - x - e_{i-1}^2 / q_{i-1} of T - x, with
// |q_i| <= pivmin replaced by -pivmin (DSTEBZ).  de[i] = (d_i, e_{i-1}^2).
//
// As quotients a step is a reciprocal and a product, 82 clocks one after the
// other.  The leading minors p_i = q_i p_{i-1} follow
//   p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}
// with one multiply-add on the chain (8 clocks), and q_i < 0 is a change of sign.
// Each of the three roundings of a step is, as in the quotient form, a relative
// change of d_i - x or e_{i-1}^2 of the order of an ulp: the count stays that of a
// nearby tridiagonal matrix.  CH steps at a time run like this, from a pair scaled
// by a power of two (exact) to order 1.  With ||T|| < 2^38 they grow by less than
// 2^670, so nothing overflows, and a pair that had underflowed would still be below
// 2^-250 at the end: then (and where ||T|| is larger, or a number is not finite) the
// CH steps are done again as quotients.  What is left per step and point is three
// operations of the double-precision pipe and one for the sign: two points per
// thread share the loads, which run half of CH ahead.  k = 200, n = 1964:
// 805 -> 411 us; k = 20, n = 316: 120 -> 69 us (643 and 106 with the range of
// every minor tested).
//
// A minor that is exactly zero (x an eigenvalue of a leading block) changes sign
// once together with its successor, whatever the sign of the zero.  As the last but
// one of a pair it leaves an infinite quotient, whose step is q = d - x: a large
// finite one gives that, the reciprocal of an infinite one would be a NaN.
constexpr int CH = 16;
constexpr int HCH = CH / 2;
constexpr int NPT = 2;

// the m steps at de as quotients, from the pair (cur, prev)
inline __host__ __device__ __noinline__ int sturm_quotients(int m, const double2* __restrict__ de, double x,
                                                            double pivmin, double& cur, double& prev) {
  double q = cur / prev;
  int cnt = 0;
  if (fabs(q) > 1e300) q = copysign(1e300, q);
  if (fabs(q) <= pivmin) {  // counted by its sign so far
    cnt = !signbit(q);
    q = -pivmin;
  }
  for (int i = 0; i < m; ++i) {
    const double2 t = de[i];
    q = fma(-t.y, recip_nr(q), t.x - x);
    if (fabs(q) <= pivmin) q = -pivmin;
    cnt += q < 0.0;
  }
  cur = q;
  prev = 1.0;
  return cnt;
}

// the high word of v, a double from its high word, the number of bits set
EXCFV_HD unsigned high_bits(double v) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(v);
#else
  unsigned long long b;
  memcpy(&b, &v, sizeof b);
  return (unsigned)(b >> 32);
#endif
}
EXCFV_HD double from_high(int hi) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(hi, 0);
#else
  const unsigned long long b = (unsigned long long)(unsigned)hi << 32;
  double v;
  memcpy(&v, &b, sizeof v);
  return v;
#endif
}
EXCFV_HD int bits_set(unsigned v) {
#ifdef __CUDA_ARCH__
  return __popc(v);
#else
  return __builtin_popcount(v);
#endif
}
EXCFV_HD int larger(int a, int b) { return a > b ? a : b; }
EXCFV_HD int smaller(int a, int b) { return a < b ? a : b; }
EXCFV_HD int hiword(double v) { return (int)(high_bits(v) & 0x7fffffffu); }

// minors: ||T|| < 2^38
EXCFV_HD void sturm_count(int n, const double2* __restrict__ de, const double (&x)[NPT], double pivmin, bool minors,
                          int (&cnt)[NPT]) {
  double cur[NPT], prev[NPT];
#pragma unroll
  for (int r = 0; r < NPT; ++r) {
    cur[r] = de[0].x - x[r];
    if (fabs(cur[r]) <= pivmin) cur[r] = -pivmin;
    prev[r] = 1.0;
    cnt[r] = cur[r] < 0.0;
  }
  int i = 1;
  if (minors) {
    double2 t[2][HCH];
#pragma unroll
    for (int u = 0; u < HCH; ++u) t[0][u] = de[smaller(i + u, n - 1)];
    for (; i + CH <= n; i += CH) {
      double c0[NPT], p0[NPT];
      unsigned sg[NPT];
#pragma unroll
      for (int r = 0; r < NPT; ++r) {
        c0[r] = cur[r]; p0[r] = prev[r];
        const int big = larger(hiword(cur[r]), hiword(prev[r])) & 0x7ff00000;
        const double sc = from_high(smaller(larger(0x7fe00000 - big, 0x00100000), 0x7fe00000));
        cur[r] *= sc; prev[r] *= sc;
        sg[r] = high_bits(cur[r]) >> 31;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int u = 0; u < HCH; ++u) t[h ^ 1][u] = de[smaller(i + (h + 1) * HCH + u, n - 1)];
#pragma unroll
        for (int u = 0; u < HCH; ++u)
#pragma unroll
          for (int r = 0; r < NPT; ++r) {
            const double nx = fma(t[h][u].x - x[r], cur[r], -(t[h][u].y * prev[r]));
            sg[r] = sg[r] << 1 | high_bits(nx) >> 31;  // the sign bits, newest last
            prev[r] = cur[r];
            cur[r] = nx;
          }
      }
#pragma unroll
      for (int r = 0; r < NPT; ++r) {
        const int big = larger(hiword(cur[r]), hiword(prev[r]));
        if (big > 0x3ff00000 - (250 << 20) && big < 0x7ff00000) {
          cnt[r] += bits_set((sg[r] ^ (sg[r] >> 1)) & ((1u << CH) - 1u));
        } else {
          cur[r] = c0[r]; prev[r] = p0[r];
          cnt[r] += sturm_quotients(CH, de + i, x[r], pivmin, cur[r], prev[r]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < NPT; ++r) cnt[r] += sturm_quotients(n - i, de + i, x[r], pivmin, cur[r], prev[r]);
}
