/*
 * fold.h — exact value of k sequential float additions, in O(binades).
 *
 * The reference rasteriser steps its edge functions incrementally: for each
 * pixel of a row it does `w += e_dx`, for each row `w_row += e_dy`, always
 * starting from the clamped bounding-box corner (rasterizer.c:1926-2151 and
 * 1015-1023).  Repeated round-to-nearest-even addition has no closed form in
 * general, so a pixel's coverage, depth and interpolation weights depend on
 * the exact fold  w_k = RN(w_{k-1} + d).  A GPU that evaluates pixels in
 * parallel must reproduce that fold without walking every intermediate step.
 *
 * Method.  Inside one binade [2^E, 2^(E+1)) (same sign) the representable
 * values are N*u with u = 2^(E-23) and integer N in [2^23, 2^24).  If the
 * exact sum N + d/u lies in the binade, rounding adds a fixed integer
 * increment Q = rne(d/u) — except for exact ties (d/u = M + 1/2), where the
 * result is always even, so after one tie-rounded step the increment is the
 * constant even value of {M, M+1}.  Hence: take three explicit steps
 * w1, w2, w3; when all three lie in one binade and w2, w3 keep one unit of
 * margin from its edges, Q = N3 - N2 is the increment of every later step
 * that stays inside [2^23+1, 2^24-1] (then the exact sum also stays inside
 * the binade, |exact - rounded| <= 1/2).  Jump there with integer
 * arithmetic, then continue with explicit steps into the next binade.
 * Zero, subnormal and non-finite values are stepped explicitly.  The cost is
 * about four additions per binade crossed instead of one per step.
 *
 * The same header is compiled for the device (kernels) and for the host
 * (unit test against the plain loop).  Besides the folds it has the division
 * by a constant, whose results are the division's.
 */
#ifndef MOPCUDA_FOLD_H
#define MOPCUDA_FOLD_H

#include <stdint.h>

#if defined(__CUDACC__)
#define MOPCUDA_HD __host__ __device__ __forceinline__
#define MOPCUDA_HD_SLOW static __host__ __device__ __noinline__
#else
#define MOPCUDA_HD static inline
#define MOPCUDA_HD_SLOW static
#include <math.h>
#include <string.h>
#endif

MOPCUDA_HD uint32_t fold_bits(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(f);
#else
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
#endif
}

MOPCUDA_HD float fold_float(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}

/* One IEEE single round-to-nearest-even addition, never contracted. */
MOPCUDA_HD float fold_fadd(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fadd_rn(a, b);
#else
  volatile float r = a + b;
  return r;
#endif
}

/* x / c for a compile-time c, by Markstein's final step (P. Markstein, IBM J.
 * Res. Dev. 34(1), 1990): q = x * RN(1/c) corrected by its exact remainder
 * rounds correctly when neither underflows.  For 2 pi and pi the sum with 0.5
 * that follows equals the division's for every float x (an underflown quotient
 * is absorbed; an infinite x gives NaN), and for 255 the bytes' quotients are
 * the division's; 3 instructions instead of a division's dozen. */
MOPCUDA_HD float div_const(float x, float c) {
  const float rc = 1.0f / c; /* folded by the compiler */
  const float q = x * rc;
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(__fmaf_rn(-q, c, x), rc, q);
#else
  return fmaf(fmaf(-q, c, x), rc, q);
#endif
}

/* A whole number of steps j with 0 <= j <= num / den, short of it by at most
 * 1 + 1.4e-6 of it, so up to 24 for the largest quotients (0 <= num, 1 <= den,
 * both below 2^24, so exact in single precision): 1e-6 of the quotient is
 * taken off before truncating, more than the approximate division and the
 * product can be above it (2 ulp and half an ulp, 3e-7).  A jump may stop short
 * of its binade's edge: the explicit steps that follow any jump cover the
 * rest. */
MOPCUDA_HD int32_t fold_room(int32_t num, int32_t den) {
#if defined(__CUDA_ARCH__)
  return (int32_t)(__fdividef((float)num, (float)den) * 0.9999990f);
#else
  return (int32_t)(((float)num / (float)den) * 0.9999990f);
#endif
}

#define FOLD_SERIAL_MAX 16

/* The binade-skipping path of fold_add for k > FOLD_SERIAL_MAX (kept out of
 * line: callers inline only the short serial loop). */
MOPCUDA_HD_SLOW float fold_add_long(float w, float d, int k) {
  uint32_t db = fold_bits(d);
  /* d = +-0, inf or NaN: after one addition the value is a fixed point. */
  if ((db & 0x7fffffffu) == 0u || (db & 0x7f800000u) == 0x7f800000u)
    return fold_fadd(w, d);
  while (k > 0) {
    uint32_t wb = fold_bits(w);
    if ((wb & 0x7f800000u) == 0x7f800000u) /* inf/NaN + finite d is stable */
      return w;
    if (k <= 3) {
      for (int i = 0; i < k; i++)
        w = fold_fadd(w, d);
      return w;
    }
    float w1 = fold_fadd(w, d);
    float w2 = fold_fadd(w1, d);
    float w3 = fold_fadd(w2, d);
    k -= 3;
    w = w3;
    uint32_t b1 = fold_bits(w1), b2 = fold_bits(w2), b3 = fold_bits(w3);
    uint32_t hi = b3 & 0xff800000u; /* sign + exponent */
    if ((b1 & 0xff800000u) != hi || (b2 & 0xff800000u) != hi)
      continue;
    uint32_t ex = (hi >> 23) & 0xffu;
    if (ex == 0u || ex == 0xffu)
      continue;
    int32_t n2 = (int32_t)((b2 & 0x007fffffu) | 0x00800000u);
    int32_t n3 = (int32_t)((b3 & 0x007fffffu) | 0x00800000u);
    const int32_t lo = 0x00800001, top = 0x00ffffff;
    if (n2 < lo || n3 < lo)
      continue;
    int32_t q = n3 - n2; /* steady increment of the magnitude */
    if (q == 0)
      return w3; /* the increment rounds away: w is a fixed point */
    int32_t room = q > 0 ? fold_room(top - n3, q) : fold_room(n3 - lo, -q);
    int32_t j = room < k ? room : k;
    if (j <= 0)
      continue;
    int32_t n = n3 + j * q; /* |j*q| < 2^24: no overflow */
    w = fold_float(hi | ((uint32_t)n & 0x007fffffu));
    k -= j;
  }
  return w;
}

/* One round of fold_add_long on (w, k), k > 0: up to three explicit steps and
 * the jump they allow.  Straight-line, so that rounds of several folds
 * interleave. */
MOPCUDA_HD void fold_round(float *w, float d, int *k) {
  const float w0 = *w;
  const float w1 = fold_fadd(w0, d), w2 = fold_fadd(w1, d), w3 = fold_fadd(w2, d);
  if (*k <= 3) {
    *w = *k == 1 ? w1 : (*k == 2 ? w2 : w3);
    *k = 0;
    return;
  }
  *w = w3;
  *k -= 3;
  const uint32_t b1 = fold_bits(w1), b2 = fold_bits(w2), b3 = fold_bits(w3);
  const uint32_t hi = b3 & 0xff800000u, ex = (hi >> 23) & 0xffu;
  if (ex == 0xffu) { /* inf / NaN + finite d is stable */
    *k = 0;
    return;
  }
  const int32_t n2 = (int32_t)((b2 & 0x007fffffu) | 0x00800000u);
  const int32_t n3 = (int32_t)((b3 & 0x007fffffu) | 0x00800000u);
  const int32_t lo = 0x00800001, top = 0x00ffffff;
  if ((b1 & 0xff800000u) != hi || (b2 & 0xff800000u) != hi || ex == 0u || n2 < lo || n3 < lo)
    return;
  const int32_t q = n3 - n2;
  if (q == 0) { /* the increment rounds away: w is a fixed point */
    *k = 0;
    return;
  }
  const int32_t room = q > 0 ? fold_room(top - n3, q) : fold_room(n3 - lo, -q);
  const int32_t j = room < *k ? room : *k;
  *w = fold_float(hi | ((uint32_t)(n3 + j * q) & 0x007fffffu));
  *k -= j;
}

/* w[e] after k sequential additions of d[e], for three folds of the same
 * length (k > FOLD_SERIAL_MAX): their rounds interleave, because each one
 * alone is a chain of dependent operations. */
MOPCUDA_HD_SLOW void fold3_add_long(float w[3], const float d[3], int k) {
  float v0 = w[0], v1 = w[1], v2 = w[2];
  int k0 = k, k1 = k, k2 = k;
  /* d = +-0, inf or NaN: after one addition the value is a fixed point */
#define FOLD3_START(v, d, kk)                                                     \
  if ((fold_bits(d) & 0x7fffffffu) == 0u || (fold_bits(d) & 0x7f800000u) == 0x7f800000u) { \
    v = fold_fadd(v, d);                                                          \
    kk = 0;                                                                       \
  } else if ((fold_bits(v) & 0x7f800000u) == 0x7f800000u)                         \
    kk = 0
  FOLD3_START(v0, d[0], k0);
  FOLD3_START(v1, d[1], k1);
  FOLD3_START(v2, d[2], k2);
#undef FOLD3_START
  while ((k0 | k1 | k2) != 0) {
    if (k0)
      fold_round(&v0, d[0], &k0);
    if (k1)
      fold_round(&v1, d[1], &k1);
    if (k2)
      fold_round(&v2, d[2], &k2);
  }
  w[0] = v0;
  w[1] = v1;
  w[2] = v2;
}

/* w after k >= 0 sequential additions of d. */
MOPCUDA_HD float fold_add(float w, float d, int k) {
  if (k <= FOLD_SERIAL_MAX) {
    /* fully unrolled and predicated: no loop and no divergence on k */
#pragma unroll
    for (int i = 0; i < FOLD_SERIAL_MAX; i++)
      if (i < k)
        w = fold_fadd(w, d);
    return w;
  }
  return fold_add_long(w, d, k);
}

#endif
