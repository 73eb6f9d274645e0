/* div_const (master-of-puppets_b200/csrc/fold.h) against the division, for the bit patterns
 * [from, to).  Built and run by tests/test_div_const.py. */
#include "fold.h"

/* Patterns whose quotient plus 0.5 differs (2 pi: two = 1, pi: 0), finite values alone; a
 * pattern of the last such run of 4,096 in bad.  The patterns per run are a simple loop, for the
 * compiler to vectorise. */
#define RUN 4096
#define CHECK(c)                                                   \
  for (uint32_t k = 0; k < RUN; k++) {                             \
    const uint32_t u = base + k;                                   \
    const float x = fold_float(u);                                 \
    const float a = div_const(x, c) + 0.5f, b = x / (c) + 0.5f;    \
    m += (a != b) & ((u & 0x7f800000u) != 0x7f800000u);            \
  }
long div_const_angles(uint64_t from, uint64_t to, int two, uint32_t *bad) {
  long n = 0;
  for (uint64_t r = from; r < to; r += RUN) {
    const uint32_t base = (uint32_t)r;
    uint32_t m = 0;
    if (two)
      CHECK(2.0f * 3.14159265f)
    else
      CHECK(3.14159265f)
    n += m;
    if (m)
      *bad = base;
  }
  return n;
}

/* Bytes whose quotient by 255 differs. */
int div_const_bytes(void) {
  int n = 0;
  for (int b = 0; b < 256; b++) {
    volatile float d = 255.0f;
    n += div_const((float)b, 255.0f) != (float)b / d;
  }
  return n;
}
