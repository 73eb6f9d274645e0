/* Host check of fold3_add_long (master-of-puppets_b200/csrc/fold.h) against
 * the plain serial loop.  Built and run by tests/test_fold3.py. */
#include "fold.h"

#include <stdint.h>
#include <string.h>

/* mismatches of n triples (w, d: 3n floats, k: n counts > 16); the first one's index in bad */
int fold3_check(int n, const float *w, const float *d, const int *k, int *bad) {
  int fails = 0;
  for (int i = 0; i < n; i++) {
    float a[3];
    memcpy(a, w + 3 * i, sizeof a);
    fold3_add_long(a, d + 3 * i, k[i]);
    int ok = 1;
    for (int e = 0; e < 3; e++) {
      volatile float b = w[3 * i + e];
      for (int s = 0; s < k[i]; s++)
        b = b + d[3 * i + e];
      const float bf = b;
      uint32_t x, y;
      memcpy(&x, &a[e], 4);
      memcpy(&y, &bf, 4);
      ok &= x == y || (a[e] != a[e] && bf != bf);
    }
    if (!ok && !fails++)
      *bad = i;
  }
  return fails;
}
