/* Device check of fold.h's folds against the plain serial loop, and of fold_room's bounds: a
 * thread per case.  Built and run by tests/test_gpu_fold.py. */
#include "fold.h"

__global__ void k_folds(int n, const float *w, const float *d, const int *k, unsigned *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  float a[3], b[3], c[3];
  for (int e = 0; e < 3; e++) {
    a[e] = b[e] = w[3 * i + e];
    c[e] = fold_add(a[e], d[3 * i + e], k[i]);
  }
  fold3_add_long(a, d + 3 * i, k[i]);
  for (int s = 0; s < k[i]; s++)
    for (int e = 0; e < 3; e++)
      b[e] = __fadd_rn(b[e], d[3 * i + e]);
  for (int e = 0; e < 3; e++) {
    const bool nan = b[e] != b[e];
    if (!(nan ? a[e] != a[e] : fold_bits(a[e]) == fold_bits(b[e])))
      atomicAdd(&bad[0], 1u);
    if (!(nan ? c[e] != c[e] : fold_bits(c[e]) == fold_bits(b[e])))
      atomicAdd(&bad[1], 1u);
  }
}

/* fold_room(num, den) is never above num / den nor further below it than its comment says */
__global__ void k_rooms(int n, const int *num, const int *den, unsigned *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const int q = num[i] / den[i], r = fold_room(num[i], den[i]);
  if (r > q)
    atomicAdd(&bad[0], 1u);
  if ((double)r < (double)q - 1.0 - 1.4e-6 * (double)q)
    atomicAdd(&bad[1], 1u);
}

extern "C" void launch_folds(int n, const float *w, const float *d, const int *k, unsigned *bad) {
  k_folds<<<(n + 127) / 128, 128>>>(n, w, d, k, bad);
}
extern "C" void launch_rooms(int n, const int *num, const int *den, unsigned *bad) {
  k_rooms<<<(n + 127) / 128, 128>>>(n, num, den, bad);
}
