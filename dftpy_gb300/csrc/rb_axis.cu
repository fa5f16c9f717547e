// Radix choice of the register-blocked FFT passes.
#include <string.h>

#include "rb_axis.h"

namespace gbrb {

// FP64: fewest stages (every further stage is one more trip of each line through
// shared memory), then the smallest largest radix (balanced stages keep every
// thread of a CTA busy).
static void search(int n, int maxr, int* cur, int depth, int* best, int& bestn) {
  static const int radices[] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  if (n == 1) {
    if (bestn == 0 || depth < bestn || (depth == bestn && cur[0] < best[0])) {
      bestn = depth;
      for (int i = 0; i < depth; ++i) best[i] = cur[i];
    }
    return;
  }
  if (depth == 8) return;
  for (int r : radices) {
    if (r > maxr || n % r) continue;
    cur[depth] = r;
    search(n / r, r, cur, depth + 1, best, bestn);
  }
}

RbAxis rb_axis(int n, bool f64, bool reverse) {
  RbAxis a;
  memset(&a, 0, sizeof(a));
  a.n = n;
  int best[8], bestn = 0;
  if (f64) {
    int cur[8];
    search(n, 16, cur, 0, best, bestn);
  } else {
    static const int order[] = {8, 4, 2, 3, 5, 7};
    int m = n;
    for (int r : order)
      while (m % r == 0 && bestn < 8) { best[bestn++] = r; m /= r; }
    if (m > 1) bestn = 0;
  }
  a.nst = bestn;
  int p = 1;
  for (int s = 0; s < bestn; ++s) {
    const int r = best[reverse ? bestn - 1 - s : s];
    a.r[s] = r;
    a.nb[s] = n / r;
    a.p[s] = p;
    a.dnb[s].set(n / r);
    a.dp[s].set(p);
    p *= r;
  }
  return a;
}

bool rb_rsqrt_length(int n) {
  return n == 32 || n == 64 || n == 96 || n == 128 || n == 160 || n == 256 || n == 360;
}

}  // namespace gbrb
