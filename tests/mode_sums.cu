// Sums of rigid-body modes as a lane of the resident solve forms them, on the
// host: argv[1] nodes of dimension 2 or 3 (argv[2]); prints the largest error
// against double sums of the exact products, relative to the sum of their
// magnitudes.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "coarse.cuh"

template <int D>
static double worst(int nodes) {
  unsigned s = 12345;
  auto next = [&] { return (double)((s = s * 1664525u + 1013904223u) >> 8) / (1 << 24) - 0.5; };
  constexpr int nr = D == 2 ? 3 : 6;
  gfea::DotAcc<float> acc[nr];
  double ref[nr] = {}, mag[nr] = {};
  for (int a = 0; a < nodes; ++a) {
    float o[D], x[D];
    for (int k = 0; k < D; ++k) {
      o[k] = (float)next();
      x[k] = (float)(next() * exp(10 * next()));
    }
    for (int m = 0; m < nr; ++m) {
      gfea::add_mode<D, float>(acc[m], m, o, x);
      const int r = m - 3, b = r == 2 ? 0 : r + 1, c = r == 0 ? 2 : r - 1;
      const double p = m < D ? x[m] : (D == 2 ? (double)o[0] * x[1] : (double)o[b] * x[c]);
      const double q = m < D ? 0 : (D == 2 ? (double)o[1] * x[0] : (double)o[c] * x[b]);
      ref[m] += p - q;
      mag[m] += fabs(p) + fabs(q);
    }
  }
  double e = 0;
  for (int m = 0; m < nr; ++m) e = fmax(e, fabs(acc[m].value() - ref[m]) / mag[m]);
  return e;
}

int main(int, char** argv) {
  const int nodes = atoi(argv[1]);
  printf("%.3e\n", atoi(argv[2]) == 2 ? worst<2>(nodes) : worst<3>(nodes));
}
