// Host driver for tests/test_ca_math_host.py: capture_f64 against
// capture_f64_general bit for bit (any NaN for any other) for truncations that
// a deck cannot give but an envelope evaluation can: negative ones, zeros and
// NaN of either sign, infinities, products that underflow. Prints "truncation
// cases wrong" per value.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "../amca3d_gb300/csrc/ca_math.h"

namespace {

unsigned long long g_state = 5;
double uni(double a, double b) {
  unsigned long long z = (g_state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return a + (b - a) * ((double)((z ^ (z >> 31)) >> 11) * 0x1.0p-53);
}

}  // namespace

int main() {
  const double truncs[] = {NAN,       -NAN,      0.0,       -0.0,      -1.0, -1e-3, INFINITY,
                           -INFINITY, 0x1p-1074, -0x1p-1074, 1e300, -1e300, 1.7320508};
  for (double t : truncs) {
    long wrong = 0;
    const long n = 40000;
    for (long i = 0; i < n; ++i) {
      const double h = 2.0e-6, L = uni(0.3, 3.0) * h;
      double m[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1}, gc[3], x[4], y[4];
      if (i & 1) {
        const double a = uni(0, 2 * M_PI), ca = cos(a), sa = sin(a);
        const double r[9] = {ca, -sa, 0, sa, ca, 0, 0, 0, 1};
        memcpy(m, r, sizeof r);
      }
      for (double &v : gc) v = uni(-0.6, 0.6) * L;
      if (i % 4 == 0) gc[1] = gc[2] = 0.0;  // on an axis,
      if (i % 8 == 0) gc[0] = L;            // at its corner: an edge length of zero
      amca::capture_f64(m, gc[0], gc[1], gc[2], L, h, t, x);
      amca::capture_f64_general(m, gc[0], gc[1], gc[2], L, h, t, y);
      bool same = true;
      for (int q = 0; q < 4; ++q) same = same && (memcmp(&x[q], &y[q], 8) == 0 || (x[q] != x[q] && y[q] != y[q]));
      wrong += !same;
    }
    std::printf("%g %ld %ld\n", t, n, wrong);
  }
  return 0;
}
