// Host driver for tests/test_hex8_bound.py: the FP32 interpolation of the
// remelting kernel (hex8_interp32, with node values and coordinates rounded to
// float as the kernel rounds them) against hex8_interp64, over the bound that
// its decisions are made with (hex8_err32), compiled from the kernels' source
// without contraction. Node values of one sign and of both, equal, at the ends
// and inside of a range of magnitudes; coordinates anywhere in [-1, 1], at its
// ends and halfway between floats; then steps uphill from the worst cases.
// Usage: hex8_bound <cases> <seed>; prints cases, cases beyond the bound and
// the largest share of it.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "../amca3d_gb300/csrc/ca_math.h"

namespace {

uint64_t g_state = 1;
uint64_t next_u64() {
  uint64_t z = (g_state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
double uni(double lo, double hi) { return lo + (hi - lo) * ((double)(next_u64() >> 11) * 0x1.0p-53); }
// a value that rounds by nearly half an ulp of its float
double halfway(double x) {
  const float f = (float)x;
  return f + 0.4999 * ((double)nextafterf(f, next_u64() & 1 ? INFINITY : -INFINITY) - f);
}

struct Case {
  double t[8], x[3];
};

double share(const Case &c) {
  float t32[8];
  for (int q = 0; q < 8; ++q) t32[q] = (float)c.t[q];
  const float v = amca::hex8_interp32(t32, (float)c.x[0], (float)c.x[1], (float)c.x[2]);
  return fabs((double)v - amca::hex8_interp64(c.t, c.x[0], c.x[1], c.x[2])) / (double)amca::hex8_err32(t32);
}

double coordinate() {
  switch (next_u64() % 5) {
    case 0: return next_u64() & 1 ? 1.0 : -1.0;
    case 1: return halfway(uni(-0.999, 0.999));
    case 2: return halfway((next_u64() & 1 ? 1.0 : -1.0) * exp2(uni(-30, -0.01)));
    default: return uni(-1, 1);
  }
}
double node(double scale, int kind) {
  const double m = next_u64() & 1 ? scale : uni(0.5, 1.0) * scale;
  const double v = kind == 0 ? m : kind == 1 ? (next_u64() & 1 ? m : -m) : uni(-1, 1) * scale;
  return next_u64() & 1 ? halfway(v) : v;
}

}  // namespace

int main(int argc, char **argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  g_state = argc > 2 ? strtoull(argv[2], nullptr, 10) : 1;
  const double scales[4] = {300.0, 1700.0, 3.0e5, 1.0e9};
  long cases = 0, beyond = 0;
  double worst = 0.0;
  auto look = [&](const Case &c) {
    const double s = share(c);
    ++cases;
    beyond += !(s <= 1.0);
    worst = s > worst ? s : worst;
    return s;
  };
  for (long i = 0; i < n; ++i) {
    const double scale = scales[next_u64() & 3];
    const int kind = (int)(next_u64() % 3);
    Case c;
    for (double &v : c.t) v = node(scale, kind);
    if (next_u64() % 8 == 0)
      for (double &v : c.t) v = c.t[0];
    for (double &v : c.x) v = coordinate();
    double s = look(c);
    if (s < 0.8 * worst || i > n / 20) continue;
    for (int step = 0; step < 2000; ++step) {  // uphill
      Case d = c;
      const int k = (int)(next_u64() % 11);
      if (k < 8) d.t[k] = next_u64() & 1 ? node(scale, kind) : d.t[k] * (1.0 + uni(-1, 1) * 0x1.0p-20);
      else d.x[k - 8] = next_u64() & 1 ? coordinate() : fmin(1.0, fmax(-1.0, d.x[k - 8] + uni(-1, 1) * 0x1.0p-18));
      const double t = look(d);
      if (t > s) {
        s = t;
        c = d;
      }
    }
  }
  printf("%ld %ld %.6f\n", cases, beyond, worst);
  return 0;
}
