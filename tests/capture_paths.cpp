// Host driver for tests/test_ca_math_host.py: capture_f64 against
// capture_f64_general bit for bit, and the bit-level FP64 helpers against the
// FP64 operations they stand for, with the kernels' own source (ca_math.h).
// Prints "name cases wrong" per group.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../amca3d_gb300/csrc/ca_math.h"

namespace {

unsigned long long g_state = 1;
unsigned long long next_u64() {
  unsigned long long z = (g_state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
double uni(double a, double b) { return a + (b - a) * ((double)(next_u64() >> 11) * 0x1.0p-53); }
bool same(double a, double b) { return memcmp(&a, &b, 8) == 0 || (a != a && b != b); }
bool same(float a, float b) { return memcmp(&a, &b, 4) == 0 || (a != a && b != b); }

void rotation(double m[9]) {
  const double a = uni(0, 2 * M_PI), b = uni(0, M_PI), c = uni(0, 2 * M_PI);
  const double ca = cos(a), sa = sin(a), cb = cos(b), sb = sin(b), cc = cos(c), sc = sin(c);
  const double r[9] = {ca * cc - sa * cb * sc, -ca * sc - sa * cb * cc, sa * sb, sa * cc + ca * cb * sc,
                       -sa * sc + ca * cb * cc, -ca * sb, sb * sc, sb * cc, cb};
  memcpy(m, r, sizeof r);
}

// kind 0: ordinary captures; 1: unrotated envelopes and offsets on axes,
// diagonals, faces and corners, with zeros of both signs; 2: two components
// of the offset a few ulps to 2^-16 apart; 3: lengths from 2^-700 to 2^300;
// 4: points a few ulps from the surface, outside included
void capture(int kind, long n) {
  long wrong = 0;
  for (long i = 0; i < n; ++i) {
    double m[9], gc[3];
    double h = next_u64() & 1 ? 2.0e-6 : 5.0e-4, L = uni(0.3, 3.0) * h;
    rotation(m);
    if (kind == 3) {
      L = ldexp(uni(1, 2), (int)(next_u64() % 1000) - 700);
      h = L * exp2(uni(-3, 3));
    }
    if (kind == 1 || next_u64() % 8 == 0)
      for (int q = 0; q < 9; ++q) m[q] = q % 4 == 0 ? 1.0 : (next_u64() & 1 ? 0.0 : -0.0);
    if (kind == 1) {
      const double v[7] = {0.0, -0.0, L, -L, L / 2, -L / 2, L / 3};
      for (int a = 0; a < 3; ++a) gc[a] = v[next_u64() % 7];
    } else {
      for (int a = 0; a < 3; ++a) gc[a] = uni(-0.7, 0.7) * L;
      if (kind == 2) {
        const int a = next_u64() % 3, b = (a + 1 + next_u64() % 2) % 3;
        gc[b] = gc[a] * (1.0 + (next_u64() % 4 == 0 ? 0.0 : exp2(uni(-52, -16)))) * (next_u64() & 1 ? 1 : -1);
      }
      if (kind == 4) {  // scaled so that |c|_1 is L up to a few ulps
        double s = 0;
        for (int k = 0; k < 3; ++k) s += fabs(gc[0] * m[k] + gc[1] * m[3 + k] + gc[2] * m[6 + k]);
        const double f = L / s * (1.0 + ((int)(next_u64() % 9) - 4) * 0x1.0p-52);
        for (int a = 0; a < 3; ++a) gc[a] *= f;
      }
    }
    const double tr[4] = {(double)sqrtf(3.0f), (double)sqrtf(2.0f) * 1.5 * 0.5, 1e-3, 1e3};
    const double t = tr[next_u64() % 4];
    double x[4], y[4];
    amca::capture_f64(m, gc[0], gc[1], gc[2], L, h, t, x);
    amca::capture_f64_general(m, gc[0], gc[1], gc[2], L, h, t, y);
    for (int q = 0; q < 4; ++q)
      if (!same(x[q], y[q])) {
        ++wrong;
        break;
      }
  }
  printf("capture%d %ld %ld\n", kind, n, wrong);
}

// a double with its last bits all ones, all zeros or random, exponent in [lo, hi]
double pick(int lo, int hi) {
  unsigned long long b = next_u64() & 0xfffffffffffffull;
  const int k = next_u64() % 4, len = (int)(next_u64() % 52);
  if (k == 1) b &= ~((1ull << len) - 1);
  if (k == 2) b |= (1ull << len) - 1;
  b |= (unsigned long long)(1023 + lo + (int)(next_u64() % (unsigned)(hi - lo + 1))) << 52;
  double x;
  memcpy(&x, &b, 8);
  return next_u64() & 1 ? x : -x;
}

void helpers(long n) {
  long w[8] = {};
  for (long i = 0; i < n; ++i) {
    const double x = pick(-500, 300), z = pick(-120, 120);
    w[0] += !same(amca::f64_third(x), x / 3);
    const float b = (float)fabs(pick(-100, 100));
    const double bd = (double)b;
    w[1] += !same(amca::pos_f32_to_f64(b), bd);
    w[2] += !same(amca::div_by_f32(x, bd, amca::recip_of_f32(b, bd)), x / bd);
    // quotients next to rounding midpoints: (odd 54-bit number) * b, rounded
    const double q = pick(-20, 20), near = fma(q, bd, 0.5 * (nextafter(q, INFINITY) - q) * bd);
    w[2] += !same(amca::div_by_f32(near, bd, amca::recip_of_f32(b, bd)), near / bd);
    w[3] += !same(amca::pos_f64_to_f32_rn(fabs(z)), (float)fabs(z));
    const float rz = amca::f64_to_f32_rz(z);
    w[4] += !(fabs((double)rz) <= fabs(z) && fabs((double)rz) >= fabs(z) * (1 - 0x1.0p-23) && (rz < 0) == (z < 0));
    const double y = next_u64() % 4 ? pick(-3, 3) : x, x2 = next_u64() % 4 ? pick(-3, 3) : x;
    w[5] += amca::f64_less(x2, y) != (x2 < y);
    const double hx = pick(-1022, 1023);
    w[6] += !same(amca::f64_half(hx), 0.5 * hx) || !same(amca::f64_half(0.0), 0.0) ||
            !same(amca::f64_half(0x1.8p-1040), 0.5 * 0x1.8p-1040);
    const int I = (int)next_u64();
    w[7] += !same(amca::cells_minus_half(I % 1000000), I % 1000000 - 0.5) || !same(amca::cells_minus_half(I), I - 0.5);
  }
  const char *name[8] = {"third", "widen", "divide", "narrow", "truncate", "less", "half", "centre"};
  for (int k = 0; k < 8; ++k) printf("%s %ld %ld\n", name[k], n, w[k]);
}

}  // namespace

int main(int argc, char **argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  g_state = argc > 2 ? strtoull(argv[2], nullptr, 10) : 1;
  for (int kind = 0; kind < 5; ++kind) capture(kind, n);
  helpers(n);
  return 0;
}
