// ca_math.h — envelope arithmetic of the CA step, shared by the CUDA kernels
// and the host engine.
//
// The FP64 routines reproduce AMCA3D's octahedron arithmetic bit for bit:
// the same operations in the same order, no fused multiply-add (device code
// is built with -fmad=false, host code with -ffp-contract=off), float square
// roots where the reference calls sqrtf on doubles.
//
//   cell centre        CA/src/CellularAutomataManager_3D.cpp:877-888
//   containment test   CA/src/Octahedron.cpp:99-128
//   decentred capture  CA/src/Octahedron.cpp:134-275, CA/src/CellularAutomataManager_3D.cpp:677-707
//   KGT velocity       CA/src/ProblemPhysics.cpp:118-135
//
// The FP32 containment pre-test decides a (cell, envelope) pair only when its
// rounding-error bound keeps it on one side of the FP64 boundary; otherwise
// the caller runs the FP64 test. Decisions therefore equal the FP64 ones.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define AMCA_HD __host__ __device__ __forceinline__
#else
#define AMCA_HD inline
#endif

#include <math.h>
#include <string.h>

namespace amca {

constexpr double kTheodorus = 1.732050807568877;  // CA/src/Octahedron.cpp:13

// Liquid cells hold -1 in the orientation field; during one generation of
// the capture sweep a liquid cell may instead hold a claim
// 0x80000000 | parity << 30 | rank (rank = position of the claiming envelope
// in the generation, which is ascending envelope id). Solid cells and the
// ghost layer hold an orientation id >= 0.
constexpr uint32_t kLiquid = 0xFFFFFFFFu;
constexpr uint32_t kClaimBit = 0x80000000u;
constexpr uint32_t kParityBit = 0x40000000u;
constexpr uint32_t kRankMask = 0x3FFFFFFFu;

AMCA_HD uint32_t claim_word(uint32_t parity, uint32_t rank) { return kClaimBit | (parity ? kParityBit : 0u) | rank; }
// liquid at the start of the current generation: -1, or a claim made in it
AMCA_HD bool is_liquid_now(uint32_t s, uint32_t parity) {
  return s == kLiquid || ((s & kClaimBit) && (((s & kParityBit) != 0) == (parity != 0)));
}

// n / d for 0 <= n < 2^31 as (n * mul) >> shift: with s = ceil(log2 d) and
// mul = ceil(2^(31+s) / d), mul * d exceeds 2^(31+s) by less than d <= 2^s, so
// n * mul / 2^(31+s) exceeds n / d by less than 1 / d.
struct FastDiv {
  uint32_t mul;
  int shift;
};
inline FastDiv fast_div(int d) {
  int s = 0;
  while ((1ll << s) < d) ++s;
  return {(uint32_t)(((1ull << (31 + s)) + (unsigned)d - 1) / (unsigned)d), 31 + s};
}
AMCA_HD int quotient(int n, FastDiv f) { return (int)(((uint64_t)(uint32_t)n * f.mul) >> f.shift); }

struct Grid {
  int nx, ny, nz;     // interior cells
  int nxg, nyg, nzg;  // with the ghost layer
  int nxyg;
  FastDiv by_x, by_xy;  // of nxg, nxyg
  double x0, y0, z0, h;
};

// FP64 on GB300: an FP64 instruction (arithmetic, comparison or conversion)
// holds a warp's scheduler for about 64 cycles however many lanes take part
// (divide: 560), against 1 for an integer or FP32 one. The helpers below do
// exact FP64 bookkeeping with integer operations on the bits instead; all of
// them return what the FP64 operation named in their comment returns.
AMCA_HD long long f64_bits(double x) {
#if defined(__CUDA_ARCH__)
  return __double_as_longlong(x);
#else
  long long b;
  memcpy(&b, &x, sizeof b);
  return b;
#endif
}
AMCA_HD double bits_f64(long long b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double(b);
#else
  double x;
  memcpy(&x, &b, sizeof x);
  return x;
#endif
}
AMCA_HD uint32_t f32_bits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(x);
#else
  uint32_t b;
  memcpy(&b, &x, sizeof b);
  return b;
#endif
}
AMCA_HD float bits_f32(uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(b);
#else
  float x;
  memcpy(&x, &b, sizeof x);
  return x;
#endif
}
AMCA_HD int f64_exponent(double x) { return (int)((unsigned long long)f64_bits(x) >> 52) & 0x7ff; }  // biased

// (double)I - 0.5: a double near 1.5 * 2^51 has a unit of 0.5, so its low bits
// count half cells; one subtraction instead of a conversion and one.
AMCA_HD double cells_minus_half(int I) { return bits_f64(0x4328000000000000ll + 2ll * I) - 3377699720527872.5; }

// get_cell_center: x0 + h*(I - 0.5) with the ghost-inclusive index I.
AMCA_HD double centre_coord(double o, double h, int I) { return o + h * cells_minus_half(I); }

// x rounded to float towards zero (within 2^-23 of x): x is 0 or normal as a
// float, or rounds as the conversion does.
AMCA_HD float f64_to_f32_rz(double x) {
  const unsigned long long b = (unsigned long long)f64_bits(x);
  const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
  if (e - 897u < 253u)
    return bits_f32((uint32_t)(b >> 32 & 0x80000000u) | ((uint32_t)(b >> 29) - (896u << 23) & 0x7fffffffu));
  return (b << 1) == 0 ? 0.0f : (float)x;
}
// (float)x for x whose float is positive and normal with room to round up
AMCA_HD float pos_f64_to_f32_rn(double x) {
  const unsigned long long b = (unsigned long long)f64_bits(x);
  return bits_f32((uint32_t)((b + 0x0fffffffull + (b >> 29 & 1ull)) >> 29) - (896u << 23));
}
// (double)x for x positive and normal
AMCA_HD double pos_f32_to_f64(float x) {
  return bits_f64(((long long)f32_bits(x) << 29) + (896ll << 52));
}
// x < y; neither is NaN, nor are they zeros of different signs
AMCA_HD bool f64_less(double x, double y) {
  const long long a = f64_bits(x), b = f64_bits(y);
  return (a ^ (a >> 63 & 0x7fffffffffffffffll)) < (b ^ (b >> 63 & 0x7fffffffffffffffll));
}
// 0.5 * x, exact unless x is subnormal or the smallest normal
AMCA_HD double f64_half(double x) {
  if (f64_exponent(x) - 2u < 0x7fcu) return bits_f64(f64_bits(x) - (1ll << 52));
  return 0.5 * x;
}
AMCA_HD double f64_fma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return fma(a, b, c);
#endif
}

// x / 3, correctly rounded (the quotient-correction step of P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990): y = RN(1/3) is within 2^-54 relative of 1/3, so q0 = RN(x y) is within
// 1 ulp of x/3, the residual x - 3 q0 is exact, and q0 plus residual * y differs
// from x/3 by less than 2^-50 ulp, while no x/3 lies nearer than 1/6 ulp to a
// rounding midpoint. x is 0 or its exponent leaves room for the residual.
AMCA_HD double f64_third(double x) {
  const double y = 0x1.5555555555555p-2;
  const double q = x * y;
  return f64_fma(f64_fma(-3.0, q, x), y, q);
}
// y within 2^-46 relative of 1 / b for a double b that holds a float: one
// Newton step from the FP32 reciprocal.
AMCA_HD double recip_of_f32(float b, double bd) {
  const double y0 = pos_f32_to_f64(1.0f / b);
  return f64_fma(y0, f64_fma(-bd, y0, 1.0), y0);
}
// x / b, correctly rounded, for that b and y: q0 is within 2^-46 of x / b, so
// the residual has under 32 significant bits and is exact, and q0 + residual *
// y is within 2^-92 of x / b; b has 24 bits, so no x / b lies within 2^-78
// relative of a rounding midpoint. x is 0 or its exponent leaves room.
AMCA_HD double div_by_f32(double x, double bd, double y) {
  const double q = x * y;
  return f64_fma(f64_fma(-bd, q, x), y, q);
}

AMCA_HD void cell_ijk(const Grid &g, int32_t id, int &I, int &J, int &K) {
  K = quotient(id, g.by_xy);
  const int r = id - K * g.nxyg;
  J = quotient(r, g.by_x);
  I = r - J * g.nxg;
}
AMCA_HD void cell_ijk(const Grid &g, int64_t id, int &I, int &J, int &K) {
  K = (int)(id / g.nxyg);
  int r = (int)(id - (int64_t)K * g.nxyg);
  J = r / g.nxg;
  I = r - J * g.nxg;
}

// Neighbour n in 0..25 in the reference's k, j, i loop order
// (CA/src/CellularAutomataManager_3D.cpp:913-925).
AMCA_HD void nbr_offset(int n, int &di, int &dj, int &dk) {
  int m = n < 13 ? n : n + 1;  // skip the centre (index 13 of 27)
  dk = m / 9 - 1;
  dj = (m / 3) % 3 - 1;
  di = m % 3 - 1;
}

// cell_is_captured in FP64. l2g is transMatrixLocal2Global (row-major);
// the global->local matrix is its transpose, summed from 0 in component order.
AMCA_HD bool is_captured_f64(const double *l2g, double gcx, double gcy, double gcz, double length) {
  if (length == 0) return false;
  double cx = 0, cy = 0, cz = 0;
  cx += gcx * l2g[0];
  cy += gcx * l2g[1];
  cz += gcx * l2g[2];
  cx += gcy * l2g[3];
  cy += gcy * l2g[4];
  cz += gcy * l2g[5];
  cx += gcz * l2g[6];
  cy += gcz * l2g[7];
  cz += gcz * l2g[8];
  return fabs(cx) + fabs(cy) + fabs(cz) <= 1.0 * length;
}

// FP32 pre-test. Returns +1 (captured), 0 (not captured) or -1 (too close to
// the boundary for FP32: use is_captured_f64). gc* are the cell-centre offsets
// from the envelope centre in FP32; err is an absolute bound on their error
// per component; m32 is l2g rounded to float.
//
// Bound: |m_ij| <= 1, so each local coordinate is a 3-term dot product whose
// FP32 evaluation errs by at most 3*u*(|gx|+|gy|+|gz|) + 3*err (u = 2^-24),
// and the final sum of three absolute values adds 2*u*(its magnitude). The
// margin used is 2^-14 relative plus 8*err per component — orders of
// magnitude above that bound and the FP64 evaluation's own error.
//
// *lower receives a lower bound of the FP64 |c'|_1 (the same FP32 estimate
// less the margin's terms for the estimate itself, plus 2^-14 of it): an
// envelope whose half-diagonal stays below it cannot contain the cell.
AMCA_HD int captured_f32_lb(const float *m32, float gx, float gy, float gz, float err, float length, float *lower) {
  float cx = gx * m32[0] + gy * m32[3] + gz * m32[6];
  float cy = gx * m32[1] + gy * m32[4] + gz * m32[7];
  float cz = gx * m32[2] + gy * m32[5] + gz * m32[8];
  float s = fabsf(cx) + fabsf(cy) + fabsf(cz);
  float scale = fabsf(gx) + fabsf(gy) + fabsf(gz);
  float margin = 6.103515625e-05f * (3.0f * scale + length) + 24.0f * err;  // 2^-14
  *lower = s - (6.103515625e-05f * (3.0f * scale + s) + 24.0f * err);
  if (s < length - margin) return 1;
  if (s > length + margin) return 0;
  return -1;
}
AMCA_HD int captured_f32(const float *m32, float gx, float gy, float gz, float err, float length) {
  float lower;
  return captured_f32_lb(m32, gx, gy, gz, err, length, &lower);
}

// CA/src/Octahedron.cpp:27-84 tables
AMCA_HD double face_normal(int q, int i) {
  // normalVector[8][3]: (+x +y +z), (-x +y +z), (-x -y +z), (+x -y +z), then z negated
  const int sx = (q == 1 || q == 2 || q == 5 || q == 6) ? -1 : 1;
  const int sy = (q == 2 || q == 3 || q == 6 || q == 7) ? -1 : 1;
  const int sz = q >= 4 ? -1 : 1;
  return (double)(i == 0 ? sx : (i == 1 ? sy : sz));
}
AMCA_HD int face_corner(int q, int i) {
  // surfaceCorner[8][3] = {0,1,4},{1,2,4},{2,3,4},{3,0,4},{0,1,5},{1,2,5},{2,3,5},{3,0,5}
  const int f = q & 3;
  if (i == 2) return q < 4 ? 4 : 5;
  return (f + i) & 3;
}
AMCA_HD double corner_unit(int c, int j) {
  // cornerCoord[6][3] = +x, +y, -x, -y, +z, -z
  switch (c) {
    case 0: return j == 0 ? 1.0 : 0.0;
    case 1: return j == 1 ? 1.0 : 0.0;
    case 2: return j == 0 ? -1.0 : 0.0;
    case 3: return j == 1 ? -1.0 : 0.0;
    case 4: return j == 2 ? 1.0 : 0.0;
    default: return j == 2 ? -1.0 : 0.0;
  }
}
// Axis of corner c (+x +y -x -y +z -z).
AMCA_HD int corner_axis(int c) { return c < 4 ? (c & 1) : 2; }
AMCA_HD double dmin_ref(double a, double b) { return (b < a) ? b : a; }  // std::min
AMCA_HD double dmax_ref(double a, double b) { return (a < b) ? b : a; }  // std::max

// plus_zero(x) == x + 0.0 (a zero of either sign becomes +0).
AMCA_HD double plus_zero(double x) {
  const long long b = f64_bits(x);
  return b == (long long)0x8000000000000000ull ? 0.0 : x;
}
// nonneg(x) == (x >= 0) for x not NaN (-0 included).
AMCA_HD bool nonneg(double x) {
  const long long b = f64_bits(x);
  return b >= 0 || b == (long long)0x8000000000000000ull;
}
// corner_unit(c, corner_axis(c)) * length: +-length (exact: a sign flip).
AMCA_HD double corner_length(int c, double length) { return (c == 2 || c == 3 || c == 5) ? -length : length; }

// Octahedron::capture decentring (CA/src/Octahedron.cpp) in the reference's
// operation order. Where a term is a product with a corner coordinate (+-1 on
// one axis, 0 on the others) the zero terms are dropped and the +-1 products
// taken as sign flips; every such rewrite is bit-identical: a sum accumulated
// from +0.0 does not depend on the signs of its zero terms (+0 + -0 = +0,
// x + -0 = x), and squares and products of zeros are zeros.
AMCA_HD void capture_f64_general(const double *l2g, double gcx, double gcy, double gcz, double length, double h,
                         double trunc_coeff, double out[4]) {
  double cx = plus_zero(gcx * l2g[0]);  // 0 + p
  double cy = plus_zero(gcx * l2g[1]);
  double cz = plus_zero(gcx * l2g[2]);
  cx += gcy * l2g[3];
  cy += gcy * l2g[4];
  cz += gcy * l2g[5];
  cx += gcz * l2g[6];
  cy += gcz * l2g[7];
  cz += gcz * l2g[8];
  const double interception = fabs(cx) + fabs(cy) + fabs(cz);
  int quad = 0;
  const bool px = nonneg(cx), py = nonneg(cy);
  if (nonneg(cz)) {
    if (px && py) quad = 0;
    else if (px && !py) quad = 3;
    else if (!px && py) quad = 1;
    else quad = 2;
  } else {
    if (px && py) quad = 4;
    else if (px && !py) quad = 7;
    else if (!px && py) quad = 5;
    else quad = 6;
  }
  const double pC[3] = {cx, cy, cz};
  const double perp = length - interception;
  // (perp * n_i) / 3 with n_i = +-1 equals +-(perp / 3) exactly (IEEE
  // division is sign-symmetric), so one division serves all three terms
  const double third = perp / 3;
  double pA[3];
  for (int i = 0; i < 3; i++) pA[i] = pC[i] + (face_normal(quad, i) > 0 ? third : -third);
  // dist[i] = ((0 + d0^2) + d1^2) + d2^2 with d_j = pA[j] - corner_j * length:
  // on corner i's axis a, d_a = pA[a] -+ length; elsewhere d_j = pA[j]
  const double sq[3] = {pA[0] * pA[0], pA[1] * pA[1], pA[2] * pA[2]};
  double dist[3];
  for (int i = 0; i < 3; i++) {
    const int id = face_corner(quad, i);
    const int a = corner_axis(id);
    const double da = pA[a] - corner_length(id, length);
    const double t0 = a == 0 ? da * da : sq[0];
    const double t1 = a == 1 ? da * da : sq[1];
    const double t2 = a == 2 ? da * da : sq[2];
    dist[i] = (t0 + t1) + t2;
  }
  // distances are +0 or positive: their order is the order of their bits
  const long long b1 = f64_bits(dist[1]), b2 = f64_bits(dist[2]);
  int cid0 = face_corner(quad, 0), cid1, cid2;
  long long mind = f64_bits(dist[0]);
  // i = 1
  if (mind > b1) {
    mind = b1;
    cid1 = cid0;
    cid0 = face_corner(quad, 1);
  } else {
    cid1 = face_corner(quad, 1);
  }
  // i = 2
  if (mind > b2) {
    mind = b2;
    cid2 = cid0;
    cid0 = face_corner(quad, 2);
  } else {
    cid2 = face_corner(quad, 2);
  }
  // |S1S2|^2 = |S1S3|^2: the three corners of a face lie on three different
  // axes, so each edge vector is +-length on two axes and +0 on the third and
  // both sums are exactly fl(L*L) + fl(L*L). S1A . S1S2 and S1A . S1S3 keep
  // their two non-zero terms, in order.
  const int a0 = corner_axis(cid0), a1 = corner_axis(cid1), a2 = corner_axis(cid2);
  const double c1v = corner_length(cid0, length);  // S1 on its axis
  const double e1 = corner_length(cid1, length);   // S2 on its axis
  const double e2 = corner_length(cid2, length);   // S3 on its axis
  const double ll = length * length;
  double n12 = ll + ll;
  double d12 = 0.0, d13 = 0.0;
  for (int i = 0; i < 3; i++) {
    const double s1a = i == a0 ? pA[i] - c1v : pA[i];
    // S2 - S1 (and S3 - S1) on axis i: +e on S2's axis, -c1 on S1's, +0 elsewhere
    if (i == a1) d12 += s1a * e1;
    else if (i == a0) d12 += s1a * (0.0 - c1v);
    if (i == a2) d13 += s1a * e2;
    else if (i == a0) d13 += s1a * (0.0 - c1v);
  }
  n12 = (double)sqrtf((float)n12);
  const double n13 = n12;
  double I0 = d12 / n12, I1 = n12 - I0;
  const double J0 = d13 / n13, J1 = n13 - J0;
  const double tv = trunc_coeff * h;
  if (I0 < tv && I1 < tv) {
    I0 = n12 * 0.5;  // == n12 / 2 exactly
    I1 = n13 * 0.5;
  }
  const double L1 = 0.5 * (dmin_ref(I0, tv) + dmin_ref(I1, tv));
  const double L2 = 0.5 * (dmin_ref(J0, tv) + dmin_ref(J1, tv));
  const double Lnew = (double)sqrtf(2.0f) * (dmax_ref(L1, L2));
  const double mag = (length - Lnew);
  // (mag * c_i) / (length * T) for the corner S1 = c: non-zero on S1's axis
  // only; the rotated offset o_k = sum_i comp_i * l2g[i + 3k] is that term + 0
  const double comp = mag * c1v / (length * kTheodorus);
  out[0] = plus_zero(comp * l2g[a0 + 0]);
  out[1] = plus_zero(comp * l2g[a0 + 3]);
  out[2] = plus_zero(comp * l2g[a0 + 6]);
  out[3] = Lnew;
}

// The face quadrant of a point (the signs of its components, -0 positive).
AMCA_HD int quadrant(double cx, double cy, double cz) {
  const bool px = nonneg(cx), py = nonneg(cy);
  const int q = px ? (py ? 0 : 3) : (py ? 1 : 2);
  return nonneg(cz) ? q : q + 4;
}

#if defined(__CUDA_ARCH__)
__device__ __noinline__ inline void capture_f64_slow(const double *l2g, double gcx, double gcy, double gcz,
                                                     double length, double h, double trunc_coeff, double out[4]) {
  capture_f64_general(l2g, gcx, gcy, gcz, length, h, trunc_coeff, out);
}
#else
inline void capture_f64_slow(const double *l2g, double gcx, double gcy, double gcz, double length, double h,
                             double trunc_coeff, double out[4]) {
  capture_f64_general(l2g, gcx, gcy, gcz, length, h, trunc_coeff, out);
}
#endif

// Octahedron::capture_cell: the new, decentred envelope for a captured cell.
// gc = cell centre - parent centre (FP64). Writes the new centre offset
// (global frame) into out[0..2] and the new half-diagonal into out[3].
//
// capture_f64_general with fewer FP64 instructions (about 60 instead of 140;
// they are what a claim phase with new envelopes spends its time on), the same
// bits in every case. Beyond the helpers above:
//  - the corners in order of distance: dist_i - dist_j = 2 L (|pA_j| - |pA_i|)
//    up to 2^-46 L^2 of rounding (each corner lies on the side of its axis that
//    pA is on), so FP32 magnitudes that differ by more than 2^-19 L order them;
//  - the edge products share S1A's term, and a sum of two terms accumulated
//    from +0.0 is plus_zero of one plus the other in either order;
//  - both edge quotients divide by the same n12, a float.
// A point outside the envelope, corners too near a tie, magnitudes near the
// ends of the exponent range and a truncation with a sign or NaN go the general
// way.
AMCA_HD void capture_f64(const double *l2g, double gcx, double gcy, double gcz, double length, double h,
                         double trunc_coeff, double out[4]) {
  double c[3];
  for (int i = 0; i < 3; ++i) c[i] = (plus_zero(gcx * l2g[i]) + gcy * l2g[3 + i]) + gcz * l2g[6 + i];
  const double interception = fabs(c[0]) + fabs(c[1]) + fabs(c[2]);
  const int quad = quadrant(c[0], c[1], c[2]);
  const double perp = length - interception;
  const int ep = f64_exponent(perp), el = f64_exponent(length);
  const double tv = trunc_coeff * h;
  // lengths between 2^-50 and 2^50; perp positive (or +0) and not vanishing;
  // a truncation that compares by its bits (no sign, no NaN)
  bool general = el - 973u > 100u || f64_bits(perp) < 0 || (ep < 400 && f64_bits(perp) != 0) ||
                 (unsigned long long)f64_bits(tv) > 0x7ff0000000000000ull;
  const double third = f64_third(perp);
  double pA[3];
  for (int i = 0; i < 3; i++) pA[i] = c[i] + (nonneg(c[i]) ? third : -third);  // the face normal's signs are c's
  float m[3];  // |pA|
  for (int i = 0; i < 3; ++i) m[i] = fabsf(f64_to_f32_rz(pA[i]));
  const float tie = 1.9073486328125e-06f * f64_to_f32_rz(length);  // 2^-19 L
  // as the reference: corner 0 against 1, then the nearer of them against 2
  const int k0 = face_corner(quad, 0), k1 = face_corner(quad, 1), k2 = face_corner(quad, 2);
  const float f0 = corner_axis(k0) == 0 ? m[0] : m[1], f1 = corner_axis(k1) == 0 ? m[0] : m[1], f2 = m[2];
  general = general || !(fabsf(f0 - f1) > tie);
  int cid0 = f0 < f1 ? k1 : k0, cid1 = f0 < f1 ? k0 : k1, cid2 = k2;
  const float near01 = f0 < f1 ? f1 : f0;
  general = general || !(fabsf(near01 - f2) > tie);
  if (near01 < f2) {
    cid2 = cid0;
    cid0 = k2;
  }
  const int a0 = corner_axis(cid0), a1 = corner_axis(cid1), a2 = corner_axis(cid2);
  const double p0 = a0 == 0 ? pA[0] : (a0 == 1 ? pA[1] : pA[2]);
  const double p1 = a1 == 0 ? pA[0] : (a1 == 1 ? pA[1] : pA[2]);
  const double p2 = a2 == 0 ? pA[0] : (a2 == 1 ? pA[1] : pA[2]);
  const double c1v = corner_length(cid0, length);  // S1 on its axis
  const double t0 = plus_zero((p0 - c1v) * -c1v);
  const double d12 = t0 + p1 * corner_length(cid1, length), d13 = t0 + p2 * corner_length(cid2, length);
  const int e12 = f64_exponent(d12), e13 = f64_exponent(d13);
  general = general || (e12 < 400 && (f64_bits(d12) << 1) != 0) || (e13 < 400 && (f64_bits(d13) << 1) != 0);
  if (general) {
    capture_f64_slow(l2g, gcx, gcy, gcz, length, h, trunc_coeff, out);
    return;
  }
  const float n12f = sqrtf(pos_f64_to_f32_rn(bits_f64(f64_bits(length * length) + (1ll << 52))));
  const double n12 = pos_f32_to_f64(n12f);
  const double y = recip_of_f32(n12f, n12);
  double I0 = div_by_f32(d12, n12, y), I1 = n12 - I0;
  const double J0 = div_by_f32(d13, n12, y), J1 = n12 - J0;
  if (f64_less(I0, tv) && f64_less(I1, tv)) {
    I0 = f64_half(n12);  // == n12 / 2
    I1 = I0;
  }
  const double s1 = (f64_less(tv, I0) ? tv : I0) + (f64_less(tv, I1) ? tv : I1);
  const double s2 = (f64_less(tv, J0) ? tv : J0) + (f64_less(tv, J1) ? tv : J1);
  const double L1 = f64_half(s1), L2 = f64_half(s2);
  const double Lnew = (double)sqrtf(2.0f) * (f64_less(L1, L2) ? L2 : L1);
  const double comp = (length - Lnew) * c1v / (length * kTheodorus);
  out[0] = plus_zero(comp * l2g[a0 + 0]);
  out[1] = plus_zero(comp * l2g[a0 + 3]);
  out[2] = plus_zero(comp * l2g[a0 + 6]);
  out[3] = Lnew;
}

#if defined(__CUDACC__)
// capture_f64 by four consecutive lanes (`mask`, the first one `base`) that
// hold the same envelope, lane base + a working on axis a = 0, 1, 2 (lane 3
// repeats axis 2) with that component gc of the offset: the same operations on
// the same values, a component or an edge each, so about 40 FP64 instructions
// in a row instead of 60. Returns the component out[a]; Lout is out[3].
__device__ __forceinline__ double capture_f64_quad(const double *l2g, int a, unsigned mask, int base, double gc,
                                                   double length, double h, double trunc_coeff, double &Lout) {
  const double gcx = __shfl_sync(mask, gc, base), gcy = __shfl_sync(mask, gc, base + 1),
               gcz = __shfl_sync(mask, gc, base + 2);
  const double c = (plus_zero(gcx * l2g[a]) + gcy * l2g[3 + a]) + gcz * l2g[6 + a];
  const double c0 = __shfl_sync(mask, c, base), c1 = __shfl_sync(mask, c, base + 1), c2 = __shfl_sync(mask, c, base + 2);
  const double interception = fabs(c0) + fabs(c1) + fabs(c2);
  const int quad = quadrant(c0, c1, c2);
  const double perp = length - interception;
  const int ep = f64_exponent(perp), el = f64_exponent(length);
  const double tv = trunc_coeff * h;
  bool general = el - 973u > 100u || f64_bits(perp) < 0 || (ep < 400 && f64_bits(perp) != 0) ||
                 (unsigned long long)f64_bits(tv) > 0x7ff0000000000000ull;
  const double third = f64_third(perp);
  const double pA = c + (nonneg(c) ? third : -third);
  const float mag = fabsf(f64_to_f32_rz(pA));
  const float m0 = __shfl_sync(mask, mag, base), m1 = __shfl_sync(mask, mag, base + 1),
              m2 = __shfl_sync(mask, mag, base + 2);
  const float tie = 1.9073486328125e-06f * f64_to_f32_rz(length);  // 2^-19 L
  const int k0 = face_corner(quad, 0), k1 = face_corner(quad, 1), k2 = face_corner(quad, 2);
  const float f0 = corner_axis(k0) == 0 ? m0 : m1, f1 = corner_axis(k1) == 0 ? m0 : m1, f2 = m2;
  general = general || !(fabsf(f0 - f1) > tie);
  int cid0 = f0 < f1 ? k1 : k0, cid1 = f0 < f1 ? k0 : k1, cid2 = k2;
  const float near01 = f0 < f1 ? f1 : f0;
  general = general || !(fabsf(near01 - f2) > tie);
  if (near01 < f2) {
    cid2 = cid0;
    cid0 = k2;
  }
  const int a0 = corner_axis(cid0);
  // edge 1-2 on the first lane, 1-3 on the others
  const int ce = a == 0 ? cid1 : cid2;
  const double p0 = __shfl_sync(mask, pA, base + a0), pe = __shfl_sync(mask, pA, base + corner_axis(ce));
  const double c1v = corner_length(cid0, length);  // S1 on its axis
  const double t0 = plus_zero((p0 - c1v) * -c1v);
  const double de = t0 + pe * corner_length(ce, length);
  const int ee = f64_exponent(de);
  general = general || (ee < 400 && (f64_bits(de) << 1) != 0);
  if (__ballot_sync(mask, general)) {
    double out[4];
    capture_f64_slow(l2g, gcx, gcy, gcz, length, h, trunc_coeff, out);
    Lout = out[3];
    return a == 0 ? out[0] : (a == 1 ? out[1] : out[2]);
  }
  const float n12f = sqrtf(pos_f64_to_f32_rn(bits_f64(f64_bits(length * length) + (1ll << 52))));
  const double n12 = pos_f32_to_f64(n12f);
  const double y = recip_of_f32(n12f, n12);
  double I0 = div_by_f32(de, n12, y), I1 = n12 - I0;
  if (a == 0 && f64_less(I0, tv) && f64_less(I1, tv)) {
    I0 = f64_half(n12);  // == n12 / 2
    I1 = I0;
  }
  const double half = f64_half((f64_less(tv, I0) ? tv : I0) + (f64_less(tv, I1) ? tv : I1));
  const double L1 = __shfl_sync(mask, half, base), L2 = __shfl_sync(mask, half, base + 1);
  const double Lnew = (double)sqrtf(2.0f) * (f64_less(L1, L2) ? L2 : L1);
  const double comp = (length - Lnew) * c1v / (length * kTheodorus);
  Lout = Lnew;
  return plus_zero(comp * l2g[a0 + 3 * a]);
}
#endif

// Hexahedral (8-node) interpolation of MapVoxelManager::evaluate_temperature
// (CA/src/MapVoxelManager.cpp:746-799) in FP64: the shape functions in the
// reference's factor order, summed from 0 in node order.
AMCA_HD double hex8_interp64(const double t[8], double xi, double eta, double zeta) {
  double s[8];
  s[0] = 0.125 * (1.0 - eta) * (1.0 - xi) * (1.0 - zeta);
  s[1] = 0.125 * (1.0 - eta) * (1.0 + xi) * (1.0 - zeta);
  s[2] = 0.125 * (1.0 + eta) * (1.0 + xi) * (1.0 - zeta);
  s[3] = 0.125 * (1.0 + eta) * (1.0 - xi) * (1.0 - zeta);
  s[4] = 0.125 * (1.0 - eta) * (1.0 - xi) * (1.0 + zeta);
  s[5] = 0.125 * (1.0 - eta) * (1.0 + xi) * (1.0 + zeta);
  s[6] = 0.125 * (1.0 + eta) * (1.0 + xi) * (1.0 + zeta);
  s[7] = 0.125 * (1.0 + eta) * (1.0 - xi) * (1.0 + zeta);
  double v = 0.0;
  for (int i = 0; i < 8; i++) v += s[i] * t[i];
  return v;
}

// FP32 estimate of hex8_interp64 from the node values and parametric
// coordinates rounded to float, and a bound on its error to decide with. With
// u = 2^-24 and M the largest node magnitude: a factor 1 +- x errs by 1.5 u (x
// rounded, then the sum), which over the eight nodes and three directions
// comes to 36 u M (the other two factors sum to 4); node values rounded 8 u M;
// three roundings per product 24 u M (the weights times 8 sum to 8); seven sums
// 56 u M; times 1/8: 15.5 u M < 2^-20 M. The bound is 2^-19 of M (plus 2^-16
// absolute, for underflow); FP64 decides closer to a threshold. A margin of
// 2^-16 sent a lane of every other warp of a melt pool's elements there.
AMCA_HD float hex8_interp32(const float t[8], float xi, float eta, float zeta) {
  const float a0 = 1.0f - eta, a1 = 1.0f + eta, b0 = 1.0f - xi, b1 = 1.0f + xi, c0 = 1.0f - zeta, c1 = 1.0f + zeta;
  return 0.125f * (a0 * b0 * c0 * t[0] + a0 * b1 * c0 * t[1] + a1 * b1 * c0 * t[2] + a1 * b0 * c0 * t[3] +
                   a0 * b0 * c1 * t[4] + a0 * b1 * c1 * t[5] + a1 * b1 * c1 * t[6] + a1 * b0 * c1 * t[7]);
}
AMCA_HD float hex8_err32(const float t[8]) {
  float mg = 0.0f;
  for (int i = 0; i < 8; ++i) mg = fmaxf(mg, fabsf(t[i]));
  return ldexpf(mg, -19) + 1.52587890625e-05f;
}

// ProblemPhysics_RappazGandin1993::compute_growth_velocity for a uniform field
AMCA_HD double kgt_velocity(double Tm, double T, double a1, double a2, double a3) {
  const double dT = Tm - T;
  double v = 0.0;
  if (dT > 0) {
    v = a1 * dT + a2 * dT * dT + a3 * dT * dT * dT;
    if (v < 0.0) v = 0.0;
  }
  return v;
}

}  // namespace amca
