// walk_fp64.cuh -- FP64 interaction and acceptance test shared by the plain
// force walk, the frozen-structure replay and the adjoint walk, so all three
// take the same decisions on the same inputs.
#pragma once

#include "nbb_internal.cuh"

namespace nbb {

// 1 / sqrt(x), square root and reciprocal each correctly rounded (the bits of
// __drcp_rn(__dsqrt_rn(x))), for x in [2^-927, 2^993): one hardware estimate
// shared by both and the residual corrections of Markstein ("Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990), 10 FP64
// operations.
//   y0      the estimate, 21 significant bits, so y0^2 is exact; r = 1 - x y0^2
//           is rounded once and |r| < 2^-19 (largest over every high word:
//           1.95 * 2^-20; the low word does not matter)
//   y       y0 (1 + r/2 + 3/8 r^2): relative error 2^-54 sqrt(x) from its
//           rounding, 5/16 |r|^3 < 2^-58 from the series (x in [1, 4))
//   g, d    x y and the residual x - g^2, each rounded once
//   s       g + d y/2, in error by less than 2^-103.5 sqrt(x) before its
//           rounding
//   e, 1/s  y + y (1 - s y), in error by less than 2^-103.5 / s before its
//           rounding
// A result rounds wrongly only when the exact value lies that close to the
// middle of two neighbours.  For the square root that takes an x with
// m^2 - x = k 2^-106 (|k| < 48, m the middle, sqrt(x) in [1, 2)), for the
// reciprocal an s with s m - 1 = k 2^-106 (|k| < 8); both sets are small
// (tests/test_inv_sqrt_rounding.py enumerates them and runs the sequence in
// exact arithmetic with every estimate of the bound): only the root s = 2 -
// 2^-52 comes out wrong (Markstein's exception), which 4 - 2^-51 has whatever
// the estimate and 4 - 2^-50 for some.  inv_sqrt_in_range leaves these two
// significands to the general form.
__device__ __forceinline__ double inv_sqrt_core(double x) {
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
  const double r = __fma_rn(-x, __dmul_rn(y0, y0), 1.0);
  const double y = __fma_rn(__fma_rn(r, 0.375, 0.5), __dmul_rn(y0, r), y0);
  const double g = __dmul_rn(x, y);
  const double d = __fma_rn(-g, g, x);
  const double half_y = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
  const double s = __fma_rn(d, half_y, g);
  return __fma_rn(__fma_rn(-s, y, 1.0), y, y);
}
// Whether inv_sqrt_core gives the right bits for x: its range, without the
// significands that may round wrongly (those with their low words are left out).
__device__ __forceinline__ bool inv_sqrt_low_word(double x) { return (unsigned)__double2loint(x) < 0xfffffffeu; }
__device__ __forceinline__ bool inv_sqrt_in_range(double x) {
  return (unsigned)(__double2hiint(x) - 0x06000000) < 0x78000000u && inv_sqrt_low_word(x);
}
static __device__ __noinline__ double inv_sqrt_general(double x) { return __drcp_rn(__dsqrt_rn(x)); }

// barnes_hut.cu:56-80, the factor G m (d^2 + eps^2)^-3/2 with the
// reference's operation order.  The reference's 1.0 / sqrt(r2) is a
// correctly rounded division of 1, which is the correctly rounded reciprocal:
// the same bits for every input.  Returns false on a singular interaction.
// gm is the product G m.
__device__ __forceinline__ bool scaled_mass_factor(double d2, double gm, double soft2, double &f) {
  const double r2 = __dadd_rn(d2, soft2);
  double inv = inv_sqrt_core(r2);
  if (!inv_sqrt_in_range(r2)) inv = inv_sqrt_general(r2);
  const double inv3 = __dmul_rn(__dmul_rn(inv, inv), inv);
  f = __dmul_rn(gm, inv3);
  return !(r2 <= 0.0);
}

// G m (d^2 + eps^2)^-3/2 d accumulated in the reference's order.  Returns
// false (and adds nothing) on a singular interaction.
__device__ __forceinline__ bool point_mass_fp64(double dx, double dy, double dz, double d2,
                                                double m, double g, double soft2, double &ax,
                                                double &ay, double &az) {
  double f;
  if (!scaled_mass_factor(d2, __dmul_rn(g, m), soft2, f)) return false;
  ax = __fma_rn(f, dx, ax);
  ay = __fma_rn(f, dy, ay);
  az = __fma_rn(f, dz, az);
  return true;
}

__device__ __forceinline__ double sqdist(double dx, double dy, double dz) {
  return __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx)));
}

// barnes_hut.cu:273-294: the acceptance test of target t at a node with
// records a = (com, mass), c = (crit, crit^2 band, box radius^2) and, at *bp,
// b = (centre, half size).  sqrt(d2) > crit is decided on d2 against crit^2
// outside a 2^-44 band and by the exact square root inside it; a node
// containing the target, or at zero distance, is never accepted.  Beyond the
// box radius (c.w: (max(crit, sqrt(3) h + |com - centre|) (1 + 2^-40))^2) no
// point of the cell lies, so the containment test can only fail there and b
// is read only inside it; the decisions are the reference's in every case.
// Returns the offset com - t and its square.
__device__ __forceinline__ bool accept_fp64(const double4 &a, const double4 *bp, const double4 &c,
                                            const double4 &t, double &dx, double &dy, double &dz,
                                            double &d2) {
  dx = __dsub_rn(a.x, t.x);
  dy = __dsub_rn(a.y, t.y);
  dz = __dsub_rn(a.z, t.z);
  d2 = sqdist(dx, dy, dz);
  bool accept = (d2 > c.z) ? true : (d2 < c.y) ? false : (__dsqrt_rn(d2) > c.x);
  if (accept && !(d2 > c.w)) {
    const double4 b = *bp;
    const bool contains = fabs(__dsub_rn(t.x, b.x)) <= b.w && fabs(__dsub_rn(t.y, b.y)) <= b.w &&
                          fabs(__dsub_rn(t.z, b.z)) <= b.w;
    accept = !contains && d2 > 0.0;
  }
  return accept;
}

}  // namespace nbb
