// Fast FP64 kernel entries for the full-kernel product K x.
//
// The product needs FP64-accurate entries (a few ulp of a kernel of the distances
// that it forms), not entries that are bit-identical to the ones ACA used, so it
// may contract into FMAs and use a cheaper exponential.  exp here follows Tang's table-driven method (P. T. P.
// Tang, "Table-driven implementation of the exponential function in IEEE
// floating-point arithmetic", ACM TOMS 15(2), 1989), in units of ln2 / T: with
// z = x T / ln2 = n + f, e^-x = 2^-(n / T) 2^(-f / T), the first factor from a
// table of correctly rounded 2^(-j/T) and an exponent shift, the second from a
// polynomial.  The unit is folded into the scale of the distances, so f = z - n is
// exact and no second multiplication by a split ln2 / T is left.  The symmetric
// forms scale the coordinates: a distance then carries an error of 2^-53 times the
// coordinates, in length scales.  The row-by-row and forest forms scale the distance
// (one more multiplication per entry): nearby coordinates subtract exactly, wherever
// the cloud lies.
//
// The product is bound by issue: an FP64 instruction takes a scheduler two cycles
// (64 lanes a cycle and SM), every other one takes one and hides behind nothing.
// So an index by FP32 and integer instructions instead of two FP64 additions
// loses, and constants that fit no operand stay in registers.  FP64 instructions of an entry, before ->
// now: Matern-3/2 in 2D 20 -> 18, Gaussian in 3D 16 -> 13.
// With the other instructions trimmed too, N = 131072 Matern-3/2 2D with 8 vectors
// 22.3 -> 20.4 ms, N = 50001 Gaussian 3D with one 2.04 -> 1.60 ms.
#pragma once

#include "kfun.h"

#if defined(__CUDACC__)
constexpr int HX_EXP2_LOG = 11;
static __device__ const double hx_exp2_table[1 << HX_EXP2_LOG] = {
#include "exp2_table.inc"
};

// A constant that stays in registers.  An FP64 instruction takes one constant
// operand; a second one of the same instruction is otherwise moved into registers
// again for every entry.
__device__ __forceinline__ double hx_in_register(double v) {
  asm volatile("" : "+d"(v));
  return v;
}

// e^-x by a table of T = 2^LOGT entries in shared memory, COPIES times side by
// side: entry j of lane l sits at j * COPIES + l % COPIES, so with 16 copies a
// lookup of 32 different entries has no bank conflicts (random entries in one
// copy cost about 6 wavefronts instead of 2).
//
// Polynomials: 2^(-f/T) - 1 = r + r^2/2 + r^3/6 (+ r^4/24), r = -f ln2 / T, with
// the first dropped term folded into the one two below it where it is smallest
// over |f| <= 1/2 (T = 2048: 7e-18, T = 256: 5e-18).
template <int LOGT, int COPIES>
struct ExpTab {
  static constexpr int T = 1 << LOGT, DOUBLES = T * COPIES;
  static constexpr double L = 0x1.62e42fefa39efp-1 / T;  // ln2 / T, exact division
  static constexpr double UNIT = 0x1.71547652b82fep+0 * T;
  static constexpr double A2 = 0.25 * L * L;  // the square of the largest |r|
  const double* p;
  double top, below, l, k375;  // the constants with more than 32 bits, and 3/8

  // tab[DOUBLES]: the caller synchronises before the first lookup.  The high word
  // of entry j is stored with j added below the exponent's unit: subtracting
  // n << (20 - LOGT), n = k T + j, takes it off again together with k.
  static __device__ __forceinline__ void fill(double* tab) {
    for (int i = threadIdx.x; i < DOUBLES; i += blockDim.x) {
      const int j = i / COPIES;
      const double v = __ldg(&hx_exp2_table[j << (HX_EXP2_LOG - LOGT)]);
      tab[i] = __hiloint2double(__double2hiint(v) + (j << (20 - LOGT)), __double2loint(v));
    }
  }
  __device__ __forceinline__ explicit ExpTab(const double* tab)
      : p(tab + (threadIdx.x & (COPIES - 1))),
        top(hx_in_register(LOGT >= 11 ? -L * L * L / 6 : L * L * L * L / 24)),
        below(hx_in_register(LOGT >= 11 ? (0.5 + 0.8284271247461901 * A2 / 24) * L * L
                                        : -(1.0 / 6 + 0.869 * A2 / 120) * L * L * L)),
        l(hx_in_register(L)),
        k375(hx_in_register(0.375)) {}

  // t = 2^-(n / T) and f of z >= 0, n = rint(z): the low word of z + 1.5 * 2^52.
  // z is clamped at 1020 T by its high word, so that 2^-n/T stays normal: from
  // x = 707 on the factor is about 1e-307.  A NaN is clamped with it: (1 + x) e^-x
  // returns the NaN of its own x, a plain e^-x the clamped value.
  __device__ __forceinline__ void split(double z, double& t, double& f) const {
    constexpr int ZMAX = (1023 + 9 + LOGT) << 20 | 0xfe000;  // high word of 1020 T
    const double zc = __hiloint2double(min(__double2hiint(z), ZMAX), __double2loint(z));
    const double t0 = zc + 0x1.8p52;
    const int n = __double2loint(t0);
    f = zc - (t0 - 0x1.8p52);
    const double v = p[(n & (T - 1)) * COPIES];
    t = __hiloint2double(__double2hiint(v) - n * (1 << (20 - LOGT)), __double2loint(v));
  }
  // (2^(-f/T) - 1) / f
  __device__ __forceinline__ double poly(double f) const {
    const double q = fma(f, top, below);
    return fma(LOGT >= 11 ? q : fma(q, f, 0.5 * L * L), f, -l);
  }
  // a e^-x
  __device__ __forceinline__ double scaled(double t, double f, double a) const {
    const double w = t * a;
    return fma(w * f, poly(f), w);
  }
  __device__ __forceinline__ double neg_exp(double z) const {
    double t, f;
    split(z, t, f);
    return fma(t * f, poly(f), t);
  }
};

// Square roots from the hardware reciprocal-square-root approximation
// (rsqrt.approx.ftz.f64, relative error below 2^-20 on this GPU).  x must be a
// positive normal number.
__device__ __forceinline__ double hx_rsqrt_seed(double x) {
  double y;
#if defined(__CUDA_ARCH__)
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#else
  y = 1.0 / sqrt(x);
#endif
  return y;
}
// sqrt(x) from the seed y0 ~ 1/sqrt(x) (relative error e ~ 2^-20) by one
// third-order correction: with y = x y0 and t = y y0 - 1 (~2e),
// sqrt(x) = y (1 + t)^(-1/2) = y (1 - t/2 + 3t^2/8 - ...), and the dropped
// term 5t^3/16 is below 2^-57.  The rounding of y enters as half its relative
// error, so the result is within 1 ulp of the correctly rounded square root
// (checked against libm's sqrt on 2e7 inputs with seeds perturbed by 2^-20).
__device__ __forceinline__ double hx_sqrt_nr(double x, double k375) {
  const double y0 = hx_rsqrt_seed(x);
  const double y = x * y0;
  const double t = fma(y, y0, -1.0);
  return fma(y, t * fma(t, k375, -0.5), y);
}
// 1/sqrt(x) likewise: y0 (1 + t)^(-1/2).
__device__ __forceinline__ double hx_rsqrt_nr(double x, double k375) {
  const double y0 = hx_rsqrt_seed(x);
  const double t = fma(x * y0, y0, -1.0);
  return fma(y0, t * fma(t, k375, -0.5), y0);
}

// Lower bound of the scaled squared distances given to hx_kernel_unit: a sum of
// squares that starts here instead of at 0 keeps the reciprocal square-root seed
// finite at r2 = 0 (the diagonal) without a per-entry max.  It moves r by less than 2^-50 units of ln2 / T (2^-58 in x), and every kernel
// value (1 - x or 1 - O(r2) there) by less than a quarter ulp.
#define HX_R2_FLOOR 0x1p-100

// Coordinates scaled by c = hx_point_scale<KTYPE>(a, E::UNIT) turn the kernel
// into a function of the scaled squared distance alone (hx_kernel_unit): one
// multiply per point instead of one per entry.  r2 >= HX_R2_FLOOR.
template <int KTYPE>
__device__ __forceinline__ double hx_point_scale(double a, double unit) {
  if (KTYPE == HX_KERNEL_GAUSSIAN) return sqrt(-a * unit);
  if (KTYPE == HX_KERNEL_MATERN32 || KTYPE == HX_KERNEL_EXPONENTIAL) return a * unit;
  return sqrt(a);  // inverse multiquadric, quadratic
}
// (1 + x) e^-x, z = x T / ln2
template <class E>
__device__ __forceinline__ double hx_matern32(double z, const E& e) {
  double t, f;
  e.split(z, t, f);
  return e.scaled(t, f, fma(z, e.l, 1.0));
}
template <int KTYPE, class E>
__device__ __forceinline__ double hx_kernel_unit(double r2, const E& e) {
  if (KTYPE == HX_KERNEL_GAUSSIAN) return e.neg_exp(r2);
  if (KTYPE == HX_KERNEL_MATERN32) return hx_matern32(hx_sqrt_nr(r2, e.k375), e);
  if (KTYPE == HX_KERNEL_INV_MULTIQUADRIC) return hx_rsqrt_nr(1.0 + r2, e.k375);
  if (KTYPE == HX_KERNEL_QUADRATIC) return 1.0 + r2;
  return e.neg_exp(hx_sqrt_nr(r2, e.k375));
}

// The same from an unscaled squared distance r2 >= HX_R2_RAW_FLOOR and c =
// hx_distance_scale<KTYPE>(a, E::UNIT): one more multiplication per entry.
#define HX_R2_RAW_FLOOR 1e-300
template <int KTYPE>
__device__ __forceinline__ double hx_distance_scale(double a, double unit) {
  if (KTYPE == HX_KERNEL_GAUSSIAN) return -a * unit;
  if (KTYPE == HX_KERNEL_MATERN32 || KTYPE == HX_KERNEL_EXPONENTIAL) return a * unit;
  return a;  // inverse multiquadric, quadratic
}
template <int KTYPE, class E>
__device__ __forceinline__ double hx_kernel_raw(double r2, double c, const E& e) {
  if (KTYPE == HX_KERNEL_GAUSSIAN) return e.neg_exp(r2 * c);
  if (KTYPE == HX_KERNEL_MATERN32) return hx_matern32(hx_sqrt_nr(r2, e.k375) * c, e);
  if (KTYPE == HX_KERNEL_INV_MULTIQUADRIC) return hx_rsqrt_nr(fma(r2, c, 1.0), e.k375);
  if (KTYPE == HX_KERNEL_QUADRATIC) return fma(r2, c, 1.0);
  return e.neg_exp(hx_sqrt_nr(r2, e.k375) * c);
}
#endif
