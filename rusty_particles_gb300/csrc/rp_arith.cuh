// Vectors and the FP64 arithmetic of the step kernels: roots and quotients from
// the hardware's seeds, conversions between float and double and comparisons on
// the integer pipe. Compiled with -fmad=false: each operation rounds by itself.
#pragma once
#include <cstdint>

namespace rp {

template <typename R>
struct T3 {
  R x, y, z;
};
template <typename R> __device__ __forceinline__ T3<R> t3(R x, R y, R z) { return T3<R>{x, y, z}; }
template <typename R> __device__ __forceinline__ T3<R> operator+(T3<R> a, T3<R> b) { return T3<R>{a.x + b.x, a.y + b.y, a.z + b.z}; }
template <typename R> __device__ __forceinline__ T3<R> operator-(T3<R> a, T3<R> b) { return T3<R>{a.x - b.x, a.y - b.y, a.z - b.z}; }
template <typename R> __device__ __forceinline__ T3<R> operator-(T3<R> a) { return T3<R>{-a.x, -a.y, -a.z}; }
template <typename R> __device__ __forceinline__ T3<R> operator*(T3<R> a, R s) { return T3<R>{a.x * s, a.y * s, a.z * s}; }
template <typename R> __device__ __forceinline__ T3<R> operator*(R s, T3<R> a) { return T3<R>{s * a.x, s * a.y, s * a.z}; }
template <typename R> __device__ __forceinline__ T3<R> operator/(T3<R> a, R s) { return T3<R>{a.x / s, a.y / s, a.z / s}; }
template <typename R> __device__ __forceinline__ R dot(T3<R> a, T3<R> b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <typename R> __device__ __forceinline__ T3<R> cross(T3<R> a, T3<R> r) {
  return T3<R>{a.y * r.z - r.y * a.z, a.z * r.x - r.z * a.x, a.x * r.y - r.x * a.y};
}
template <typename R> __device__ __forceinline__ R len(T3<R> a) { return sqrt(dot(a, a)); }
template <typename R, typename S> __device__ __forceinline__ T3<R> cvt(T3<S> a) { return T3<R>{(R)a.x, (R)a.y, (R)a.z}; }

using V = T3<double>;
using Vf = T3<float>;
__device__ __forceinline__ V vmk(double x, double y, double z) { return V{x, y, z}; }
// isfinite(x), x == 0 and 0.0 + x from the bits, off the FP64 pipe
__device__ __forceinline__ bool finite_bits(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ double plus_zero(double x) { return is_zero(x) ? 0.0 : x; }
// whether any component has a bit other than its sign set (is not +-0)
__device__ __forceinline__ bool some_bits(V a) {
  return ((__double_as_longlong(a.x) | __double_as_longlong(a.y) | __double_as_longlong(a.z)) << 1) != 0;
}
__device__ __forceinline__ float plus_zero(float x) { return (__float_as_int(x) << 1) == 0 ? 0.0f : x; }

constexpr double kPi = 3.14159265358979323846;

// float -> double, exactly, on the integer pipe: the exponent is re-biased
// (+896) and the mantissa shifted into place; a subnormal's leading one becomes
// the implicit one. A conversion instruction would run on the FP64 pipe, and
// costs it an issue slot even where a predicate turns it off.
__device__ __forceinline__ double f2d_exact(float f) {
  const uint32_t u = __float_as_uint(f);
  uint32_t m = u & 0x7FFFFFFFu, e = 896u << 20;
  if (m < 0x00800000u) {  // zero or subnormal
    const uint32_t up = __clz(m) - 8u;
    m = m ? m << up : 0u;  // (bit 23 adds one to the exponent)
    e = m ? (896u - up) << 20 : 0u;
  } else if (m >= 0x7F800000u) {
    e = (2047u - 255u) << 20;
  }
  return __hiloint2double((int)((u & 0x80000000u) | ((m >> 3) + e)), (int)(m << 29));
}

// -------------------------------------------- FP64 roots and quotients
// GB300's FP64 pipe takes a warp instruction every 16 clocks of an SM, and the
// library's sqrt, 1/x and a/b measured 144, 178 and about 190 of them (9, 11
// and 12 FP64 instructions) in kernels that this pipe bounds. Here the
// hardware's seeds (rsqrt / rcp.approx.ftz.f64: MUFU instructions, off that
// pipe) take one third-order step (Householder: y (1 + e/2 + 3 e^2/8) with
// e = 1 - x y^2, and y (1 + e + e^2) with e = 1 - x y), and the result is
// corrected by its exact residual (Markstein 1990: x - s^2 and a - b q are
// representable): 8 FP64 instructions for a root, 2 more for its reciprocal, 6
// for a quotient. Together with the integer comparisons below this took the pair
// kernel of a 1,048,576-sphere Hertz bed from 206 to 194 million FP64 thread
// instructions (461 to 435 us), and the reference's JKR Newton on 262,144 spheres
// from 2.82 to 2.67 ms a step. Zero, negative, infinite, NaN and very large or
// small arguments go to the library.
//
// The results are the correctly rounded ones, as the library's are:
// * Root: before its last rounding it is within 2^-51 ulp, and the numbers whose
//   root lies closer than 2^-50 ulp to a midpoint are among the M^2 + M + j with
//   |j| < 16 (M + 1/2 the midpoint).
// * Quotient: the seed is good to 2^-19.94 (2^-20.04 where the divisor's mantissa
//   starts with five ones; every upper word measured, the lower one is not read),
//   so y is within 0.5 + 2^52 seed^3 = 0.5045 (0.5036) ulp of 1/b and q + r y
//   within 2^-51 ulp of a/b. It can round the wrong way only with a midpoint that
//   close, which is half or three halves of an ulp from q; three halves need a
//   y, and so the mantissas of a and b, above 1.985. Such quotients go to the
//   library; without that, 28 of 8 million operands built to lie next to a
//   midpoint came out an ulp off. The test costs the reference's JKR Newton, four
//   quotients a round, 2.7 % (262,144 spheres, 1489 to 1530 us a call of 8 steps).
// * Reciprocal of the root: one correction from within two ulp misses 1/s only
//   where s m = 2^106 - 1 for a 54-bit m, that is for s = 2 - 2^-52 and its
//   multiples by powers of two, which go to the library.
// tests/test_gpu_arithmetic.py tries the operands next to the midpoints.
__device__ __forceinline__ bool exponent_in(double x, uint32_t lo, uint32_t hi) {
  return (uint32_t)__double2hiint(x) - lo < hi - lo;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rcp_step(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// sqrt(x) and 1/sqrt(x) to an ulp (2^-766 <= x < 2^767; not checked)
__device__ __forceinline__ double sqrt_step(double x, double& inv) {
  const double y = rsqrt_seed(x);
  const double r = x * y;
  const double e = fma(-r, y, 1.0);
  const double q = e * fma(e, 0.375, 0.5);
  inv = fma(y, q, y);
  const double s = fma(r, q, r);
  const double half_inv = __hiloint2double(__double2hiint(inv) - 0x00100000, __double2loint(inv));
  return fma(fma(-s, s, x), half_inv, s);
}
constexpr uint32_t EXP_LO = 0x10100000u, EXP_HI = 0x6FE00000u;      // 2^-766 .. 2^767
constexpr uint32_t QUOT_LO = 0x30000000u, QUOT_HI = 0x4FF00000u;    // 2^-255 .. 2^256
__device__ __forceinline__ double sqrt_rn(double x) {
  if (!exponent_in(x, EXP_LO, EXP_HI)) return sqrt(x);
  double inv;
  return sqrt_step(x, inv);
}
__device__ __forceinline__ float sqrt_rn(float x) { return sqrt(x); }
// sqrt(x) and the rounded 1/sqrt(x) of that rounded root
__device__ __forceinline__ double sqrt_rn(double x, double& inv) {
  // (the roots that round to s = 2 - 2^-52 are those of the last two x below a power of four)
  if (!exponent_in(x, EXP_LO, EXP_HI) || (uint32_t)__double2loint(x) >= 0xFFFFFFFCu) {
    const double s = sqrt(x);
    inv = 1.0 / s;
    return s;
  }
  double y;
  const double s = sqrt_step(x, y);
  inv = fma(y, fma(-s, y, 1.0), y);
  return s;
}
// Whether the corrected quotient of a and b may lie next to a midpoint (q before
// the correction, r = a - b q): |r| = b ulp(q) / 2 to one unit of the upper word,
// or three times that. (|r| = b ulp(q), an exact quotient missed by one, is common
// where a wall's normal is formed along an axis: taken for a midpoint it cost a
// bed of 1,000 spheres 25.1 -> 27.0 us a step.)
__device__ __forceinline__ bool near_midpoint(double a, double b, double q, double r) {
  const uint32_t hr = (uint32_t)__double2hiint(r) & 0x7FFFFFFFu, hb = (uint32_t)__double2hiint(b) & 0x7FFFFFFFu,
                 ha = (uint32_t)__double2hiint(a), eq = (uint32_t)__double2hiint(q) & 0x7FF00000u;
  return hr - hb - eq + (1076u << 20) + 1u < 3u ||
         ((ha & hb & 0x000FC000u) == 0x000FC000u && (hr & 0x7FF00000u) + (52u << 20) >= (ha & 0x7FF00000u));
}
// a / b, rounded the other way at most next to a midpoint: for physical mode's
// fused law, which has no counterpart to agree with bit for bit
__device__ __forceinline__ double div_near(double a, double b) {
  if (!(exponent_in(fabs(a), QUOT_LO, QUOT_HI) && exponent_in(fabs(b), QUOT_LO, QUOT_HI))) return a / b;
  const double y = rcp_step(b);
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ double div_rn(double a, double b) {
  if (!(exponent_in(fabs(a), QUOT_LO, QUOT_HI) && exponent_in(fabs(b), QUOT_LO, QUOT_HI))) return a / b;
  const double y = rcp_step(b);
  const double q = a * y;
  const double r = fma(-b, q, a);
  if (near_midpoint(a, b, q, r)) return a / b;
  return fma(r, y, q);
}
__device__ __forceinline__ float div_rn(float a, float b) { return a / b; }
// a / b for each component (b > 0), the divisor's reciprocal formed once. A
// plane's normal along an axis leaves zeros: they are their own quotients.
__device__ __forceinline__ V div_rn(V a, double b) {
  const bool zx = is_zero(a.x), zy = is_zero(a.y), zz = is_zero(a.z);
  if (!((zx || exponent_in(fabs(a.x), QUOT_LO, QUOT_HI)) && (zy || exponent_in(fabs(a.y), QUOT_LO, QUOT_HI)) &&
        (zz || exponent_in(fabs(a.z), QUOT_LO, QUOT_HI)) && exponent_in(b, QUOT_LO, QUOT_HI)))
    return a / b;
  const double y = rcp_step(b);
  const V q = vmk(a.x * y, a.y * y, a.z * y);
  const V r = vmk(fma(-b, q.x, a.x), fma(-b, q.y, a.y), fma(-b, q.z, a.z));
  if (near_midpoint(a.x, b, q.x, r.x) || near_midpoint(a.y, b, q.y, r.y) || near_midpoint(a.z, b, q.z, r.z)) return a / b;
  return vmk(zx ? a.x : fma(r.x, y, q.x), zy ? a.y : fma(r.y, y, q.y), zz ? a.z : fma(r.z, y, q.z));
}
// Comparisons of FP64 values as integers, off the FP64 pipe (a comparison
// there costs as much as an addition): the bits of non-negative values order
// as the values do.
// max(x, 0), 0 for NaN (as fmax)
__device__ __forceinline__ double relu(double x) {
  const long long b = __double_as_longlong(x);
  return b > 0 && b <= 0x7FF0000000000000ll ? x : 0.0;
}
__device__ __forceinline__ float relu(float x) { return fmax(x, 0.0f); }
// a < b for a >= 0 or NaN (false, whichever its sign: inf - inf has it set) and
// b >= 0. As unsigned words, a NaN of either sign lies above infinity.
__device__ __forceinline__ bool less_nn(double a, double b) {
  return (unsigned long long)__double_as_longlong(a) < (unsigned long long)__double_as_longlong(b);
}
__device__ __forceinline__ bool less_nn(float a, float b) { return a < b; }
// x <= 0 (false for NaN)
__device__ __forceinline__ bool not_positive(double x) {
  const long long b = __double_as_longlong(x);
  return b <= 0 && (unsigned long long)b <= 0xFFF0000000000000ull;
}
__device__ __forceinline__ bool not_positive(float x) { return x <= 0.0f; }
// whether an overlap exceeds 0.2 min(r_i, r_j); below an eighth of both radii
// the exponents decide it
__device__ __forceinline__ bool is_excess(double overlap, double ri, double rj) {
  if (__double2hiint(overlap) + 0x00300000 < min(__double2hiint(ri), __double2hiint(rj))) return false;
  return overlap > 0.2 * fmin(ri, rj);
}
__device__ __forceinline__ bool is_excess(float overlap, float ri, float rj) { return overlap > 0.2f * fmin(ri, rj); }
__device__ __forceinline__ double dot_fma(V a, V b) { return fma(a.z, b.z, fma(a.y, b.y, a.x * b.x)); }
// a x b, each component one product and one fused multiply-add
__device__ __forceinline__ V cross_fma(V a, V b) {
  return V{fma(a.y, b.z, -(b.y * a.z)), fma(a.z, b.x, -(b.z * a.x)), fma(a.x, b.y, -(b.x * a.y))};
}
__device__ __forceinline__ V mad(double s, V a, V b) { return V{fma(s, a.x, b.x), fma(s, a.y, b.y), fma(s, a.z, b.z)}; }

// double -> float, rounded to nearest even, on the integer pipe, for every input. A conversion
// instruction runs on the FP64 pipe, and takes it as long where a predicate
// turns it off: leaving the rare inputs to one saved nothing. The mixed pair law
// narrows 13 values a contact (58 FP64-pipe instructions with conversions),
// the integrator 3 a particle: the pair kernel of a million-sphere hopper 196 to
// 171 us, its mixed step 395 to 372, the FP64 step 629 to 623, a gas of a million
// 259 to 254, a mixed drum of 4.2 million 1346 to 1253.
__device__ __forceinline__ uint32_t d2f_odd(uint32_t hi, uint32_t lo) {
  const uint32_t e = hi & 0x7FFFFFFFu;
  if (e >= 0x47F00000u)  // 2^128 and above, infinity, NaN
    return e > 0x7FF00000u || (e == 0x7FF00000u && lo != 0u) ? 0x7FFFFFFFu : 0x7F800000u;
  const uint32_t down = 926u - (e >> 20);  // bits below the unit 2^-149
  if (down > 54u) return 0u;
  const unsigned long long m = ((unsigned long long)((e & 0x000FFFFFu) | 0x00100000u) << 32) | lo;
  return (uint32_t)((m + ((1ull << (down - 1u)) - 1ull) + ((m >> down) & 1ull)) >> down);
}
template <typename R> __device__ __forceinline__ R narrow(double x) { return x; }
__device__ __forceinline__ float d2f_exact(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x), e = hi & 0x7FFFFFFFu;
  const uint32_t f = ((e - 0x38000000u) << 3) | (lo >> 29);
  uint32_t r = f + (((lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (f & 1u)) >> 29);
  if (e - 0x38100000u >= 0x47F00000u - 0x38100000u) r = d2f_odd(hi, lo);
  return __uint_as_float(r | (hi & 0x80000000u));
}
template <> __device__ __forceinline__ float narrow<float>(double x) { return d2f_exact(x); }
template <typename R> __device__ __forceinline__ T3<R> narrow(V a) { return T3<R>{narrow<R>(a.x), narrow<R>(a.y), narrow<R>(a.z)}; }

}  // namespace rp
