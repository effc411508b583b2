// phase.cuh — v3's phases, angles, square roots and reciprocals in few FP64
// instructions.  Plain functions of their arguments (the host tests compile
// them with stand-ins for the intrinsics), to be built without multiply-add
// contraction.
#pragma once

namespace sfft {

// ----------------------------------------------------------------- phases --
//
// cos and sin of an angle held as a fraction of a turn in 64-bit fixed point,
// and the fraction of a double angle of any size (M. Payne and R. Hanek,
// "Radian reduction for trigonometric functions", SIGNUM Newsletter 18,
// 1983): the angle's mantissa times a 128-bit window of 1 / (2 pi), in integer
// arithmetic, of which the fraction's top 64 bits are kept.  The fraction's
// nearest 1024th of a turn comes from a table, the rest (under 0.0031 rad)
// from the Taylor terms that reach 1e-17.  13 FP64 instructions against more
// than 40 in sincos (and its slow path beyond 1e5 rad, which the comb's phase
// arguments of up to 2 pi n take); the arguments' own rounding, which the
// reference's results contain, is untouched.  Largest error against 113-bit
// arithmetic over 10^6 arguments of 1e-3 to 1e15 rad: 1.13e-16 (a correctly
// rounded value: 0.56e-16; CUDA states 2 units in the last place, 2.2e-16).

constexpr int TRIG_BITS = 10;  // V3Dev::trig: (cos, sin)(2 pi i / 1024)

__device__ __forceinline__ double2 cis_turn(const double2 *trig, unsigned long long fr) {
  const unsigned long long up = fr + (1ull << (63 - TRIG_BITS));
  const double2 t = trig[(int)(up >> (64 - TRIG_BITS))];
  // the rest, in (-2^53, 2^53] units of 2^-64 turn; as a double through the mantissa of 1.5 2^52
  const long long rest = (long long)(fr - (up & ~((1ull << (64 - TRIG_BITS)) - 1)));
  const double x =
      __dadd_rn(__longlong_as_double(0x4338000000000000ll + (rest >> 2)), -6755399441055744.0) * 1.3624486320346218e-18;
  const double s = x * x;
  const double sn = fma(x * s, fma(s, 1.0 / 120, -1.0 / 6), x);  // sin x
  const double cm = s * fma(s, 1.0 / 24, -0.5);                  // cos x - 1
  return make_double2(t.x + fma(t.x, cm, -(t.y * sn)), t.y + fma(t.y, cm, t.x * sn));
}

// The fraction of a turn of `a` radians (|a| < 2^110).
__device__ __forceinline__ unsigned long long turn_of(double a) {
  constexpr unsigned long long R0 = 0x28be60db9391054aull, R1 = 0x7f09d5f47d4d3770ull, R2 = 0x36d8a5664f10e410ull;  // 1 / (2 pi)
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  const int ex = (int)((b >> 52) & 0x7ff);
  const unsigned long long M = (b & 0xfffffffffffffull) | (1ull << 52);
  const int e = ex - 1075;  // |a| = M 2^e
  unsigned long long hi, lo;
  if (e > 0) {
    hi = e < 64 ? (R0 << e) | (R1 >> (64 - e)) : R1 << (e - 64);
    lo = e < 64 ? (R1 << e) | (R2 >> (64 - e)) : R2 << (e - 64);
  } else if (e > -64) {
    hi = R0 >> -e;
    lo = e ? (R1 >> -e) | (R0 << (64 + e)) : R1;
  } else {
    hi = 0;
    lo = e > -128 ? R0 >> (-e - 64) : 0;
  }
  const unsigned long long fr = __umul64hi(M, lo) + M * hi;
  return (long long)b < 0 ? 0ull - fr : fr;
}

__device__ __forceinline__ double2 cis(const double2 *trig, double a) { return cis_turn(trig, turn_of(a)); }

// e^{i (a + k b)}, the angle not rounded to a double in between.
__device__ __forceinline__ double2 cis_step(const double2 *trig, double a, int k, double b) {
  const double kd = (double)k, hi = kd * b, lo = fma(kd, b, -hi);
  const unsigned long long fr = turn_of(a) + turn_of(hi) + (unsigned long long)__double2ll_rn(lo * 2935890503282001226.0);
  return cis_turn(trig, fr);
}

// atan2(y, x).  An FP32 arctangent names the nearest 1024th of a turn, the
// vector is turned back by it (table), and the remaining angle, under 0.0035
// rad, is the series of its tangent; the quotient's FP32 reciprocal is
// corrected to FP64.  About 20 FP64 instructions; largest error over 10^6
// vectors 3.3e-16 rad (half a unit in the last place of pi is 2.2e-16).
// Magnitudes outside 2^+-60 take the library function.
__device__ __forceinline__ double angle_of(const double2 *trig, double y, double x) {
  const int ey = (__double2hiint(y) >> 20) & 0x7ff, exx = (__double2hiint(x) >> 20) & 0x7ff, m = max(ey, exx);
  if (m < 1023 - 60 || m > 1023 + 60) return atan2(y, x);
  const float af = atan2f((float)y, (float)x);
  const int k = __float2int_rn(af * 162.97466172610083f);  // 1024 / (2 pi)
  const double2 t = trig[k & 1023];
  const double u = fma(x, t.x, y * t.y), v = fma(y, t.x, -(x * t.y));
  const double r = (double)(1.0f / (float)u);
  const double q0 = v * r, q = fma(fma(-q0, u, v), r, q0);
  const double s = q * q, d = fma(q * s, fma(s, 0.2, -1.0 / 3), q);
  const double kd = (double)k;
  return fma(kd, 0.006135923151542565, fma(kd, 2.391888279584674e-19, d));
}

// sqrt(a) and 1 / a for positive a of 2^+-60, from FP32 seeds by Newton steps
// with exact FMA remainders (8 and 6 FP64 instructions); the library's beyond.
__device__ __forceinline__ bool seedable(double a) {
  const int e = __double2hiint(a) >> 20;
  return e > 1023 - 60 && e < 1023 + 60;
}
__device__ __forceinline__ double sqrt_of(double a) {
  if (!seedable(a)) return sqrt(a);
  const double y = (double)rsqrtf((float)a);
  double g = a * y, h = 0.5 * y;
  const double e = fma(-g, h, 0.5);
  g = fma(g, e, g);
  h = fma(h, e, h);
  return fma(fma(-g, g, a), h, g);
}
__device__ __forceinline__ double recip_of(double a) {
  if (!seedable(a)) return 1. / a;
  const double y = (double)(1.0f / (float)a), r = fma(fma(-a, y, 1.0), y, y);
  return fma(fma(-a, r, 1.0), r, r);
}

}  // namespace sfft
