// v3's phase functions (csrc/phase.cuh) on the host: stand-ins for the device's
// intrinsics, and their errors against arithmetic of 113 bits.
#include <algorithm>
#include <cmath>
#include <cstring>

#ifdef __x86_64__
#include <quadmath.h>
typedef __float128 Q;
static Q qcos(Q a) { return cosq(a); }
static Q qsin(Q a) { return sinq(a); }
static Q qatan2(Q y, Q x) { return atan2q(y, x); }
static Q qsqrt(Q a) { return sqrtq(a); }
#else  // aarch64: long double has 113 bits
typedef long double Q;
static Q qcos(Q a) { return cosl(a); }
static Q qsin(Q a) { return sinl(a); }
static Q qatan2(Q y, Q x) { return atan2l(y, x); }
static Q qsqrt(Q a) { return sqrtl(a); }
#endif

#define __device__
#define __forceinline__ inline
struct double2 {
  double x, y;
};
static double2 make_double2(double x, double y) { return {x, y}; }
static unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
static double __longlong_as_double(long long a) {
  double d;
  memcpy(&d, &a, 8);
  return d;
}
static long long __double_as_longlong(double a) {
  long long d;
  memcpy(&d, &a, 8);
  return d;
}
static int __double2hiint(double a) { return (int)(__double_as_longlong(a) >> 32); }
static long long __double2ll_rn(double a) { return llrint(a); }
static int __float2int_rn(float a) { return (int)lrintf(a); }
static double __dadd_rn(double a, double b) { return a + b; }
static float rsqrtf(float a) { return 1.0f / sqrtf(a); }
using std::fma;
using std::max;

#include "phase.cuh"

namespace {

double2 table[1 << sfft::TRIG_BITS];
const Q TURN = 2 * (Q)3.141592653589793115997963468544185161590576171875 + 2 * (Q)1.2246467991473531772e-16;

double apart(Q a, Q b) { return fabs((double)(a - b)); }
double apart(double2 c, Q a) { return std::max(apart(qcos(a), c.x), apart(qsin(a), c.y)); }

}  // namespace

extern "C" {

// (cos, sin)(2 pi i / 1024), rounded to doubles
void phase_table() {
  for (int i = 0; i < 1 << sfft::TRIG_BITS; i++) {
    const int o = i >> 7, k = i & 127, j = o & 1 ? 128 - k : k;  // within an octant
    const Q a = TURN * j / 1024;
    const double c = (double)qcos(a), s = (double)qsin(a);
    const bool swap = !(o == 0 || o == 7 || o == 3 || o == 4);
    table[i] = make_double2((o >= 2 && o < 6 ? -1 : 1) * (swap ? s : c), (o >= 4 ? -1 : 1) * (swap ? c : s));
  }
}

double phase_cis(double a) { return apart(sfft::cis(table, a), (Q)a); }
double phase_step(double a, int k, double b) { return apart(sfft::cis_step(table, a, k, b), (Q)a + (Q)k * b); }
void phase_step_value(double a, int k, double b, double *re, double *im) {
  const double2 c = sfft::cis_step(table, a, k, b);
  *re = c.x;
  *im = c.y;
}
double phase_angle(double y, double x) {
  const double e = apart(qatan2(y, x), sfft::angle_of(table, y, x));
  return std::min(e, fabs(e - (double)TURN));  // -pi and pi are one angle
}
double phase_sqrt(double a) { return (double)fabs((double)(sfft::sqrt_of(a) / qsqrt(a) - 1)); }
double phase_recip(double a) { return (double)fabs((double)((Q)sfft::recip_of(a) * a - 1)); }

}  // extern "C"
