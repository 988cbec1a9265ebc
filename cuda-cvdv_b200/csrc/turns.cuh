// Phases counted in turns, reduced mod 1 before their sine and cosine.
//
// A phase of c x with x = dx u / 2 (u = 2 n - N + 1, dx^2 = 2 pi / N) is c lin_turns(N) u
// turns, one of c x^2 is c u^2 / (4 N), and a transform twiddle is a fraction of 4 N.  In
// complex128 a sum of them is kept in two words: the products' low halves, the sum's
// rounding and the constant's second word, which a last first-order step adds to the sine
// and cosine.  In one word the sum's rounding (up to 2^-54 turns, 3.5e-16 radians) comes
// back up to 31 times where a thread's running product repeats a step, and the constant's
// grows with the angle.  Relative error of a displacement by 0.7 - 0.4i of random amplitudes,
// one word -> two: 6.2e-15 -> 0.9e-15 on 2^11 points, 1.2e-14 -> 0.7e-15 on 2^13.  Complex64
// keeps one word: its amplitudes round to 6e-8.
#pragma once

#include "cvdv_internal.cuh"

namespace cvdv {

// Turns of the phase x per unit of u on 2^logN points, 1 / (2 sqrt(2 pi N)), as hi + lo.
struct LinTurns {
  double hi, lo;
};
__host__ __device__ constexpr LinTurns lin_turns(int logN) {
  LinTurns t = (logN & 1) ? LinTurns{0.14104739588693907, 1.916932451645735e-18}
                          : LinTurns{0.19947114020071635, -1.246163601138865e-17};
  for (int k = 0; k < logN / 2; ++k) t = LinTurns{0.5 * t.hi, 0.5 * t.lo};
  return t;
}

template <typename C>
struct Turns;

template <>
struct Turns<double2> {
  double hi = 0.0, lo = 0.0;  // hi in -1/2 .. 1/2
  // q m turns, q = (qh, ql); m an integer that a double holds
  __device__ __forceinline__ void add(double qh, double ql, double m) {
    const double p = qh * m, r = p - rint(p);  // (the difference is exact)
    add_hi(r);
    lo += fma(ql, m, fma(qh, m, -p));
  }
  __device__ __forceinline__ void add_hi(double r) {  // r in -1/2 .. 1/2
    const double s = hi + r, b = s - hi;
    lo += (hi - (s - b)) + (r - b);
    hi = s - rint(s);
  }
  // a coefficient times a two-word constant
  static __device__ __forceinline__ void scale(double a, double ch, double cl, double& qh, double& ql) {
    qh = a * ch;
    ql = fma(a, cl, fma(a, ch, -qh));
  }
  __device__ __forceinline__ Turns times(double n) const {  // n a small power of two
    Turns t;
    t.hi = n * hi;
    t.hi -= rint(t.hi);
    t.lo = n * lo;
    return t;
  }
  __device__ __forceinline__ double2 root() const {
    const double h = hi + lo, l = lo - (h - hi);
    // (a low word that is still no rounding belongs to 2^53 turns and more: no digit of
    // the angle is left, and the first-order step would change the modulus)
    const double d = fabs(l) < 1e-8 ? 2.0 * CVDV_PI * l : 0.0;
    double s, c;
    sincospi(2.0 * (h - rint(h)), &s, &c);
    return make_double2(fma(-d, s, c), fma(d, c, s));
  }
};

template <>
struct Turns<float2> {
  double v = 0.0;
  __device__ __forceinline__ void add(double qh, double, double m) { v += fma(qh, m, -rint(qh * m)); }
  __device__ __forceinline__ void add_hi(double r) { v += r; }
  static __device__ __forceinline__ void scale(double a, double ch, double, double& qh, double& ql) {
    qh = a * ch;
    ql = 0.0;
  }
  __device__ __forceinline__ Turns times(double n) const {
    Turns t;
    t.v = n * v;
    return t;
  }
  __device__ __forceinline__ double2 root() const {
    double s, c;
    sincospi(2.0 * v, &s, &c);
    return make_double2(c, s);
  }
};

}  // namespace cvdv
