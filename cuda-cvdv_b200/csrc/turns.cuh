// Phases counted in turns, reduced mod 1 before their sine and cosine.
//
// A phase of c x with x = dx u / 2 (u = 2 n - N + 1, dx^2 = 2 pi / N) is c lin_turns(N) u
// turns, one of c x^2 is c u^2 / (4 N), and a transform twiddle is a fraction of 4 N.  A
// product q m is reduced exactly where its rounding is kept (LOW) and q has two words: in one
// word the constant's rounding grows with the angle (a displacement by 0.7 - 0.4i of random
// amplitudes on 2^11 points, relative error 6.2e-15 -> 0.9e-15).  Complex64 needs no low word:
// its amplitudes round to 6e-8.
//
// A sum of phases in one word rounds to 2^-54 turns (3.5e-16 radians), which a thread's running
// product repeats once a step: Turns1 serves tables and runs of 8 points in batches, Turns2
// keeps the sum's rounding too, for programs and longer runs in complex128 (a displacement by
// 5.3 - 4.7i on 2^13 points 4.3e-15 with Turns1, below 3.7e-15 with Turns2; one by 0.7 - 0.4i in a
// batch of 2^8-point rows 2.0e-15 and 0.7e-15).  On runs of 8 Turns2 gains little (0.5e-15)
// and costs a small batch 8 % of its time (5 circuits of 19 gates 362 us against 333).
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

// A coefficient times a two-word constant, in two words.
struct TurnRate {
  double hi, lo;
};
__device__ __forceinline__ TurnRate turn_rate(double a, double ch, double cl) {
  const double h = a * ch;
  return {h, fma(a, cl, fma(a, ch, -h))};
}

__device__ __forceinline__ double2 turn_root(double v) {
  double s, c;
  sincospi(2.0 * v, &s, &c);
  return make_double2(c, s);
}

template <bool LOW>
struct Turns1 {
  double v;
  __device__ __forceinline__ explicit Turns1(double r = 0.0) : v(r) {}
  __device__ __forceinline__ void add(TurnRate q, double m) {  // q m turns; m an integer that a double holds
    if constexpr (LOW) {
      const double p = q.hi * m;  // (p - rint(p) is exact)
      const double s = v + ((p - rint(p)) + fma(q.lo, m, fma(q.hi, m, -p)));
      v = s - rint(s);
    } else {
      v += fma(q.hi, m, -rint(q.hi * m));
    }
  }
  __device__ __forceinline__ Turns1 times(double n) const { return Turns1(n * v); }
  __device__ __forceinline__ double2 root() const { return turn_root(v); }
};

struct Turns2 {
  double hi, lo;
  __device__ __forceinline__ explicit Turns2(double r = 0.0) : hi(r), lo(0.0) {}  // r in -1/2 .. 1/2
  __device__ __forceinline__ void add(TurnRate q, double m) {
    const double p = q.hi * m, r = p - rint(p);
    const double s = hi + r, b = s - hi;
    lo += (hi - (s - b)) + (r - b);
    lo += fma(q.lo, m, fma(q.hi, m, -p));
    hi = s - rint(s);
  }
  __device__ __forceinline__ Turns2 times(double n) const {  // n a small power of two
    Turns2 t(n * hi);
    t.hi -= rint(t.hi);
    t.lo = n * lo;
    return t;
  }
  __device__ __forceinline__ double2 root() const {
    const double h = hi + lo, l = lo - (h - hi);
    // (a low word that is still no rounding belongs to 2^53 turns and more: no digit of
    // the angle is left, and the first-order step would change the modulus)
    const double d = fabs(l) < 1e-8 ? 2.0 * CVDV_PI * l : 0.0;
    const double2 w = turn_root(h - rint(h));
    return make_double2(fma(-d, w.y, w.x), fma(d, w.x, w.y));
  }
};

}  // namespace cvdv
