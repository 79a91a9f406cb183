// Cells of the wave-cell expansion (fj_expand.cu): which cell a station lies
// in at a frequency, and where in it. Host and device code, so that a CPU test
// can run the kernels' own rule (tests/cell_rule_check.cpp).
//
// x = r f / hu (hu: a cell's length in u = r f). Cells of the J basis are
// [i, i + 1). DY (the Y basis is asked for): the cells below x = 1 are
// [2^(i-24), 2^(i-23)), the others follow.
#pragma once

#include <math.h>
#include <string.h>

#if defined(__CUDACC__)
#define XP_HD __host__ __device__ __forceinline__
#else
#define XP_HD inline
#endif

namespace ccfj {
namespace xp {

// Intervals up to this share of a cell are short: whole in the cell of their
// far end. A cell's polynomials live on [-kShort, 1] of it; the middle of that
// is kCentre, and t = (x - middle) kPerHalf.
constexpr float kShort = 0.0625f;
constexpr float kCentre = 0.46875f;
constexpr float kPerHalf = 1.8823529f;
constexpr double kCellPhase = 9.8;  // radians of a cell at the slowest velocity
constexpr int kDyadic = 24;         // halved cells below the first (Y basis)

XP_HD int float_bits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_int(x);
#else
  int i;
  memcpy(&i, &x, sizeof(i));
  return i;
#endif
}
XP_HD float bits_float(int i) {
#if defined(__CUDA_ARCH__)
  return __int_as_float(i);
#else
  float x;
  memcpy(&x, &i, sizeof(x));
  return x;
#endif
}

// x as a double-float product of r and fx = f / hu (not fused into what
// follows: every kernel forms the same fx and the same x).
struct Fx {
  float hi, lo;
};
XP_HD Fx make_fx(float f, double inv_hu) {
#if defined(__CUDA_ARCH__)
  const double v = __dmul_rn((double)f, inv_hu);
#else
  const double v = (double)f * inv_hu;
#endif
  Fx x;
  x.hi = (float)v;
  x.lo = (float)(v - (double)x.hi);
  return x;
}

// x = p + l: l holds p's rounding (up to half a spacing of p) and r fx.lo (up
// to one more), so it can carry x across an integer in either direction.
struct Place {
  float p, l;
};
XP_HD Place place_of(float r, Fx fx) {
  Place x;
#if defined(__CUDA_ARCH__)
  x.p = __fmul_rn(r, fx.hi);
#else
  x.p = r * fx.hi;
#endif
  x.l = fmaf(r, fx.lo, fmaf(r, fx.hi, -x.p));
  return x;
}

// The one rule of the cells: x has reached `end`.
XP_HD bool reached(Place x, float end) { return (x.p - end) + x.l >= 0.0f; }

// The cell that holds x, and x's place in it from kCentre (so that its
// rounding is smallest, -kCentre .. 1 - kCentre). The cell never decreases
// with r, and is the one that a walk over the cells by reached() ends in: the
// moments of a chunk of stations are found by such a walk, the cells that its
// neighbours share with it by this function.
template <bool DY>
XP_HD int locate(float r, Fx fx, float& v) {
  const Place x = place_of(r, fx);
  float c = floorf(x.p);
  if (!reached(x, c))
    c -= 1.0f;
  else if (reached(x, c + 1.0f))
    c += 1.0f;
  if (!DY || c >= 1.0f) {
    v = (x.p - (c + kCentre)) + x.l;
    return (int)c + (DY ? kDyadic - 1 : 0);
  }
  // x < 1: [len, 2 len) with len the power of two at or below x
  float len = bits_float(float_bits(x.p) & 0x7f800000);
  if (x.p >= 1.0f) len = 0.5f;  // x just below 1
  if (!reached(x, len)) len *= 0.5f;
  v = ((x.p - len * (1.0f + kCentre)) + x.l) / len;
  const int e = (float_bits(len) >> 23) - 127;  // -24 .. -1
  return e + kDyadic > 0 ? e + kDyadic : 0;
}
template <bool DY>
XP_HD float cell_len(int cell) {
  return DY && cell < kDyadic ? bits_float((cell - kDyadic + 127) << 23) : 1.0f;
}
template <bool DY>
XP_HD float cell_begin(int cell) {
  if (!DY) return (float)cell;
  return cell < kDyadic ? cell_len<DY>(cell) : (float)(cell - kDyadic + 1);
}

}  // namespace xp
}  // namespace ccfj
