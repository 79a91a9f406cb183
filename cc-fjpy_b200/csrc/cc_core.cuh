// Arithmetic of the cross-correlation front end (xcorr.cu), written once
// for the device kernels and for host-side checks: every function here
// compiles with nvcc (host and device) and with a plain C++ compiler, where
// the tests drive it thread by thread.
//
// The reference computes, for every station pair, the average over the
// overlapping windows both stations keep of conj(X_a) X_b, where X is the
// (optionally one-bit, optionally whitened) real FFT of a window at bins
// j*fstride (src/CrossCorr.cpp:33-159). Here:
//
// * shift_range: the shifts k a station keeps form one interval [lo, hi]
//   (both tests of src/CrossCorr.cpp:88-95 are monotone in k), so a pair's
//   count is the length of the intersection of two intervals;
// * the real FFT of N = 2M samples is a complex FFT of z[m] = x[2m] +
//   i x[2m+1] (M points, self-sorting Stockham passes of radix 2, 3, 4, 5
//   or 8) followed by the split
//     X[k] = (Z[k] + conj Z[M-k]) / 2 - (i/2) e^{-i pi k/M} (Z[k] - conj Z[M-k]);
// * whiten: X / max(|X|, 1e-8) in float32, as the reference;
// * gram_step: one thread's share of a 16 x 16 station tile of
//   conj(X_a) X_b for one frequency lane.
//
// The device kernel transforms a folded window where it can: with g the
// common divisor of the bins' stride and M, the bins of x at multiples of g
// are all the bins of the 2M/g samples sum_t x[n + 2M t/g].
#pragma once

#include <math.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define CC_HD __host__ __device__ __forceinline__
#else
#define CC_HD inline
#endif

namespace ccfj {
namespace xc {

struct alignas(8) Cpx {
  float re, im;
};

CC_HD Cpx cpx(float re, float im) {
  Cpx c;
  c.re = re;
  c.im = im;
  return c;
}
CC_HD Cpx cadd(Cpx a, Cpx b) { return cpx(a.re + b.re, a.im + b.im); }
CC_HD Cpx csub(Cpx a, Cpx b) { return cpx(a.re - b.re, a.im - b.im); }
CC_HD Cpx cmul(Cpx a, Cpx b) { return cpx(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re); }
CC_HD Cpx cscale(Cpx a, float s) { return cpx(a.re * s, a.im * s); }
// -i * a
CC_HD Cpx cmul_negi(Cpx a) { return cpx(a.im, -a.re); }
CC_HD Cpx cconj(Cpx a) { return cpx(a.re, -a.im); }

// ------------------------------------------------------------ small DFTs
// Forward DFT of R points in place, natural order:
// X[q] = sum_r v[r] exp(-2 pi i r q / R).
template <int R>
CC_HD void dft(Cpx* v);

template <>
CC_HD void dft<2>(Cpx* v) {
  const Cpx a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

template <>
CC_HD void dft<4>(Cpx* v) {
  const Cpx t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
  const Cpx t2 = cadd(v[1], v[3]), t3 = cmul_negi(csub(v[1], v[3]));
  v[0] = cadd(t0, t2);
  v[2] = csub(t0, t2);
  v[1] = cadd(t1, t3);
  v[3] = csub(t1, t3);
}

template <>
CC_HD void dft<8>(Cpx* v) {
  // even and odd halves, then X[q] = E[q] + W8^q O[q], X[q+4] = E[q] - W8^q O[q]
  Cpx e[4] = {v[0], v[2], v[4], v[6]};
  Cpx o[4] = {v[1], v[3], v[5], v[7]};
  dft<4>(e);
  dft<4>(o);
  const float h = 0.70710678118654752f;  // 1/sqrt(2)
  const Cpx w1 = cmul(o[1], cpx(h, -h));
  const Cpx w2 = cmul_negi(o[2]);
  const Cpx w3 = cmul(o[3], cpx(-h, -h));
  v[0] = cadd(e[0], o[0]);
  v[4] = csub(e[0], o[0]);
  v[1] = cadd(e[1], w1);
  v[5] = csub(e[1], w1);
  v[2] = cadd(e[2], w2);
  v[6] = csub(e[2], w2);
  v[3] = cadd(e[3], w3);
  v[7] = csub(e[3], w3);
}

template <>
CC_HD void dft<3>(Cpx* v) {
  // w = exp(-2 pi i / 3) = -1/2 - i sqrt(3)/2
  const float s3 = 0.86602540378443865f;
  const Cpx s = cadd(v[1], v[2]);
  const Cpx d = cscale(cmul_negi(csub(v[1], v[2])), s3);
  const Cpx m = csub(v[0], cscale(s, 0.5f));
  v[0] = cadd(v[0], s);
  v[1] = cadd(m, d);
  v[2] = csub(m, d);
}

template <>
CC_HD void dft<5>(Cpx* v) {
  // cos and sin of 2 pi / 5 and 4 pi / 5
  const float c1 = 0.30901699437494742f, s1 = 0.95105651629515357f;
  const float c2 = -0.80901699437494742f, s2 = 0.58778525229247313f;
  const Cpx s14 = cadd(v[1], v[4]), d14 = csub(v[1], v[4]);
  const Cpx s23 = cadd(v[2], v[3]), d23 = csub(v[2], v[3]);
  const Cpx x0 = v[0];
  const Cpx m1 = cadd(x0, cadd(cscale(s14, c1), cscale(s23, c2)));
  const Cpx m2 = cadd(x0, cadd(cscale(s14, c2), cscale(s23, c1)));
  const Cpx n1 = cmul_negi(cadd(cscale(d14, s1), cscale(d23, s2)));
  const Cpx n2 = cmul_negi(csub(cscale(d14, s2), cscale(d23, s1)));
  v[0] = cadd(x0, cadd(s14, s23));
  v[1] = cadd(m1, n1);
  v[4] = csub(m1, n1);
  v[2] = cadd(m2, n2);
  v[3] = csub(m2, n2);
}

// ------------------------------------------------------ Stockham passes
// One pass of radix R over M points, done by butterflies t = 0 .. M/R - 1
// after Ns points have been combined (Ns = product of the earlier radices).
// Butterfly t reads src[t + r M/R], twiddles input r by
// exp(-2 pi i (t mod Ns) r / (Ns R)) = tw[(t mod Ns) r M / (Ns R)], with
// tw[u] = exp(-2 pi i u / M), and writes dst[(t / Ns) Ns R + t mod Ns + q Ns].
// After the last pass (Ns R = M) dst holds the DFT in natural order. The
// load and the rest are separate so that a caller can run the pass in place
// (every load before any store).
// src and dst are pointers or anything that indexes like one (the device
// kernel's skewed shared array).
template <int R, class Src>
CC_HD void bf_load(Src src, int M, int t, Cpx* v) {
  const int stride = M / R;
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = src[t + r * stride];
}

// The twiddles w[r] = w[1]^r of a butterfly, 0 < r < R, from the powers that a
// table holds: 1, 2 and (radix 8) 4; the others as products of those (one or
// two products deep).
template <int R>
CC_HD void twiddle_powers(Cpx* w) {
  if (R >= 4) w[3 % R] = cmul(w[1], w[2 % R]);
  if (R == 5) w[4 % R] = cmul(w[2 % R], w[2 % R]);
  if (R == 8) {
    w[5 % R] = cmul(w[4 % R], w[1]);
    w[6 % R] = cmul(w[4 % R], w[2 % R]);
    w[7 % R] = cmul(w[4 % R], w[3 % R]);
  }
}

// Powers that the table of a pass holds
CC_HD constexpr int twiddle_rows(int R) { return R == 8 ? 3 : R >= 3 ? 2 : 1; }

// Butterfly t = tq Ns + jn with its twiddles (unread for jn = 0)
template <int R, class Dst>
CC_HD void bf_twiddled(Dst dst, int Ns, int tq, int jn, const Cpx* w, Cpx* v) {
  if (jn != 0) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], w[r]);
  }
  dft<R>(v);
  const int base = tq * Ns * R + jn;
#pragma unroll
  for (int r = 0; r < R; ++r) dst[base + r * Ns] = v[r];
}

// From the pass's own table, whose row i holds the powers 2^i of its Ns
// twiddles: neighbouring butterflies read neighbouring entries.
template <int R, class Dst>
CC_HD void bf_rows(Dst dst, int Ns, int tq, int jn, const Cpx* rows, Cpx* v) {
  Cpx w[R];
  if (jn != 0) {
#pragma unroll
    for (int i = 0; i < twiddle_rows(R); ++i) w[1 << i] = rows[i * Ns + jn];
    twiddle_powers<R>(w);
  }
  bf_twiddled<R>(dst, Ns, tq, jn, w, v);
}

// The same from the one table tw[u] = exp(-2 pi i u / M) of every pass (the host
// replay's form)
template <int R>
CC_HD void bf_finish(Cpx* dst, int M, int Ns, const Cpx* tw, int t, Cpx* v) {
  const int jn = t % Ns;
  const int step = (M / (Ns * R)) * jn;
  Cpx w[R];
  if (jn != 0) {
    for (int i = 0; i < twiddle_rows(R); ++i) w[1 << i] = tw[step << i];
    twiddle_powers<R>(w);
  }
  bf_twiddled<R>(dst, Ns, t / Ns, jn, w, v);
}

// Radices of a self-sorting plan for M points: 8s, then a 4 or 2, then 3s
// and 5s. Returns the number of passes, or 0 when M has another prime
// factor (or needs more than kMaxPasses passes).
constexpr int kMaxPasses = 24;
CC_HD int fft_plan(int M, int* radix) {
  if (M < 2) return 0;
  int n = 0;
  while (M % 8 == 0 && n < kMaxPasses) {
    radix[n++] = 8;
    M /= 8;
  }
  if (M % 4 == 0 && n < kMaxPasses) {
    radix[n++] = 4;
    M /= 4;
  }
  if (M % 2 == 0 && n < kMaxPasses) {
    radix[n++] = 2;
    M /= 2;
  }
  while (M % 3 == 0 && n < kMaxPasses) {
    radix[n++] = 3;
    M /= 3;
  }
  while (M % 5 == 0 && n < kMaxPasses) {
    radix[n++] = 5;
    M /= 5;
  }
  return M == 1 ? n : 0;
}

// Bin k (0 <= k <= M) of the real FFT of 2M samples from the complex FFT Z
// of z[m] = x[2m] + i x[2m+1]; wk = exp(-i pi k / M).
template <class Src>
CC_HD Cpx real_bin(Src Z, int M, int k, Cpx wk) {
  const Cpx a = Z[k == M ? 0 : k];
  const Cpx b = cconj(Z[k == 0 ? 0 : M - k]);
  const Cpx s = cscale(cadd(a, b), 0.5f);
  const Cpx d = cscale(csub(a, b), 0.5f);
  return cadd(s, cmul_negi(cmul(wk, d)));
}

// X / max(|X|, 1e-8) with float32 sqrt and division (src/CrossCorr.cpp:104-110);
// std::max(a, b) is (a < b) ? b : a, so a NaN magnitude stays NaN
CC_HD Cpx whiten(Cpx x) {
  float a = sqrtf(x.re * x.re + x.im * x.im);
  a = a < 1e-8f ? 1e-8f : a;
  return cpx(x.re / a, x.im / a);
}

CC_HD float onebit(float x) { return x > 0.f ? 1.f : (x < 0.f ? -1.f : 0.f); }

// ------------------------------------------------------- window geometry
// floor(a / b) and ceil(a / b) for b > 0
CC_HD long long floor_div(long long a, long long b) {
  return a >= 0 ? a / b : -((-a + b - 1) / b);
}
CC_HD long long ceil_div(long long a, long long b) { return -floor_div(-a, b); }

// The shifts k in [0, nshifts) with k*steplen >= start and
// k*steplen + fftlen < end (src/CrossCorr.cpp:88-95), as [*lo, *hi];
// empty when *lo > *hi. steplen > 0 unless nshifts == 1.
CC_HD void shift_range(long long nshifts, long long steplen, long long fftlen, long long start,
                       long long end, long long* lo, long long* hi) {
  if (nshifts <= 1) {
    const bool keep = nshifts == 1 && 0 >= start && fftlen < end;
    *lo = 0;
    *hi = keep ? 0 : -1;
    return;
  }
  long long a = start <= 0 ? 0 : ceil_div(start, steplen);
  long long b = floor_div(end - fftlen - 1, steplen);
  if (b > nshifts - 1) b = nshifts - 1;
  *lo = a;
  *hi = b;
}

// Windows both stations keep
CC_HD int pair_count(int lo_a, int hi_a, int lo_b, int hi_b) {
  const int lo = lo_a > lo_b ? lo_a : lo_b;
  const int hi = hi_a < hi_b ? hi_a : hi_b;
  return hi >= lo ? hi - lo + 1 : 0;
}

// --------------------------------------------------------- pair products
// Station tiles of kTile x kTile and kLanes frequencies; a CTA of
// kGramThreads threads: warp w owns tile rows 4w .. 4w+3, lane j frequency
// j of the tile, and every column b. Four rows by sixteen columns read 20
// values of shared memory for 64 products (two rows read 18 for 32).
constexpr int kTile = 16;
constexpr int kLanes = 32;
constexpr int kGramThreads = 128;
constexpr int kRowsPerWarp = kTile / (kGramThreads / 32);  // 4

// acc += conj(a) x, the two halves of each step as a pair: (re, im) gains
// a.re (x.re, x.im), then a.im (x.im, -x.re). On the device a pair is one packed
// instruction of two fused multiply-adds, and the operands are built once for
// the products that share them.
#if defined(__CUDA_ARCH__)
typedef unsigned long long Two;
__device__ __forceinline__ Two two(float lo, float hi) {
  Two v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void fma_two(Cpx& acc, Two p, Two q) {
  Two c = two(acc.re, acc.im);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(p), "l"(q));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(acc.re), "=f"(acc.im) : "l"(c));
}
#else
typedef Cpx Two;
CC_HD Two two(float lo, float hi) { return cpx(lo, hi); }
CC_HD void fma_two(Cpx& acc, Two p, Two q) {
  acc.re += p.re * q.re;
  acc.im += p.im * q.im;
}
#endif

// One shift: xa = the tile's a rows [kTile][kLanes], xb its b rows. halves:
// bit h = columns 8h .. 8h+7 are wanted.
CC_HD void gram_step(const Cpx* xa, const Cpx* xb, int warp, int lane,
                     Cpx (&acc)[kRowsPerWarp][kTile], unsigned halves = 3u) {
  Two re[kRowsPerWarp], im[kRowsPerWarp];
#pragma unroll
  for (int ra = 0; ra < kRowsPerWarp; ++ra) {
    const Cpx a = xa[(warp * kRowsPerWarp + ra) * kLanes + lane];
    re[ra] = two(a.re, a.re);
    im[ra] = two(a.im, a.im);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!(halves >> h & 1u)) continue;
#pragma unroll
    for (int b = h * kTile / 2; b < (h + 1) * kTile / 2; ++b) {
      const Cpx x = xb[b * kLanes + lane];
      const Two q = two(x.re, x.im), turned = two(x.im, -x.re);
#pragma unroll
      for (int ra = 0; ra < kRowsPerWarp; ++ra) fma_two(acc[ra][b], re[ra], q);
#pragma unroll
      for (int ra = 0; ra < kRowsPerWarp; ++ra) fma_two(acc[ra][b], im[ra], turned);
    }
  }
}

// The stored value of a pair: (initial + sum) / count, the reference's
// in-place accumulation followed by its division (src/CrossCorr.cpp:122-144).
// The FP32 quotient as an FP64 product with inv = 1 / count, rounded once more:
// a quotient of two 24-bit numbers lies at least 2^-49 of itself from the middle
// between two floats, so the rounding is that of the division.
CC_HD Cpx pair_value(Cpx init, Cpx sum, double inv) {
  return cpx((float)((double)(init.re + sum.re) * inv), (float)((double)(init.im + sum.im) * inv));
}
CC_HD Cpx pair_value(Cpx init, Cpx sum, int count) {
  return pair_value(init, sum, 1.0 / (double)count);
}

}  // namespace xc
}  // namespace ccfj
