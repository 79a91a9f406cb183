// Ambient-noise cross-correlation on the device: the reference's
// CrossCorrelation (src/CrossCorr.cpp:33-159), which produces the
// cross-spectra that fj_noise takes.
//
// Three kernels per call:
//   xc_spectra_kernel   one CTA per (shift, station) window: its samples
//                       (one-bit on load; folded to the wanted bins' period)
//                       as complex points in shared memory, self-sorting
//                       Stockham passes of radix 8/4/2/3/5 in place, then
//                       the real-FFT split at bins j*fstride, whitening, and
//                       a store to X[k][i][j] (complex FP32, frequency
//                       fastest, rows padded to 32; zeros for a window that
//                       the station does not keep);
//   xc_spectra_direct_kernel   the same bins by a direct transform (FP64
//                       accumulation) for windows the shared-memory FFT
//                       does not take (odd, longer than 16384 samples, or
//                       a prime factor above 5 in F/2);
//   xc_gram_kernel      per 16 x 16 station tile and 32 frequencies, the
//                       sums over shifts of conj(X_a) X_b, staged 2 shifts
//                       at a time in shared memory; windows a station does
//                       not keep are zero in X, so the sums need no mask,
//                       and each pair's count is the overlap of two shift
//                       intervals. The epilogue divides and stores every
//                       pair of the caller's list that falls in the tile.
// The arithmetic lives in cc_core.cuh and the planning in cc_plan.h, which
// the tests also run on the host.
#include <algorithm>
#include <string>
#include <vector>

#include "cc_core.cuh"
#include "cc_plan.h"
#include "ccfj_core.cuh"
#include "fj_frontend.cuh"

namespace ccfj {
namespace xc {

// exp(-2 pi i u / n) for u < count, from FP64 sincospi
__global__ void xc_twiddle_kernel(int n, int count, Cpx* __restrict__ out) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= count) return;
  double s, c;
  sincospi(-2.0 * (double)u / (double)n, &s, &c);
  out[u] = cpx((float)c, (float)s);
}

// The tables of the Stockham passes, one after the other (see bf_rows), then
// the M + 1 factors exp(-i pi k / M) of the real transform's split
struct PassTables {
  int M, npass;
  int radix[kMaxPasses], at[kMaxPasses + 1];  // at[npass]: the split's factors
};

static PassTables pass_tables(int M, int npass, const int* radix) {
  PassTables t = {};
  t.M = M;
  t.npass = npass;
  int Ns = 1;
  for (int p = 0; p < npass; ++p) {
    t.radix[p] = radix[p];
    t.at[p + 1] = t.at[p] + twiddle_rows(radix[p]) * Ns;
    Ns *= radix[p];
  }
  return t;
}

__global__ void xc_pass_tables_kernel(PassTables t, Cpx* __restrict__ out) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u > t.at[t.npass] + t.M) return;
  int p = 0, Ns = 1;
  for (; p < t.npass && u >= t.at[p + 1]; ++p) Ns *= t.radix[p];
  const int v = u - t.at[p];
  double s, c;
  if (p < t.npass)
    sincospi(-2.0 * (double)((v % Ns) << (v / Ns)) / (double)(Ns * t.radix[p]), &s, &c);
  else
    sincospi(-(double)v / (double)t.M, &s, &c);
  out[u] = cpx((float)c, (float)s);
}

struct SpecJob {
  const float* data;      // [nsta][npts]
  long long npts;
  long long steplen;
  int F, M;
  int fold;               // parts of the window that are added (2M fold = F)
  int npass_r[5];         // passes of radix 8, 4, 2, 3, 5, in that order
  const Cpx* tw;          // the passes' tables, one after the other (Stockham), or [F] (direct)
  const Cpx* twh;         // [M + 1] exp(-i pi k/M) (Stockham)
  const int* lo;          // [nsta] kept shifts
  const int* hi;
  int nf, fstride, whiten, onebit;
  int nsta, ldj;
  Cpx* X;                 // [nshifts][nsta][ldj]
};

// The points in shared memory, one slot skipped after every 16: the first
// passes store at strides of 2, 4 and 8 points, which would otherwise meet
// in the same banks (16 pairs of banks of 8 bytes).
struct Skew {
  Cpx* p;
  __device__ __forceinline__ Cpx& operator[](int i) const { return p[i + (i >> 4)]; }
};
static int skewed(int m) { return m + m / 16 + 1; }

// One in-place Stockham pass over s[0 .. M): every thread loads all of its
// butterflies' inputs, then (after the barrier) twiddles, transforms and
// stores them. t / Ns by the high word of a product: exact for t Ns < 2^32
// (here below 2^26).
template <int R, int T>
__device__ __forceinline__ void spec_pass(Skew s, int M, int& Ns, const Cpx*& tw) {
  constexpr int B = (kFftPoints + R - 1) / R;
  Cpx v[B][R];
  const int nb = M / R;
  const unsigned inv = 0xffffffffu / (unsigned)Ns + 1u;  // ceil(2^32 / Ns); 0 for Ns = 1
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const int t = threadIdx.x + b * T;
    if (t < nb) bf_load<R>(s, M, t, v[b]);
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const int t = threadIdx.x + b * T;
    if (t < nb) {
      const int tq = Ns == 1 ? t : (int)__umulhi((unsigned)t, inv);
      bf_rows<R>(s, Ns, tq, t - tq * Ns, tw, v[b]);
    }
  }
  __syncthreads();
  tw += twiddle_rows(R) * Ns;
  Ns *= R;
}

// sum += v, what the rounding loses into low.
__device__ __forceinline__ void add_exact(float& sum, float& low, float v) {
  const float t = sum + v, b = t - sum;
  low += (sum - (t - b)) + (v - b);
  sum = t;
}
__device__ __forceinline__ void add_exact(Cpx& sum, Cpx& low, Cpx v) {
  add_exact(sum.re, low.re, v.re);
  add_exact(sum.im, low.im, v.im);
}

// What bounds it: issue, about half of it the passes (index arithmetic, twiddles
// and transforms), then the reads of the overlapping windows (each sample once
// per window that holds it, from L2). Both shrink when the wanted bins lie
// fstride apart: the window is folded to 2M samples on load (SpecJob::fold parts
// added, with the roundings carried along or, more than four, in FP64, so that
// the sum rounds once), which leaves the transform of the wanted bins
// alone. 100 stations x 51 windows of 14400 samples, every third bin: 317 us
// without the fold, 135 with it, 119 with each pass's twiddles in their own rows
// (one table of all had a line per lane), 105 with samples loaded in pairs; the
// carried roundings add 8.
template <int T>
__global__ void __launch_bounds__(T, 1024 / T) xc_spectra_kernel(SpecJob j) {
  extern __shared__ Cpx smem[];  // [skewed(M)]
  const Skew s{smem};
  const int k = blockIdx.x, i = blockIdx.y;
  Cpx* out = j.X + ((long long)k * j.nsta + i) * j.ldj;
  if (k < j.lo[i] || k > j.hi[i]) {  // not kept: nothing to the sums
    for (int q = threadIdx.x; q < j.ldj; q += T) out[q] = cpx(0.f, 0.f);
    return;
  }
  // a kept window lies inside the record: k*steplen + F <= npts
  const float* x = j.data + (long long)i * j.npts + (long long)k * j.steplen;
  const long long F2 = 2 * j.M;
  // sample 2m and 2m + 1 of a part of the window, in one load where the
  // window's start allows it (the parts lie an even number of samples apart)
  const bool even = ((uintptr_t)x & 7u) == 0;
  auto samples = [&](const float* at) {
    Cpx v;
    if (even)
      v = *reinterpret_cast<const Cpx*>(at);
    else
      v = cpx(at[0], at[1]);
    return j.onebit ? cpx(onebit(v.re), onebit(v.im)) : v;
  };
  if (j.fold <= 4) {
#pragma unroll 4
    for (int m = threadIdx.x; m < j.M; m += T) {
      const float* at = x + 2 * m;
      Cpx a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = u < j.fold ? samples(at + u * F2) : cpx(0.f, 0.f);
      Cpx sum = a[0], low = cpx(0.f, 0.f);
      if (j.fold > 1) add_exact(sum, low, a[1]);
      if (j.fold > 2) add_exact(sum, low, a[2]);
      if (j.fold > 3) add_exact(sum, low, a[3]);
      s[m] = cadd(sum, low);
    }
  } else {
    for (int m = threadIdx.x; m < j.M; m += T) {
      const float* at = x + 2 * m;
      double re = 0.0, im = 0.0;
#pragma unroll 8
      for (int t = 0; t < j.fold; ++t, at += F2) {
        const Cpx v = samples(at);
        re += (double)v.re;
        im += (double)v.im;
      }
      s[m] = cpx((float)re, (float)im);
    }
  }
  __syncthreads();
  // the plan's passes in its order: 8s, a 4 or a 2, 3s, 5s (one loop per
  // radix keeps each radix's registers apart)
  int Ns = 1;
  const Cpx* tw = j.tw;
  for (int p = 0; p < j.npass_r[0]; ++p) spec_pass<8, T>(s, j.M, Ns, tw);
  for (int p = 0; p < j.npass_r[1]; ++p) spec_pass<4, T>(s, j.M, Ns, tw);
  for (int p = 0; p < j.npass_r[2]; ++p) spec_pass<2, T>(s, j.M, Ns, tw);
  for (int p = 0; p < j.npass_r[3]; ++p) spec_pass<3, T>(s, j.M, Ns, tw);
  for (int p = 0; p < j.npass_r[4]; ++p) spec_pass<5, T>(s, j.M, Ns, tw);
  for (int q = threadIdx.x; q < j.ldj; q += T) {
    Cpx v = cpx(0.f, 0.f);
    if (q < j.nf) {
      const int k = q * j.fstride;  // <= M (checked by the plan)
      v = real_bin(s, j.M, k, j.twh[k]);
      if (j.whiten) v = whiten(v);
    }
    out[q] = v;
  }
}

template <int T>
static int launch_spectra(const SpecJob& j, unsigned nshifts, cudaStream_t s) {
  const size_t smem = (size_t)skewed(j.M) * sizeof(Cpx);
  CCFJ_CUDA_TRY(cudaFuncSetAttribute(xc_spectra_kernel<T>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  xc_spectra_kernel<T><<<dim3(nshifts, j.nsta), T, smem, s>>>(j);
  count_launch();
  CCFJ_LAUNCH_CHECK("xc_spectra_kernel");
  return CCFJ_OK;
}

constexpr int kDirectThreads = 128;

__global__ void __launch_bounds__(kDirectThreads) xc_spectra_direct_kernel(SpecJob j) {
  const int k = blockIdx.x, i = blockIdx.y;
  const int q = blockIdx.z * kDirectThreads + threadIdx.x;
  if (q >= j.ldj) return;
  Cpx* out = j.X + ((long long)k * j.nsta + i) * j.ldj;
  // not kept, or the row's padding, which the pair products read too
  if (k < j.lo[i] || k > j.hi[i] || q >= j.nf) {
    out[q] = cpx(0.f, 0.f);
    return;
  }
  const float* x = j.data + (long long)i * j.npts + (long long)k * j.steplen;
  const long long bin = (long long)q * j.fstride;  // <= F/2 < F
  double re = 0.0, im = 0.0;
  long long ph = 0;  // bin*n mod F
  for (int n = 0; n < j.F; ++n) {
    float v = x[n];
    if (j.onebit) v = onebit(v);
    const Cpx t = j.tw[ph];
    re += (double)v * (double)t.re;
    im += (double)v * (double)t.im;
    ph += bin;
    if (ph >= j.F) ph -= j.F;
  }
  Cpx v = cpx((float)re, (float)im);
  if (j.whiten) v = whiten(v);
  out[q] = v;
}

struct GramJob {
  const Cpx* X;
  int nsta, ldj, nf;
  const Tile* tiles;
  const int* lo;
  const int* hi;
  const int* pmap;   // [nsta * nsta]
  const int* pnext;  // [npairs]
  float* out_re;
  float* out_im;
  long long out_ld;  // floats between pairs
  int out_es;        // floats between bins
  int accumulate;
  int paired;        // re and im are neighbours and 8-byte aligned
};

constexpr int kGramStages = 3;
typedef Cpx GramRows[kShiftChunk][2][kTile][kLanes];  // 16 KiB

// What bounds it: the FP32 pipe (four multiply-adds a product, as two packed
// instructions: 40 us of the case below), then issue and the copies' latency
// with 12 warps per SM, whose sums fill the registers. The rows of the next
// shifts are copied (cp.async) while the present ones are multiplied; a half
// tile of columns that no pair wants is left out, and the epilogue looks its
// pairs up by lanes and divides by a product in FP64. 100 stations, 4950 pairs x
// 1000 bins x 51 shifts: 99 us; 192 us with copies through registers, a lookup
// per pair and an FP32 division (128 us of those when nothing hid them).
__global__ void __launch_bounds__(kGramThreads, 3) xc_gram_kernel(GramJob g) {
  extern __shared__ Cpx smem[];
  GramRows* xs = reinterpret_cast<GramRows*>(smem);  // [kGramStages]
  const Tile t = g.tiles[blockIdx.x];
  const int j0 = blockIdx.y * kLanes;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  // the pair, the next pair of the same stations and 1 / count at this lane's
  // two (row, column) places: rows 0-1 of the warp's four, then rows 2-3
  int pr[2], nx[2];
  double inv[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int a = t.a0 + warp * kRowsPerWarp + 2 * h + lane / kTile;
    const int b = t.b0 + lane % kTile;
    pr[h] = nx[h] = -1;
    inv[h] = 0.0;
    if (a < g.nsta && b < g.nsta) {
      pr[h] = g.pmap[(long long)a * g.nsta + b];
      const int cnt = pair_count(g.lo[a], g.hi[a], g.lo[b], g.hi[b]);
      if (cnt == 0) pr[h] = -1;
      inv[h] = 1.0 / (double)cnt;
      if (pr[h] >= 0) nx[h] = g.pnext[pr[h]];
    }
  }
  const unsigned want = __ballot_sync(0xffffffffu, pr[0] >= 0 || pr[1] >= 0);
  const unsigned halves = ((want & 0x00ff00ffu) ? 1u : 0u) | ((want & 0xff00ff00u) ? 2u : 0u);

  Cpx acc[kRowsPerWarp][kTile];
#pragma unroll
  for (int ra = 0; ra < kRowsPerWarp; ++ra)
#pragma unroll
    for (int b = 0; b < kTile; ++b) acc[ra][b] = cpx(0.f, 0.f);

  // Shifts kc .. kc + kShiftChunk - 1 into a stage, 16 bytes a copy: this
  // thread's part of rows r and r + 8 of both sides. Past the last station the
  // last one is copied (no pair is looked up there), past the last shift the
  // last one (not multiplied).
  constexpr int kPer = kLanes / 2;                // copies a row
  constexpr int kStep = kGramThreads / kPer;      // rows at once
  constexpr int kRows = 2 * kTile / kStep;        // copies of a thread for a shift
  const int l = 2 * (threadIdx.x % kPer), r = threadIdx.x / kPer;
  const long long shift = (long long)g.nsta * g.ldj;
  const Cpx* from[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int row = i * kStep + r;
    const int st = (row < kTile ? t.a0 : t.b0 - kTile) + row;
    from[i] = g.X + (long long)min(st, g.nsta - 1) * g.ldj + j0 + l;
  }
  auto fetch = [&](int stage, int kc) {
#pragma unroll
    for (int kk = 0; kk < kShiftChunk; ++kk) {
      const long long at = min(kc + kk, t.k1) * shift;
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const unsigned dst = (unsigned)__cvta_generic_to_shared(&xs[stage][kk][0][i * kStep + r][l]);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(from[i] + at)
                     : "memory");
      }
    }
  };
  int fill = t.k0;
#pragma unroll
  for (int i = 0; i < kGramStages - 1; ++i, fill += kShiftChunk) {
    if (fill <= t.k1) fetch(i, fill);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  int stage = 0, into = kGramStages - 1;
  for (int kc = t.k0; kc <= t.k1; kc += kShiftChunk, fill += kShiftChunk) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kGramStages - 2) : "memory");
    __syncthreads();  // this stage is in, and the one before it has been read
    if (fill <= t.k1) fetch(into, fill);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll 1
    for (int kk = 0; kk < min(kShiftChunk, t.k1 - kc + 1); ++kk)
      gram_step(&xs[stage][kk][0][0][0], &xs[stage][kk][1][0][0], warp, lane, acc, halves);
    stage = stage + 1 == kGramStages ? 0 : stage + 1;
    into = into + 1 == kGramStages ? 0 : into + 1;
  }

  // A row of sums at a time through shared memory, so that the stores are a
  // loop: written out for all 64 sums they did not fit the instruction cache
  // (the waits for instructions were a third of the kernel).
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  Cpx* mine = smem + warp * kTile * kLanes + lane;
  const int j = j0 + lane;
#pragma unroll
  for (int ra = 0; ra < kRowsPerWarp; ++ra) {
#pragma unroll
    for (int b = 0; b < kTile; ++b) mine[b * kLanes] = acc[ra][b];
#pragma unroll 2
    for (int b = 0; b < kTile; ++b) {
      const int from = (ra & 1) * kTile + b;
      int p = __shfl_sync(0xffffffffu, pr[ra / 2], from);
      const int next = __shfl_sync(0xffffffffu, nx[ra / 2], from);
      const double one = __shfl_sync(0xffffffffu, inv[ra / 2], from);
      if (p < 0 || j >= g.nf) continue;
      const Cpx sum = mine[b * kLanes];
      for (bool first = true; p >= 0; p = first ? next : g.pnext[p], first = false) {
        float* re = g.out_re + (long long)p * g.out_ld + (long long)j * g.out_es;
        float* im = g.out_im + (long long)p * g.out_ld + (long long)j * g.out_es;
        const Cpx init = g.accumulate ? cpx(*re, *im) : cpx(0.f, 0.f);
        const Cpx v = pair_value(init, sum, one);
        if (g.paired) {
          *reinterpret_cast<Cpx*>(re) = v;
        } else {
          *re = v.re;
          *im = v.im;
        }
      }
    }
  }
}

template <typename T>
static T* upload(Scratch& sc, const std::vector<T>& v, cudaStream_t s, int* status) {
  T* d = sc.get_n<T>(v.empty() ? 1 : v.size());
  if (!d) {
    *status = CCFJ_ERR_ALLOC;
    return nullptr;
  }
  if (!v.empty()) {
    cudaError_t e = cudaMemcpyAsync(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) {
      *status = set_error(CCFJ_ERR_CUDA, "cudaMemcpyAsync (plan upload): %s", cudaGetErrorString(e));
      return nullptr;
    }
  }
  return d;
}

static int twiddles(Cpx* out, int n, int count, cudaStream_t s) {
  xc_twiddle_kernel<<<div_up(count, 256), 256, 0, s>>>(n, count, out);
  count_launch();
  CCFJ_LAUNCH_CHECK("xc_twiddle_kernel");
  return CCFJ_OK;
}

static int run(const ccfj_cc_args& a, cudaStream_t s) {
  CCFJ_REQUIRE(a.struct_size == (int)sizeof(ccfj_cc_args),
               "ccfj_cc_v1: struct_size=%d, expected %d", a.struct_size, (int)sizeof(ccfj_cc_args));
  CCFJ_REQUIRE(a.data != nullptr, "ccfj_cc_v1: data is NULL");
  Plan p;
  std::string err;
  const int pst = make_plan(a, &p, &err, false);
  if (pst != CCFJ_OK) return set_error(pst, "ccfj_cc_v1: %s", err.c_str());
  const long long nout = (long long)a.npairs * a.nf;
  CCFJ_REQUIRE(nout == 0 || (a.out_re && (a.out_layout == 1 || a.out_im)),
               "ccfj_cc_v1: output pointer is NULL");
  CCFJ_REQUIRE(a.nf <= 65535LL * kLanes, "ccfj_cc_v1: nf=%d too large", a.nf);
  CCFJ_REQUIRE(p.nwindows <= 0x7fffffff, "ccfj_cc_v1: too many windows");
  const long long nrec = (long long)a.nsta * a.npts;
  if (!a.device_ptrs && a.onebit)  // the reference rewrites the caller's samples
    for (long long n = 0; n < nrec; ++n) a.data[n] = onebit(a.data[n]);
  if (nout == 0) return CCFJ_OK;  // no pairs or no bins: nothing for the device

  Scratch sc(s);
  int status = CCFJ_OK;
  const float* d_data = a.data;
  if (!a.device_ptrs) {
    float* d = sc.get_n<float>(nrec);
    if (!d) return CCFJ_ERR_ALLOC;
    const int cst = copy_from_host(d, a.data, nrec * sizeof(float), s);
    if (cst != CCFJ_OK) return cst;
    d_data = d;
  }
  // outputs: planes (re, im) [npairs][nf] or interleaved complex [npairs][nf]
  const size_t plane = (size_t)nout * sizeof(float);
  float* d_re = a.out_re;
  float* d_im = a.out_layout == 1 ? (a.out_re ? a.out_re + 1 : nullptr) : a.out_im;
  if (!a.device_ptrs && nout > 0) {
    if (a.out_layout == 1) {
      d_re = sc.get_n<float>(2 * nout);
      if (!d_re) return CCFJ_ERR_ALLOC;
      d_im = d_re + 1;
    } else {
      d_re = sc.get_n<float>(nout);
      d_im = sc.get_n<float>(nout);
      if (!d_re || !d_im) return CCFJ_ERR_ALLOC;
    }
  }
  if (nout > 0) {
    if (a.accumulate && !a.device_ptrs) {
      if (a.out_layout == 1) {
        CCFJ_CUDA_TRY(cudaMemcpyAsync(d_re, a.out_re, 2 * plane, cudaMemcpyHostToDevice, s));
      } else {
        CCFJ_CUDA_TRY(cudaMemcpyAsync(d_re, a.out_re, plane, cudaMemcpyHostToDevice, s));
        CCFJ_CUDA_TRY(cudaMemcpyAsync(d_im, a.out_im, plane, cudaMemcpyHostToDevice, s));
      }
    } else if (!a.accumulate && !p.every_pair) {  // what the products don't store
      if (a.out_layout == 1) {
        CCFJ_CUDA_TRY(cudaMemsetAsync(d_re, 0, 2 * plane, s));
      } else {
        CCFJ_CUDA_TRY(cudaMemsetAsync(d_re, 0, plane, s));
        CCFJ_CUDA_TRY(cudaMemsetAsync(d_im, 0, plane, s));
      }
    }
  }

  if (nout > 0 && !p.tiles.empty()) {
    // window spectra
    const size_t xcount = (size_t)p.nshifts * a.nsta * p.ldj;
    Cpx* X = sc.get_n<Cpx>(xcount);
    if (!X) return CCFJ_ERR_ALLOC;
    const int* d_lo = upload(sc, p.lo, s, &status);
    const int* d_hi = d_lo ? upload(sc, p.hi, s, &status) : nullptr;
    if (!d_hi) return status;
    SpecJob j = {};
    j.data = d_data;
    j.npts = a.npts;
    j.steplen = a.steplen;
    j.F = p.F;
    j.M = p.M;
    j.fold = 1;
    j.fstride = a.fstride;
    int npass = p.npass;
    int radix[kMaxPasses];
    std::copy(p.radix, p.radix + kMaxPasses, radix);
    if (p.stockham) {
      // Bins at multiples of g (a divisor of M) are the bins of the window
      // folded to F / g samples: one pass over the window instead of a
      // transform of all of it (xc_spectra_kernel has the figures).
      int g = p.M, b = a.fstride;
      while (b != 0) {
        const int rest = g % b;
        g = b;
        b = rest;
      }
      if (g > 1 && p.M / g >= 2) {
        j.M = p.M / g;
        j.fold = g;
        j.fstride = a.fstride / g;
        npass = fft_plan(j.M, radix);
      }
    }
    for (int i = 0; i < npass; ++i) {
      const int r = radix[i];
      ++j.npass_r[r == 8 ? 0 : r == 4 ? 1 : r == 2 ? 2 : r == 3 ? 3 : 4];
    }
    j.lo = d_lo;
    j.hi = d_hi;
    j.nf = a.nf;
    j.whiten = a.whiten ? 1 : 0;
    j.onebit = a.onebit ? 1 : 0;
    j.nsta = a.nsta;
    j.ldj = p.ldj;
    j.X = X;
    const unsigned nshifts = (unsigned)p.nshifts;
    if (p.stockham) {
      const PassTables t = pass_tables(j.M, npass, radix);
      const int ntab = t.at[npass] + j.M + 1;
      Cpx* tw = sc.get_n<Cpx>(ntab);
      if (!tw) return CCFJ_ERR_ALLOC;
      xc_pass_tables_kernel<<<div_up(ntab, 128), 128, 0, s>>>(t, tw);
      count_launch();
      CCFJ_LAUNCH_CHECK("xc_pass_tables_kernel");
      j.tw = tw;
      j.twh = tw + t.at[npass];
      // the fewest threads that hold the points: more windows per SM, whose
      // loads and passes overlap
      const int e = j.M <= 128 * kFftPoints   ? launch_spectra<128>(j, nshifts, s)
                    : j.M <= 256 * kFftPoints ? launch_spectra<256>(j, nshifts, s)
                                              : launch_spectra<512>(j, nshifts, s);
      if (e) return e;
    } else {
      Cpx* tw = sc.get_n<Cpx>(p.F);
      if (!tw) return CCFJ_ERR_ALLOC;
      if (int e = twiddles(tw, p.F, p.F, s)) return e;
      j.tw = tw;
      xc_spectra_direct_kernel<<<dim3(nshifts, a.nsta, div_up(p.ldj, kDirectThreads)),
                                 kDirectThreads, 0, s>>>(j);
      count_launch();
      CCFJ_LAUNCH_CHECK("xc_spectra_direct_kernel");
    }
    // pair products
    const Tile* d_tiles = upload(sc, p.tiles, s, &status);
    const int* d_pmap = d_tiles ? upload(sc, p.pmap, s, &status) : nullptr;
    const int* d_pnext = d_pmap ? upload(sc, p.pnext, s, &status) : nullptr;
    if (!d_pnext) return status;
    GramJob g = {};
    g.X = X;
    g.nsta = a.nsta;
    g.ldj = p.ldj;
    g.nf = a.nf;
    g.tiles = d_tiles;
    g.lo = d_lo;
    g.hi = d_hi;
    g.pmap = d_pmap;
    g.pnext = d_pnext;
    g.out_re = d_re;
    g.out_im = d_im;
    g.out_ld = a.out_layout == 1 ? 2LL * a.nf : a.nf;
    g.out_es = a.out_layout == 1 ? 2 : 1;
    g.accumulate = a.accumulate ? 1 : 0;
    g.paired = a.out_layout == 1 && (uintptr_t)d_re % sizeof(Cpx) == 0 ? 1 : 0;
    const size_t smem = kGramStages * sizeof(GramRows);
    CCFJ_CUDA_TRY(cudaFuncSetAttribute(xc_gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
    xc_gram_kernel<<<dim3((unsigned)p.tiles.size(), div_up(a.nf, kLanes)), kGramThreads, smem, s>>>(g);
    count_launch();
    CCFJ_LAUNCH_CHECK("xc_gram_kernel");
  }

  if (!a.device_ptrs) {
    int st = CCFJ_OK;
    if (nout > 0 && a.out_layout == 1) {
      st = copy_to_host(a.out_re, d_re, 2 * plane, 0, s);
    } else if (nout > 0) {
      st = copy_to_host(a.out_re, d_re, plane, 0, s);
      if (st == CCFJ_OK) st = copy_to_host(a.out_im, d_im, plane, 0, s);
    } else {
      CCFJ_CUDA_TRY(cudaStreamSynchronize(s));
    }
    if (st != CCFJ_OK) return st;
  }
  return CCFJ_OK;
}

// Records to dispersion spectrum: the cross-correlation writes its
// complex64 cross-spectra into device scratch, and the transform reads
// their real parts there (perm, r, f, c and out as the caller gives them).
static int cc_fj_noise(const ccfj_cc_args& cc, const ccfj_fj_args& fj, cudaStream_t s) {
  CCFJ_REQUIRE(cc.struct_size == (int)sizeof(ccfj_cc_args),
               "ccfj_cc_fj_noise_v1: cc struct_size=%d, expected %d", cc.struct_size,
               (int)sizeof(ccfj_cc_args));
  CCFJ_REQUIRE(!cc.accumulate, "ccfj_cc_fj_noise_v1: cc->accumulate must be 0");
  CCFJ_REQUIRE(cc.device_ptrs == fj.device_ptrs,
               "ccfj_cc_fj_noise_v1: cc->device_ptrs (%d) != fj->device_ptrs (%d)",
               cc.device_ptrs, fj.device_ptrs);
  CCFJ_REQUIRE(cc.data != nullptr, "ccfj_cc_fj_noise_v1: data is NULL");
  CCFJ_REQUIRE(fj.nr == cc.npairs && fj.nf == cc.nf,
               "ccfj_cc_fj_noise_v1: fj nr=%d nf=%d must equal the pairs (%d) and bins (%d)",
               fj.nr, fj.nf, cc.npairs, cc.nf);
  CCFJ_REQUIRE(fj.mode == CCFJ_MODE_J || fj.mode == CCFJ_MODE_J_MINUS_Y,
               "ccfj_cc_fj_noise_v1: mode must be CCFJ_MODE_J (func 0) or CCFJ_MODE_J_MINUS_Y "
               "(func 1)");
  CCFJ_REQUIRE(cc.npairs >= 1 && cc.nf >= 1, "ccfj_cc_fj_noise_v1: npairs=%d nf=%d", cc.npairs,
               cc.nf);
  Scratch sc(s);
  CallFlag flag(s);
  FjChoice choice;
  if (!cc.device_ptrs && !(choice.err = flag.word())) return CCFJ_ERR_ALLOC;
  float* spec = sc.get_n<float>(2 * (size_t)cc.npairs * cc.nf);
  if (!spec) return CCFJ_ERR_ALLOC;
  ccfj_cc_args c = cc;
  c.device_ptrs = 1;
  c.out_layout = 1;
  c.out_re = spec;
  c.out_im = nullptr;
  const long long nrec = (long long)cc.nsta * cc.npts;
  if (!cc.device_ptrs) {  // the records cross to the device once
    CCFJ_REQUIRE(cc.nsta >= 1 && cc.npts >= 1, "ccfj_cc_fj_noise_v1: nsta=%d npts=%d", cc.nsta,
                 cc.npts);
    float* d = sc.get_n<float>(nrec);
    if (!d) return CCFJ_ERR_ALLOC;
    const int cst = copy_from_host(d, cc.data, nrec * sizeof(float), s);
    if (cst != CCFJ_OK) return cst;
    c.data = d;
  }
  ccfj_fj_args f = fj;
  f.u[0] = spec;
  f.u[1] = nullptr;
  f.u_ld = 2LL * cc.nf;
  f.u_rows = cc.npairs;
  f.u_es = 2;
  f.u_ncols = cc.nf;
  f.fstride = 1;
  f.hilbert = fj.mode == CCFJ_MODE_J_MINUS_Y ? 1 : 0;
  f.col_begin = 0;
  f.nf_total = 0;
  f.device_ptrs = 1;
  int st = fj_validate(&f);
  if (st != CCFJ_OK) return st;
  if (!fj.device_ptrs) {  // the small per-pair and grid arrays, and the result
    float* dr = sc.get_n<float>(fj.nr);
    float* df = sc.get_n<float>(fj.nf);
    float* dc = sc.get_n<float>(fj.nc);
    float* dout = sc.get_n<float>((size_t)fj.nc * fj.nf);
    long long* dp = fj.perm ? sc.get_n<long long>(fj.nr) : nullptr;
    if (!dr || !df || !dc || !dout || (fj.perm && !dp)) return CCFJ_ERR_ALLOC;
    if (fj.perm)
      for (int i = 0; i < fj.nr; ++i)
        CCFJ_REQUIRE(fj.perm[i] >= 0 && fj.perm[i] < fj.nr,
                     "ccfj_cc_fj_noise_v1: perm[%d]=%lld out of range", i, fj.perm[i]);
    CCFJ_CUDA_TRY(cudaMemcpyAsync(dr, fj.r, sizeof(float) * fj.nr, cudaMemcpyHostToDevice, s));
    CCFJ_CUDA_TRY(cudaMemcpyAsync(df, fj.f, sizeof(float) * fj.nf, cudaMemcpyHostToDevice, s));
    CCFJ_CUDA_TRY(cudaMemcpyAsync(dc, fj.c, sizeof(float) * fj.nc, cudaMemcpyHostToDevice, s));
    if (dp)
      CCFJ_CUDA_TRY(cudaMemcpyAsync(dp, fj.perm, sizeof(long long) * fj.nr, cudaMemcpyHostToDevice,
                                    s));
    f.r = dr;
    f.f = df;
    f.c = dc;
    f.out = dout;
    f.perm = dp;
  }
  st = run(c, s);
  if (st != CCFJ_OK) return st;
  st = fj_device(f, s, choice);
  if (st != CCFJ_OK || fj.device_ptrs) return st;
  st = copy_to_host(fj.out, f.out, sizeof(float) * fj.nc * fj.nf, 0, s);
  return st != CCFJ_OK ? st : flag.status("ccfj_cc_fj_noise_v1");
}

}  // namespace xc
}  // namespace ccfj

CCFJ_API int ccfj_cc_fj_noise_v1(const ccfj_cc_args* cc, const ccfj_fj_args* fj, void* stream) {
  ccfj::clear_error();
  if (!cc || !fj) return ccfj::set_error(CCFJ_ERR_INVALID, "ccfj_cc_fj_noise_v1: NULL args");
  if (fj->struct_size != (int)sizeof(ccfj_fj_args))
    return ccfj::set_error(CCFJ_ERR_INVALID, "ccfj_cc_fj_noise_v1: fj struct_size=%d, expected %d",
                           fj->struct_size, (int)sizeof(ccfj_fj_args));
  return ccfj::xc::cc_fj_noise(*cc, *fj, (cudaStream_t)stream);
}

CCFJ_API int ccfj_cc_v1(const ccfj_cc_args* args, void* stream) {
  ccfj::clear_error();
  if (!args) return ccfj::set_error(CCFJ_ERR_INVALID, "ccfj_cc_v1: args is NULL");
  return ccfj::xc::run(*args, (cudaStream_t)stream);
}

CCFJ_API int CrossCorrelation(ccfj_cc_data d) {
  ccfj_cc_args a = {};
  a.struct_size = (int)sizeof(a);
  a.nsta = d.nsta;
  a.npts = d.npts;
  a.nf = d.nf;
  a.npairs = d.npairs;
  a.fstride = d.fstride;
  a.fftlen = d.fftlen;
  a.steplen = d.steplen;
  a.onebit = d.ifonebit;
  a.whiten = d.ifspecwhitenning;
  a.device_ptrs = 0;
  a.accumulate = 1;
  a.out_layout = 0;
  a.pairs = d.Pairs;
  a.startend = d.startend;
  a.data = d.data;
  a.out_re = d.ncfsr;
  a.out_im = d.ncfsi;
  return ccfj_cc_v1(&a, nullptr);
}
