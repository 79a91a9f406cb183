// Wave-cell expansion of the F-J transform.
//
// Both forms of the transform (src/FJcpu.cpp:230-419) are linear functionals
// of the function r -> Z0(k r), k = 2 pi f / c:
//
//   itype 1   out(c, f) = sum over intervals of int (g_A + b (r - r_A)) r Z0(k r) dr
//   itype 0   out(c, f) = sum over stations of g w Z0(k r)
//
// and k r = 2 pi u / c depends on u = r f alone. So the axis of u is cut into
// cells on which Z0 is a polynomial to FP32 rounding at every velocity of the
// call: cells of 9.8 radians at the slowest velocity and 16 Chebyshev terms
// (the series of a wave over +-5.2 radians has the coefficients 2 J_n(5.2):
// 1e-7 at n = 16, at the slowest velocity alone). With Z0(2 pi u / c) = sum_n E[c][cell, n] T_n,
// the transform is a matrix product
//
//   out[c, f] = sum_{cell, n} E[c][cell, n] W[cell, n][f]
//
// of a matrix E that is the same for every frequency, every set of a batch
// and every input, and the moments W of the spectra over the cells, which
// know nothing of the velocities:
//
//   W[cell, n][f] = int over the cell of g(r) r T_n dr.
//
// A short interval belongs to the cell of its far end, so the polynomials
// reach 1/16 of a cell below their cell (10.4 radians in all).
//
// The direct kernels evaluate the special functions once per (pair, f, c);
// here they are evaluated once per (cell node, c), the pairs are visited once
// per f, and the rest is multiply-adds. The number of cells of a frequency,
// f (r_max - r_min) / h, does not depend on the number of pairs.
//
// An interval that spans whole cells would add up as much over them as it
// cancels again (its integral is that of a wave), in FP32. It is integrated in
// closed form between the first and the last cell end inside it:
//
//   int (g_A + s (r - r_A)) r Z0(k r) dr = [g r Z1 / k + s (r Z0 / k^2 - B / k^3)]
//
// (B the integral of Z0): two more rows of E per cell, V their weights, and
// nothing in the cells between.
//
// Where the Y basis is asked for, the first cell is cut in half again and
// again towards u = 0 (kDyadic cells), so that the singularity of Y0 stays a
// cell length away from every cell.
//
// Kernels of a call, in order:
//   xp_columns_kernel  which columns take the expansion, cell range per tile
//                      of 128 frequencies; checks that r ascends
//   xp_scan_kernel     where each tile's W blocks and GEMM units begin
//   xp_basis_kernel    E
//   xp_moments_kernel  W, in chunks of stations; the cells that a chunk
//                      shares with its neighbours go to head / tail parts
//   xp_join_kernel     adds those parts in chunk order
//   xp_gemm_kernel     the product on the tensor cores, in units of (128
//                      velocities x 128 columns x a run of cells)
//   xp_finish_kernel   adds a column's units in order, |.| and normalisation
//
// Measured against the direct kernels on one B200 (device-resident call):
// 19,900 pairs x 2048 f x 1000 c 61.3 -> 0.98 ms, 200 x 512 x 300 0.215 ->
// 0.091 ms, 128 subarrays of 50-20,000 pairs (512 f x 500 c) 196 -> 3.6 ms; the
// error against 64-bit quadrature 1.1e-6 -> 2e-7 of the spectrum (2-norm).
//
// Every sum is in an order fixed by the sizes, so results do not depend on
// scheduling, nor on which frequencies share a call.
#include <algorithm>
#include <cmath>

#include "fj_cell.h"
#include "fj_cells.cuh"
#include "fj_expand.cuh"
#include "fj_tcgen05.cuh"

namespace ccfj {

namespace {

using namespace xp;

constexpr int kNodes = 16;          // Chebyshev terms of a cell
// Cells of one frequency: 2048 are 3190 wavelengths of the slowest velocity.
// Columns with more go to the direct kernels.
constexpr int kMaxCells = 2048;
constexpr int kTileCols = 128;      // frequencies of a W tile and GEMM column tile
constexpr int kTileRows = 128;      // velocities of a GEMM tile
constexpr int kGroup = 4;           // tiles begin and end with groups of cells
constexpr int kEndRows = 2;         // rows of a cell's end
constexpr int kEndFloats = kTileCols * kGroup * kEndRows;  // one (tile, group, input) of V
constexpr int kBlockFloats = kTileCols * kNodes;  // one (tile, cell, input) of W

struct XpTile {
  int lo, hi;    // cells [lo, hi) of the tile's columns, whole groups
  long long w;   // first W block (cell blocks of one input)
  long long unit;  // first GEMM unit
};

struct XpPlan {
  double hu, inv_hu;  // cell length in u = r f, and its inverse
  long long units;
  long long blocks;   // W blocks of an input
  long long left;     // columns left to the direct kernels
  int lo, hi;         // cells of E
};

constexpr int kBad = 1 << 30;
struct XpDev {
  const float* rs;
  const float* wtr;
  const long long* off;
  int nsets;
  long long total;
  int nf, nc, ncp;       // ncp: velocities padded to GEMM tiles
  const float* f;
  const float* c;
  InDesc in[2];
  float* out;
  int normalize;
  int ft;                // column tiles of a set
  int chunk;             // stations of a moments chunk
  double nf_all;         // frequencies of the whole problem
  double cells_in_time;  // a column with fewer takes the expansion (worth_cells)
  int mtiles;            // velocity tiles
  int run;               // cells of a GEMM unit
  int nsrc, nacc;        // products of a result, results of a column
  int has_ends;          // itype 1: V and Eend are in use
  int cells_cap;
  int tile_cells;        // a tile of a set of n pairs has at most n / 4 + this many
  long long blocks_cap, units_cap, slots;
  unsigned char* use;
  XpPlan* plan;
  XpTile* tile;
  // [nsets * ft] columns of the tile that go direct; kBad: the tile's part of
  // r is out of order, or a velocity is not positive and finite
  int* direct;
  int* set_bad;          // [nsets] some tile of the set is bad: all its columns go direct
  int* slot_set;         // [slot] the set of a moments chunk
  float* E;              // [basis][cell][velocity tile][128][16]
  float* Eend;           // [basis][group][velocity tile][128][cell of the group][2]
  float* W;              // [block][input][128][16]
  float* V;              // [group][input][128][cell of the group][2]
  int* unit_tile;        // [unit]
  unsigned char* ends;   // [group] some column has weights in V
  float* part;           // [unit][128][128]
  float* head;           // [slot][nf][input][16]
  float* tail;
  int2* span;            // [slot][nf] first and last cell of a chunk
  unsigned int* err;     // the call's flag of the product's waits, or NULL
  long long wait_cycles;
  int no_load;           // self-test: the product's operands never come
};

__device__ __forceinline__ long long set_begin(const XpDev& d, int b) { return d.off ? d.off[b] : 0; }
__device__ __forceinline__ long long set_end(const XpDev& d, int b) {
  return d.off ? d.off[b + 1] : d.total;
}

// Slot of a set's first chunk: sets' slots do not overlap, since a set of n
// pairs has at most n / chunk + 1 chunks.
__device__ __forceinline__ long long slot_begin(const XpDev& d, int b) {
  return set_begin(d, b) / d.chunk + b;
}
__device__ __forceinline__ int chunks_of(const XpDev& d, long long n) {
  return max(1, (int)((n - 1 + d.chunk - 1) / d.chunk));
}

// ------------------------------------------------------------------- plan
// Whether the expansion is worth its launches for a set of n pairs: they take
// about 45 us together, and the direct kernels walk the pairs one after the
// other at 1 to 1.5 us a pair (60 pairs x 40 f x 50 c: 98 us, 58 us here), or
// are bound by their terms (6e6: 50 us). Decided by the whole problem's sizes,
// so that frequency windows, blocks and sets of a batch decide alike.
constexpr double kAnyCost = 4e8;  // issue slots, 20 us
__host__ __device__ inline bool worth(double n, double per_pair) {
  return n >= 48.0 || (n >= 2.0 && n * per_pair >= 6e6);
}

// Whether a column with this many cells takes the expansion. Two estimates:
//
// Throughput, for a chip that is full: multiply-adds of the expansion against
// those of the direct kernel (56 issue slots a term measured on short
// intervals, 250 where most are long against the wavelength; itype 0 has no
// intervals, and its sparse columns count 250 in batches and below 48 pairs
// alone). A problem whose columns all cost little keeps them together: the
// direct kernels' time is the walk over the pairs, for one column too.
//
// Latency, for one transform: both ways are chains, of launches here, of pairs
// there, and a problem with columns on both sides of the line pays for both. A
// column takes the expansion if a problem that had this one as its highest
// frequency would be computed in less time (cells_in_time()), or up to 1.3 times as
// long. Not where a column has many more cells than pairs (earthquake records
// over thousands of km): such problems have columns beyond any line, and more
// of them on this side made them slower.
//
// Of 1683 transforms drawn at random (2-19,900 pairs, half of them of up to 600
// pairs, where the line lies), 135 took more than 15% longer than the direct
// kernels alone with the first estimate only (an itype 0 case 2.7 times as
// long), 85 with both; 77 became more than 15% faster and 1 slower (66 pairs x
// 906 f x 38 c 164 -> 89 us, 95 by the direct kernels; 182 pairs x 208 f x 23 c,
// itype 0, 118 -> 79 us, 101 directly). Still slower than directly: problems
// whose upper frequencies go direct while the lower ones do not (156 records x
// 320 f x 43 c 306 us, 187 directly).
constexpr double kMargin = 1.3;
constexpr double kDense = 6.5;
__device__ __forceinline__ bool worth_cells(const XpDev& d, int itype, int cells_of_column,
                                            double n) {
  const double cells = cells_of_column;
  const double grid =
      (cells + kGroup) * kNodes * ((double)d.ncp * d.nsrc * d.nacc + 200.0) + 200.0 * n;
  const bool sparse = cells > n;
  const double direct =
      n * d.nc * d.nsrc * (sparse && (itype == 1 || n < 48.0 || d.off) ? 250.0 : 56.0);
  if (grid < direct || grid * d.nf_all < kAnyCost) return true;
  return cells < d.cells_in_time && cells * d.nacc <= kDense * n;
}

// One CTA of 128 threads per (set, 128 frequencies).
template <int MODE, int ITYPE>
__global__ void xp_columns_kernel(XpDev d) {
  constexpr bool DY = ModeTraits<MODE>::WY;
  constexpr int kWarps = kTileCols / 32;
  __shared__ float red[kWarps];
  __shared__ int ired[kWarps][3];
  const int t = threadIdx.x, b = blockIdx.y;
  float lo = INFINITY;  // the slowest velocity
  bool fine = true;
  for (int j = t; j < d.nc; j += kTileCols) {
    const float v = d.c[j];
    fine = fine && v > 0.0f && v < INFINITY;
    lo = fminf(lo, v);
  }
  // this tile's share of the set's distances: finite and ascending
  const long long o = set_begin(d, b), n = set_end(d, b) - o;
  for (long long i = blockIdx.x * kTileCols + t; i < n; i += (long long)d.ft * kTileCols) {
    const float v = d.rs[o + i];
    fine = fine && v >= 0.0f && v < INFINITY && (i == 0 || v >= d.rs[o + i - 1]);
  }
  for (int s = 16; s > 0; s >>= 1) lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, s));
  fine = __all_sync(0xffffffffu, fine);
  if ((t & 31) == 0) {
    red[t >> 5] = lo;
    ired[t >> 5][2] = fine;
  }
  __syncthreads();
  for (int w = 0; w < kWarps; ++w) {
    lo = fminf(lo, red[w]);
    fine = fine && ired[w][2];
  }
  const double hu = kCellPhase / fjs::kTwoPi * (double)lo, inv_hu = 1.0 / hu;
  const int tile = b * d.ft + blockIdx.x;
  if (tile == 0 && t == 0) {
    d.plan->hu = hu;
    d.plan->inv_hu = inv_hu;
  }
  const int fi = blockIdx.x * kTileCols + t;
  int first = 0, last = 0;
  bool use = false;
  if (fine && fi < d.nf && worth((double)n, d.nf_all * d.nc)) {
    const float fl = d.f[fi];
    const float r0 = d.rs[o], r1 = d.rs[o + n - 1];
    if (fl == 0.0f) {
      // itype 1: the column is NaN; itype 0: Z0(0) everywhere
      use = ITYPE == 1 || !DY;
      last = ITYPE == 1 ? 0 : 1;
    } else if (fl >= 1e-20f && fl < INFINITY) {
      const double x0 = (double)r0 * fl * inv_hu, x1 = (double)r1 * fl * inv_hu;
      if (x1 < (double)(d.cells_cap - kGroup - (DY ? kDyadic : 0)) && (!DY || x0 >= 0x1p-23)) {
        const Fx fx = make_fx(fl, inv_hu);
        float rel;
        first = locate<DY>(r0, fx, rel);
        last = locate<DY>(r1, fx, rel) + 1;
        use = worth_cells(d, ITYPE, last - first, (double)n);
      }
    }
  }
  if (blockIdx.x == 0) {  // the set's slots of moments chunks
    const long long s0 = slot_begin(d, b), s1 = b + 1 < d.nsets ? slot_begin(d, b + 1) : d.slots;
    for (long long s = s0 + t; s < s1; s += kTileCols) d.slot_set[s] = b;
  }
  const bool has = use && last > first;
  int mn = has ? first : 0x7fffffff, mx = has ? last : 0;
  for (int s = 16; s > 0; s >>= 1) {
    mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, s));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, s));
  }
  if ((t & 31) == 0) {
    ired[t >> 5][0] = mn;
    ired[t >> 5][1] = mx;
  }
  __syncthreads();
  for (int w = 0; w < kWarps; ++w) {
    mn = min(mn, ired[w][0]);
    mx = max(mx, ired[w][1]);
  }
  if (mx <= mn) mn = mx = 0;
  mn &= ~(kGroup - 1);
  mx = (mx + kGroup - 1) & ~(kGroup - 1);
  // a tile with more cells than its share of W goes direct (see layout())
  if (mx - mn > n / 4 + d.tile_cells) {
    use = false;
    mn = mx = 0;
  }
  if (fi < d.nf) d.use[(long long)b * d.nf + fi] = use;
  const int left = __syncthreads_count(fi < d.nf && !use);
  if (t == 0) {
    d.direct[tile] = fine ? left : kBad;
    d.tile[tile].lo = mn;
    d.tile[tile].hi = mx;
  }
}

// Runs of cells [lo, hi): they end at multiples of d.run, so that a column's
// sum does not depend on the tile it is in.
__device__ __forceinline__ int runs_of(const XpDev& d, int lo, int hi) {
  return hi > lo ? (hi + d.run - 1) / d.run - lo / d.run : 0;
}

// One CTA: exclusive sums over the tiles. The columns of a set with distances
// out of order go direct, those of the other sets don't depend on it.
__global__ void __launch_bounds__(1024) xp_scan_kernel(XpDev d) {
  __shared__ long long sw[32], su[32];
  __shared__ int slo[32], shi[32];
  __shared__ long long sleft[32];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int ntile = d.nsets * d.ft;
  long long bw = 0, bu = 0;
  int lo = 0x7fffffff, hi = 0;
  long long left = 0;
  for (int b = t; b < d.nsets; b += 1024) d.set_bad[b] = 0;
  __syncthreads();
  bool bad = false;
  for (int i = t; i < ntile; i += 1024)
    if (d.direct[i] & kBad) {
      d.set_bad[i / d.ft] = 1;
      bad = true;
    }
  bad = __syncthreads_or(bad);
  for (int i0 = 0; i0 < ntile; i0 += 1024) {
    const int i = i0 + t;
    long long w = 0, u = 0;
    if (i < ntile) {
      if (bad && d.set_bad[i / d.ft]) {
        d.tile[i].lo = d.tile[i].hi = 0;
        d.direct[i] = min(kTileCols, d.nf - i % d.ft * kTileCols);
      }
      const int a = d.tile[i].lo, z = d.tile[i].hi;
      w = z - a;
      u = (long long)d.nacc * d.mtiles * runs_of(d, a, z);
      if (z > a) {
        lo = min(lo, a);
        hi = max(hi, z);
      }
      left += d.direct[i];
    }
    long long iw = w, iu = u;
    for (int s = 1; s < 32; s <<= 1) {
      const long long pw = __shfl_up_sync(0xffffffffu, iw, s), pu = __shfl_up_sync(0xffffffffu, iu, s);
      if (lane >= s) {
        iw += pw;
        iu += pu;
      }
    }
    if (lane == 31) {
      sw[wid] = iw;
      su[wid] = iu;
    }
    __syncthreads();
    long long ow = bw, ou = bu;
    for (int k = 0; k < wid; ++k) {
      ow += sw[k];
      ou += su[k];
    }
    if (i < ntile) {
      d.tile[i].w = ow + iw - w;
      d.tile[i].unit = ou + iu - u;
    }
    for (int k = 0; k < 32; ++k) {
      bw += sw[k];
      bu += su[k];
    }
    __syncthreads();
  }
  for (int s = 16; s > 0; s >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, s));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, s));
    left += __shfl_xor_sync(0xffffffffu, left, s);
  }
  if (lane == 0) {
    slo[wid] = lo;
    shi[wid] = hi;
    sleft[wid] = left;
  }
  __syncthreads();
  left = 0;
  for (int k = 0; k < 32; ++k) {
    lo = min(lo, slo[k]);
    hi = max(hi, shi[k]);
    left += sleft[k];
  }
  // (always so: the tiles' shares add up to less)
  const bool ok = bw <= d.blocks_cap && bu <= d.units_cap;
  if (t == 0) {
    d.plan->units = ok ? bu : 0;
    d.plan->blocks = ok ? bw : 0;
    d.plan->left = ok ? left : (long long)d.nsets * d.nf;
    d.plan->lo = ok && hi > lo ? lo : 0;
    d.plan->hi = ok && hi > lo ? hi : 0;
  }
  __syncthreads();
  if (ok) {
    for (int i = t; i < ntile; i += 1024) {
      const int runs = runs_of(d, d.tile[i].lo, d.tile[i].hi);
      int* u = d.unit_tile + d.tile[i].unit;
      for (int k = 0; k < d.nacc * d.mtiles * runs; ++k) u[k] = i;
    }
  }
  if (!ok || bad) {
    const long long ncol = (long long)d.nsets * d.nf;
    for (long long i = t; i < ncol; i += 1024)
      if (!ok || d.set_bad[i / d.nf]) d.use[i] = 0;
  }
}

// ------------------------------------------------------------------ basis
// J0 and Y0 (END: J1, Y1 and the integrals B too) at x = 2 pi cyc >= 8 to about
// 1e-9 of the amplitude, in FP64 (k r reaches 1e4 rad, and E is rounded to FP32
// once): as eval_station_f64, with shorter polynomials and 1 / sqrt(x) by a
// Newton step from FP32 instead of its divisions and square root (the basis of
// 1005 cells x 1000 velocities took 164 us with that, 89 us with this).
template <bool END>
__device__ __forceinline__ void eval_large(double x, double cyc, ZB<double>& J, ZB<double>& Y) {
  const double n = rint(cyc);
  const double a = 4.0 * (cyc - n) - 0.5;
  const double qf = rint(a);
  const int q = (int)qf;
  const double v = a - qf, v2 = v * v;
  constexpr double csn[] = FJC_M64_SIN;
  constexpr double ccs[] = FJC_M64_COS;
  const double s = v * fjs::horner(csn, v2), c = fjs::horner(ccs, v2);
  double sn = q & 1 ? c : s, cs = q & 1 ? s : c;
  if (q & 2) sn = -sn;
  if ((q + 1) & 2) cs = -cs;
  double y = rsqrtf((float)x);
  y = y * fma(-0.5 * x * y, y, 1.5);
  const double s8 = 8.0 * y * y, z = s8 * s8, m = fjs::kSqrt2OverPi * y;
  constexpr double cp[] = FJC_M64_L_P0;
  constexpr double cq[] = FJC_M64_L_Q0;
  const double P = fjs::horner(cp, z) * m, Q = fjs::horner(cq, z) * (s8 * m);
  J.z0 = P * cs - Q * sn;
  Y.z0 = P * sn + Q * cs;
  if (END) {
    constexpr double cp1[] = FJC_M64_L_P1;
    constexpr double cq1[] = FJC_M64_L_Q1;
    constexpr double cr0[] = FJC_M64_L_RHO0;
    constexpr double cr1[] = FJC_M64_L_RHO1;
    const double P1 = fjs::horner(cp1, z) * m, Q1 = fjs::horner(cq1, z) * (s8 * m);
    const double rho0 = fjs::horner(cr0, z), rho1 = fjs::horner(cr1, z) * s8;
    J.z1 = P1 * sn + Q1 * cs;
    Y.z1 = Q1 * sn - P1 * cs;
    J.b = 1.0 + J.z1 * rho0 - J.z0 * rho1;
    Y.b = Y.z1 * rho0 - Y.z0 * rho1;
  }
}

// E: the values of Z0 at the cell's 16 Chebyshev nodes to coefficients. T_4..T_7 and T_12..T_15
// carry a minus sign here and in the moments, where it saves the negation of
// the paired recurrence. One thread per (velocity, cell).
template <int MODE, int ITYPE>
__global__ void __launch_bounds__(kTileRows) xp_basis_kernel(XpDev d) {
  using MT = ModeTraits<MODE>;
  constexpr bool DY = MT::WY;
  __shared__ double dct[kNodes / 2][kNodes];  // [node][term]; node 15 - m by the term's parity
  __shared__ double node[kNodes / 2];         // from the cell's middle
  const int t = threadIdx.x;
  if (t < kNodes / 2 * kNodes) {
    const int m = t / kNodes, n = t % kNodes;
    const double v = cospi(n * (m + 0.5) / kNodes) * (n == 0 ? 1.0 : 2.0) / kNodes;
    dct[m][n] = n & 4 ? -v : v;
  }
  if (t < kNodes / 2) node[t] = cospi((t + 0.5) / kNodes) / (double)kPerHalf;
  __syncthreads();
  if (ITYPE == 1) {
    // V and its flags, which the moments write only where there are end rows
    const long long n4 = d.plan->blocks / kGroup * MT::NIN * (kEndFloats / 4);
    const long long id = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * kTileRows + t;
    const long long all = (long long)gridDim.x * gridDim.y * kTileRows;
    for (long long i = id; i < n4; i += all)
      reinterpret_cast<float4*>(d.V)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (long long i = id; i < d.plan->blocks / kGroup; i += all) d.ends[i] = 0;
  }
  const int lo = d.plan->lo, hi = d.plan->hi;
  const double hu = d.plan->hu;
  const int j = blockIdx.x * kTileRows + t;
  const double per_c = j < d.nc ? hu / (double)d.c[j] : 0.0;  // cycles per cell
  for (int cell = lo + blockIdx.y; cell < hi; cell += gridDim.y) {
    double eJ[kNodes], eY[kNodes];
#pragma unroll
    for (int n = 0; n < kNodes; ++n) eJ[n] = eY[n] = 0.0;
    const double x0 = cell_begin<DY>(cell), len = cell_len<DY>(cell);
    if (j < d.nc) {
      auto values = [&](double at, double& J0, double& Y0) {
        const double cyc = fma(len, at, x0) * per_c, x = fjs::kTwoPi * cyc;
        ZB<double> J{}, Y{};
        if (x >= 8.0)
          eval_large<false>(x, cyc, J, Y);
        else
          fjs::eval_station_f64<MT::WJ, MT::WY, false>(x, cyc, J, Y);
        J0 = J.z0;
        Y0 = Y.z0;
      };
#pragma unroll 1
      for (int m = 0; m < kNodes / 2; ++m) {
        double ja = 0.0, ya = 0.0, jb = 0.0, yb = 0.0;
        values(kCentre + node[m], ja, ya);
        values(kCentre - node[m], jb, yb);
        const double js = ja + jb, jd = ja - jb, ys = ya + yb, yd = ya - yb;
#pragma unroll
        for (int n = 0; n < kNodes; ++n) {
          const double w = dct[m][n];
          if (MT::WJ) eJ[n] = fma(w, n & 1 ? jd : js, eJ[n]);
          if (MT::WY) eY[n] = fma(w, n & 1 ? yd : ys, eY[n]);
        }
      }
    }
    const long long plane = (long long)d.cells_cap * kNodes * d.ncp;
    float4* e = reinterpret_cast<float4*>(
        d.E + (((long long)cell * d.mtiles + blockIdx.x) * kTileRows + t) * kNodes);
#pragma unroll
    for (int n = 0; n < kNodes; n += 4) {
      if (MT::WJ)
        e[n / 4] = make_float4((float)eJ[n], (float)eJ[n + 1], (float)eJ[n + 2], (float)eJ[n + 3]);
      if (MT::WY)
        e[(MT::WJ ? plane / 4 : 0) + n / 4] =
            make_float4((float)eY[n], (float)eY[n + 1], (float)eY[n + 2], (float)eY[n + 3]);
    }
    if (ITYPE == 1) {
      // the cell's end, with r in cells and k = 2 pi per_c
      ZB<double> J{}, Y{};
      double r1 = 0.0, r2J = 0.0, r2Y = 0.0, r1Y = 0.0;
      if (j < d.nc) {
        const double x = x0 + len, cyc = x * per_c, ik = 1.0 / (fjs::kTwoPi * per_c);
        if (cyc >= 8.0 / fjs::kTwoPi)
          eval_large<true>(fjs::kTwoPi * cyc, cyc, J, Y);
        else
          fjs::eval_station_f64<MT::WJ, MT::WY, true>(fjs::kTwoPi * cyc, cyc, J, Y);
        r1 = x * J.z1 * ik;
        r2J = (x * J.z0 - J.b * ik) * ik * ik;
        r1Y = x * Y.z1 * ik;
        r2Y = (x * Y.z0 - Y.b * ik) * ik * ik;
      }
      const long long eplane = (long long)d.cells_cap * kEndRows * d.ncp;
      float* v = d.Eend +
                 (((long long)(cell / kGroup) * d.mtiles + blockIdx.x) * kTileRows + t) *
                     (kGroup * kEndRows) +
                 (cell & (kGroup - 1)) * kEndRows;
      if (MT::WJ) *reinterpret_cast<float2*>(v) = make_float2((float)r1, (float)r2J);
      if (MT::WY)
        *reinterpret_cast<float2*>(v + (MT::WJ ? eplane : 0)) = make_float2((float)r1Y, (float)r2Y);
    }
  }
}

// ---------------------------------------------------------------- moments
// acc[m] += a (T_2m, T_2m+1) (signed as above) at t. The pairs follow the
// recurrence of step 2, T_{n+2} = 2 T_2 T_n - T_{n-2}; the signs turn it into
// R_{m+1} = -+ (2 T_2) R_m + R_{m-1}. With one input the recurrence runs on
// a R_m itself.
template <int NIN>
__device__ __forceinline__ void add_point(float2 (&acc)[NIN][kNodes / 2], float t,
                                          const float (&a)[NIN]) {
  const float dt = t + t;
  const float t2 = fmaf(dt, t, -1.0f);
  const float t3 = fmaf(dt, t2, -t);
  const float2 s = fjs::psplat(t2 + t2), ns = fjs::psplat(-(t2 + t2));
  float2 p = make_float2(1.0f, t), q = make_float2(t2, t3);
  if (NIN == 1) {
    p = make_float2(a[0], a[0] * t);
    q = make_float2(a[0] * t2, a[0] * t3);
  }
#pragma unroll
  for (int m = 0; m < kNodes / 2; ++m) {
    if (NIN == 1) {
      acc[0][m] = fjs::padd(acc[0][m], p);
    } else {
#pragma unroll
      for (int k = 0; k < NIN; ++k) acc[k][m] = fjs::pfma(fjs::psplat(a[k]), p, acc[k][m]);
    }
    const float2 n = fjs::pfma(m & 1 ? s : ns, q, p);  // R_{m+2}
    p = q;
    q = n;
  }
}

// Gauss rules of 5 and 9 points, one after the other: (x, weight).
__constant__ float2 kRule[14] = {
    {-0.906179846f, 0.236926885f}, {-0.538469310f, 0.478628670f}, {0.0f, 0.568888889f},
    {0.538469310f, 0.478628670f},  {0.906179846f, 0.236926885f},
    {-0.968160240f, 0.081274388f}, {-0.836031107f, 0.180648161f}, {-0.613371433f, 0.260610696f},
    {-0.324253423f, 0.312347077f}, {0.0f, 0.330239355f},          {0.324253423f, 0.312347077f},
    {0.613371433f, 0.260610696f},  {0.836031107f, 0.180648161f},  {0.968160240f, 0.081274388f}};

// One point of a piece: its middle tm and half length th in the cell's t, in r
// rm and hr; the spectrum's value gm at the middle and its rise gh over half
// the piece.
template <int NIN>
__device__ __forceinline__ void piece_point(float2 (&acc)[NIN][kNodes / 2], float x, float w,
                                            float tm, float th, float rm, float hr,
                                            const float (&gm)[NIN], const float (&gh)[NIN]) {
  float a[NIN];
  const float rw = fmaf(hr, x, rm) * (hr * w);
#pragma unroll
  for (int k = 0; k < NIN; ++k) a[k] = fmaf(gh[k], x, gm[k]) * rw;
  add_point<NIN>(acc, fmaf(th, x, tm), a);
}

// A CTA is one warp; it takes 32 frequencies and a chunk of stations. Chunk q
// visits the stations after q chunk up to (q + 1) chunk (chunk 0 of itype 0 its
// first station too), and for itype 1 the intervals that end there. Its lanes
// keep the 16 moments of the cell they are in; a finished cell that the chunk
// has to itself goes to W, the first one to head, the last one to tail (their
// numbers to span).
//
// An interval (or the piece of it in one cell) takes the Gauss rule of 2, 3, 5
// or 9 points by its length d in cells: each rule is at most 5e-8 of the
// integral off where the next one begins, at 0.1, 0.6, 2.5 and 9.8 radians. A
// short interval is not cut at a cell's end: since the lanes' cells end at
// different stations, cutting each one ran two pieces in nearly every step.
//
// Bound by issue (66% of the slots at 19,900 pairs x 2048 f, with 17 warps an SM)
// and the FMA pipe's throttle: 15 paired multiply-adds and about as many other
// instructions a point, 2 or 3 points for most intervals. The spectra come in by cp.async,
// 16 stations ahead; unrolling the stations instead (loads into registers)
// left the warps waiting for instructions as long as they issued. A lane of
// short intervals follows its cell by one compare with the next one's start
// (locate() only after a long interval), and the zeros of V come from the basis
// kernel: 19,900 pairs x 2048 f 472 us with a locate() and V in every step,
// 435 us so; 20 subarrays 1884 and 1755 us.
constexpr int kMomStations = 16;
template <int NIN>
struct MomStage {
  float g[NIN][kMomStations][32];  // [station][frequency]
  float4 st[kMomStations];  // r, the interval's length, 1 / max(length, 0.1), trapezoid weight
};

template <int NIN, int ITYPE, bool DY>
__global__ void __launch_bounds__(32, NIN == 1 ? 24 : 16) xp_moments_kernel(XpDev d, int ftiles) {
  __shared__ __align__(16) MomStage<NIN> stage[2];
  __shared__ float2 rule[14];
  __shared__ float2 tot[NIN][kNodes / 2][32];  // sums of earlier stations of the lane's cell
  const int lane = threadIdx.x;
  const long long slot = blockIdx.x / ftiles;
  const int fi = (int)(blockIdx.x % ftiles) * 32 + lane;
  const int b = d.slot_set[slot];
  const long long o = set_begin(d, b);
  const int n = (int)(set_end(d, b) - o);
  const int q = (int)(slot - slot_begin(d, b));
  if (q >= chunks_of(d, n)) return;
  const bool mine = fi < d.nf && d.use[(long long)b * d.nf + fi] != 0 &&
                    !(ITYPE == 1 && d.f[fi] == 0.0f);
  if (__all_sync(0xffffffffu, !mine)) return;
  if (lane < 14) rule[lane] = kRule[lane];
  const int fc = min(fi, d.nf - 1);
  const float fl = mine ? d.f[fc] : 0.0f;
  const Fx fx = make_fx(fl, d.plan->inv_hu);
  const float huf = ITYPE == 1 ? (float)(d.plan->hu / (double)(mine ? fl : 1.0f)) : 0.0f;
  const XpTile tile = d.tile[b * d.ft + fc / kTileCols];
  const int s0 = q * d.chunk, s1 = min(s0 + d.chunk, n - 1);
  const float* const rs = d.rs + o;
  float2 acc[NIN][kNodes / 2];
#pragma unroll
  for (int k = 0; k < NIN; ++k)
#pragma unroll
    for (int m = 0; m < kNodes / 2; ++m) acc[k][m] = make_float2(0.f, 0.f);
  bool more = false;  // tot holds part of the cell's sums
  float vA;
  int cell = locate<DY>(rs[s0], fx, vA);
  const int cell0 = cell;
  float base_x = cell_begin<DY>(cell);
  const long long edge = ((slot * d.nf + fc) * NIN) * kNodes;
  // where the current cell goes, and the next one
  float* here = d.head + edge;
  long long here_step = kNodes;
  float* next = d.W + (tile.w + cell + 1 - tile.lo) * NIN * kBlockFloats + (fc & (kTileCols - 1)) * kNodes;
  float* const V = d.V + (tile.w / kGroup) * NIN * kEndFloats + (fc & (kTileCols - 1)) * kGroup * kEndRows;
  auto store = [&](float* base, long long step) {
    if (more) {
#pragma unroll
      for (int k = 0; k < NIN; ++k)
#pragma unroll
        for (int m = 0; m < kNodes / 2; ++m) acc[k][m] = fjs::padd(acc[k][m], tot[k][m][lane]);
      more = false;
    }
#pragma unroll
    for (int k = 0; k < NIN; ++k) {
      float4* p = reinterpret_cast<float4*>(base + k * step);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        p[m] = make_float4(acc[k][2 * m].x, acc[k][2 * m].y, acc[k][2 * m + 1].x,
                           acc[k][2 * m + 1].y);
        acc[k][2 * m] = acc[k][2 * m + 1] = make_float2(0.f, 0.f);
      }
    }
  };
  auto flush = [&]() {  // the cell is finished
    store(here, here_step);
    here = next;
    here_step = kBlockFloats;
    next += NIN * kBlockFloats;
    ++cell;
    if (DY)
      base_x = cell_begin<DY>(cell);
    else
      base_x += 1.0f;
  };
  const float* u[NIN];
#pragma unroll
  for (int k = 0; k < NIN; ++k) u[k] = d.in[k].p + (long long)fc * d.in[k].cs;
  auto row_of = [&](int k, int i) -> long long {
    const long long* perm = d.in[k].perm;
    return (perm ? __ldg(perm + o + i) : o + i) * d.in[k].ld;
  };
  // stations base .. base + 15 (each lane one station's numbers, all lanes
  // every station's spectrum)
  auto load = [&](int base, int buf) {
    const int i = min(base + (lane & (kMomStations - 1)), s1);
    const float r = rs[i];
    const float D = ITYPE == 1 ? r - rs[i - 1] : 0.0f;
    if (lane < kMomStations)
      stage[buf].st[lane] = make_float4(r, D, 1.0f / fmaxf(D, 0.1f), ITYPE == 0 ? d.wtr[o + i] : 0.0f);
    long long row[NIN];
#pragma unroll
    for (int k = 0; k < NIN; ++k) row[k] = row_of(k, i);
    const int cnt = min(kMomStations, s1 - base + 1);
    for (int j = 0; j < cnt; ++j)
#pragma unroll
      for (int k = 0; k < NIN; ++k)
        cp_async4(&stage[buf].g[k][j][lane], u[k] + __shfl_sync(0xffffffffu, row[k], j));
    cp_async_commit();
  };
  if (s0 + 1 <= s1) load(s0 + 1, 0);
  float gA[NIN];
#pragma unroll
  for (int k = 0; k < NIN; ++k) gA[k] = __ldg(u[k] + row_of(k, s0));
  if (ITYPE == 0 && q == 0 && mine) {
    float a[NIN];
#pragma unroll
    for (int k = 0; k < NIN; ++k) a[k] = gA[k] * d.wtr[o];
    add_point<NIN>(acc, vA * kPerHalf, a);
  }
  int buf = 0;
  for (int base = s0 + 1; base <= s1; base += kMomStations, buf ^= 1) {
    if (base + kMomStations <= s1)
      load(base + kMomStations, buf ^ 1);
    else
      cp_async_commit();  // one group per round keeps the count below
    cp_async_wait<1>();
    __syncwarp();
    const int cnt = mine ? min(kMomStations, s1 - base + 1) : 0;
    const int mark = cell;
#pragma unroll 1
    for (int j = 0; j < cnt; ++j) {
      const float4 st = stage[buf].st[j];
      const float rB = st.x, D = st.y;
      float gB[NIN], gm[NIN], gh[NIN], vB;
#pragma unroll
      for (int k = 0; k < NIN; ++k) gB[k] = stage[buf].g[k][j][lane];
      // itype 1: a short interval whole, in the cell of its far end; a long one
      // from its beginning to the first cell end, from the last cell end on,
      // and between the two in closed form. (Lanes that end a cell do so before
      // all lanes' points.)
      float dB = D * fx.hi;
      int cB = 0;
      const bool dyadic = DY && cell < kDyadic;
      if (dyadic) {
        cB = locate<DY>(rB, fx, vB);
        dB /= cell_len<DY>(cB);
      }
      if (ITYPE == 0 || dB <= kShort) {
        if (dyadic) {
#pragma unroll 1
          while (cell < cB) flush();
        } else {
          // the station's cell and place, as locate() finds them, from the cell
          // that the lane is in
          const Place x = place_of(rB, fx);
#pragma unroll 1
          while (reached(x, base_x + 1.0f)) flush();
          vB = (x.p - (base_x + kCentre)) + x.l;
        }
        if (ITYPE == 0) {
#pragma unroll
          for (int k = 0; k < NIN; ++k) gm[k] = gB[k] * st.w;
          add_point<NIN>(acc, vB * kPerHalf, gm);
        } else {
          const float hr = 0.5f * D, th = 0.5f * kPerHalf * dB;
          const float tm = fmaf(vB, kPerHalf, -th), rm = rB - hr;
#pragma unroll
          for (int k = 0; k < NIN; ++k) {
            // over the reference's floor of an interval (src/FJcpu.cpp:259)
            gh[k] = (gB[k] - gA[k]) * (st.z * hr);
            gm[k] = gA[k] + gh[k];
          }
          if (dB <= 0.01f) {
            piece_point<NIN>(acc, -0.577350269f, 1.0f, tm, th, rm, hr, gm, gh);
            piece_point<NIN>(acc, 0.577350269f, 1.0f, tm, th, rm, hr, gm, gh);
          } else {
            piece_point<NIN>(acc, -0.774596669f, 0.555555556f, tm, th, rm, hr, gm, gh);
            piece_point<NIN>(acc, 0.0f, 0.888888889f, tm, th, rm, hr, gm, gh);
            piece_point<NIN>(acc, 0.774596669f, 0.555555556f, tm, th, rm, hr, gm, gh);
          }
        }
      } else {
        if (!dyadic) cB = locate<DY>(rB, fx, vB);
        const int span = cB - cell;
#pragma unroll 1
        for (int step = 0;; ++step) {
          const bool cross = step < span;
          float hr = 0.0f;
          if (!cross || step == 0) {
            const float va = step == 0 ? vA : -kCentre;
            const float w = (cross ? 1.0f - kCentre : vB) - va;  // in cells
            const float cl = cell_len<DY>(cell);
            hr = span == 0 ? 0.5f * D : 0.5f * w * cl * huf;
            const float th = 0.5f * kPerHalf * w, tm = fmaf(va, kPerHalf, th);
            const float rm = fmaf(cl, fmaf(0.5f, w, va) + kCentre, cell_begin<DY>(cell)) * huf;
#pragma unroll
            for (int k = 0; k < NIN; ++k) {
              const float sl = (gB[k] - gA[k]) * st.z;
              gm[k] = fmaf(sl, cross || span == 0 ? hr : D - hr, gA[k]);
              gh[k] = sl * hr;
            }
            const bool five = w <= 0.25f;
#pragma unroll 1
            for (int i = five ? 0 : 5; i < (five ? 5 : 14); ++i)
              piece_point<NIN>(acc, rule[i].x, rule[i].y, tm, th, rm, hr, gm, gh);
          }
          if (!cross) break;
          if (span > 1 && (step == 0 || step == span - 1)) {
            // the cell end's weights: the spectrum's line there, from A, or from B
            // back, and its slope
            const int at = cell - tile.lo;
            float* v = V + (long long)(at / kGroup) * (NIN * kEndFloats) + (at & (kGroup - 1)) * kEndRows;
            const float back = (vB + kCentre) * cell_len<DY>(cB) * huf;
            const float h2 = step == 0 ? -huf * huf : huf * huf;
#pragma unroll
            for (int k = 0; k < NIN; ++k) {
              const float sl = (gB[k] - gA[k]) * st.z;
              *reinterpret_cast<float2*>(v + k * kEndFloats) =
                  make_float2(h2 * fmaf(sl, step == 0 ? 2.0f * hr : D - back, gA[k]), h2 * huf * sl);
            }
            d.ends[(tile.w + at) / kGroup] = 1;
          }
          flush();
        }
      }
#pragma unroll
      for (int k = 0; k < NIN; ++k) gA[k] = gB[k];
      vA = vB;
    }
    // many stations to a cell (low frequencies): sums of 16 stations, added up
    if (cell == mark) {
#pragma unroll
      for (int k = 0; k < NIN; ++k)
#pragma unroll
        for (int m = 0; m < kNodes / 2; ++m) {
          tot[k][m][lane] = more ? fjs::padd(tot[k][m][lane], acc[k][m]) : acc[k][m];
          acc[k][m] = make_float2(0.f, 0.f);
        }
      more = true;
    }
    __syncwarp();  // the stage is filled again
  }
  if (!mine) return;
  store((cell == cell0 ? d.head : d.tail) + edge, kNodes);
  d.span[slot * d.nf + fi] = make_int2(cell0, cell);
}

// Adds the parts of the cells that lie across chunk boundaries, in chunk
// order, and clears the cells of the tile that a column does not reach. That is
// shared by a chunk for 32 cells, up to kClear chunks: by the first and the last
// one alone it was a chain of stores as long as the tile (279 records x 105 f
// over 1116 cells: 71 us, 20 us so). Bound by latency, so six CTAs an SM: with the
// registers for four, 128 subarrays took 50 us longer. Four threads per (slot,
// frequency). The first chunk that begins in a cell adds all that the cell got:
// the tail of the chunk before it, its own head, and the heads of the chunks
// after it that begin in the same cell.
constexpr int kClear = 32;
template <int NIN, int ITYPE, bool DY>
__global__ void __launch_bounds__(256, 6) xp_join_kernel(XpDev d) {
  const int n4 = threadIdx.x & 3;
  const int fi = blockIdx.y * 64 + (threadIdx.x >> 2);
  const long long slot = blockIdx.x;
  if (fi >= d.nf) return;
  const int b = d.slot_set[slot];
  const int n = (int)(set_end(d, b) - set_begin(d, b));
  const int q = (int)(slot - slot_begin(d, b)), nch = chunks_of(d, n);
  if (q >= nch || !d.use[(long long)b * d.nf + fi]) return;
  if (ITYPE == 1 && d.f[fi] == 0.0f) return;
  const int2* span = d.span + slot * d.nf + fi;  // of chunk q + i: span[i nf]
  const int2 me = span[0];
  const int before = q > 0 ? span[-(long long)d.nf].x : -1;
  if (before == me.x && q != nch - 1 && q >= kClear) return;
  const XpTile tile = d.tile[b * d.ft + fi / kTileCols];
  float* const col = d.W + (fi & (kTileCols - 1)) * kNodes + n4 * 4;
  auto put = [&](int cell, int k, float4 v) {
    *reinterpret_cast<float4*>(col + ((tile.w + cell - tile.lo) * NIN + k) * kBlockFloats) = v;
  };
  const long long step = (long long)d.nf * NIN * kNodes;
  const long long at = ((slot * d.nf + fi) * NIN) * kNodes + n4 * 4;
  auto add = [](float4& v, const float* p) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p));
    v = make_float4(v.x + a.x, v.y + a.y, v.z + a.z, v.w + a.w);
  };
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const int share = min(nch, max(1, min(kClear, (tile.hi - tile.lo) / 32)));
  if (q < share) {
    const int first = span[-(long long)q * d.nf].x, last = span[(long long)(nch - 1 - q) * d.nf].y;
    for (int c = tile.lo + q; c < tile.hi; c += share)
      if (c < first || c > last) {
#pragma unroll
        for (int k = 0; k < NIN; ++k) put(c, k, zero);
      }
  }
  if (before == me.x && q != nch - 1) return;
  if (before != me.x) {
#pragma unroll
    for (int k = 0; k < NIN; ++k) {
      float4 v = zero;
      if (q > 0) add(v, d.tail + at - step + k * kNodes);
      add(v, d.head + at + k * kNodes);
      // eight chunks' loads at a time (many stations to a cell: low frequencies)
      for (int c = 1; q + c < nch; c += 8) {
        float4 h[8];
        bool in[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int cc = min(c + i, nch - 1 - q);
          in[i] = q + c + i < nch && span[(long long)cc * d.nf].x == me.x;
          h[i] = __ldg(reinterpret_cast<const float4*>(d.head + at + cc * step + k * kNodes));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (in[i]) v = make_float4(v.x + h[i].x, v.y + h[i].y, v.z + h[i].z, v.w + h[i].w);
        if (!in[7]) break;
      }
      put(me.x, k, v);
    }
  }
  if (q == nch - 1) {
    if (me.y != me.x) {
#pragma unroll
      for (int k = 0; k < NIN; ++k) {
        float4 v = zero;
        add(v, d.tail + at + k * kNodes);
        put(me.y, k, v);
      }
    }
  }
}

// ------------------------------------------------------------------- GEMM
// Units of 128 velocities x 128 columns x up to `run` cells on the tensor
// cores, kind::tf32. An FP32 operand x is split into hi (its 11 leading bits,
// rounded) and lo = x - hi, which keep 22 of its 24 bits and all of its range
// (no scales, as a split into fp16 halves would need), and the product is
// hi hi + hi lo + lo hi with FP32 accumulation. The tensor core truncates each
// sum, so hi hi is taken out of tensor memory after every group of four cells
// (8 steps) and added in FP32 registers; the two small products, 2^-11 of it,
// have an accumulator of their own that is read once, at the unit's end.
//
// One persistent CTA per SM, by warps: 8 that drain tensor memory (each 32
// rows x 64 columns of the totals), 8 that bring the operands in (global to
// registers, split, to shared memory as 8 x 16 byte core matrices), one that
// issues the MMAs. Four stages of one step each: a cell (K = 16) or a group's
// end rows (K = 8). No unit is full: at 19,900 pairs x 2048 f x 1000 c (335 us; 884
// us with FP32 multiply-adds, 128 x 64 tiles, 8 x 8 a thread, paired) the tensor
// pipe is active 36% of the time, the loaders' stores (32 KB a step) and the
// drains take 39% of the shared memory's wavefronts beside the 48 KB a step that
// the MMAs read, and the largest stall is the loaders' wait for L2.
//
// Every wait is bounded. One that runs out sets `abort`, the other roles then
// run out or see it, the unit's sums become NaN, and g_xp_error and the call's
// own flag are set.
__device__ unsigned int g_xp_error = 0;
constexpr int kDrainWarps = 8, kLoadWarps = 8;
constexpr int kGemmThreads = 32 * (kDrainWarps + kLoadWarps + 1);
constexpr int kStages = 4;
constexpr int kLbo = kTileRows * 16 + 32;       // bytes between core matrices along K (padded)
constexpr int kPlane = 4 * kLbo;                // one operand's hi or lo part, K = 16
constexpr int kStageBytes = 4 * kPlane;         // A hi, A lo, B hi, B lo
constexpr int kGemmSmem = kStages * kStageBytes + 1024;
static_assert(kTileRows == kTileCols, "one loader serves both operands");

__device__ __forceinline__ uint32_t instr_desc_tf32() {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(kTileCols >> 3) << 17) |
         ((uint32_t)(kTileRows >> 4) << 24);
}
__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}
// x rounded to 11 bits (half up; a NaN or an infinity stays one), and the rest
__device__ __forceinline__ void split_tf32(float x, float& hi, float& lo) {
  hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
  lo = x - hi;
}

// A unit: its tile, velocity tile, result and cells.
struct Unit {
  XpTile tile;
  int mt, q, c0, c1;
  unsigned ends;  // its groups that have end rows
};
__device__ __forceinline__ Unit unit_at(const XpDev& d, long long unit) {
  Unit u;
  u.tile = d.tile[d.unit_tile[unit]];
  const int rest = (int)(unit - u.tile.unit);
  u.mt = rest % d.mtiles;
  u.q = (rest / d.mtiles) % d.nacc;
  const int run = u.tile.lo / d.run + rest / (d.mtiles * d.nacc);
  u.c0 = max(u.tile.lo, run * d.run);
  u.c1 = min((run + 1) * d.run, u.tile.hi);
  const int g = u.c0 + (threadIdx.x & 31) * kGroup;
  u.ends = __ballot_sync(0xffffffffu, d.has_ends && g < u.c1 &&
                                          d.ends[(u.tile.w + g - u.tile.lo) / kGroup] != 0);
  return u;
}
// The steps of a unit: a group's four cells (sub 0 .. 3) and, if it has them,
// its end rows (sub 4, cell then the first one after the group), each for
// every source.
struct Step {
  int cell, sub, src;
};
template <int NSRC>
__device__ __forceinline__ Step next_step(Step p, const Unit& u) {
  if (++p.src < NSRC) return p;
  p.src = 0;
  if (p.sub < kGroup) ++p.cell;
  ++p.sub;
  if (p.sub == kGroup && !(u.ends >> ((p.cell - u.c0) / kGroup - 1) & 1)) ++p.sub;
  if (p.sub > kGroup) p.sub = 0;
  return p;
}
__device__ __forceinline__ bool in_unit(const Step& p, const Unit& u) {
  return p.cell < u.c1 || p.sub == kGroup;
}

template <int NSRC>
__global__ void __launch_bounds__(kGemmThreads, 1) xp_gemm_kernel(XpDev d) {
  extern __shared__ __align__(1024) unsigned char smem[];
  // full[4] empty[4] acc_full[2] acc_empty[2] low_empty done
  __shared__ __align__(8) uint64_t bars[2 * kStages + 6];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  uint64_t* const full = bars;
  uint64_t* const empty = bars + kStages;
  uint64_t* const acc_full = bars + 2 * kStages;
  uint64_t* const acc_empty = acc_full + 2;
  uint64_t* const low_empty = acc_full + 4;
  uint64_t* const done = acc_full + 5;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kMmaWarp = kDrainWarps + kLoadWarps;
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      tc::mbar_init(full + i, kLoadWarps);
      tc::mbar_init(empty + i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(acc_full + i, 1);
      tc::mbar_init(acc_empty + i, kDrainWarps);
    }
    tc::mbar_init(low_empty, kDrainWarps);
    tc::mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc::smem_u32(&tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const long long units = d.plan->units;
  const int nin = d.nacc > NSRC ? d.nacc : NSRC;

  // false (for the whole warp) once a wait has run out anywhere
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    bool ok = true;
    if (!tc::mbar_try_wait(bar, parity)) {
      const long long t0 = clock64();
      while (ok && !tc::mbar_try_wait(bar, parity))
        if (abort_flag || clock64() - t0 > d.wait_cycles) ok = false;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) abort_flag = 1;
    return ok;
  };

  if (warp < kDrainWarps) {
    // ---------------------------------------------------------------- drain
    const int half = warp >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * 64);
    uint32_t groups = 0, n = 0;
    bool ok = true;
    for (long long unit = blockIdx.x; unit < units; unit += gridDim.x, ++n) {
      const Unit u = unit_at(d, unit);
      float tot[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) tot[j] = 0.0f;
      auto add = [&](uint32_t column) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          float v[16];
          tc::tmem_ld16(lane_base + column + h * 16, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) tot[h * 16 + j] += v[j];
        }
      };
      for (int c = u.c0; ok && c < u.c1; c += kGroup, ++groups) {
        const uint32_t b = groups & 1;
        ok = wait(acc_full + b, (groups >> 1) & 1);
        if (!ok) break;
        tc::tc_fence_after();
        add(b * kTileCols);
        if (c + kGroup >= u.c1) {  // the unit's last group: its commit covers the low products
          add(2 * kTileCols);
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(low_empty);
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty + b);
      }
      float4* o = reinterpret_cast<float4*>(d.part + unit * (kTileRows * kTileCols) +
                                            row * kTileCols + half * 64);
      const float bad = __int_as_float(0x7fffffff);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        o[j] = ok ? make_float4(tot[4 * j], tot[4 * j + 1], tot[4 * j + 2], tot[4 * j + 3])
                  : make_float4(bad, bad, bad, bad);
    }
  } else if (warp < kMmaWarp) {
    // ----------------------------------------------------------------- load
    const int lt = tid - 32 * kDrainWarps;
    const long long plane = (long long)d.cells_cap * kNodes * d.ncp;
    uint32_t it = 0;
    bool ok = true;
    for (long long unit = d.no_load ? units : blockIdx.x; ok && unit < units; unit += gridDim.x) {
      const Unit u = unit_at(d, unit);
      struct Raw {
        float4 a[2], b[2];
      };
      auto fetch = [&](const Step& p, Raw& r) {
        const int in = NSRC == 2 && p.src ? 1 - u.q : u.q;
        if (p.sub < kGroup) {
          const float4* e = reinterpret_cast<const float4*>(
              d.E + (p.src ? plane : 0) +
              ((long long)p.cell * d.mtiles + u.mt) * (kTileRows * kNodes));
          const float4* w = reinterpret_cast<const float4*>(
              d.W + ((u.tile.w + p.cell - u.tile.lo) * nin + in) * kBlockFloats);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            r.a[i] = __ldg(e + lt + i * 256);
            r.b[i] = __ldg(w + lt + i * 256);
          }
        } else {
          const int g = p.cell - kGroup;
          r.a[0] = __ldg(reinterpret_cast<const float4*>(
                             d.Eend + (p.src ? plane / kNodes * kEndRows : 0) +
                             ((long long)(g / kGroup) * d.mtiles + u.mt) *
                                 (kTileRows * kGroup * kEndRows)) + lt);
          r.b[0] = __ldg(reinterpret_cast<const float4*>(
                             d.V + ((u.tile.w + g - u.tile.lo) / kGroup * nin + in) * kEndFloats) + lt);
        }
      };
      // splits and stores a step; false when a wait ran out
      auto put = [&](const Step& p, const Raw& r) {
        const uint32_t s = it % kStages;
        if (it >= kStages && !wait(empty + s, (it / kStages - 1) & 1)) return false;
        const float sg = NSRC == 2 && p.src && u.q == 0 ? -1.0f : 1.0f;
        unsigned char* st = smem + s * kStageBytes;
        const bool ends = p.sub == kGroup;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (i == 1 && ends) break;
          const int v = lt + i * 256;
          const int off = ends ? (v & 1) * kLbo + (v >> 1) * 16 : (v & 3) * kLbo + (v >> 2) * 16;
          float4 h, l;
          split_tf32(r.a[i].x, h.x, l.x);
          split_tf32(r.a[i].y, h.y, l.y);
          split_tf32(r.a[i].z, h.z, l.z);
          split_tf32(r.a[i].w, h.w, l.w);
          *reinterpret_cast<float4*>(st + off) = h;
          *reinterpret_cast<float4*>(st + kPlane + off) = l;
          split_tf32(sg * r.b[i].x, h.x, l.x);
          split_tf32(sg * r.b[i].y, h.y, l.y);
          split_tf32(sg * r.b[i].z, h.z, l.z);
          split_tf32(sg * r.b[i].w, h.w, l.w);
          *reinterpret_cast<float4*>(st + 2 * kPlane + off) = h;
          *reinterpret_cast<float4*>(st + 3 * kPlane + off) = l;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(full + s);
        ++it;
        return true;
      };
      // the loads run three steps ahead of their use (a step's MMAs take less
      // than the latency of L2)
      Raw raw[3];
      Step at[3];
      at[0] = Step{u.c0, 0, 0};
      bool on[3] = {true, false, false};
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        if (i > 0 && on[i - 1]) {
          at[i] = next_step<NSRC>(at[i - 1], u);
          on[i] = in_unit(at[i], u);
        }
        if (on[i]) fetch(at[i], raw[i]);
      }
      while (ok && on[0]) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if (!on[i]) break;
          if (!(ok = put(at[i], raw[i]))) break;
          const int last = (i + 2) % 3;  // the furthest step that is fetched
          on[i] = on[last];
          if (on[i]) {
            at[i] = next_step<NSRC>(at[last], u);
            on[i] = in_unit(at[i], u);
            if (on[i]) fetch(at[i], raw[i]);
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ MMA
    // One thread. The descriptors differ in their address field alone, so a
    // step's are sums of 32-bit words (formed anew for each MMA they took
    // longer than the MMAs).
    const uint32_t idesc = instr_desc_tf32();
    const uint64_t desc0 = tc::smem_desc(smem, kLbo, 128);
    const uint32_t desc_hi = (uint32_t)(desc0 >> 32);
    const uint32_t low = tmem + 2 * kTileCols;
    uint32_t it = 0, groups = 0, n = 0;
    int ok = 1;
    auto wait1 = [&](uint64_t* bar, uint32_t parity) {
      if (tc::mbar_try_wait(bar, parity)) return true;
      const long long t0 = clock64();
      while (!tc::mbar_try_wait(bar, parity))
        if (abort_flag || clock64() - t0 > d.wait_cycles) {
          abort_flag = 1;
          return false;
        }
      return true;
    };
    for (long long unit = blockIdx.x; ok && unit < units; unit += gridDim.x, ++n) {
      const Unit u = unit_at(d, unit);
      if (lane == 0) {
        if (n > 0) ok = wait1(low_empty, (n - 1) & 1);
        uint32_t low_on = 0;
        for (int c = u.c0; ok && c < u.c1; c += kGroup, ++groups) {
          const uint32_t top = tmem + (groups & 1) * kTileCols;
          if (groups >= 2 && !(ok = wait1(acc_empty + (groups & 1), ((groups >> 1) - 1) & 1))) break;
          const int cells = kGroup * NSRC;
          const int steps = cells + ((u.ends >> ((c - u.c0) / kGroup)) & 1 ? NSRC : 0);
          uint32_t top_on = 0;
          for (int step = 0; step < steps; ++step, ++it) {
            const uint32_t s = it % kStages;
            if (!(ok = wait1(full + s, (it / kStages) & 1))) break;
            // the loaders' stores before the tensor core's reads; here rather than
            // in the loaders, where the fence would wait for their loads in flight
            tc::fence_async_smem();
            tc::tc_fence_after();
            const uint32_t ah = (uint32_t)desc0 + s * (kStageBytes >> 4);
            auto desc = [&](uint32_t at) { return ((uint64_t)desc_hi << 32) | at; };
            auto mma3 = [&](uint32_t k, uint32_t on_low, uint32_t on_top) {
              const uint64_t dah = desc(ah + k), dal = desc(ah + k + (kPlane >> 4));
              const uint64_t dbh = desc(ah + k + 2 * (kPlane >> 4)), dbl = desc(ah + k + 3 * (kPlane >> 4));
              mma_tf32(low, dal, dbh, idesc, on_low);
              mma_tf32(low, dah, dbl, idesc, 1u);
              mma_tf32(top, dah, dbh, idesc, on_top);
            };
            mma3(0, low_on, top_on);
            if (step < cells) mma3(2 * kLbo >> 4, 1u, 1u);
            tc::mma_commit(empty + s);
            low_on = top_on = 1;
          }
          if (ok) tc::mma_commit(acc_full + (groups & 1));
        }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
    }
    if (!ok) {
      // no MMA may be in flight when the tensor memory goes
      if (lane == 0) {
        tc::mma_commit(done);
        tc::mbar_wait(done, 0, tc::kWaitCycles);
      }
      __syncwarp();
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_flag) {
    if (!d.no_load) atomicOr(&g_xp_error, 1u);
    if (d.err) *static_cast<volatile unsigned int*>(d.err) = 1u;  // host memory
  }
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// ----------------------------------------------------------------- finish
// The units of a result added in order, the mode's magnitude, NaN at f = 0
// (itype 1, as the reference's 1/k), and the normalisation with Python's
// builtin max (see fj_normalize_kernel). A CTA takes 8 columns (one 32-byte
// sector of a row) of one set, so that 512 frequencies still make 64 CTAs, or
// 32 where that leaves enough CTAs (128 subarrays x 512 f x 500 c: 400 us with
// 8). A thread keeps its velocities' values in registers where they fit (2048
// or 1024 velocities). Bound by the latency of the units' loads: 16 in flight
// where few columns leave few CTAs and short runs make many units (140 f x 197 c
// over 1436 cells: 57 us with 4, 34 with 16).
constexpr int kFinThreads = 1024;
template <int MODE, int ITYPE, int kFinCols>
__global__ void __launch_bounds__(kFinThreads) xp_finish_kernel(XpDev d) {
  constexpr int kFinRows = kFinThreads / kFinCols, kFinKeep = kFinCols == 8 ? 16 : 32;
  constexpr int kWarpRows = 32 / kFinCols, kAhead = 16;
  constexpr int NACC = ModeTraits<MODE>::NACC;
  __shared__ float red[kFinRows / kWarpRows][kFinCols];
  const int fi = blockIdx.x * kFinCols + threadIdx.x, b = blockIdx.y;
  const bool mine = fi < d.nf && d.use[(long long)b * d.nf + min(fi, d.nf - 1)] != 0;
  if (!__syncthreads_or(mine)) return;
  const XpTile tile = d.tile[b * d.ft + (blockIdx.x * kFinCols) / kTileCols];
  const int nrun = runs_of(d, tile.lo, tile.hi);
  const bool nan_col = ITYPE == 1 && mine && d.f[fi] == 0.0f;
  float* o = d.out + (long long)b * d.nc * d.nf + fi;
  auto value = [&](int c) {
    float v[2] = {0.f, 0.f};
#pragma unroll
    for (int q = 0; q < NACC; ++q) {
      const float* p = d.part +
                       (tile.unit + q * d.mtiles + c / kTileRows) * (kTileRows * kTileCols) +
                       (c % kTileRows) * kTileCols + (fi & (kTileCols - 1));
      const long long step = (long long)d.mtiles * NACC * kTileRows * kTileCols;
      int s = 0;
      if (kFinCols == 8)
        for (; s + kAhead <= nrun; s += kAhead) {
          float t[kAhead];
#pragma unroll
          for (int i = 0; i < kAhead; ++i) t[i] = p[(s + i) * step];
#pragma unroll
          for (int i = 0; i < kAhead; ++i) v[q] += t[i];
        }
#pragma unroll 4
      for (; s < nrun; ++s) v[q] += p[s * step];
    }
    if (nan_col) return __int_as_float(0x7fffffff);
    return NACC == 1 ? v[0] : sqrtf(v[0] * v[0] + v[1] * v[1]);
  };
  float keep[kFinKeep];
  const bool in_regs = d.nc <= kFinRows * kFinKeep;
  float m = -INFINITY;
  if (mine) {
    if (in_regs) {
#pragma unroll
      for (int i = 0; i < kFinKeep; ++i) {
        const int c = threadIdx.y + i * kFinRows;
        if (c < d.nc) {
          keep[i] = value(c);
          m = fmaxf(m, fabsf(keep[i]));
        }
      }
    } else {
      for (int c = threadIdx.y; c < d.nc; c += kFinRows) {
        const float v = value(c);
        o[(long long)c * d.nf] = v;
        m = fmaxf(m, fabsf(v));
      }
    }
  }
#pragma unroll
  for (int s = kFinCols; s < 32; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
  if (threadIdx.y % kWarpRows == 0) red[threadIdx.y / kWarpRows][threadIdx.x] = m;
  __shared__ float first[kFinCols];
  if (threadIdx.y == 0 && mine) first[threadIdx.x] = fabsf(in_regs ? keep[0] : o[0]);
  __syncthreads();
  if (!mine) return;
  float div = 1.0f;
  if (d.normalize) {
    for (int y = 0; y < kFinRows / kWarpRows; ++y) m = fmaxf(m, red[y][threadIdx.x]);
    const float f0 = first[threadIdx.x];
    div = isnan(f0) ? f0 : m;
  }
  if (in_regs) {
#pragma unroll
    for (int i = 0; i < kFinKeep; ++i) {
      const int c = threadIdx.y + i * kFinRows;
      if (c < d.nc) o[(long long)c * d.nf] = d.normalize ? keep[i] / div : keep[i];
    }
  } else if (d.normalize) {
    for (int c = threadIdx.y; c < d.nc; c += kFinRows) o[(long long)c * d.nf] /= div;
  }
}

// ------------------------------------------------------------------- host
int nin_of(int mode) { return mode == CCFJ_MODE_J || mode == CCFJ_MODE_Y ? 1 : 2; }
int nsrc_of(int mode) { return mode == CCFJ_MODE_J_MINUS_Y || mode == CCFJ_MODE_ABS_H ? 2 : 1; }
int nacc_of(int mode) { return mode == CCFJ_MODE_ABS_J || mode == CCFJ_MODE_ABS_H ? 2 : 1; }

// The cells of the highest frequency of one transform at which the expansion
// takes kMargin times the direct kernels' time; none for a batch, whose sets run
// side by side. The constants (microseconds) are a fit to one B200's times of
// the transforms that worth_cells() names: half of the predictions are within
// 12% of the direct kernels' time and 8% of the expansion's, nine in ten within
// 50% and 25%.
double cells_in_time(const XpProblem& p, const XpDev& d) {
  if (p.off) return 0.0;
  const int nin = nin_of(p.mode);
  const bool trapezoid = p.itype == 0, two = d.nsrc == 2;
  const double n = (double)p.total, nf = p.nf_all;
  const double launches = 60.0 + (trapezoid ? 0.0 : 8.0) + 20.0 * (nin - 1) +
                          2.0 * std::min(d.chunk, 32) * nin;
  // half the cells of the highest frequency in the product and the moments (a
  // linear grid's mean), all of them in the basis
  const double per_cell =
      0.5 * (4.9e-3 * div_up(p.nf_all, kTileCols) * d.mtiles * d.nacc * d.nsrc + 5.5e-5 * nf * nin) +
      1.7e-4 * d.ncp + (trapezoid ? 0.0 : 0.035);
  // The direct kernels: a walk over the pairs (in as many station ranges as their
  // untuned choice, split_for()) or their terms, whichever is longer.
  const double ctas = (double)div_up(p.nc, trapezoid ? 32 : 16) * div_up(p.nf_all, 32);
  double ranges = 1.0;
  for (int k = 2; k <= 4; ++k)
    if (k * ctas <= 444.0 && n >= 64.0 * k) ranges = k;
  const double walk = n / ranges * (trapezoid ? (two ? 0.95 : 0.85) : (two ? 1.5 : 1.0));
  const double terms =
      n * nf * p.nc * 1e-8 * (trapezoid ? (two ? 350.0 : 126.0) : (two ? 1100.0 : 500.0));
  const double direct = 34.0 + 20.0 * (nin - 1) + std::pow(std::pow(walk, 4) + std::pow(terms, 4), 0.25);
  return (kMargin * direct - launches) / per_cell;
}

size_t round256(size_t v) { return (v + 255) & ~size_t(255); }

// Sizes, and places relative to `base`; returns the bytes needed.
size_t layout(const XpProblem& p, void* base, XpDev* out) {
  XpDev d{};
  d.rs = p.rs;
  d.wtr = p.wtr;
  d.off = p.off;
  d.nsets = p.nsets;
  d.total = p.total;
  d.nf = p.nf;
  d.nc = p.nc;
  d.f = p.f;
  d.c = p.c;
  d.in[0] = p.in[0];
  d.in[1] = p.in[1];
  d.out = p.out;
  d.normalize = p.normalize;
  d.err = p.err;
  d.wait_cycles = tc::kWaitCycles;
  d.ft = (int)div_up(p.nf, kTileCols);
  d.mtiles = (int)div_up(p.nc, kTileRows);
  d.ncp = d.mtiles * kTileRows;
  d.nsrc = nsrc_of(p.mode);
  d.nacc = nacc_of(p.mode);
  d.has_ends = p.itype == 1;
  d.nf_all = p.nf_all;
  const int nin = nin_of(p.mode);
  const bool batch = p.off != nullptr;
  // Stations of a moments chunk: long chunks leave fewer shared cells to
  // join, short ones keep the SMs busy when there are few pairs.
  if (batch)
    d.chunk = p.total_all >= 100000 ? 128 : 32;
  else
    d.chunk = p.total <= 128 ? 4 : p.total <= 1024 ? 8 : p.total <= 2048 ? 16 : p.total <= 4096 ? 32 : p.total <= 8192 ? 64 : 128;
  // Shorter runs of cells where the tiles alone leave SMs idle.
  const long long mn = (long long)div_up(p.nf_all, kTileCols) * d.mtiles * d.nacc;
  d.run = batch || mn >= 96 ? 64 : mn >= 32 ? 32 : mn >= 12 ? 16 : 8;
  // No column that the plan takes (xp_columns_kernel) has more cells than this.
  d.cells_in_time = cells_in_time(p, d);
  const double most =
      std::max(std::max((double)p.total_all * p.nc * d.nsrc * 250.0, kAnyCost / p.nf_all) /
                   (kNodes * ((double)d.ncp * d.nsrc * d.nacc + 200.0)),
               d.cells_in_time);
  // Nor does W get more than the direct kernels' interval data and 512 MiB (all
  // cells of 4096 frequencies): of more frequencies, those with many cells go
  // direct. By the whole problem's sizes, for its windows to decide alike.
  const double fit = ((double)p.total * p.nf_all * 16 + (512 << 20)) / (kBlockFloats * 4) /
                     div_up(p.nf_all, kTileCols);
  d.cells_cap = (int)std::min({(double)kMaxCells, 2 * kGroup + kDyadic + most,
                               batch ? (double)kMaxCells : std::max(64.0, fit)}) &
                ~(kGroup - 1);
  const long long ntile = (long long)p.nsets * d.ft;
  long long cells = ntile * d.cells_cap;
  d.tile_cells = d.cells_cap;
  if (batch) {
    // W of a tile of n pairs: as much as the direct kernels' interval data (n / 4
    // blocks) and tile_cells more. Its own share, and not what other sets leave,
    // so that a set's columns go the same way whatever sets it shares a call or
    // a group of a host batch with. tile_cells: 384, as long as that comes to
    // less than 4 GiB and a quarter of the interval data together, or 64 MiB in
    // all. (Of 400 batches of 4 to 64 sets of 20-4000 pairs, drawn at random,
    // 320 left no tile out that 64 MiB beside the interval data had held for all
    // tiles together, 256 left out tiles of three; 500 sets of 50-200 pairs x
    // 512 f, r to 300 km at 1 Hz: at most 192.)
    const long long block = (long long)kBlockFloats * 4;
    const long long ntile_all = (long long)p.nsets_all * d.ft;
    const long long more = (4ll << 30) / block / nin + (long long)p.total_all * p.nf * 4 / block;
    d.tile_cells = (int)std::min<long long>(
        kMaxCells, std::max(std::min(384ll, more / ntile_all), (64ll << 20) / block / ntile_all));
    cells = std::min(cells, (p.total / 4 + (long long)p.nsets * d.tile_cells) * d.ft);
  }
  cells &= ~(long long)(kGroup - 1);
  d.blocks_cap = cells;
  d.units_cap = (long long)d.nacc * d.mtiles * (cells / d.run + 2 * ntile);
  d.slots = p.total / d.chunk + p.nsets + 1;
  size_t at = 0;
  auto place = [&](size_t bytes) {
    const size_t o = at;
    at += round256(bytes);
    return static_cast<char*>(base) + o;
  };
  d.use = reinterpret_cast<unsigned char*>(place((size_t)p.nsets * p.nf));
  d.plan = reinterpret_cast<XpPlan*>(place(sizeof(XpPlan)));
  d.tile = reinterpret_cast<XpTile*>(place(sizeof(XpTile) * ntile));
  d.direct = reinterpret_cast<int*>(place(sizeof(int) * ntile));
  d.set_bad = reinterpret_cast<int*>(place(sizeof(int) * (size_t)p.nsets));
  d.slot_set = reinterpret_cast<int*>(place(sizeof(int) * (size_t)d.slots));
  const int nbasis = d.nsrc;
  d.E = reinterpret_cast<float*>(place(sizeof(float) * (size_t)nbasis * d.cells_cap * kNodes * d.ncp));
  d.W = reinterpret_cast<float*>(place(sizeof(float) * (size_t)cells * nin * kBlockFloats));
  if (d.has_ends) {
    d.Eend = reinterpret_cast<float*>(
        place(sizeof(float) * (size_t)nbasis * d.cells_cap * kEndRows * d.ncp));
    d.V = reinterpret_cast<float*>(place(sizeof(float) * (size_t)(cells / kGroup) * nin * kEndFloats));
    d.ends = reinterpret_cast<unsigned char*>(place((size_t)(cells / kGroup)));
  }
  d.unit_tile = reinterpret_cast<int*>(place(sizeof(int) * (size_t)d.units_cap));
  d.part = reinterpret_cast<float*>(
      place(sizeof(float) * (size_t)d.units_cap * kTileRows * kTileCols));
  const size_t edge = sizeof(float) * (size_t)d.slots * p.nf * nin * kNodes;
  d.head = reinterpret_cast<float*>(place(edge));
  d.tail = reinterpret_cast<float*>(place(edge));
  d.span = reinterpret_cast<int2*>(place(sizeof(int2) * (size_t)d.slots * p.nf));
  *out = d;
  return at;
}

template <int MODE, int ITYPE>
int plan_mode(const XpDev& d, cudaStream_t s) {
  xp_columns_kernel<MODE, ITYPE><<<dim3(d.ft, d.nsets), kTileCols, 0, s>>>(d);
  count_launch();
  CCFJ_LAUNCH_CHECK("xp_columns_kernel");
  xp_scan_kernel<<<1, 1024, 0, s>>>(d);
  count_launch();
  CCFJ_LAUNCH_CHECK("xp_scan_kernel");
  return CCFJ_OK;
}

template <int MODE, int ITYPE>
int run_mode(const XpDev& d, cudaStream_t s) {
  using MT = ModeTraits<MODE>;
  constexpr int NIN = MT::NIN;
  constexpr bool DY = MT::WY;
  constexpr int NSRC = MT::WJ && MT::WY ? 2 : 1;
  int dev = 0, sms = 148;
  CCFJ_CUDA_TRY(cudaGetDevice(&dev));
  CCFJ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  prof_begin(s);
  const int by = std::max(1, std::min(d.cells_cap, 16 * sms / d.mtiles));
  xp_basis_kernel<MODE, ITYPE><<<dim3(d.mtiles, by), kTileRows, 0, s>>>(d);
  count_launch();
  CCFJ_LAUNCH_CHECK("xp_basis_kernel");
  const int ftiles = (int)div_up(d.nf, 32);
  const long long warps = d.slots * ftiles;
  xp_moments_kernel<NIN, ITYPE, DY><<<(unsigned)warps, 32, 0, s>>>(d, ftiles);
  count_launch();
  CCFJ_LAUNCH_CHECK("xp_moments_kernel");
  xp_join_kernel<NIN, ITYPE, DY>
      <<<dim3((unsigned)d.slots, div_up(d.nf, 64)), 256, 0, s>>>(d);
  count_launch();
  CCFJ_LAUNCH_CHECK("xp_join_kernel");
  const int grid = (int)std::min<long long>(d.units_cap, sms);
  CCFJ_CUDA_TRY(cudaFuncSetAttribute(xp_gemm_kernel<NSRC>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
  xp_gemm_kernel<NSRC><<<grid, kGemmThreads, kGemmSmem, s>>>(d);
  count_launch();
  CCFJ_LAUNCH_CHECK("xp_gemm_kernel");
  prof_end(s);
  if ((long long)d.nsets * div_up(d.nf, 32) >= 4 * sms)
    xp_finish_kernel<MODE, ITYPE, 32>
        <<<dim3(div_up(d.nf, 32), d.nsets), dim3(32, kFinThreads / 32), 0, s>>>(d);
  else
    xp_finish_kernel<MODE, ITYPE, 8>
        <<<dim3(div_up(d.nf, 8), d.nsets), dim3(8, kFinThreads / 8), 0, s>>>(d);
  count_launch();
  CCFJ_LAUNCH_CHECK("xp_finish_kernel");
  return CCFJ_OK;
}

template <int ITYPE>
int dispatch(const XpDev& d, int mode, bool plan, cudaStream_t s) {
  switch (mode) {
#define CCFJ_XP(M) \
  case M:          \
    return plan ? plan_mode<M, ITYPE>(d, s) : run_mode<M, ITYPE>(d, s)
    CCFJ_XP(CCFJ_MODE_J);
    CCFJ_XP(CCFJ_MODE_Y);
    CCFJ_XP(CCFJ_MODE_J_MINUS_Y);
    CCFJ_XP(CCFJ_MODE_ABS_J);
    CCFJ_XP(CCFJ_MODE_ABS_H);
#undef CCFJ_XP
  }
  return set_error(CCFJ_ERR_INVALID, "bad mode %d", mode);
}

}  // namespace

bool xp_eligible(long long total, int nsets, int nf_all, int nc) {
  // (a batch's largest set may hold nearly all pairs; the plan decides set by set)
  return nsets <= 65535 && nf_all <= 65535 * 8 && worth((double)total, (double)nf_all * nc);
}

// A call that is being captured gets its memory when the graph is launched, too
// late to do without the workspace. So the workspace has to fit, with what the
// call has already asked for, into what the device has free now. (What earlier
// graphs hold and don't use counts as taken: the device still reports it as used
// after they have run.)
static bool captured_without_memory(size_t bytes, cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (!s || allocator_hooked() || cudaStreamIsCapturing(s, &cs) != cudaSuccess ||
      cs == cudaStreamCaptureStatusNone)
    return false;
  size_t free_bytes = 0, all = 0;
  if (cudaMemGetInfo(&free_bytes, &all) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return bytes > free_bytes;
}

int xp_plan(const XpProblem& p, Scratch& sc, cudaStream_t s, XpWork* w, bool* ok) {
  XpDev d;
  *ok = false;
  const size_t bytes = layout(p, nullptr, &d);
  if (d.slots > 0x7fffffffll || d.slots * div_up(p.nf, 32) > 0x7fffffffll) return CCFJ_OK;
  if (captured_without_memory(bytes + sc.bytes(), s)) return CCFJ_OK;
  void* base = sc.get(bytes);
  if (!base) {
    clear_error();
    return CCFJ_OK;
  }
  layout(p, base, &d);
  w->base = base;
  w->use = d.use;
  w->left = &d.plan->left;
  *ok = true;
  return p.itype == 1 ? dispatch<1>(d, p.mode, true, s) : dispatch<0>(d, p.mode, true, s);
}

int xp_sticky_error(cudaStream_t s, bool* failed) {
  unsigned int h = 0;
  const unsigned int zero = 0;
  CCFJ_CUDA_TRY(cudaMemcpyFromSymbolAsync(&h, g_xp_error, sizeof(h), 0, cudaMemcpyDeviceToHost, s));
  CCFJ_CUDA_TRY(cudaStreamSynchronize(s));
  if (h) CCFJ_CUDA_TRY(cudaMemcpyToSymbol(g_xp_error, &zero, sizeof(zero)));
  *failed = h != 0;
  return CCFJ_OK;
}

int xp_self_test(cudaStream_t s, int* status) {
  Scratch sc(s);
  CallFlag flag(s);
  XpDev d{};
  d.plan = sc.get_n<XpPlan>(1);
  d.tile = sc.get_n<XpTile>(1);
  d.unit_tile = sc.get_n<int>(1);
  d.part = sc.get_n<float>(kTileRows * kTileCols);
  d.err = flag.word();
  if (!d.plan || !d.tile || !d.unit_tile || !d.part || !d.err) return CCFJ_ERR_ALLOC;
  // one unit of one group of cells
  XpPlan plan{};
  plan.units = 1;
  XpTile tile{};
  tile.hi = kGroup;
  const int unit_tile = 0;
  CCFJ_CUDA_TRY(cudaMemcpyAsync(d.plan, &plan, sizeof(plan), cudaMemcpyHostToDevice, s));
  CCFJ_CUDA_TRY(cudaMemcpyAsync(d.tile, &tile, sizeof(tile), cudaMemcpyHostToDevice, s));
  CCFJ_CUDA_TRY(cudaMemcpyAsync(d.unit_tile, &unit_tile, sizeof(int), cudaMemcpyHostToDevice, s));
  CCFJ_CUDA_TRY(cudaMemsetAsync(d.part, 0, sizeof(float) * kTileRows * kTileCols, s));
  d.mtiles = d.nacc = d.nsrc = 1;
  d.run = kGroup;
  d.wait_cycles = 2000000;  // ~1 ms
  d.no_load = 1;
  CCFJ_CUDA_TRY(cudaFuncSetAttribute(xp_gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kGemmSmem));
  xp_gemm_kernel<1><<<1, kGemmThreads, kGemmSmem, s>>>(d);
  count_launch();
  CCFJ_LAUNCH_CHECK("xp_gemm_kernel (self-test)");
  float sum = 0.0f;
  CCFJ_CUDA_TRY(cudaMemcpyAsync(&sum, d.part, sizeof(sum), cudaMemcpyDeviceToHost, s));
  CCFJ_CUDA_TRY(cudaStreamSynchronize(s));
  *status = flag.status("self-test");
  if (sum == sum)
    return set_error(CCFJ_ERR_CUDA, "self-test: the product gave a number without its operands");
  return CCFJ_OK;
}

int xp_run(const XpProblem& p, const XpWork& w, cudaStream_t s) {
  XpDev d;
  layout(p, w.base, &d);
  return p.itype == 1 ? dispatch<1>(d, p.mode, false, s) : dispatch<0>(d, p.mode, false, s);
}

}  // namespace ccfj

CCFJ_API int ccfj_self_test_product_timeout(void* stream) {
  ccfj::clear_error();
  int status = CCFJ_OK;
  const int st = ccfj::xp_self_test((cudaStream_t)stream, &status);
  if (st != CCFJ_OK) return st;
  if (status != CCFJ_ERR_TIMEOUT)
    return ccfj::set_error(CCFJ_ERR_CUDA, "self-test: the product did not report its timeout");
  ccfj::clear_error();
  return CCFJ_OK;
}
