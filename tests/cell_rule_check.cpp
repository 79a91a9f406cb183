// Host checks of the expansion's cell rule (csrc/fj_cell.h): locate() against
// the walk over the cells that the moments kernel takes.
#include <cstdint>

#include "fj_cell.h"

using namespace ccfj::xp;

namespace {
constexpr double kTwoPi = 6.283185307179586476925286766559;

uint64_t next(uint64_t& s) {  // splitmix64
  uint64_t z = (s += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
double uniform(uint64_t& s) { return (next(s) >> 11) * 0x1p-53; }

template <bool DY>
int walk(float r, Fx fx, int from, float& v) {
  const Place x = place_of(r, fx);
  float begin = cell_begin<DY>(from);
  for (; reached(x, begin + 1.0f); begin += 1.0f) ++from;
  v = (x.p - (begin + kCentre)) + x.l;
  return from;
}

// Cells of r by locate() and by walks that begin one, two and three cells
// below: 1 where they differ in the cell or the place.
template <bool DY>
int differs(float r, Fx fx) {
  float v, w;
  const int cell = locate<DY>(r, fx, v);
  const int first = DY ? kDyadic : 0;
  for (int back = 0; back <= 3; ++back) {
    if (cell - back < first) break;
    if (walk<DY>(r, fx, cell - back, w) != cell || w != v) return 1;
  }
  return 0;
}
}  // namespace

extern "C" {

double cell_hu(float cmin) { return kCellPhase / kTwoPi * (double)cmin; }

// Disagreements among n random (r, f): half of them with r f within a few
// spacings of a whole number of cells.
long long cell_disagreements(long long n, uint64_t seed, float cmin) {
  const double hu = cell_hu(cmin), inv_hu = 1.0 / hu;
  long long bad = 0;
  for (long long i = 0; i < n; ++i) {
    const float f = (float)(0.005 + 2.0 * uniform(seed));
    const Fx fx = make_fx(f, inv_hu);
    float r = (float)(500.0 + 4e5 * uniform(seed));
    if (i & 1) {
      r = (float)((1.0 + (double)(next(seed) % 1500)) * hu / f);
      const int steps = (int)(next(seed) % 5) - 2;
      for (int k = 0; k < (steps < 0 ? -steps : steps); ++k) r = nextafterf(r, steps < 0 ? 0.0f : 1e30f);
    }
    bad += differs<false>(r, fx) + differs<true>(r, fx);
  }
  return bad;
}

// The smallest cells' r (a whole number of cells at f, or a neighbour of it)
// for which the product's float lies below the cell that x has reached, that
// is, where p + l carries over an integer: up to `max` of them with r in
// [r0, r1), ascending.
int cell_carries(float f, float cmin, float r0, float r1, int max, float* out) {
  const double hu = cell_hu(cmin);
  const Fx fx = make_fx(f, 1.0 / hu);
  int n = 0;
  for (double m = floor(r0 * (double)f / hu) + 1.0; n < max; m += 1.0) {
    float r = (float)(m * hu / f);
    if (r >= r1) break;
    r = nextafterf(nextafterf(r, 0.0f), 0.0f);
    for (int k = 0; k < 5; ++k, r = nextafterf(r, 1e30f)) {
      const Place x = place_of(r, fx);
      if (r >= r0 && r < r1 && floorf(x.p) == (float)(m - 1.0) && reached(x, (float)m)) {
        out[n++] = r;
        break;
      }
    }
  }
  return n;
}

int cell_locate(float r, float f, float cmin, int dy) {
  const Fx fx = make_fx(f, 1.0 / cell_hu(cmin));
  float v;
  return dy ? locate<true>(r, fx, v) : locate<false>(r, fx, v);
}
int cell_walk(float r, float f, float cmin, int dy, int from) {
  const Fx fx = make_fx(f, 1.0 / cell_hu(cmin));
  float v;
  return dy ? walk<true>(r, fx, from, v) : walk<false>(r, fx, from, v);
}
}
