// Wave-cell expansion of the FP32 transform (fj_expand.cu): host interface.
#pragma once

#include "ccfj_core.cuh"
#include "fj_frontend.cuh"

namespace ccfj {

// One transform, or a batch of sets that share f and c, as the expansion
// reads it (every pointer is device memory).
struct XpProblem {
  const float* rs;       // [total] distances, ascending within each set
  const float* wtr;      // [total] trapezoid weights (itype 0)
  const long long* off;  // [nsets + 1], or NULL for one set of `total` pairs
  int nsets;
  long long total;
  int nf, nc;
  const float* f;
  const float* c;
  int itype, mode;
  InDesc in[2];
  float* out;  // [nsets][nc][nf]
  int normalize;
  // frequencies, pairs and sets of the whole problem that this one is a window
  // or a group of sets of
  int nf_all;
  long long total_all;
  int nsets_all;
  unsigned int* err;  // set when a bounded wait of the product runs out, or NULL
};

// What the host sized and where it lies in the call's scratch.
struct XpWork {
  const unsigned char* use;  // [nsets][nf] 1: the expansion computes the column
  const long long* left;     // how many columns it leaves
  void* base;
};

// Whether a problem of these sizes runs the expansion at all. Decided from
// the sizes of the whole problem alone, so that frequency windows and blocks
// of one problem decide alike.
bool xp_eligible(long long total, int nsets, int nf_all, int nc);
// Reserves the scratch and runs the plan (which columns take the expansion).
// ok = false (and no error) where the memory cannot be had: the caller then
// computes every column directly.
int xp_plan(const XpProblem& p, Scratch& sc, cudaStream_t s, XpWork* w, bool* ok);
// Waits for `s`, reads the process-wide flag of the product's bounded waits
// (set when one ran out: that unit's columns are NaN) and clears it.
int xp_sticky_error(cudaStream_t s, bool* failed);
// Self-test of those waits: one CTA of the product whose operands never come,
// with a ~1 ms limit, as a host-memory call reads it: *status becomes
// CCFJ_ERR_TIMEOUT where the kernel gave up and set the call's flag.
int xp_self_test(cudaStream_t s, int* status);
// Computes the columns the plan chose, normalised if asked.
int xp_run(const XpProblem& p, const XpWork& w, cudaStream_t s);

}  // namespace ccfj
