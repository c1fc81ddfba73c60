// mom_rows.cuh -- the stored rows of a momentum sector's apply.
//
// A row of H in a momentum sector takes, per spin flip of its representative,
// the rank of the flipped state (two tables), that state's map entry (its
// representative j and the translation t reaching it) and n_j before it can
// ask for x_j: four dependent loads per term, none of which depends on x.  A
// handle forms them once, when it is made and when its couplings change, and
// keeps one 32-bit entry per term:
//     j | idx << jbits,   idx = (ratio * n_val + v) * n_trans + t
// with v the index of the term's element among the couplings' distinct
// elements and `ratio` that of n_j / n_i among the ratios that occur (0: 1);
// cf[idx] is the term's coefficient phase_t * (element * ratio).  The entries
// of 32 consecutive rows (a slice) lie side by side, entry e of row i at
// (off[i / 32] + e) * 32 + i % 32, so that a warp reads them as whole lines,
// each slice as wide as its longest row; kMomRowPad fills the shorter ones.
// The terms stay in the order of the walk, and so do the bits of the result.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "momentum.cuh"

namespace aed {

constexpr uint32_t kMomRowPad = 0xffffffffu;

// What a first pass over the rows finds: the distinct normalisations (bits of
// the doubles, 0: none), and used[a] bit b: a term of a row of normalisation
// a with n_j = normalisation b.
struct MomRowMarks {
  unsigned long long norm[kMomRowNorms];
  uint32_t used[kMomRowNorms];
  uint32_t many;  // more normalisations than slots
  unsigned long long total;  // sum of the slices' widths (mom_row_scan_kernel)
};

struct MomRowSpec {
  int n_val = 0, n_trans = 0, jbits = 0;
  double val[kMomRowVals];  // the distinct elements
  double norm[kMomRowNorms];
  uint8_t ridx[kMomRowNorms][kMomRowNorms];  // index of the ratio norm[b] / norm[a]
  uint8_t vid[kMaxBonds];                    // spin 1/2: the element of each flip
};

__device__ __forceinline__ int mom_norm_slot(const double* norm, double n) {
  int s = 0;
  while (s < kMomRowNorms - 1 && norm[s] != n) ++s;
  return s;
}

// A term with map entry e (not kMomNone) in a row of normalisation ni.
__device__ __forceinline__ void mom_row_mark(MomRowMarks* __restrict__ marks, const double* __restrict__ norm,
                                             double ni, uint32_t e) {
  const double nj = __ldg(norm + (e & ((1u << kMomRepBits) - 1u)));
  if (nj == ni) return;
  const double* slots = reinterpret_cast<const double*>(marks->norm);
  const int a = mom_norm_slot(slots, ni), b = mom_norm_slot(slots, nj);
  if (!(*(volatile uint32_t*)(marks->used + a) >> b & 1u)) atomicOr(marks->used + a, 1u << b);
}

__device__ __forceinline__ uint32_t mom_row_entry(const MomRowSpec& spec, const double* __restrict__ norm, double ni,
                                                  int v, uint32_t e) {
  const uint32_t j = e & ((1u << kMomRepBits) - 1u), t = e >> kMomRepBits;
  const double nj = __ldg(norm + j);
  const int r = nj == ni ? 0 : spec.ridx[mom_norm_slot(spec.norm, ni)][mom_norm_slot(spec.norm, nj)];
  return j | ((uint32_t)((r * spec.n_val + v) * spec.n_trans) + t) << spec.jbits;
}

// The build's host steps (momentum.cu), around the two passes over the rows.
// kMomRowsNone: an entry cannot hold the sector's indices, or there is no
// memory for the rows; the apply walks the representatives.
constexpr int kMomRowsNone = 1;
int mom_rows_begin(const double* norm, int64_t dim, MomRowStore& rs, cudaStream_t st);
int mom_rows_plan(const MomParams& mp, int64_t dim, MomRowSpec& spec, MomRowStore& rs, cudaStream_t st);
void mom_rows_done(const MomRowSpec& spec, int64_t dim, const double* diag, MomRowStore& rs);

}  // namespace aed
