// tri_step.h -- plan and launch of the lock-step triangular solves
// (tri_step.cuh has the kernel and its reasons).
#pragma once

#include "gblap_internal.h"
#include "sptrsv.h"

namespace gb {

constexpr int kStepDeps = 4;          // dependencies a row may have
constexpr int kStepPageShift = 7;
constexpr int kStepPage = 1 << kStepPageShift;  // rows of a staged page
constexpr int kStepMaxPages = 32;     // staged pages, at most
constexpr int kStepMaxWarps = 8;      // solver warps, at most
constexpr int kStepLoaders = 4;      // warps gathering right-hand sides by page
constexpr int kStepChunkWarps = 6;   // warps streaming rows in natural order
constexpr int kStepChunk = 32 * kStepChunkWarps;  // rows of one of their passes
constexpr unsigned kStepNone = 0xffffu;  // a row no later tile needs

// One page of kStepPage rows: per row {place 0 | place 1 << 16, place 2 |
// place 3 << 16, row within the tile | export << 16, FP32: 1/d}, then (FP64)
// 1/d, then the coefficients l/d in 16-byte columns.
//
// Staging depth: solving a page's last row needs the pages up to two steps
// past it ready: 32*nw rows each, so at most 6 pages on with 8 warps -- below
// the least ring of 8.
template <typename T>
struct StepPageGeom;
template <>
struct StepPageGeom<float> {
  static constexpr int dinv = 0;  // in the row's first 16 bytes
  static constexpr int coef = kStepPage * 16;
  static constexpr int bytes = kStepPage * 32;
  static constexpr int slot = bytes + kStepPage * 4;  // staged: with the scaled right-hand sides
};
template <>
struct StepPageGeom<double> {
  static constexpr int dinv = kStepPage * 16;
  static constexpr int coef = kStepPage * 24;
  static constexpr int bytes = kStepPage * 56;
  static constexpr int slot = bytes + kStepPage * 8;
};

// warps polling the mailbox of the previous cluster
__host__ __device__ constexpr int step_importers(bool nat) { return nat ? 3 : 4; }
// threads of a launch: solvers, loaders, page warp, gate, stager, importers
constexpr int step_threads(bool nat, int nw) {
  return (nw + (nat ? kStepChunkWarps : kStepLoaders) + 3 + step_importers(nat)) * 32;
}
__host__ __device__ inline int step_chunks(int rows) { return (rows + kStepChunk - 1) / kStepChunk; }
// A row's own place in natural order: lines skewed by three banks each, since
// a level of a grid walks its rows with a stride of one line less one.
__host__ __device__ inline int step_place(int i) { return (i & ~31) | ((i + 3 * (i >> 5)) & 31); }

struct StepTile {
  int row0;    // first row of the tile
  int npos;    // its rows
  int page0, npages;
  int step0, nsteps;
  int nexp;    // rows the next tile depends on
  int thr0;    // first of its chunks' thresholds
};

// The strict one-sided part of a full CSR pattern (the plans' test hooks);
// diag_src is the row.
TriDeps deps_of_part(int n, const int* ia, const int* ja, bool lower);

// Builds the plan for values of `elem` bytes where the factor allows it
// (every row within kStepDeps dependencies, all within one tile or the tile
// before, shared memory for the previous tile's exports) and a solve is
// estimated at limit_us or less; plan->fits and plan->on say.
// lev: the rows' global levels, nlev of them.
int step_plan_build(const TriDeps& d, const std::vector<int>& lev, int nlev, int elem, double limit_us, StepPlan* plan);
// That estimate; negative where the factor does not allow the form.
double step_plan_estimate(const TriDeps& d, const std::vector<int>& lev, int nlev, int elem);
void step_plan_free(StepPlan* plan);
// Writes the coefficients and reciprocal diagonals from the value arrays.
int step_plan_fill(const StepPlan* plan, const double* ent_src, const double* diag_src, cudaStream_t s);
// The mailboxes at the sentinel: once per solve, since a launch that timed
// out may leave values behind.
int step_plan_reset(const StepPlan* plan, cudaStream_t s);
// y = T^{-1} rhs unless *done; rhs in T, or FP64 rounded to FP32.
template <typename T, typename TR>
int step_solve(const StepPlan& plan, const TR* rhs, T* y, const int* done, int* err, cudaStream_t s);

}  // namespace gb
