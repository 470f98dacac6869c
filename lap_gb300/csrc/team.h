// team.h -- whole PCG recurrences (line_jacobi, none) in one launch
// (team.cu has the kernel and its reasons).
#pragma once

#include <vector>

#include "gblap_internal.h"

namespace gb {

struct PcgState;

// Blocks of one launch, by system: blocks [cta0[s], cta0[s+1]) hold system
// s's rows, kTeamThreads * rows of them each.
struct TeamPlan {
  bool on = false;
  int ctas = 0, rows = 0;   // blocks; rows of a thread (1 to 4)
  size_t smem = 0;          // bytes of matrix entries kept in shared memory (0: none)
  int max_nnz = 0;          // most entries of a block
  long long nnz = 0;        // entries in all
  size_t debug_smem = 0;    // test hook: bytes to ask for at least, past what the device gives every block
  int systems = 0;
  int *cta_sys = nullptr, *cta0 = nullptr;  // device [ctas], [systems + 2] (the last twice)
  int debug_block = -1, debug_sys = 0;      // test hook: a block that leaves at once, and its system
  double *mail = nullptr;        // device: per system [blocks][4][blocks][2]
  long long *mail0 = nullptr;    // device [systems]
  long long mail_len = 0;
};

constexpr int kTeamThreads = 256;
constexpr size_t kTeamMaxSmem = 200 * 1024;
constexpr int kTeamMaxRow = 64;  // entries of a row (a thread sums its rows alone)

// Plans `count` systems of rows [row_off[s], row_off[s+1]) with global row
// pointers ia (host); plan->on says whether all their blocks fit the device
// at once and no row is too long.
int team_plan_build(int count, const std::vector<int>& row_off, const int* ia, TeamPlan* plan);
void team_plan_free(TeamPlan* plan);
// Test hook: block `block` (-1: none) belongs to a system past the last whose
// state, states[systems], is done, and leaves at once without a word to its team.
int team_debug_silent(TeamPlan* plan, int block, PcgState* states);

// Vectors and matrix of the systems, concatenated; columns local to the
// system.  d_r null: no preconditioner (w is r).
template <typename T, typename TA>
struct TeamData {
  const int *ia, *ja;
  const TA* a;
  const T* d_r;
  T *x, *r, *w, *p, *q;
  const int* row_off;  // null: one system from row 0
  int n;               // rows in all
  PcgState* st;        // [systems], and one more for the test hook
  double* hist;        // one system: residual history (st->hist_len entries), or null
  int roll_done;       // rho rolls in the last iteration too (the single-system recurrence's convention)
  int* err;
};

// Whether the one launch is the faster way: past these entries the loops' kernels,
// which stage rows by whole lines, win over threads that read their own rows.
// An iteration, loop -> one launch, us.  FP64, one system: 27-point 70^3 (9.0M
// entries) 88 -> 82, 74^3 (10.6M) 94 -> 106, a band of 25 on 400k rows (10.0M)
// 89 -> 97; a batch's loop has four launches: 109 -> 97, a band of 33 there
// (13.2M) 139 -> 140, split 117 -> 132, and 10.0M 95 -> 85.  FP32: a band of 25 on
// 200k rows (5.0M) 43 -> 37, random 12 on 400k (5.2M) 60 -> 60, 27-point 60^3
// (5.6M) 46 -> 42, a band of 33 (6.6M) 47 -> 53.
template <typename T, typename TA>
bool team_runs(const TeamPlan& plan, bool batch) {
  const long long most = sizeof(T) == 4 ? 5800000 : sizeof(TA) == 4 ? 10000000 : batch ? 12000000 : 9000000;
  return plan.on && plan.nnz <= most;
}

// Runs every system's recurrence from its state until it is done (or its
// state says it is), as the loops of update / spmv_pq kernels do.
// GB_NOT_SUPPORTED, with nothing of the state touched, where it is not the
// faster way or the device refuses the launch (fewer SMs for this context than
// when the plan was made): the caller then runs the loop.
template <typename T, typename TA>
int team_loop(const TeamPlan& plan, const TeamData<T, TA>& d, cudaStream_t s);

}  // namespace gb
