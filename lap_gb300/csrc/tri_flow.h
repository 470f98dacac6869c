// tri_flow.h -- plan of the value-polling triangular solves (tri_flow.cuh has
// the kernel and its reasons, tri_plan.cu which factors take them).
#pragma once

#include <vector>

#include "gblap_internal.h"
#include "sptrsv.h"

namespace gb {

// Sources of a lane's coefficient (FlowPlan::vsrc) besides an entry's index.
constexpr int kFlowNoDep = -1;
constexpr int kFlowPartSum = -2;  // a part's sum: coefficient 1

// The host layout: 32 lanes a record.
struct FlowLayout {
  int nrec = 0, nslots = 0, nlev = 0;
  std::vector<int> col;    // value the lane reads: < n a row's, n + i part i's, -1 none
  std::vector<int> out;    // node the lane belongs to: < n a row, n + i part i, -1 none
  std::vector<int> lanes;  // [nrec] lanes of each of its nodes
  std::vector<int> vsrc, dsrc;
};
void flow_layout(const TriDeps& d, FlowLayout* L);

int flow_plan_build(const TriDeps& d, int elem, FlowPlan* plan);
void flow_plan_free(FlowPlan* plan);
// Writes the coefficients l/d and reciprocal diagonals from the value arrays.
int flow_plan_fill(const FlowPlan* plan, const double* ent_src, const double* diag_src, cudaStream_t s);
// The parts' slots and the counters: once per solve, since a launch that
// timed out may leave values behind.
int flow_plan_reset(const FlowPlan* plan, cudaStream_t s);

}  // namespace gb
