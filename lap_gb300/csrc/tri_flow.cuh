// tri_flow.cuh -- triangular solves of factors with many or far dependencies
// (power-law graphs, random labellings): every value through L2.
//
// A record is a warp's work: nodes of one level, each with a lane per
// dependency (a power of two up to 32).  A lane polls its own value -- the
// sentinel says not yet -- and the node's lanes sum by shuffles as soon as the
// last one has arrived, whatever the record's other nodes wait for.  A row of
// more than 32 dependencies has its earliest ones summed by part nodes of 32
// placed at their own levels, so that what is left after the last dependency
// arrives is one poll, one sum of 32 and one store.  Warps take records in
// level order by ticket: a record waits only on lower ones, the lowest
// unfinished one always belongs to a running warp, and so no two blocks need
// to be resident at once.
//
// Bound by the chain of levels: a level takes 0.9 us in FP64 and 0.7 us in
// FP32 (an L2 round trip of the poll, five shuffle sums, the store on its way
// to L2).  131k-row Chung-Lu factor of 166 levels and hubs of 10,240
// dependencies: lower / upper 594 / 1241 us on the records, 157 / 149 us here
// (FP32 549 / 1362 -> 115 / 125 us); its 35 MB of FP64 records are 5 us.
// Eight warps an SM poll without crowding the L2: 16 warps cost 0-4% more, 32
// 5-10%, 4 warps 10% on 131k rows (too few for a wide level).
#pragma once

#include "gb_common.cuh"
#include "gblap_internal.h"

namespace gb {

constexpr int kFlowThreads = 256;

template <typename T>
struct FlowArgs {
  int n, nrec;
  const int* col;
  const int* out;
  const int* lanes;
  const T* val;
  const T* dinv;
  T* y;
  T* part;
  unsigned* ticket;  // [0] next record, [1] blocks gone
  int* err;
};

template <typename T, typename OP>
__global__ void __launch_bounds__(kFlowThreads) tri_flow_kernel(const FlowArgs<T> F, OP op) {
  op.begin();
  if (!op.active()) return;
  const int lane = threadIdx.x & 31;
  auto ticket = [&] {
    unsigned t = 0;
    if (lane == 0) t = atomicAdd(&F.ticket[0], 1u);
    return t;
  };
  const unsigned nrec = (unsigned)F.nrec;
  unsigned rec = __shfl_sync(~0u, ticket(), 0);
  int col = -1, out = -1, lanes = 32;
  T val = T(0), dinv = T(0);
  auto fetch = [&](unsigned q, int& c, int& o, int& g, T& v, T& di) {
    const size_t i = (size_t)q * 32 + lane;
    c = __ldg(F.col + i);
    o = __ldg(F.out + i);
    g = __ldg(F.lanes + q);
    v = __ldg(F.val + i);
    di = __ldg(F.dinv + i);
  };
  if (rec < nrec) fetch(rec, col, out, lanes, val, dinv);
  bool failed = false;
  while (rec < nrec && !failed) {
    // the next record's data while this one waits
    const unsigned tn = ticket();
    const bool dep = col >= 0, from_part = col >= F.n;
    const T* p = from_part ? F.part + (col - F.n) : F.y + col;
    T v = T(0);
    if (dep) v = ld_relaxed(p);
    const bool first = (lane & (lanes - 1)) == 0;
    const bool row = first && out >= 0 && out < F.n;
    typename OP::Pre pr;
    typename OP::DPre dp;
    if (row) {
      pr = op.pre(out);
      dp = op.dpre(out);
    }
    const unsigned next = __shfl_sync(~0u, tn, 0);
    int ncol = -1, nout = -1, nlanes = 32;
    T nval = T(0), ndinv = T(0);
    if (next < nrec) fetch(next, ncol, nout, nlanes, nval, ndinv);
    const unsigned mine = (lanes == 32 ? ~0u : (1u << lanes) - 1u) << (lane & ~(lanes - 1));
    bool miss = dep && is_sentinel(v), open = out >= 0;
    SpinClock clk;
    unsigned polls = 0;
    while (true) {
      const unsigned m = __ballot_sync(~0u, miss);
      const bool ready = open && (m & mine) == 0u;
      if (__any_sync(~0u, ready)) {
        T s = miss ? T(0) : val * v;
        for (int o = lanes >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(~0u, s, o);
        if (ready && first) {
          if (row) {
            const T yv = publishable(fma_rn(op.rhs(out, pr), dinv, -s));
            st_relaxed(F.y + out, yv);
            op.done(out, yv, dp);
          } else {
            st_relaxed(F.part + (out - F.n), publishable(s));
          }
        }
        if (ready) open = false;
      }
      if (m == 0u) break;
      if (miss) {
        v = ld_relaxed(p);
        miss = is_sentinel(v);
      }
      if ((++polls & kPollCheck) == 0u && __any_sync(~0u, clk.expired(F.err))) {
        failed = true;
        break;
      }
    }
    if (from_part && !failed) st_relaxed(F.part + (col - F.n), sentinel<T>());  // read once; ready for the next solve
    rec = next;
    col = ncol;
    out = nout;
    lanes = nlanes;
    val = nval;
    dinv = ndinv;
  }
  __syncthreads();
  // the last block to leave resets the counters for the next launch
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&F.ticket[1], 1u) == gridDim.x - 1u) {
      F.ticket[0] = 0u;
      F.ticket[1] = 0u;
      __threadfence();
    }
  }
}

template <typename T, typename OP>
int flow_launch(const FlowPlan& p, T* y, int* err, OP op, cudaStream_t s) {
  if (!p.on || p.elem != (int)sizeof(T)) return GB_NOT_SUPPORTED;
  FlowArgs<T> F;
  F.n = p.n;
  F.nrec = p.nrec;
  F.col = p.col;
  F.out = p.out;
  F.lanes = p.lanes;
  F.val = (const T*)p.val;
  F.dinv = (const T*)p.dinv;
  F.y = y;
  F.part = (T*)p.part;
  F.ticket = p.ticket;
  F.err = err;
  constexpr int warps = kFlowThreads / 32;
  // Two blocks an SM where a level holds more than half of one block's records
  // an SM (FP64 lower solve of 1M-row Chung-Lu 444 -> 340 us, 800k-row kNN 199
  // -> 150, 200k-row 73 -> 62), one where levels are narrow and more warps only
  // poll (131k-row Chung-Lu 157 either way, 20k-row kNN 37 against 39 us).
  const int per_sm = 2LL * p.nrec > (long long)p.nlev * warps * device_sm_count() ? 2 : 1;
  const int grid = std::max(1, std::min((p.nrec + warps - 1) / warps, per_sm * device_sm_count()));
  tri_flow_kernel<T, OP><<<grid, kFlowThreads, 0, s>>>(F, op);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

}  // namespace gb
