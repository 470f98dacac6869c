// tri_flow.cu -- layout, values and reset of the value-polling solves
// (tri_flow.cuh).
#include <algorithm>

#include "gb_common.cuh"
#include "kernels.h"
#include "tri_flow.h"
#include "tri_step.h"

namespace gb {

void flow_layout(const TriDeps& d, FlowLayout* L) {
  const int n = d.n;
  // Nodes: rows, and parts as they are cut.  lev: longest chain below a node.
  struct Dep {
    int lev, id, src;
  };
  std::vector<int> lev(n), part_row;               // part_row[i]: the row part i belongs to
  std::vector<std::vector<Dep>> long_deps;         // of parts and of rows cut
  std::vector<int> row_long(n, -1), part_long, part_lev;
  std::vector<Dep> w;
  int nlev = 0;
  for (int q = 0; q < n; ++q) {
    const int i = d.lower ? q : n - 1 - q;
    const int k0 = d.row_ptr[i], k1 = d.row_ptr[i + 1];
    int l = 0;
    if (k1 - k0 <= 32) {
      for (int k = k0; k < k1; ++k) l = std::max(l, lev[d.dep_col[k]] + 1);
    } else {
      w.clear();
      for (int k = k0; k < k1; ++k) w.push_back({lev[d.dep_col[k]], d.dep_col[k], d.dep_src[k]});
      auto earlier = [](const Dep& a, const Dep& b) { return a.lev < b.lev; };
      std::stable_sort(w.begin(), w.end(), earlier);
      // the 32 earliest into a part, which takes its place among the rest;
      // the last part takes only as many as leave 32
      size_t h = 0;
      while (w.size() - h > 32) {
        const size_t take = std::min<size_t>(32, w.size() - h - 31);
        const int pl = w[h + take - 1].lev + 1, id = (int)part_row.size();
        long_deps.emplace_back(w.begin() + h, w.begin() + h + take);
        part_row.push_back(i);
        part_long.push_back((int)long_deps.size() - 1);
        part_lev.push_back(pl);
        nlev = std::max(nlev, pl + 1);
        h += take;
        const Dep me = {pl, n + id, kFlowPartSum};
        w.insert(std::upper_bound(w.begin() + h, w.end(), me, earlier), me);
      }
      long_deps.emplace_back(w.begin() + h, w.end());
      row_long[i] = (int)long_deps.size() - 1;
      l = w.back().lev + 1;
    }
    lev[i] = l;
    nlev = std::max(nlev, l + 1);
  }
  const int np = (int)part_row.size(), total = n + np;
  auto deps_of = [&](int id) {
    if (id < n) return row_long[id] < 0 ? d.row_ptr[id + 1] - d.row_ptr[id] : (int)long_deps[row_long[id]].size();
    return (int)long_deps[part_long[id - n]].size();
  };
  // buckets by level, then by lanes of a node (32, 16, .. 1)
  auto bucket_of = [&](int id) {
    int g = 0;
    while ((1 << g) < deps_of(id)) ++g;
    return (size_t)(id < n ? lev[id] : part_lev[id - n]) * 6 + (5 - g);
  };
  std::vector<int> ptr((size_t)nlev * 6 + 1, 0), ids(total);
  for (int id = 0; id < total; ++id) ptr[bucket_of(id) + 1]++;
  for (size_t b = 0; b < (size_t)nlev * 6; ++b) ptr[b + 1] += ptr[b];
  {
    std::vector<int> fill(ptr.begin(), ptr.end() - 1);
    for (int id = 0; id < total; ++id) ids[fill[bucket_of(id)]++] = id;
  }
  L->nslots = np;
  L->nlev = nlev;
  L->nrec = 0;
  for (size_t b = 0; b < (size_t)nlev * 6; ++b) {
    const int g = 1 << (5 - b % 6), per = 32 / g, cnt = ptr[b + 1] - ptr[b];
    L->nrec += (cnt + per - 1) / per;
  }
  const size_t len = (size_t)L->nrec * 32;
  L->col.assign(len, -1);
  L->out.assign(len, -1);
  L->vsrc.assign(len, kFlowNoDep);
  L->dsrc.assign(len, -1);
  L->lanes.assign(L->nrec, 32);
  size_t rec = 0;
  for (size_t b = 0; b < (size_t)nlev * 6; ++b) {
    const int g = 1 << (5 - b % 6), per = 32 / g;
    for (int p = ptr[b]; p < ptr[b + 1]; p += per, ++rec) {
      L->lanes[rec] = g;
      for (int u = 0; u < per && p + u < ptr[b + 1]; ++u) {
        const int id = ids[p + u], owner = id < n ? id : part_row[id - n];
        const size_t at = rec * 32 + (size_t)u * g;
        for (int k = 0; k < g; ++k) {
          L->out[at + k] = id;
          L->dsrc[at + k] = d.diag_src[owner];
        }
        const int lg = id < n ? row_long[id] : part_long[id - n];
        if (lg < 0) {
          for (int k = d.row_ptr[id], j = 0; k < d.row_ptr[id + 1]; ++k, ++j) {
            L->col[at + j] = d.dep_col[k];
            L->vsrc[at + j] = d.dep_src[k];
          }
        } else {
          for (size_t j = 0; j < long_deps[lg].size(); ++j) {
            L->col[at + j] = long_deps[lg][j].id;
            L->vsrc[at + j] = long_deps[lg][j].src;
          }
        }
      }
    }
  }
}

template <typename V>
static int upload(V** dst, const std::vector<V>& v) {
  GB_CUDA_TRY(cudaMalloc(dst, sizeof(V) * std::max<size_t>(v.size(), 1)));
  if (!v.empty()) GB_CUDA_TRY(cudaMemcpy(*dst, v.data(), sizeof(V) * v.size(), cudaMemcpyHostToDevice));
  return GB_OK;
}

int flow_plan_build(const TriDeps& d, int elem, FlowPlan* plan) {
  FlowLayout L;
  flow_layout(d, &L);
  plan->elem = elem;
  plan->n = d.n;
  plan->nrec = L.nrec;
  plan->nslots = L.nslots;
  plan->nlev = L.nlev;
  GB_TRY(upload(&plan->col, L.col));
  GB_TRY(upload(&plan->out, L.out));
  GB_TRY(upload(&plan->lanes, L.lanes));
  GB_TRY(upload(&plan->vsrc, L.vsrc));
  GB_TRY(upload(&plan->dsrc, L.dsrc));
  const size_t len = std::max<size_t>(L.col.size(), 1);
  GB_CUDA_TRY(cudaMalloc(&plan->val, len * elem));
  GB_CUDA_TRY(cudaMalloc(&plan->dinv, len * elem));
  GB_CUDA_TRY(cudaMalloc(&plan->part, std::max<size_t>(L.nslots, 1) * (size_t)elem));
  GB_CUDA_TRY(cudaMalloc(&plan->ticket, sizeof(unsigned) * 2));
  plan->on = true;
  GB_TRY(flow_plan_reset(plan, 0));
  GB_CUDA_TRY(cudaStreamSynchronize(0));
  return GB_OK;
}

void flow_plan_free(FlowPlan* p) {
  void* ptrs[] = {p->col, p->out, p->lanes, p->vsrc, p->dsrc, p->val, p->dinv, p->part, p->ticket};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  *p = FlowPlan();
}

// 1/d, and each coefficient times it in FP64, rounded once (as the records'
// FMA form).
template <typename T>
__global__ void flow_fill_kernel(long long len, const int* __restrict__ vsrc, const int* __restrict__ dsrc,
                                 const double* __restrict__ ent, const double* __restrict__ dg, T* val, T* dinv) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < len;
       i += (long long)gridDim.x * blockDim.x) {
    const int ds = dsrc[i], vs = vsrc[i];
    const double d = ds >= 0 ? dg[ds] : 0.0;
    const double di = d != 0.0 ? 1.0 / d : 0.0;
    dinv[i] = (T)di;
    val[i] = vs >= 0 ? (T)(ent[vs] * di) : vs == kFlowPartSum ? T(1) : T(0);
  }
}

int flow_plan_fill(const FlowPlan* p, const double* ent, const double* dg, cudaStream_t s) {
  const long long len = (long long)p->nrec * 32;
  if (len <= 0) return GB_OK;
  const int grid = std::max(1, std::min(device_sm_count() * 8, ceil_div(len, 256)));
  if (p->elem == 8)
    flow_fill_kernel<double><<<grid, 256, 0, s>>>(len, p->vsrc, p->dsrc, ent, dg, (double*)p->val, (double*)p->dinv);
  else
    flow_fill_kernel<float><<<grid, 256, 0, s>>>(len, p->vsrc, p->dsrc, ent, dg, (float*)p->val, (float*)p->dinv);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

int flow_plan_reset(const FlowPlan* p, cudaStream_t s) {
  if (!p->on) return GB_OK;
  GB_CUDA_TRY(cudaMemsetAsync(p->ticket, 0, sizeof(unsigned) * 2, s));
  if (p->nslots == 0) return GB_OK;
  return p->elem == 8 ? fill_sentinel_dev(p->nslots, (double*)p->part, s)
                      : fill_sentinel_dev(p->nslots, (float*)p->part, s);
}

}  // namespace gb

extern "C" int gb_debug_flow_plan(int n, const int* ia_host, const int* ja_host, int lower, int* info, int* col,
                                  int* out, int* vsrc, int* dsrc, int* lanes) {
  if (n <= 0 || !ia_host || !ja_host || !info) return GB_BAD_INPUT;
  gb::FlowLayout L;
  gb::flow_layout(gb::deps_of_part(n, ia_host, ja_host, lower != 0), &L);
  info[0] = L.nrec;
  info[1] = L.nslots;
  info[2] = L.nlev;
  if (col) std::copy(L.col.begin(), L.col.end(), col);
  if (out) std::copy(L.out.begin(), L.out.end(), out);
  if (vsrc) std::copy(L.vsrc.begin(), L.vsrc.end(), vsrc);
  if (dsrc) std::copy(L.dsrc.begin(), L.dsrc.end(), dsrc);
  if (lanes) std::copy(L.lanes.begin(), L.lanes.end(), lanes);
  return GB_OK;
}
