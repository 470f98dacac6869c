// tri_step.cu -- plan, value fill and launch of the lock-step triangular
// solves (tri_step.cuh).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "tri_step.cuh"

namespace gb {

namespace {

// opt-in shared memory per block, less the kernel's static part
constexpr size_t kStepMaxSmem = 231168;

template <typename V>
int upload(V** dst, const std::vector<V>& src) {
  const size_t bytes = sizeof(V) * std::max<size_t>(src.size(), 1);
  GB_CUDA_TRY(cudaMalloc(dst, bytes));
  if (!src.empty()) GB_CUDA_TRY(cudaMemcpy(*dst, src.data(), sizeof(V) * src.size(), cudaMemcpyHostToDevice));
  return GB_OK;
}

size_t page_bytes(int elem) { return elem == 8 ? StepPageGeom<double>::bytes : StepPageGeom<float>::bytes; }

size_t smem_bytes(int elem, bool nat, int np, int window, int inbox, int max_steps, int max_pages, int chunks) {
  return (size_t)np * (page_bytes(elem) + (nat ? 0 : (size_t)kStepPage * elem)) + (size_t)(window + inbox + 2) * elem +
         2 * (size_t)(max_steps + 4 + max_pages + chunks);
}

// The kernel a plan runs, for split-precision (FP64) or same-type right-hand sides.
template <typename T, typename TR>
void (*kernel_of(bool nat, int k))(const StepArgs<T>, const TR*) {
  if (nat)
    return k <= 2   ? tri_step_kernel<T, TR, 2, true>
           : k == 3 ? tri_step_kernel<T, TR, 3, true>
                    : tri_step_kernel<T, TR, 4, true>;
  return k <= 2   ? tri_step_kernel<T, TR, 2, false>
         : k == 3 ? tri_step_kernel<T, TR, 3, false>
                  : tri_step_kernel<T, TR, 4, false>;
}

template <typename T, typename TR>
int set_attributes() {
  for (int v = 0; v < 2 * (kStepDeps - 1); ++v) {
    auto f = kernel_of<T, TR>(v & 1, 2 + v / 2);
    GB_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStepMaxSmem));
    GB_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
  return GB_OK;
}

// Once per device: the attributes belong to the current device's context.
int prepare_device() {
  static std::mutex mu;
  static unsigned long long done = 0;
  int dev = 0;
  GB_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && (done >> dev & 1ull)) return GB_OK;
  GB_TRY((set_attributes<float, double>()));
  GB_TRY((set_attributes<float, float>()));
  GB_TRY((set_attributes<double, double>()));
  if (dev < 64) done |= 1ull << dev;
  return GB_OK;
}

template <typename K>
int active_clusters(K kern, int cl, int threads, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(cl);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int active = 0;
  if (cudaOccupancyMaxActiveClusters(&active, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return active;
}

int clusters_of(const StepPlan& p, int cl) {
  const int th = step_threads(p.nat, p.nw);
  return p.elem == 8 ? active_clusters(kernel_of<double, double>(p.nat, p.k), cl, th, p.smem)
                     : active_clusters(kernel_of<float, double>(p.nat, p.k), cl, th, p.smem);
}

// Estimated cycles of one step of a level of `width` rows, fitted on 128^3,
// 64^3, 97 x 61 x 83 and 1000 x 700 grids cut into tiles of 1 to 44 bands
// (FP32: 165 at 32 rows, 200 at 64, 310 at 128, 700 at 256; FP64: 320 at 16,
// 380 at 64, 550 at 128, 1000 at 256).
double step_cycles(int elem, int width) {
  const double w = width;
  return (elem == 8 ? 300.0 + 1.1 * w : 140.0 + 0.5 * w) + 0.0065 * w * w;
}
constexpr double kHopCycles = 250.0;      // more for a step whose inputs come from the previous tile
constexpr double kCrossCycles = 2000.0;   // and from another cluster, through L2
constexpr int kResidentTiles = 140;       // about what clusters of 8 to 16 place on 152 SMs
// Seconds a resident tile may wait for the one before it, by the estimate: a
// wait ends at one second (kSpinBudgetNs).  A path of 9M rows, FP64, in the
// tallest tiles there are is 146 of 61,697 steps, all running, and the last
// would wait 1.1 s.
constexpr double kStepMaxWait = 0.4;

// Tiles of a cluster, as far as can be said before the device is asked.
int cluster_guess(int ntiles) { return ntiles <= 16 ? ntiles : ntiles <= 112 ? 16 : 10; }

int warps_for(int width) { return width <= 32 ? 1 : width <= 64 ? 2 : width <= 128 ? 4 : kStepMaxWarps; }

// The host image of a plan.
struct StepLayout {
  int k = 0, ntiles = 0, tile_rows = 0, nw = 0, np = 0, window = 0, nexp_max = 0, max_steps = 0, max_pages = 0, max_chunks = 0;
  int width = 1;  // widest level of a tile
  bool nat = false;
  long long npages = 0;
  size_t smem = 0;
  std::vector<StepTile> tiles;
  std::vector<unsigned short> ends, needs, thr;
  std::vector<unsigned> meta;     // [npages * kStepPage * 4]
  std::vector<int> psrc, pdiag;
};

constexpr int kMaxRows = 65000;  // rows of a tile and its exports are 16-bit numbers

// Tile heights to try: multiples of the band (the farthest a dependency lies
// in index), so that a tile depends on itself and the tile before only;
// cheapest first by an estimate of the dependency chain: the hops between
// tiles, the steps within them, the crossings between clusters and the page
// stream.  Empty where a row has too many dependencies.
std::vector<int> step_heights(const TriDeps& d, const std::vector<int>& lev, int nlev, int elem, int* kmax) {
  const int n = d.n;
  int band = 1;
  *kmax = 0;
  for (int i = 0; i < n; ++i) {
    const int b = d.row_ptr[i], e = d.row_ptr[i + 1];
    *kmax = std::max(*kmax, e - b);
    if (*kmax > kStepDeps) return {};
    for (int k = b; k < e; ++k) band = std::max(band, std::abs(i - d.dep_col[k]));
  }
  struct Cand {
    int rows;
    double cost;
  };
  std::vector<Cand> cands;
  std::vector<int> count(nlev, 0);
  for (int m = 1;; m = m < 4 ? m + 1 : m + m / 4) {
    const long long want = (long long)band * m;
    const bool whole = want >= n;
    const int rows = whole ? n : (int)std::min<long long>(want, kMaxRows + 1);
    if (rows > kMaxRows) break;
    const int nt = (n + rows - 1) / rows;
    int span = 1, width = 1;  // levels and widest level of a few tiles
    for (int t = 0; t < std::min(nt, 4); ++t) {
      const int q = nt <= 4 ? t : (int)((long long)t * (nt - 1) / 3);
      const int r0 = q * rows, r1 = std::min(n, r0 + rows);
      int lo = nlev, hi = 0;
      for (int i = r0; i < r1; ++i) {
        lo = std::min(lo, lev[i]);
        hi = std::max(hi, lev[i]);
        width = std::max(width, ++count[lev[i]]);
      }
      span = std::max(span, hi - lo + 1);
      for (int i = r0; i < r1; ++i) count[lev[i]] = 0;
    }
    const int cl = cluster_guess(nt);
    double cost = step_cycles(elem, width) * std::max(span, nlev) + kHopCycles * (nt - 1) +
                  kCrossCycles * ((nt + cl - 1) / cl - 1);
    // clusters that are not resident start when an earlier one has ended
    // (1000 x 700 FP32: 175 tiles 328 us, 88 tiles 189 us)
    cost *= (nt + kResidentTiles - 1) / kResidentTiles;
    const double chain = std::min<double>(nlev, (double)std::min(nt, kResidentTiles) * span);
    if (chain * step_cycles(elem, std::min(width, 32 * kStepMaxWarps)) < kStepMaxWait * 2e9) cands.push_back({rows, cost});
    if (whole) break;
  }
  std::stable_sort(cands.begin(), cands.end(), [](const Cand& a, const Cand& b) { return a.cost < b.cost; });
  std::vector<int> h;
  for (const Cand& c : cands) h.push_back(c.rows);
  return h;
}

// Estimated microseconds of a solve laid out so, launch apart: the chain of
// steps, hops and crossings as above, but of the steps that there are (a wide
// level is several), and a tile's own rows on their way into its SM, which a
// tile of few steps waits for (1.3 ns a row).  Against measured, split lower
// solves: shuffled 100^2 33 / 31, 200^2 111 / 110, red-black 100^2 30 / 25,
// 20^3 14 / 8, 160^3 446 / 420 us; it errs upwards on grids.
double step_estimate(const StepLayout& L, int n, int nlev, int elem) {
  const int cl = cluster_guess(L.ntiles);
  double cycles = step_cycles(elem, std::min(L.width, 32 * L.nw)) * std::max(nlev, L.max_steps) +
                  kHopCycles * (L.ntiles - 1) + kCrossCycles * ((L.ntiles + cl - 1) / cl - 1);
  if (L.ntiles > kResidentTiles) cycles *= 2.0;  // 148 x 148 x 300 took 1.0 times, 160^3 1.9, 1000 x 700 on 175 tiles 2.2
  return cycles / 2000.0 + 0.0013 * std::min(L.tile_rows, n);
}

// Lays the factor out in tiles of R rows; false where that does not fit.
bool step_layout(const TriDeps& d, const std::vector<int>& lev, int nlev, int elem, int kmax, int R, StepLayout* L) {
  *L = StepLayout();
  const int n = d.n, nt = (n + R - 1) / R;
  auto tile_at = [&](int q) { return d.lower ? q : nt - 1 - q; };
  std::vector<unsigned char> need(n, 0);  // rows the next tile depends on
  for (int i = 0; i < n; ++i)
    for (int k = d.row_ptr[i]; k < d.row_ptr[i + 1]; ++k) {
      const int c = d.dep_col[k];
      if (c / R == i / R) continue;
      if (std::abs(c / R - i / R) != 1) return false;
      need[c] = 1;
    }
  std::vector<int> pos(n), order(n), lptr, fill;
  std::vector<unsigned short> expo(n);
  int width = 1;
  L->tiles.resize(nt);
  for (int q = 0; q < nt; ++q) {
    const int t0 = tile_at(q) * R, t1 = std::min(n, t0 + R);
    int lo = nlev, hi = 0;
    for (int i = t0; i < t1; ++i) {
      lo = std::min(lo, lev[i]);
      hi = std::max(hi, lev[i]);
    }
    lptr.assign(hi - lo + 2, 0);
    for (int i = t0; i < t1; ++i) lptr[lev[i] - lo + 1]++;
    for (int l = 0; l <= hi - lo; ++l) {
      width = std::max(width, lptr[l + 1]);
      lptr[l + 1] += lptr[l];
    }
    fill.assign(lptr.begin(), lptr.end() - 1);
    for (int i = t0; i < t1; ++i) {
      const int p = fill[lev[i] - lo]++;
      pos[i] = p;
      order[t0 + p] = i;
    }
    int ex = 0;
    for (int p = 0; p < t1 - t0; ++p) {
      const int i = order[t0 + p];
      expo[i] = need[i] ? (unsigned short)ex++ : (unsigned short)kStepNone;
    }
    L->nexp_max = std::max(L->nexp_max, ex);
    L->tiles[q] = {t0, t1 - t0, (int)L->npages, (t1 - t0 + kStepPage - 1) / kStepPage, 0, 0, ex, (int)L->thr.size()};
    // a chunk (in the order rows are loaded) may be stored once its last row is solved
    for (int c = 0; c < step_chunks(t1 - t0); ++c) {
      int last = 0;
      for (int o = c * kStepChunk; o < std::min(t1 - t0, (c + 1) * kStepChunk); ++o)
        last = std::max(last, pos[d.lower ? t0 + o : t1 - 1 - o] + 1);
      L->thr.push_back((unsigned short)last);
    }
    L->max_chunks = std::max(L->max_chunks, step_chunks(t1 - t0));
    L->npages += L->tiles[q].npages;
  }
  L->width = width;
  L->nw = warps_for(width);
  const int per = 32 * L->nw;
  std::vector<int> step_end(R);
  int reach = 1;  // places of own values that must be live at once
  for (StepTile& t : L->tiles) {
    t.step0 = (int)L->ends.size();
    for (int p = 0; p < t.npos;) {
      const int l = lev[order[t.row0 + p]];
      int e = p;
      while (e < t.npos && e - p < per && lev[order[t.row0 + e]] == l) ++e;
      for (int u = p; u < e; ++u) step_end[u] = e;
      L->ends.push_back((unsigned short)e);
      p = e;
    }
    t.nsteps = (int)L->ends.size() - t.step0;
    int need = 0;  // chunks loaded before the rows of the pages so far may be read
    for (int p = 0; p < t.npos; ++p) {
      const int o = order[t.row0 + p] - t.row0;
      need = std::max(need, (d.lower ? o : t.npos - 1 - o) / kStepChunk + 1);
      if ((p + 1) % kStepPage == 0 || p + 1 == t.npos) L->needs.push_back((unsigned short)need);
    }
    L->max_pages = std::max(L->max_pages, t.npages);
    L->max_steps = std::max(L->max_steps, t.nsteps);
    // a place is written again `window` positions later: in a later step
    // than every reader's
    for (int i = t.row0; i < t.row0 + t.npos; ++i)
      for (int k = d.row_ptr[i]; k < d.row_ptr[i + 1]; ++k) {
        const int c = d.dep_col[k];
        if (c >= t.row0 && c < t.row0 + t.npos) reach = std::max(reach, step_end[pos[i]] - pos[c]);
      }
  }
  // The rows' own places in natural order where levels are wide and all of
  // them fit beside the inbox: right-hand sides and solutions then move by
  // whole lines (128^3 split lower solve 91 us, 124 in a window).  Else a
  // window in step order, its right-hand sides gathered row by row: with one
  // solver warp the chain is all, and the window's is shorter by an LDS and
  // an address (1000 x 700: 161 us, 180 in natural order).
  bool fits = false;
  for (int form = L->nw > 1 ? 0 : 1; form < 2 && !fits; ++form) {
    L->nat = form == 0;
    L->window = 32;
    if (L->nat) L->window = (R + 31) & ~31;
    else while (L->window < reach) L->window <<= 1;
    if (L->window + L->nexp_max + 1 > 65535) continue;
    for (L->np = kStepMaxPages; L->np >= 8 && !fits; L->np /= 2) {
      L->smem = smem_bytes(elem, L->nat, L->np, L->window, L->nexp_max, L->max_steps, L->max_pages, L->max_chunks);
      fits = L->smem <= kStepMaxSmem;
      if (fits) break;
    }
  }
  if (!fits) return false;
  L->k = std::max(2, kmax);
  L->ntiles = nt;
  L->tile_rows = R;
  const size_t rows = (size_t)L->npages * kStepPage;
  L->meta.assign(rows * 4, 0);
  L->psrc.assign(rows * kStepDeps, -1);
  L->pdiag.assign(rows, -1);
  const unsigned zero = (unsigned)(L->window + L->nexp_max);
  for (const StepTile& t : L->tiles)
    for (int p = 0; p < t.npages * kStepPage; ++p) {
      const size_t P = (size_t)t.page0 * kStepPage + p;
      unsigned place[kStepDeps] = {zero, zero, zero, zero}, who = kStepNone << 16;
      if (p < t.npos) {
        const int i = order[t.row0 + p];
        L->pdiag[P] = d.diag_src[i];
        who = (unsigned)(L->nat ? step_place(i - t.row0) : i - t.row0) | (unsigned)expo[i] << 16;
        int u = 0;
        for (int own = 0; own < 2; ++own)  // other tiles' terms first, each kind in column order
          for (int k = d.row_ptr[i]; k < d.row_ptr[i + 1]; ++k) {
            const int c = d.dep_col[k];
            const bool in = c >= t.row0 && c < t.row0 + t.npos;
            if (in != (own == 1)) continue;
            place[u] = !in      ? (unsigned)(L->window + expo[c])
                       : L->nat ? (unsigned)step_place(c - t.row0)
                                : (unsigned)pos[c] & (unsigned)(L->window - 1);
            L->psrc[P * kStepDeps + u] = d.dep_src[k];
            ++u;
          }
      }
      L->meta[P * 4] = place[0] | place[1] << 16;
      L->meta[P * 4 + 1] = place[2] | place[3] << 16;
      L->meta[P * 4 + 2] = who;
    }
  return true;
}

}  // namespace

double step_plan_estimate(const TriDeps& d, const std::vector<int>& lev, int nlev, int elem) {
  int kmax = 0;
  StepLayout L;
  for (int R : step_heights(d, lev, nlev, elem, &kmax))
    if (step_layout(d, lev, nlev, elem, kmax, R, &L)) return step_estimate(L, d.n, nlev, elem);
  return -1.0;
}

int step_plan_build(const TriDeps& d, const std::vector<int>& lev, int nlev, int elem, double limit_us, StepPlan* plan) {
  *plan = StepPlan();
  int kmax = 0;
  StepLayout L;
  for (int R : step_heights(d, lev, nlev, elem, &kmax)) {
    if (!step_layout(d, lev, nlev, elem, kmax, R, &L)) continue;
    plan->fits = true;
    if (step_estimate(L, d.n, nlev, elem) > limit_us) return GB_OK;
    plan->elem = elem;
    plan->k = L.k;
    plan->ntiles = L.ntiles;
    plan->tile_rows = L.tile_rows;
    plan->nw = L.nw;
    plan->np = L.np;
    plan->window = L.window;
    plan->nexp_max = L.nexp_max;
    plan->max_steps = L.max_steps;
    plan->max_pages = L.max_pages;
    plan->nat = L.nat;
    plan->n = d.n;
    plan->lower = d.lower;
    plan->npages = L.npages;
    plan->smem = L.smem;
    GB_TRY(prepare_device());
    // Cluster size: all tiles in one cluster where they fit; else the
    // largest size of which every group is resident at once (a boundary
    // between clusters costs a round trip through L2); else the most tiles.
    int best = 0, best_tiles = 0;
    for (int cl = std::min(L.ntiles, 16); cl >= 1; --cl) {
      const int groups = (L.ntiles + cl - 1) / cl, act = clusters_of(*plan, cl);
      if (act >= groups) {
        best = cl;
        break;
      }
      if (act * cl > best_tiles) {
        best_tiles = act * cl;
        best = cl;
      }
    }
    if (best < 1) continue;
    plan->cluster = best;
    plan->ngroups = (L.ntiles + best - 1) / best;
    StepTile* dt = nullptr;
    GB_TRY(upload(&dt, L.tiles));
    plan->tiles = dt;
    GB_TRY(upload(&plan->ends, L.ends));
    GB_TRY(upload(&plan->psrc, L.psrc));
    if (L.nat) {
      GB_TRY(upload(&plan->needs, L.needs));
      GB_TRY(upload(&plan->thr, L.thr));
      GB_TRY(upload(&plan->dsrc, d.diag_src));
      GB_CUDA_TRY(cudaMalloc(&plan->dinv, (size_t)d.n * elem));
    }
    GB_TRY(upload(&plan->pdiag, L.pdiag));
    const size_t PB = page_bytes(elem);
    GB_CUDA_TRY(cudaMalloc(&plan->pages, (size_t)L.npages * PB));
    GB_CUDA_TRY(cudaMemset(plan->pages, 0, (size_t)L.npages * PB));
    GB_CUDA_TRY(cudaMemcpy2D(plan->pages, PB, L.meta.data(), kStepPage * 16, kStepPage * 16, (size_t)L.npages,
                             cudaMemcpyHostToDevice));
    GB_CUDA_TRY(cudaMalloc(&plan->mail, std::max<size_t>((size_t)plan->ngroups * L.nexp_max * elem, 16)));
    GB_CUDA_TRY(cudaMalloc(&plan->ticket, sizeof(unsigned)));
    GB_CUDA_TRY(cudaMemset(plan->ticket, 0, sizeof(unsigned)));
    plan->on = true;
    GB_TRY(step_plan_reset(plan, 0));
    GB_CUDA_TRY(cudaStreamSynchronize(0));
    return GB_OK;
  }
  return GB_OK;
}

void step_plan_free(StepPlan* p) {
  void* ptrs[] = {p->tiles, p->ends, p->pages, p->psrc, p->pdiag, p->mail, p->ticket, p->needs, p->thr, p->dsrc, p->dinv};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  *p = StepPlan();
}

// One thread per staged row: 1/d, and each coefficient times it in FP64,
// rounded once (as the records' FMA form).
template <typename T>
__global__ void step_fill_kernel(long long rows, const int* __restrict__ psrc, const int* __restrict__ pdiag,
                                 const double* __restrict__ ent, const double* __restrict__ dg,
                                 unsigned char* pages) {
  for (long long P = blockIdx.x * (long long)blockDim.x + threadIdx.x; P < rows;
       P += (long long)gridDim.x * blockDim.x) {
    const int src = pdiag[P];
    if (src < 0) continue;
    const double d = dg[src];
    const double dinv = d != 0.0 ? 1.0 / d : 0.0;
    const int4 k = *reinterpret_cast<const int4*>(psrc + P * kStepDeps);
    const double l0 = k.x >= 0 ? ent[k.x] * dinv : 0.0, l1 = k.y >= 0 ? ent[k.y] * dinv : 0.0;
    const double l2 = k.z >= 0 ? ent[k.z] * dinv : 0.0, l3 = k.w >= 0 ? ent[k.w] * dinv : 0.0;
    unsigned char* pg = pages + (P / kStepPage) * StepPageGeom<T>::bytes;
    const int e = (int)(P % kStepPage);
    if constexpr (sizeof(T) == 4) {
      reinterpret_cast<float*>(pg + e * 16)[3] = (float)dinv;
      *reinterpret_cast<float4*>(pg + StepPageGeom<T>::coef + e * 16) =
          make_float4((float)l0, (float)l1, (float)l2, (float)l3);
    } else {
      *reinterpret_cast<double*>(pg + StepPageGeom<T>::dinv + e * 8) = dinv;
      *reinterpret_cast<double2*>(pg + StepPageGeom<T>::coef + e * 16) = make_double2(l0, l1);
      *reinterpret_cast<double2*>(pg + StepPageGeom<T>::coef + kStepPage * 16 + e * 16) = make_double2(l2, l3);
    }
  }
}

template <typename T>
__global__ void step_dinv_kernel(int n, const int* __restrict__ dsrc, const double* __restrict__ dg, T* dinv) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double d = dg[dsrc[i]];
    dinv[i] = (T)(d != 0.0 ? 1.0 / d : 0.0);
  }
}

int step_plan_fill(const StepPlan* p, const double* ent, const double* dg, cudaStream_t s) {
  const long long rows = p->npages * kStepPage;
  if (rows <= 0) return GB_OK;
  const int grid = std::max(1, std::min(device_sm_count() * 8, ceil_div(rows, 256)));
  if (p->elem == 8)
    step_fill_kernel<double><<<grid, 256, 0, s>>>(rows, p->psrc, p->pdiag, ent, dg, p->pages);
  else
    step_fill_kernel<float><<<grid, 256, 0, s>>>(rows, p->psrc, p->pdiag, ent, dg, p->pages);
  GB_CUDA_TRY(cudaGetLastError());
  if (p->nat) {
    if (p->elem == 8) step_dinv_kernel<double><<<grid, 256, 0, s>>>(p->n, p->dsrc, dg, (double*)p->dinv);
    else step_dinv_kernel<float><<<grid, 256, 0, s>>>(p->n, p->dsrc, dg, (float*)p->dinv);
    GB_CUDA_TRY(cudaGetLastError());
  }
  return GB_OK;
}

int step_plan_reset(const StepPlan* p, cudaStream_t s) {
  if (!p->on || p->ngroups < 2) return GB_OK;
  const int cnt = p->ngroups * p->nexp_max;
  GB_CUDA_TRY(cudaMemsetAsync(p->ticket, 0, sizeof(unsigned), s));
  return p->elem == 8 ? fill_sentinel_dev(cnt, (double*)p->mail, s) : fill_sentinel_dev(cnt, (float*)p->mail, s);
}

template <typename T, typename TR>
int step_solve(const StepPlan& p, const TR* rhs, T* y, const int* done, int* err, cudaStream_t s) {
  if (!p.on || p.elem != (int)sizeof(T)) return GB_NOT_SUPPORTED;
  auto kern = kernel_of<T, TR>(p.nat, p.k);
  const int threads = step_threads(p.nat, p.nw);
  int clusters = p.ngroups;
  if (p.ngroups > 1) clusters = std::max(1, std::min(p.ngroups, active_clusters(kern, p.cluster, threads, p.smem)));
  StepArgs<T> A;
  A.ntiles = p.ntiles;
  A.ngroups = p.ngroups;
  A.nw = p.nw;
  A.np = p.np;
  A.window = p.window;
  A.inbox = p.nexp_max;
  A.np_shift = p.np == 32 ? 5 : p.np == 16 ? 4 : 3;
  // every cluster claims until none is left, or once where all are resident
  A.claims = (unsigned)(clusters == p.ngroups ? p.ngroups : p.ngroups + clusters);
  A.tiles = (const StepTile*)p.tiles;
  A.ends = p.ends;
  A.needs = p.needs;
  A.thr = p.thr;
  A.dinv = (const T*)p.dinv;
  A.lower = p.lower;
  A.max_steps = p.max_steps;
  A.max_pages = p.max_pages;
  A.pages = p.pages;
  A.mail = (T*)p.mail;
  A.ticket = p.ticket;
  A.y = y;
  A.err = err;
  A.done = done;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(clusters * p.cluster);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, (const StepArgs<T>)A, rhs));
  return GB_OK;
}
TriDeps deps_of_part(int n, const int* ia, const int* ja, bool lower) {
  TriDeps d;
  d.n = n;
  d.lower = lower;
  d.row_ptr.assign(n + 1, 0);
  d.diag_src.resize(n);
  for (int i = 0; i < n; ++i) {
    d.diag_src[i] = i;
    for (int k = ia[i]; k < ia[i + 1]; ++k)
      if ((lower && ja[k] < i) || (!lower && ja[k] > i)) {
        d.dep_col.push_back(ja[k]);
        d.dep_src.push_back(k);
      }
    d.row_ptr[i + 1] = (int)d.dep_col.size();
  }
  return d;
}

// The host layout for the strict one-sided part of a full CSR pattern.
int step_layout_debug(int n, const int* ia, const int* ja, int lower, int elem, int tile_rows, int* info, int* tiles,
                      unsigned short* ends, unsigned* meta, int* src, unsigned short* needs, unsigned short* thr) {
  const TriDeps d = deps_of_part(n, ia, ja, lower != 0);
  std::vector<int> lev(n, 0);
  int nlev = 0;
  for (int q = 0; q < n; ++q) {
    const int i = lower ? q : n - 1 - q;
    for (int k = d.row_ptr[i]; k < d.row_ptr[i + 1]; ++k) lev[i] = std::max(lev[i], lev[d.dep_col[k]] + 1);
    nlev = std::max(nlev, lev[i] + 1);
  }
  int kmax = 0;
  std::vector<int> heights = step_heights(d, lev, nlev, elem, &kmax);
  if (tile_rows > 0 && !heights.empty()) heights.assign(1, std::min(tile_rows, kMaxRows));
  StepLayout L;
  bool ok = false;
  for (int R : heights)
    if ((ok = step_layout(d, lev, nlev, elem, kmax, R, &L))) break;
  if (!ok) return GB_NOT_SUPPORTED;
  const int v[12] = {L.ntiles, L.tile_rows, L.nw,        L.np,        L.window,
                     L.nexp_max, L.max_steps, (int)L.npages, (int)L.ends.size(), (int)L.smem, L.nat, (int)L.thr.size()};
  std::copy(v, v + 12, info);
  if (tiles) memcpy(tiles, L.tiles.data(), sizeof(StepTile) * L.tiles.size());
  if (ends) std::copy(L.ends.begin(), L.ends.end(), ends);
  if (meta) std::copy(L.meta.begin(), L.meta.end(), meta);
  if (src) std::copy(L.psrc.begin(), L.psrc.end(), src);
  if (needs) std::copy(L.needs.begin(), L.needs.end(), needs);
  if (thr) std::copy(L.thr.begin(), L.thr.end(), thr);
  return GB_OK;
}

template int step_solve<float, double>(const StepPlan&, const double*, float*, const int*, int*, cudaStream_t);
template int step_solve<float, float>(const StepPlan&, const float*, float*, const int*, int*, cudaStream_t);
template int step_solve<double, double>(const StepPlan&, const double*, double*, const int*, int*, cudaStream_t);

}  // namespace gb

extern "C" int gb_debug_step_plan(int n, const int* ia_host, const int* ja_host, int lower, int elem_bytes,
                                  int tile_rows, int* info, int* tiles, unsigned short* ends, unsigned* meta,
                                  int* src, unsigned short* needs, unsigned short* thr) {
  if (n <= 0 || !ia_host || !ja_host || !info || (elem_bytes != 4 && elem_bytes != 8)) return GB_BAD_INPUT;
  return gb::step_layout_debug(n, ia_host, ja_host, lower, elem_bytes, tile_rows, info, tiles, ends, meta, src,
                               needs, thr);
}
