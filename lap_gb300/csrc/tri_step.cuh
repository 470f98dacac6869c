// tri_step.cuh -- the PCG's triangular solves, marched level by level.
//
// The form of tri_kernel.cuh's solve for factors whose rows have at most
// kStepDeps dependencies, all of them near in index (grids, banded and other
// locally numbered sparse graphs): y_i = rhs_i/d_i - sum (l_ij/d_i) y_j, FMA
// form, the same terms in the same order (other tiles' first, then the
// tile's own, each in column order).
//
// What bounds it: the chain of levels.  A level is a few dozen to a few
// hundred rows whose inputs are the level before; bytes and FMAs are far
// from any limit.  The record kernel lets 13 warps chase records and waits
// per value, and a record's own ~2,500 cycles of code, not the hand-off,
// set its pace (about 1,080 cycles a level on 128^3).  Here everything that
// is not the chain is done by other warps beforehand, and the chain itself
// is as short as it can be made:
//   * a tile is solved by `nw` solver warps in lock step: one STEP is up to
//     32*nw rows of one level, a named barrier ends it.  The barrier makes
//     the tile's values plain shared-memory loads -- no sentinel, no poll,
//     no counter -- and frees staged rows and value slots without further
//     signalling;
//   * a row is two or three 16-byte loads from the staged page: its values'
//     places in shared memory (resolved at plan time: the tile's own window,
//     the inbox, or a zero), its coefficients, and its scaled right-hand
//     side.  They are loaded one step ahead;
//   * loader warps gather the right-hand side pages ahead and scale it, so
//     neither the gather's latency nor FP64 conversions are on the chain;
//   * the rows' static data is one stream of kStepPage-row pages in step
//     order, copied by TMA into a ring (a barrier per page, counts of loaded pages and of solved rows);
//   * a tile depends on the previous tile only.  That tile pushes the values
//     its successor needs into the successor's inbox: through distributed
//     shared memory inside a cluster, through a small mailbox in global
//     memory between clusters (import warps poll it and put the sentinel
//     back, so no output vector needs a sentinel fill).
//
// Measured against the record kernel, whole solves to 1e-12: 128^3 IC(0) split
// 189.9 -> 104.4 ms, FP64 240.2 -> 137.3 ms; 64^3 with a refactorisation
// 130.3 -> 32.9 ms; Gauss-Seidel on 97 x 61 x 83 164.2 -> 54.3 ms (its planes
// fit no power-of-two tile); 1000 x 700 forward + adjoint 132.0 -> 84.9 ms.
//
// Progress: a tile depends only on the tile before it, groups of tiles are
// claimed by ticket in order by running clusters, and every staged page's
// inputs are released by steps that do not need it.  Every wait is bounded
// (SpinClock); after one gave up, the warps keep the barriers' count and
// nothing else, so the launch ends and the error word says why.
#pragma once

#include "gb_common.cuh"
#include "kernels.h"
#include "tri_kernel.cuh"
#include "tri_step.h"

namespace gb {

constexpr int kStepLoaders = 8;    // warps gathering right-hand sides
constexpr int kStepImporters = 2;  // warps polling the mailbox of the previous cluster
constexpr int kStepImportBatch = 8;
constexpr int kStepMaxThreads = (kStepMaxWarps + kStepLoaders + 2 + kStepImporters) * 32;

template <typename T>
struct StepArgs {
  int ntiles, ngroups, nw, np, np_shift, window, inbox;
  unsigned claims;                        // ticket claims of one launch (it wraps to 0)
  const StepTile* __restrict__ tiles;     // [ntiles]
  const unsigned short* __restrict__ ends;  // steps' end positions, tile after tile
  const unsigned char* __restrict__ pages;
  T* mail;           // [ngroups][nexp_max], sentinel between launches
  unsigned* ticket;
  T* y;
  int* err;
  const int* done;   // nonzero: the recurrence has stopped, nothing to do
};

__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

// Shared-memory accesses by 32-bit address; volatile, so that they stay in
// the order written around the barriers.
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ unsigned lds_u16(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void lds_value(uint32_t a, float& v) {
  asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void lds_value(uint32_t a, double& v) {
  asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
template <typename T>
__device__ __forceinline__ T* cluster_ptr(T* p, unsigned rank) {
  unsigned long long r;
  asm volatile("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
  return reinterpret_cast<T*>(r);
}

// Predicated forms: a branch around one store costs the chain more than the
// store.
__device__ __forceinline__ void sts_value_if(bool on, uint32_t a, float v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.volatile.shared.f32 [%1], %2;\n}" ::"r"((int)on),
               "r"(a), "f"(v)
               : "memory");
}
__device__ __forceinline__ void sts_value_if(bool on, uint32_t a, double v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.volatile.shared.f64 [%1], %2;\n}" ::"r"((int)on),
               "r"(a), "d"(v)
               : "memory");
}
// An export: to the next tile's inbox (its generic address) or the mailbox.
__device__ __forceinline__ void st_export_if(bool on, float* p, float v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.relaxed.gpu.f32 [%1], %2;\n}" ::"r"((int)on), "l"(p),
               "f"(v)
               : "memory");
}
__device__ __forceinline__ void st_export_if(bool on, double* p, double v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.relaxed.gpu.f64 [%1], %2;\n}" ::"r"((int)on), "l"(p),
               "d"(v)
               : "memory");
}
__device__ __forceinline__ void st_global_if(bool on, float* p, float v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.global.f32 [%1], %2;\n}" ::"r"((int)on), "l"(p),
               "f"(v)
               : "memory");
}
__device__ __forceinline__ void st_global_if(bool on, double* p, double v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.global.f64 [%1], %2;\n}" ::"r"((int)on), "l"(p),
               "d"(v)
               : "memory");
}
__device__ __forceinline__ void sts_s32_if(bool on, uint32_t a, int v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.volatile.shared.s32 [%1], %2;\n}" ::"r"((int)on),
               "r"(a), "r"(v)
               : "memory");
}
// One look at a phase, without try_wait's suspension.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* b, unsigned parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Named barrier 1 among `threads` threads; true when any brought `bad`.
__device__ __forceinline__ int ld_acquire_cta(uint32_t a) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_cta(uint32_t a, int v) {
  asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ bool bar_any(int threads, bool bad) {
  int any;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n barrier.cta.red.or.pred q, 1, %2, p;\n selp.s32 %0, 1, 0, q;\n}"
      : "=r"(any)
      : "r"((int)bad), "r"(threads)
      : "memory");
  return any != 0;
}

// Out of line: a value the previous tile has not pushed yet; the sentinel
// when the wait gave up.
template <typename T>
__device__ __noinline__ T step_wait_value(uint32_t a, int* err) {
  SpinClock clk;
  for (unsigned polls = 1;; ++polls) {
    T v;
    lds_value(a, v);
    if (!is_sentinel(v)) return v;
    if ((polls & 255u) == 0u && clk.expired(err)) return v;
  }
}

// A row as the solver holds it: where its values lie, its coefficients and
// its scaled right-hand side.
template <typename T, int K>
struct StepRow {
  uint32_t at[K];
  T l[K];
  T acc;
  unsigned s01, s23, le;
};

// Where a tile's staged data lies in shared memory (32-bit addresses).
struct StepShared {
  uint32_t ring, vals, ends, prog, loaded;
};

// One solver warp's part of a tile.  K: the most dependencies a row has.
// Per step and warp: the row's values (LDS), the next step's row (LDS, off
// the chain), K FMAs, the value's store, the barrier.  The gate warp has seen
// to the next step's pages.  False when a wait gave up.
template <typename T, int K>
__device__ __forceinline__ bool step_solve_tile(const StepArgs<T>& A, const StepTile& ti, unsigned base, int first,
                                                const StepShared& S, T* out) {
  using G = StepPageGeom<T>;
  const unsigned npm = (unsigned)A.np - 1u;
  const unsigned wmask = (unsigned)A.window - 1u;
  const int threads = (A.nw + 1) * 32;  // solvers and gate
  T* const yt = A.y + ti.row0;
  // the row at position a + first of [a, b), from its staged page; past b
  // the last one again, which is then not stored
  auto load = [&](StepRow<T, K>& r, int a, int b) {
    const unsigned p = (unsigned)min(a + first, b - 1);
    const uint32_t pg = S.ring + ((base + (p >> kStepPageShift)) & npm) * G::slot;
    const uint32_t e = p & (kStepPage - 1);
    const uint4 m = lds128(pg + e * 16);
    const uint4 c = lds128(pg + G::coef + e * 16);
    if constexpr (sizeof(T) == 4) {
      r.l[0] = __uint_as_float(c.x);
      r.l[1] = __uint_as_float(c.y);
      if constexpr (K > 2) r.l[2] = __uint_as_float(c.z);
      if constexpr (K > 3) r.l[3] = __uint_as_float(c.w);
    } else {
      r.l[0] = __hiloint2double((int)c.y, (int)c.x);
      r.l[1] = __hiloint2double((int)c.w, (int)c.z);
      if constexpr (K > 2) {
        const uint4 d = lds128(pg + G::coef + kStepPage * 16 + e * 16);
        r.l[2] = __hiloint2double((int)d.y, (int)d.x);
        if constexpr (K > 3) r.l[3] = __hiloint2double((int)d.w, (int)d.z);
      }
    }
    lds_value(pg + G::bytes + e * (uint32_t)sizeof(T), r.acc);
    r.s01 = m.x;
    r.s23 = m.y;
    r.le = m.z;
  };
  auto decode = [&](StepRow<T, K>& r) {
    r.at[0] = S.vals + (r.s01 & 0xffffu) * (uint32_t)sizeof(T);
    r.at[1] = S.vals + (r.s01 >> 16) * (uint32_t)sizeof(T);
    if constexpr (K > 2) r.at[2] = S.vals + (r.s23 & 0xffffu) * (uint32_t)sizeof(T);
    if constexpr (K > 3) r.at[3] = S.vals + (r.s23 >> 16) * (uint32_t)sizeof(T);
  };
  int a = 0, b = (int)lds_u16(S.ends), nb = (int)lds_u16(S.ends + 2);
  uint32_t ep = S.ends + 4;
  // one step: solves `c`, stages the next into `n`; false when a wait gave up
  auto step = [&](StepRow<T, K>& c, StepRow<T, K>& n) -> bool {
    T v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) lds_value(c.at[k], v[k]);
    const int nnb = (int)lds_u16(ep);  // the list ends in copies of the last end
    ep += 2;
    load(n, b, nb);
    bool bad = false, miss = false;  // only the inbox's places can hold the sentinel
#pragma unroll
    for (int k = 0; k < K; ++k) miss |= is_sentinel(v[k]);
    if (miss) {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (is_sentinel(v[k])) {
          v[k] = step_wait_value<T>(c.at[k], A.err);
          bad = bad || is_sentinel(v[k]);
        }
    }
    // an FMA never returns the sentinel (a signalling NaN)
    T acc = c.acc;
#pragma unroll
    for (int k = 0; k < K; ++k) acc = fma_rn(-c.l[k], v[k], acc);
    decode(n);  // beside the FMAs: its loads are back with the values
    const int p = a + first;
    const bool on = p < b;
    sts_value_if(on, S.vals + ((unsigned)p & wmask) * (uint32_t)sizeof(T), acc);
    const unsigned ex = c.le >> 16;
    st_export_if(on && ex != kStepNone, out + ex, acc);
    const bool any = bar_any(threads, bad);
    st_global_if(on, yt + (c.le & 0xffffu), acc);
    a = b;
    b = nb;
    nb = nnb;
    return !any;
  };
  StepRow<T, K> r0, r1;
  if (bar_any(threads, false)) return false;  // the first two steps' pages are there
  load(r0, a, b);
  decode(r0);
  for (int s = 0; s < ti.nsteps; s += 2) {  // an odd count's last step is empty
    if (!step(r0, r1)) return false;
    if (!step(r1, r0)) return false;
  }
  return true;
}

// The gate warp: waits for the pages of the rows the solvers load next, joins
// the steps' barriers and publishes how far they are.
template <typename T>
__device__ __forceinline__ bool step_gate_tile(const StepArgs<T>& A, const StepTile& ti, int lane,
                                               const StepShared& S) {
  const int threads = (A.nw + 1) * 32;
  int avail = 0;  // pages known to be ready
  // Loader w finishes pages (w >> 2) + k * (kStepLoaders / 4) in order and
  // counts them: the first page one of them still owes ends what is ready.
  auto pages = [&](int b) -> bool {
    const int need = (b - 1) >> kStepPageShift;
    if (need < avail) return true;
    SpinClock clk;
    for (unsigned polls = 1;; ++polls) {
      int owed = 0x7fffffff;
      if (lane < kStepLoaders) owed = (lane >> 2) + ld_acquire_cta(S.loaded + lane * 4) * (kStepLoaders / 4);
      avail = (int)__reduce_min_sync(0xffffffffu, (unsigned)owed);
      if (need < avail) return true;
      const bool stop = (polls & 255u) == 0u && clk.expired(A.err);
      if (__any_sync(0xffffffffu, stop)) return false;
    }
  };
  bool bad = !pages((int)lds_u16(S.ends + 2));
  if (bar_any(threads, bad)) return false;
  uint32_t ep = S.ends;
  for (int s = 0; s < ((ti.nsteps + 1) & ~1); ++s, ep += 2) {
    bad = !pages((int)lds_u16(ep + 4));
    if (bar_any(threads, bad)) return false;
    sts_s32_if(lane == 0, S.prog, (int)lds_u16(ep));
  }
  return true;
}

// One loader warp: a quarter of every (kStepLoaders / 4)-th page, in batches
// of the pages that have landed (kBatch at most): all of a batch's gathers in
// flight together, then one release for the batch -- a release with gathers
// outstanding waits for them (one page at a time: ~450 cycles a page).
template <typename T, typename TR>
__device__ __forceinline__ bool step_load_rhs(const StepArgs<T>& A, const StepTile& ti, unsigned base, int lw, int lane,
                                              unsigned char* ring, const TR* __restrict__ rhs, uint64_t* full,
                                              uint32_t loaded) {
  using G = StepPageGeom<T>;
  constexpr int kBatch = 4, kStride = kStepLoaders / 4;
  const unsigned npm = (unsigned)A.np - 1u;
  const int e = (lw & 3) * 32 + lane;
  const TR* const rt = rhs + ti.row0;
  int count = 0;  // pages finished
  for (int pg = lw >> 2; pg < ti.npages;) {
    TR r[kBatch];
    T dv[kBatch];
    bool in[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int p = pg + j * kStride;
      const unsigned u = base + (unsigned)p, slot = u & npm, par = (u >> A.np_shift) & 1u;
      in[j] = p < ti.npages && (j == 0 || in[j > 0 ? j - 1 : 0]);
      if (in[j]) {
        if (j == 0) {
          if (!__all_sync(0xffffffffu, mbar_wait(&full[slot], par, A.err))) return false;
        } else {
          in[j] = __all_sync(0xffffffffu, mbar_test_wait(&full[slot], par)) != 0;
        }
      }
      r[j] = TR(0);
      dv[j] = T(0);
      if (in[j]) {
        const unsigned char* pb = ring + slot * G::slot;
        const uint4 m = *reinterpret_cast<const uint4*>(pb + e * 16);
        if constexpr (sizeof(T) == 4) dv[j] = __uint_as_float(m.w);
        else dv[j] = *reinterpret_cast<const double*>(pb + G::dinv + e * 8);
        if (p * kStepPage + e < ti.npos) r[j] = __ldg(rt + (m.z & 0xffffu));
      }
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j)
      if (in[j]) {
        const unsigned slot = (base + (unsigned)pg) & npm;
        reinterpret_cast<T*>(ring + slot * G::slot + G::bytes)[e] = (T)r[j] * dv[j];
        pg += kStride;
        ++count;
      }
    __syncwarp();
    if (lane == 0) st_release_cta(loaded, count);
  }
  return true;
}

// The page warp's wait until `rows` of the tile are solved (bounded).  Its
// reads are of shared memory the solvers have finished with, so the order
// the barrier gives is all that is needed before the page is overwritten.
__device__ __forceinline__ bool step_wait_rows(const int* prog, int rows, int* err) {
  SpinClock clk;
  for (unsigned polls = 1; *(const volatile int*)prog < rows; ++polls) {
    if ((polls & 255u) == 0u && clk.expired(err)) return false;
    __nanosleep(32);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  return true;
}

// rhs: the right-hand side (TR; rounded to T), natural row order.
template <typename T, typename TR, int K>
__global__ void __launch_bounds__(kStepMaxThreads, 1) tri_step_kernel(const StepArgs<T> A, const TR* __restrict__ rhs) {
  using G = StepPageGeom<T>;
  extern __shared__ __align__(128) unsigned char step_smem[];
  unsigned char* ring = step_smem;                                        // np pages, each with its scaled rhs
  T* vals = reinterpret_cast<T*>(step_smem + (size_t)A.np * G::slot);      // window | inbox | zero
  unsigned short* ends = reinterpret_cast<unsigned short*>(vals + A.window + A.inbox + 2);
  __shared__ __align__(8) uint64_t full[kStepMaxPages];
  __shared__ int s_loaded[kStepLoaders];  // pages of the current tile each loader warp has finished
  __shared__ int s_prog;  // rows of the current tile solved
  __shared__ unsigned s_issued[kStepMaxPages];  // last stream page copied into each slot
  __shared__ int s_group;
  if (*A.done != 0) return;  // the whole grid: nothing writes it meanwhile
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned rank = cluster_rank(), cl = cluster_size();
  if (threadIdx.x == 0) {
    for (int s = 0; s < A.np; ++s) {
      mbar_init(&full[s], 1);
      s_issued[s] = ~0u;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    vals[A.window + A.inbox] = T(0);
  }
  const int prod = A.nw + kStepLoaders, import0 = prod + 2;
  unsigned base = 0;  // pages of earlier tiles streamed by this CTA
  bool failed = false;
  for (bool first = true;; first = false) {
    // claim the next group of cl tiles; meanwhile every inbox is emptied
    if (!first && A.claims == (unsigned)A.ngroups) break;  // one claim per cluster: no further group
    if (rank == 0 && threadIdx.x == 0) s_group = A.ngroups > 1 ? (int)atomicInc(A.ticket, A.claims - 1u) : (first ? 0 : 1);
    for (int i = threadIdx.x; i < A.inbox; i += blockDim.x) vals[A.window + i] = sentinel<T>();
    cluster_sync_all();
    const int g = ld_cluster_s32(cluster_map(&s_group, 0));
    if (g >= A.ngroups) {  // the same for the whole cluster
      cluster_sync_all();  // every CTA has read rank 0's claim before that CTA leaves
      break;
    }
    const int q = g * (int)cl + (int)rank;
    if (q < A.ntiles) {
      const StepTile ti = A.tiles[q];
      for (int i = threadIdx.x; i < ti.nsteps + 3; i += blockDim.x)
        ends[i] = A.ends[ti.step0 + min(i, ti.nsteps - 1)];
      if (threadIdx.x < kStepLoaders) s_loaded[threadIdx.x] = 0;
      if (threadIdx.x == 0) s_prog = 0;
      // where the next tile expects this one's exports
      T* out = rank + 1 < cl ? cluster_ptr(vals + A.window, q + 1 < A.ntiles ? rank + 1 : rank)
                             : A.mail + (size_t)g * A.inbox;
      const StepShared S{smem_u32(ring), smem_u32(vals), smem_u32(ends), smem_u32(&s_prog), smem_u32(s_loaded)};
      __syncthreads();
      if (wid < A.nw) {
        if (!failed)
          failed = !step_solve_tile<T, K>(A, ti, base, (int)threadIdx.x, S, out);
      } else if (wid < prod) {
        failed = !step_load_rhs<T, TR>(A, ti, base, wid - A.nw, lane, ring, rhs, full,
                                        smem_u32(s_loaded + (wid - A.nw)));
      } else if (wid == prod) {
        // one lane, in page order: lanes of one warp waiting on different
        // barriers would hold each other up (a try_wait suspends the warp)
        if (lane == 0) {
          const unsigned char* src = A.pages + (size_t)ti.page0 * G::bytes;
          for (int pg = 0; pg < ti.npages; ++pg) {
            const unsigned u = base + (unsigned)pg, slot = u & ((unsigned)A.np - 1u);
            // the slot's page of the lap before: read by every warp
            if (!step_wait_rows(&s_prog, (pg - A.np + 1) * kStepPage, A.err)) {
              failed = true;
              break;
            }
            mbar_expect_tx(&full[slot], G::bytes);
            tma_load_1d(ring + slot * G::slot, src + (size_t)pg * G::bytes, G::bytes, &full[slot]);
            s_issued[slot] = u;
            // L2 ahead of the ring: the stream is read once per launch
            if (pg + A.np < ti.npages) tma_prefetch_l2(src + (size_t)(pg + A.np) * G::bytes, G::bytes);
          }
        }
        __syncwarp();
      } else if (wid == prod + 1) {
        if (!failed) failed = !step_gate_tile<T>(A, ti, lane, S);
      } else if (rank == 0 && g > 0) {
        // the previous cluster's last tile: its exports, in its step order
        const T* mail = A.mail + (size_t)(g - 1) * A.inbox;
        const int cnt = A.tiles[q - 1].nexp;
        constexpr int kLane = kStepImporters * 32;
        for (int i0 = (wid - import0) * 32 + lane; i0 < cnt && !failed; i0 += kLane * kStepImportBatch) {
          unsigned pend = 0;
#pragma unroll
          for (int j = 0; j < kStepImportBatch; ++j) pend |= i0 + j * kLane < cnt ? 1u << j : 0u;
          SpinClock clk;
          for (unsigned polls = 1; pend; ++polls) {
            T v[kStepImportBatch];
#pragma unroll
            for (int j = 0; j < kStepImportBatch; ++j)
              if (pend >> j & 1u) v[j] = ld_relaxed(mail + i0 + j * kLane);
#pragma unroll
            for (int j = 0; j < kStepImportBatch; ++j)
              if ((pend >> j & 1u) && !is_sentinel(v[j])) {
                *(volatile T*)(vals + A.window + i0 + j * kLane) = v[j];
                st_relaxed(const_cast<T*>(mail) + i0 + j * kLane, sentinel<T>());
                pend &= ~(1u << j);
              }
            if (pend && (polls & 63u) == 0u && clk.expired(A.err)) {
              failed = true;
              break;
            }
          }
        }
        __syncwarp();
      }
      base += (unsigned)ti.npages;
    }
    __syncthreads();
    cluster_sync_all();  // the group's pushes are complete before any inbox is emptied or freed
  }
  // every issued copy lands before the shared memory goes away: only the last
  // copy into each slot can still be in flight (after a timeout)
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int s = 0; s < A.np; ++s) {
      const unsigned u = s_issued[s];
      if (u == ~0u) continue;
      const uint64_t w0 = globaltimer_ns();
      while (!mbar_try_wait(&full[s], (u >> A.np_shift) & 1u) && globaltimer_ns() - w0 < kSpinBudgetNs) {
      }
    }
  }
}

}  // namespace gb
