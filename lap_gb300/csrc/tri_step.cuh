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
// is as short as it can be made (165 to 310 cycles a level of 32 to 128
// rows, FP32):
//   * a tile is solved by `nw` solver warps in lock step: one STEP is up to
//     32*nw rows of one level, a named barrier ends it.  The barrier makes
//     the tile's values plain shared-memory loads -- no sentinel, no poll,
//     no counter -- and frees staged rows and value places without further
//     signalling;
//   * a row is two or three 16-byte loads from the staged page: its values'
//     places in shared memory (resolved at plan time: its tile's own, the
//     inbox, or a zero) and its coefficients.  They are loaded one step
//     ahead;
//   * the rows' static data is one stream of kStepPage-row pages in step
//     order, copied by TMA into a ring by the page warp;
//   * right-hand sides are scaled into place by loader warps.  In natural
//     order (NAT: wide levels) each row has its own place in shared memory,
//     which holds its scaled right-hand side and then its value, so both
//     move by whole lines; else a loader gathers a page's right-hand sides
//     row by row, and solvers store their values row by row;
//   * the stager warp counts the rows whose data is there, and the gate warp
//     joins the solvers' barrier only once the next rows are: solver warps
//     check nothing and branch on nothing;
//   * a tile depends on the previous tile only.  That tile pushes the values
//     its successor needs into the successor's inbox: through distributed
//     shared memory inside a cluster (~450 cycles), through a small mailbox
//     in global memory between clusters (~1 us; import warps poll it and put
//     the sentinel back, so no output vector needs a sentinel fill).
//
// Measured against the record kernel, IC(0) solves (lower / upper with r'w):
// 128^3 split 200 / 248 -> 88 / 106 us, FP64 271 / 337 -> 142 / 158 us; 64^3
// split 243 / 245 -> 38 / 48 us; 97 x 61 x 83 207 / 253 -> 49 / 60 us (its
// planes fit no power-of-two tile); 1000 x 700 377 / 383 -> 151 / 164 us.
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

constexpr int kStepImportDepth = 3;  // groups of the mailbox an import warp keeps in flight
constexpr int kStepMaxThreads = 20 * 32;
static_assert(kStepMaxThreads >= step_threads(true, kStepMaxWarps) && kStepMaxThreads >= step_threads(false, kStepMaxWarps),
              "the widest launch");

template <typename T>
struct StepArgs {
  int ntiles, ngroups, nw, np, np_shift, window, inbox, max_steps, max_pages;
  unsigned claims;                        // ticket claims of one launch (it wraps to 0)
  const StepTile* __restrict__ tiles;     // [ntiles]
  const unsigned short* __restrict__ ends;  // steps' end positions, tile after tile
  const unsigned short* __restrict__ needs;  // NAT: chunks loaded before a page's rows may be read
  const unsigned short* __restrict__ thr;    // NAT: positions solved before a chunk may be stored
  const T* __restrict__ dinv;                // NAT: 1/d, natural row order
  int lower;
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
__device__ __forceinline__ void sts_s32(uint32_t a, int v) {
  asm volatile("st.volatile.shared.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
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
__device__ __forceinline__ int ld_acquire_cta(uint32_t a) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_cta(uint32_t a, int v) {
  asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ int lds_s32(uint32_t a) {
  int v;
  asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
// The steps' barrier, of the solver warps and the gate.  (A barrier that also
// reduces a predicate, barrier.red, cost 90-400 cycles more a step: 1000 x
// 700 solve 503 us against 189, 128^3 127 against 90.)
__device__ __forceinline__ void step_barrier(int threads) {
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}
__device__ __forceinline__ void st_release_if(bool on, uint32_t a, int v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.release.cta.shared::cta.b32 [%1], %2;\n}" ::"r"((int)on),
               "r"(a), "r"(v)
               : "memory");
}

// A row as the solver holds it: where its values lie, its coefficients and
// its scaled right-hand side.
template <typename T, int K>
struct StepRow {
  uint32_t at[K], own;
  T l[K];
  T acc;
  unsigned s01, s23, le;
};

// Where a tile's staged data lies in shared memory (32-bit addresses).
struct StepShared {
  uint32_t ring, vals, ends, prog, staged, loaded, late;
};

// One solver warp's part of a tile.  K: the most dependencies a row has.
// Per step and warp: the row's values (LDS), the next step's row (LDS, off
// the chain), K FMAs, the value's store, the barrier -- and no branch but the
// rare wait for a value: each one costs the chain tens of cycles (a check of
// the staged rows and a page-wise progress word here instead of in the gate:
// 1000 x 700 solve 337 us against 189).  So nothing here fails: a value
// waited for in vain is taken as NaN and marks the tile late, and rows that
// were not staged in time are whatever the ring holds -- always rows of this
// plan, whose places are in bounds; the error word is set either way.
template <typename T, int K, bool NAT>
__device__ __forceinline__ void step_solve_tile(const StepArgs<T>& A, const StepTile& ti, unsigned base, int first,
                                                const StepShared& S, T* out) {
  using G = StepPageGeom<T>;
  constexpr uint32_t kSlot = NAT ? G::bytes : G::slot;
  const unsigned npm = (unsigned)A.np - 1u;
  const unsigned wmask = (unsigned)A.window - 1u;
  const int threads = (A.nw + 1) * 32;  // solvers and gate
  T* const yt = A.y + ti.row0;
  // the row at position a + first of [a, b), from its staged page; past b
  // the last one again, which is then not stored
  auto load = [&](StepRow<T, K>& r, int a, int b) {
    const unsigned p = (unsigned)min(a + first, b - 1);
    const uint32_t pg = S.ring + ((base + (p >> kStepPageShift)) & npm) * kSlot;
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
    if constexpr (!NAT) lds_value(pg + G::bytes + e * (uint32_t)sizeof(T), r.acc);
    r.s01 = m.x;
    r.s23 = m.y;
    r.le = m.z;
  };
  auto decode = [&](StepRow<T, K>& r) {
    r.at[0] = S.vals + (r.s01 & 0xffffu) * (uint32_t)sizeof(T);
    r.at[1] = S.vals + (r.s01 >> 16) * (uint32_t)sizeof(T);
    if constexpr (K > 2) r.at[2] = S.vals + (r.s23 & 0xffffu) * (uint32_t)sizeof(T);
    if constexpr (K > 3) r.at[3] = S.vals + (r.s23 >> 16) * (uint32_t)sizeof(T);
    if constexpr (NAT) r.own = S.vals + (r.le & 0xffffu) * (uint32_t)sizeof(T);
  };
  int a = 0, b = (int)lds_u16(S.ends), nb = (int)lds_u16(S.ends + 2);
  uint32_t ep = S.ends + 4;
  // one step: solves `c`, loads the next rows into `n`
  auto step = [&](StepRow<T, K>& c, StepRow<T, K>& n) {
    T v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) lds_value(c.at[k], v[k]);
    if constexpr (NAT) lds_value(c.own, c.acc);  // the scaled rhs, until the row is solved
    const int nnb = (int)lds_u16(ep);  // the list ends in copies of the last end
    ep += 2;
    load(n, b, nb);
    bool miss = false;  // only the inbox's places can hold the sentinel
#pragma unroll
    for (int k = 0; k < K; ++k) miss |= is_sentinel(v[k]);
    if (miss) {
      SpinClock clk;
      for (unsigned polls = 1; miss; ++polls) {
        miss = false;
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (is_sentinel(v[k])) {
            lds_value(c.at[k], v[k]);
            miss |= is_sentinel(v[k]);
          }
        if (miss && (polls & 255u) == 0u && (lds_s32(S.late) != 0 || clk.expired(A.err))) {
          sts_s32(S.late, 1);
          miss = false;  // the sentinel is a NaN
        }
      }
    }
    // an FMA never returns the sentinel (a signalling NaN)
    T acc = c.acc;
#pragma unroll
    for (int k = 0; k < K; ++k) acc = fma_rn(-c.l[k], v[k], acc);
    decode(n);  // beside the FMAs: its loads are back with the values
    const int p = a + first;
    const bool on = p < b;
    sts_value_if(on, NAT ? c.own : S.vals + ((unsigned)p & wmask) * (uint32_t)sizeof(T), acc);
    const unsigned ex = c.le >> 16;
    st_export_if(on && ex != kStepNone, out + ex, acc);
    step_barrier(threads);
    if constexpr (!NAT) st_global_if(on && (c.le & 0xffffu) < (unsigned)ti.npos, yt + (c.le & 0xffffu), acc);
    a = b;
    b = nb;
    nb = nnb;
  };
  StepRow<T, K> r0, r1;
  step_barrier(threads);  // the first two steps' rows are staged
  load(r0, a, b);
  decode(r0);
  for (int s = 0; s < ti.nsteps; s += 2) {  // an odd count's last step is empty
    step(r0, r1);
    step(r1, r0);
  }
}

// The gate warp: joins the steps' barriers, which it enters only once the
// rows of the step after next are staged, and publishes how far the steps
// are.  It does nothing else: with the stager's work in it it took ~340
// cycles a step and set the pace.
template <typename T>
__device__ __forceinline__ bool step_gate_tile(const StepArgs<T>& A, const StepTile& ti, int lane,
                                               const StepShared& S) {
  const int threads = (A.nw + 1) * 32;
  int staged = 0;
  bool ok = true;
  auto wait = [&](int end) {
    SpinClock clk;
    for (unsigned polls = 1; ok; ++polls) {
      staged = ld_acquire_cta(S.staged);
      if (staged >= end) return;
      if ((polls & 255u) == 0u && clk.expired(A.err)) ok = false;
    }
    staged = 0x7fffffff;  // gave up: the solvers run on unguarded
  };
  int b = (int)lds_u16(S.ends), nb = (int)lds_u16(S.ends + 2), nnb = (int)lds_u16(S.ends + 4);
  if (nb > staged) wait(nb);
  step_barrier(threads);
  uint32_t at = S.ends + 6;
  const int steps = (ti.nsteps + 1) & ~1;
  for (int s = 0; s < steps; ++s, at += 2) {
    if (nnb > staged) wait(nnb);
    step_barrier(threads);
    st_release_if(lane == 0, S.prog, b);
    b = nb;
    nb = nnb;
    nnb = (int)lds_u16(at);
  }
  return ok;
}

// The stager warp: publishes how many rows are staged, page by page -- landed
// (NAT; the loaders have seen to it otherwise) and with their scaled
// right-hand sides in place.
template <typename T, bool NAT>
__device__ __forceinline__ bool step_stage_tile(const StepArgs<T>& A, const StepTile& ti, unsigned base, int lane,
                                                const StepShared& S, const unsigned short* needs, uint64_t* full) {
  constexpr int kLoaders = NAT ? kStepChunkWarps : kStepLoaders;
  int avail = 0;  // NAT: chunks loaded; else pages with their right-hand sides
  for (int page = 0; page < ti.npages; ++page) {
    if constexpr (NAT) {
      const unsigned u = base + (unsigned)page, slot = u & ((unsigned)A.np - 1u);
      if (!__all_sync(0xffffffffu, mbar_wait(&full[slot], (u >> A.np_shift) & 1u, A.err))) return false;
    }
    const int need = NAT ? (int)needs[page] : page + 1;
    if (avail < need) {  // the least of the loader warps' counts
      SpinClock clk;
      for (unsigned polls = 1;; ++polls) {
        const int c = lane < kLoaders ? ld_acquire_cta(S.loaded + lane * 4) : 0x7fffffff;
        avail = (int)__reduce_min_sync(0xffffffffu, (unsigned)c);
        if (avail >= need) break;
        const bool stop = (polls & 255u) == 0u && clk.expired(A.err);
        if (__any_sync(0xffffffffu, stop)) return false;
      }
    }
    if (!NAT) page = avail - 1;  // as many as they have finished
    if (lane == 0) st_release_cta(S.staged, (page + 1) * kStepPage);
  }
  return true;
}

// Natural order (NAT): the rows' scaled right-hand sides go into the rows'
// own places in row order, by whole lines; once the rows of a chunk are
// solved the same warps write them out, by whole lines.
template <typename T, typename TR>
__device__ __forceinline__ bool step_stream_rows(const StepArgs<T>& A, const StepTile& ti, int lw, int lane, T* vals,
                                                 const unsigned short* thr, const int* prog,
                                                 const TR* __restrict__ rhs, uint32_t loaded) {
  constexpr int kBatch = 4;
  const int chunks = step_chunks(ti.npos);
  const TR* const rt = rhs + ti.row0;
  const T* const dt = A.dinv + ti.row0;
  for (int c0 = 0; c0 < chunks; c0 += kBatch) {
    TR r[kBatch];
    T dv[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int o = (c0 + j) * kStepChunk + lw * 32 + lane;
      if (c0 + j < chunks && o < ti.npos) {
        const int i = A.lower ? o : ti.npos - 1 - o;
        r[j] = __ldg(rt + i);
        dv[j] = __ldg(dt + i);
      }
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int o = (c0 + j) * kStepChunk + lw * 32 + lane;
      if (c0 + j < chunks && o < ti.npos) {
        const int i = A.lower ? o : ti.npos - 1 - o;
        vals[step_place(i)] = (T)r[j] * dv[j];
      }
    }
    __syncwarp();
    if (lane == 0) st_release_cta(loaded, min(c0 + kBatch, chunks));
  }
  T* const yt = A.y + ti.row0;
  for (int c = 0; c < chunks; ++c) {
    const int need = thr[c];
    SpinClock clk;
    bool ok = true;
    for (unsigned polls = 1; ld_acquire_cta(smem_u32(prog)) < need; ++polls) {
      if ((polls & 255u) == 0u && clk.expired(A.err)) {
        ok = false;
        break;
      }
      __nanosleep(64);
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    const int o = c * kStepChunk + lw * 32 + lane;
    if (o < ti.npos) {
      const int i = A.lower ? o : ti.npos - 1 - o;
      yt[i] = vals[step_place(i)];
    }
  }
  return true;
}

// One loader warp (!NAT): a quarter of every page, in batches
// of the pages that have landed (kBatch at most): all of a batch's gathers in
// flight together, then one release for the batch -- a release with gathers
// outstanding waits for them (one page at a time: ~450 cycles a page).
template <typename T, typename TR>
__device__ __forceinline__ bool step_load_rhs(const StepArgs<T>& A, const StepTile& ti, unsigned base, int lw, int lane,
                                              unsigned char* ring, const TR* __restrict__ rhs, uint64_t* full,
                                              uint32_t loaded) {
  using G = StepPageGeom<T>;
  static_assert(kStepLoaders * 32 == kStepPage, "a loader warp takes a quarter of each page");
  constexpr int kBatch = 4;
  const unsigned npm = (unsigned)A.np - 1u;
  const int e = lw * 32 + lane;
  const TR* const rt = rhs + ti.row0;
  for (int pg = 0; pg < ti.npages;) {
    TR r[kBatch];
    T dv[kBatch];
    bool in[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int p = pg + j;
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
        ++pg;
      }
    __syncwarp();
    if (lane == 0) st_release_cta(loaded, pg);
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
template <typename T, typename TR, int K, bool NAT>
__global__ void __launch_bounds__(kStepMaxThreads, 1) tri_step_kernel(const StepArgs<T> A, const TR* __restrict__ rhs) {
  using G = StepPageGeom<T>;
  extern __shared__ __align__(128) unsigned char step_smem[];
  constexpr uint32_t kSlot = NAT ? G::bytes : G::slot;
  constexpr int kLoaders = NAT ? kStepChunkWarps : kStepLoaders;
  unsigned char* ring = step_smem;                                     // np pages (!NAT: with their scaled rhs)
  T* vals = reinterpret_cast<T*>(step_smem + (size_t)A.np * kSlot);     // own places | inbox | zero
  unsigned short* ends = reinterpret_cast<unsigned short*>(vals + A.window + A.inbox + 2);
  unsigned short* needs = ends + A.max_steps + 4;                       // NAT
  unsigned short* thr = needs + A.max_pages;                            // NAT
  __shared__ __align__(8) uint64_t full[kStepMaxPages];
  __shared__ int s_loaded[kLoaders];  // pages of the current tile each loader warp has finished
  __shared__ int s_late;  // a value of the current tile was waited for in vain
  __shared__ int s_prog, s_staged;  // rows of the current tile solved, and staged
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
  // rows that are never staged (a timeout) must still be in bounds
  for (unsigned i = threadIdx.x; i < A.np * kSlot / 16u; i += blockDim.x) reinterpret_cast<uint4*>(ring)[i] = make_uint4(0, 0, 0, 0);
  const int prod = A.nw + kLoaders, import0 = prod + 3;
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
      for (int i = threadIdx.x; i < ti.nsteps + 4; i += blockDim.x)
        ends[i] = A.ends[ti.step0 + min(i, ti.nsteps - 1)];
      if constexpr (NAT) {
        for (int i = threadIdx.x; i < ti.npages; i += blockDim.x) needs[i] = A.needs[ti.page0 + i];
        for (int i = threadIdx.x; i < step_chunks(ti.npos); i += blockDim.x) thr[i] = A.thr[ti.thr0 + i];
      }
      if (threadIdx.x < kLoaders) s_loaded[threadIdx.x] = 0;
      if (threadIdx.x == 0) s_prog = s_staged = s_late = 0;
      // where the next tile expects this one's exports
      T* out = rank + 1 < cl ? cluster_ptr(vals + A.window, q + 1 < A.ntiles ? rank + 1 : rank)
                             : A.mail + (size_t)g * A.inbox;
      const StepShared S{smem_u32(ring), smem_u32(vals), smem_u32(ends), smem_u32(&s_prog), smem_u32(&s_staged),
                         smem_u32(s_loaded), smem_u32(&s_late)};
      __syncthreads();
      if (wid < A.nw) {
        step_solve_tile<T, K, NAT>(A, ti, base, (int)threadIdx.x, S, out);
      } else if (wid < prod) {
        const uint32_t count = smem_u32(s_loaded + (wid - A.nw));
        if constexpr (NAT)
          failed = !step_stream_rows<T, TR>(A, ti, wid - A.nw, lane, vals, thr, &s_prog, rhs, count);
        else
          failed = !step_load_rhs<T, TR>(A, ti, base, wid - A.nw, lane, ring, rhs, full, count);
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
            tma_load_1d(ring + slot * kSlot, src + (size_t)pg * G::bytes, G::bytes, &full[slot]);
            s_issued[slot] = u;
            // L2 ahead of the ring: the stream is read once per launch
            if (pg + A.np < ti.npages) tma_prefetch_l2(src + (size_t)(pg + A.np) * G::bytes, G::bytes);
          }
        }
        __syncwarp();
      } else if (wid == prod + 1) {
        failed = !step_gate_tile<T>(A, ti, lane, S) || failed;
      } else if (wid == prod + 2) {
        if (!failed) failed = !step_stage_tile<T, NAT>(A, ti, base, lane, S, needs, full);
      } else if (rank == 0 && g > 0) {
        // the previous cluster's last tile: its exports, in its step order
        T* mail = A.mail + (size_t)(g - 1) * A.inbox;
        const int cnt = A.tiles[q - 1].nexp;
        // A warp takes every kWarps-th group of 32 and keeps kDepth groups'
        // loads in flight; what has arrived goes into the inbox at once, and
        // the warp moves on past the leading groups that are complete.
        // (Per-lane places with their own polls ran into one L2 round trip a
        // place: 4-5 us behind, against ~1.)
        constexpr int kWarps = step_importers(NAT), kDepth = kStepImportDepth;
        SpinClock clk;
        int grp = wid - import0;
        for (unsigned polls = 1; grp * 32 < cnt; ++polls) {
          T v[kDepth];
#pragma unroll
          for (int j = 0; j < kDepth; ++j)
            v[j] = ld_relaxed(mail + min((grp + j * kWarps) * 32 + lane, cnt - 1));
          int lead = 0;
#pragma unroll
          for (int j = 0; j < kDepth; ++j) {
            const int at = (grp + j * kWarps) * 32 + lane;
            const bool here = !is_sentinel(v[j]);
            sts_value_if(here && at < cnt, smem_u32(vals + A.window) + (uint32_t)at * (uint32_t)sizeof(T), v[j]);
            const bool all = __all_sync(0xffffffffu, here);
            if (lead == j && all) {
              if (at < cnt) st_relaxed(mail + at, sentinel<T>());
              ++lead;
            }
          }
          grp += lead * kWarps;
          if (lead) clk = SpinClock();
          else if ((polls & 63u) == 0u && __any_sync(0xffffffffu, clk.expired(A.err))) {
            failed = true;
            break;
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
