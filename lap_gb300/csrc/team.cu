// team.cu -- whole PCG recurrences with line_jacobi or no preconditioner in
// one launch, for systems that fit the device's blocks at once.
//
// What bounds a small system's iteration as two (batches: four) launches is
// the launches: 256 x 256 took 23.4 us an iteration, of which the FP64 work
// is 1.6 us and the bytes, all in L2, less.  Here a team of blocks per system
// runs the recurrence by itself: a thread keeps its rows' r, p and q in
// registers, a block its matrix entries in shared memory where they fit, only
// w goes through L2.  The team meets twice an iteration -- at p'q and at r'r,
// r'w -- and both meetings are the reduction itself: each block sends
// its partial sums to every other, polls its own mail (value as flag) and adds
// them in the same order, so all of them hold the same scalars and take the
// same decisions, and results do not depend on timing.
//
// Mail: a block has a place for every peer's pair of sums in each of four
// sets used in turn, and only the block itself reads them (all blocks polling
// one array of slots cost 256 x 256 6 us an iteration more).  Meeting t uses
// set t mod 4; the reader puts the sentinel back at once, and the next write
// of that set comes two releases later.  The second meeting of an iteration
// releases the new w (fence before the sums).
//
// Measured, an iteration: 256 x 256 FP64 23.6 -> 11.1 us, 1,024 rows 19.5 ->
// 6.6 us, 64^3 35.8 -> 20.6 us; 48 kNN systems of 1,000 to 20,000 rows 50.8
// -> 30.4 us.  Past the device's blocks (467,000 rows) the captured loop's
// bandwidth kernels are as fast: 700 x 700 42.6 us either way.
//
// All blocks must run at once (cooperative launch).  Every poll is bounded;
// when one gives up the block leaves, the others' polls end the same way, and
// the error word says why.
#include <algorithm>
#include <mutex>

#include "gb_common.cuh"
#include "kernels.h"
#include "pcg_state.cuh"
#include "team.h"

namespace gb {

namespace {

constexpr int kTeamWarps = kTeamThreads / 32;  // worker warps; one more does the scalars

__device__ __forceinline__ void team_bar(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(kTeamThreads + 32) : "memory");
}

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Sums of two values over the warp in six adds' time instead of ten: after
// the first exchange lanes 0-15 hold a's halves and lanes 16-31 b's.
// Valid: a in lane 0, b in lane 16.
__device__ __forceinline__ double warp_sum2(double a, double b, int lane) {
  const double keep = lane & 16 ? b : a, give = lane & 16 ? a : b;
  double v = keep + __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void st_pair(double* p, double a, double b) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ void ld_pair(const double* p, double& a, double& b) {
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "l"(p) : "memory");
}

// The scalar warp's half of a meeting: adds the block's warps' partials
// (part[NV][warps]), writes the sums into every block's mail, reads its own.
// sum: this lane's share, peers lane, lane + 32, ...  False when a poll gave up.
template <int NV>
__device__ __forceinline__ bool team_exchange(const double* part, unsigned round, bool release, double* mail, int me,
                                              int k, int lane, double (&sum)[NV], int* err) {
  double v[2] = {0.0, 0.0};
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i] = lane < kTeamWarps ? part[i * kTeamWarps + lane] : 0.0;
#pragma unroll
    for (int o = kTeamWarps / 2; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    v[i] = publishable(__shfl_sync(0xffffffffu, v[i], 0));
  }
  const size_t set = (size_t)(round & 3u) * 2 * k;  // [block][set][peer][2]
  if (release) fence_gpu();
  for (int s = lane; s < k; s += 32) st_pair(mail + (size_t)s * 8 * k + set + 2 * me, v[0], v[1]);
  bool ok = true;
#pragma unroll
  for (int i = 0; i < NV; ++i) sum[i] = 0.0;
  double* const mine = mail + (size_t)me * 8 * k + set;
  constexpr int kIn = 4;
  for (int s0 = lane; s0 < k; s0 += 32 * kIn) {
    double x[kIn][2];
#pragma unroll
    for (int u = 0; u < kIn; ++u) {
      x[u][0] = x[u][1] = 0.0;
      if (s0 + 32 * u < k) ld_pair(mine + 2 * (s0 + 32 * u), x[u][0], x[u][1]);
    }
    SpinClock clk;
    for (unsigned polls = 1;; ++polls) {
      bool miss = false;
#pragma unroll
      for (int u = 0; u < kIn; ++u)
        if (is_sentinel(x[u][0]) || is_sentinel(x[u][1])) {
          ld_pair(mine + 2 * (s0 + 32 * u), x[u][0], x[u][1]);
          miss = miss || is_sentinel(x[u][0]) || is_sentinel(x[u][1]);
        }
      if (!miss) break;
      if ((polls & 255u) == 0u && clk.expired(err)) {
        ok = false;
        break;
      }
    }
#pragma unroll
    for (int u = 0; u < kIn; ++u)
      if (s0 + 32 * u < k) st_pair(mine + 2 * (s0 + 32 * u), sentinel<double>(), sentinel<double>());
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (s0 == lane) sum[i] = x[0][i];
      else sum[i] += x[0][i];
#pragma unroll
      for (int u = 1; u < kIn; ++u)
        if (s0 - lane + 32 * u < k) sum[i] += x[u][i];  // uniform: no adds for groups there are not
    }
  }
  return __all_sync(0xffffffffu, ok) != 0;
}

template <typename T, typename TA>
struct TeamArgs {
  TeamData<T, TA> d;
  const int *cta_sys, *cta0;
  double* mail;
  const long long* mail0;  // [systems] first element of the system's mail
  int cached;  // cached: entries a block has room for in shared memory
};

template <typename T, typename TA, int R>
__global__ void __launch_bounds__(kTeamThreads + 32, R >= 3 ? 3 : 2) team_pcg_kernel(const TeamArgs<T, TA> A) {
  extern __shared__ __align__(16) unsigned char team_smem[];
  __shared__ double part[2 * kTeamWarps];
  __shared__ double s_alpha, s_beta;
  __shared__ int s_go, s_done;  // meeting outcomes: 0: go on, else leave
  const TeamData<T, TA>& D = A.d;
  const int sys = A.cta_sys[blockIdx.x], c0 = A.cta0[sys], k = A.cta0[sys + 1] - c0;
  PcgState* const S = D.st + sys;
  if (S->done) return;  // the whole team: its blocks write S only after every block has met
  const int row0 = D.row_off ? D.row_off[sys] : 0;
  const int end = D.row_off ? D.row_off[sys + 1] : D.n;
  const int first_row = row0 + ((int)blockIdx.x - c0) * kTeamThreads * R;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int iter = S->iter;
  // the block's entries, from shared memory where they fit
  const int e0 = D.ia[first_row], e1 = D.ia[min(first_row + kTeamThreads * R, end)];
  const bool cached = A.cached && e1 - e0 <= A.cached;
  TA* const sa = reinterpret_cast<TA*>(team_smem);
  int* const sj = reinterpret_cast<int*>(sa + A.cached);
  if (cached)
    for (int e = e0 + threadIdx.x; e < e1; e += kTeamThreads + 32) {
      sa[e - e0] = D.a[e];
      sj[e - e0] = D.ja[e];
    }
  __syncthreads();

  if (wid == kTeamWarps) {
    // The scalar warp: FP64 divisions and roots are some twenty instructions
    // on a pipe that takes 64 cycles a warp for each, so one warp does them,
    // and those the next product does not need while the others compute it.
    double rho = S->rho, rho_prev = S->rho_prev, rr = S->rr, pq = S->pq;
    const double tolrel = S->tolrel;
    const int maxit = S->maxit, hist_len = D.hist ? S->hist_len : 0;
    int done = 0, flag = S->flag, status = S->status;
    const bool lead = (int)blockIdx.x == c0 && lane == 0;
    double* const mail = A.mail + A.mail0[sys];
    const int me = (int)blockIdx.x - c0;
    if (lane == 0) {
      s_beta = iter == 0 ? 0.0 : rho / rho_prev;
      s_done = 0;
    }
    team_bar(3);
    for (unsigned round = 0; !done; round += 2) {
      team_bar(1);  // p'q partials are there
      double m1[1], m2[2];
      bool ok = team_exchange<1>(part, round, false, mail, me, k, lane, m1, D.err);
      pq = warp_sum(m1[0]);
      const double alpha = rho / pq;
      if (!ok) {
        done = 1;
        status = GB_TIMEOUT;
      } else if (!(pq > 0.0 && isfinite(alpha))) {
        done = 1;
        flag = 2;
        status = GB_BREAKDOWN;
      }
      if (lane == 0) {
        s_alpha = alpha;
        s_go = done;
      }
      team_bar(2);
      if (done) break;
      team_bar(1);  // r'r, r'w partials, and w is stored
      ok = team_exchange<2>(part, round + 1, true, mail, me, k, lane, m2, D.err);
      fence_gpu();  // the other blocks' w, read by every worker below
      if (lane == 0) s_go = !ok;
      team_bar(2);  // workers start on the next product
      if (!ok) {
        done = 1;
        status = GB_TIMEOUT;
        break;
      }
      const double both = warp_sum2(m2[0], m2[1], lane);
      rr = __shfl_sync(0xffffffffu, both, 0);
      const double rw = __shfl_sync(0xffffffffu, both, 16);
      // cg.c's stopping rule, as pcg_check
      const double res = sqrt(rr);
      ++iter;
      if (lead && iter < hist_len) D.hist[iter] = res;
      if (!(res == res) || isinf(res)) {
        done = 1;
        flag = 2;
        status = GB_BREAKDOWN;
      } else if (res < tolrel) {
        done = 1;
        flag = 0;
        status = GB_OK;
      } else if (iter > maxit) {
        done = 1;
        flag = 1;
        status = GB_MAXIT;
      }
      if (!done || D.roll_done) {
        rho_prev = rho;
        rho = rw;
      }
      const double beta = rho / rho_prev;
      if (lane == 0) {
        s_beta = beta;
        s_done = done;
      }
      team_bar(3);
    }
    if (lead) {
      S->rho = rho;
      S->rho_prev = rho_prev;
      S->rr = rr;
      S->pq = pq;
      S->iter = iter;
      S->flag = flag;
      S->status = status;
      S->done = 1;
    }
    return;
  }

  const TA* const av = cached ? sa : D.a;
  const int* const jv = cached ? sj : D.ja;
  const int shift = cached ? e0 : 0;
  const T* const w = D.w + row0;
  int g[R], rs[R], re[R];
  T r[R], p[R], q[R], wi[R];
  int longest = 0;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    g[j] = first_row + j * kTeamThreads + (int)threadIdx.x;
    const bool own = g[j] < end;
    if (!own) g[j] = -1;
    rs[j] = own ? D.ia[g[j]] - shift : 0;
    re[j] = own ? D.ia[g[j] + 1] - shift : 0;
    longest = max(longest, re[j] - rs[j]);
    r[j] = own ? D.r[g[j]] : T(0);
    wi[j] = own && D.d_r ? D.d_r[g[j]] * r[j] : r[j];
    p[j] = own && iter > 0 ? D.p[g[j]] : T(0);
    q[j] = own && iter > 0 ? D.q[g[j]] : T(0);
  }
  for (;; ++iter) {
    // A w: all rows' entries in step, so that R rows' gathers are in flight
    TA s[R];
    T dr[R], xo[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      s[j] = TA(0);
      dr[j] = g[j] >= 0 && D.d_r ? __ldg(D.d_r + g[j]) : T(1);
      xo[j] = g[j] >= 0 ? D.x[g[j]] : T(0);
    }
    constexpr int kStep = R >= 3 ? 2 : 4;
    for (int e = 0; e < longest; e += kStep) {
      TA a[R][kStep], v[R][kStep];
#pragma unroll
      for (int j = 0; j < R; ++j)
#pragma unroll
        for (int u = 0; u < kStep; ++u) {
          const bool in = rs[j] + e + u < re[j];
          a[j][u] = in ? av[rs[j] + e + u] : TA(0);
          v[j][u] = in ? (TA)ld_relaxed(w + jv[rs[j] + e + u]) : TA(0);
        }
#pragma unroll
      for (int j = 0; j < R; ++j)
#pragma unroll
        for (int u = 0; u < kStep; ++u)
          if (rs[j] + e + u < re[j]) s[j] = fma_rn(a[j][u], v[j][u], s[j]);
    }
    team_bar(3);  // beta, and whether the last iteration was the last
    if (s_done) break;
    const bool first = iter == 0;
    const T beta = (T)s_beta;
    double m = 0.0;
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (g[j] >= 0) {
        p[j] = first ? wi[j] : fma_rn(beta, p[j], wi[j]);
        q[j] = first ? (T)s[j] : fma_rn(beta, q[j], (T)s[j]);
        m = fma((double)p[j], (double)q[j], m);
      }
    m = warp_sum(m);
    if (lane == 0) part[wid] = m;
    team_bar(1);
    team_bar(2);
    if (s_go) break;
    const T al = (T)s_alpha, nal = -al;
    double m0 = 0.0, m1 = 0.0;
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (g[j] >= 0) {
        r[j] = fma_rn(nal, q[j], r[j]);
        wi[j] = D.d_r ? dr[j] * r[j] : r[j];
        D.w[g[j]] = wi[j];
        m0 = fma((double)r[j], (double)r[j], m0);
        m1 = fma((double)r[j], (double)wi[j], m1);
      }
    m0 = warp_sum2(m0, m1, lane);
    if ((lane & 15) == 0) part[(lane >> 4) * kTeamWarps + wid] = m0;
    team_bar(1);
#pragma unroll
    for (int j = 0; j < R; ++j)  // while the team meets
      if (g[j] >= 0) D.x[g[j]] = fma_rn(al, p[j], xo[j]);
    team_bar(2);
    if (s_go) break;
  }
#pragma unroll
  for (int j = 0; j < R; ++j)
    if (g[j] >= 0) {
      D.r[g[j]] = r[j];
      D.p[g[j]] = p[j];
      D.q[g[j]] = q[j];
    }
}

template <typename T, typename TA>
void (*team_kernel(int rows))(const TeamArgs<T, TA>) {
  return rows == 1 ? team_pcg_kernel<T, TA, 1> : rows == 2 ? team_pcg_kernel<T, TA, 2>
         : rows == 3 ? team_pcg_kernel<T, TA, 3> : team_pcg_kernel<T, TA, 4>;
}

// Blocks of every instantiation of `rows` rows a thread that fit the device.
int resident(int rows, size_t smem) {
  const void* k[3] = {(const void*)team_kernel<double, double>(rows), (const void*)team_kernel<float, float>(rows),
                      (const void*)team_kernel<double, float>(rows)};
  int least = 1 << 30;
  for (const void* f : k) {
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTeamMaxSmem) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, kTeamThreads + 32, smem) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    least = std::min(least, per);
  }
  return least * device_sm_count();
}

template <typename V>
int to_device(V** dst, const std::vector<V>& src) {
  GB_CUDA_TRY(cudaMalloc(dst, sizeof(V) * src.size()));
  GB_CUDA_TRY(cudaMemcpy(*dst, src.data(), sizeof(V) * src.size(), cudaMemcpyHostToDevice));
  return GB_OK;
}

}  // namespace

int team_plan_build(int count, const std::vector<int>& row_off, const int* ia, TeamPlan* p) {
  *p = TeamPlan();
  const int n = row_off[count];
  for (int i = 0; i < n; ++i)
    if (ia[i + 1] - ia[i] > kTeamMaxRow) return GB_OK;
  // Rows of a thread: those that leave the fewest to the fullest SM (its two
  // FP64 lanes a cycle are what its blocks share), in the fewest blocks.
  const int sms = device_sm_count();
  auto blocks = [&](int rows) {
    long long c = 0;
    for (int s = 0; s < count; ++s) c += (row_off[s + 1] - row_off[s] + kTeamThreads * rows - 1) / (kTeamThreads * rows);
    return c;
  };
  int rows = 0;
  long long best = 0, c = 0;
  for (int r = 4; r >= 1; --r) {
    const long long b = blocks(r), per_sm = (b + sms - 1) / sms;
    if (per_sm > (r >= 3 ? 3 : 2)) continue;
    if (rows == 0 || per_sm * r < best) {
      rows = r;
      best = per_sm * r;
      c = b;
    }
  }
  if (rows == 0) return GB_OK;
  std::vector<int> cta_sys, cta0{0};
  std::vector<long long> mail0;
  for (int s = 0; s < count; ++s) {
    for (int i = row_off[s]; i < row_off[s + 1]; i += kTeamThreads * rows) {
      cta_sys.push_back(s);
      p->max_nnz = std::max(p->max_nnz, ia[std::min(i + kTeamThreads * rows, row_off[s + 1])] - ia[i]);
    }
    cta0.push_back((int)cta_sys.size());
    const long long k = cta0[s + 1] - cta0[s];
    mail0.push_back(p->mail_len);
    p->mail_len += 8 * k * k;
  }
  p->rows = rows;
  p->ctas = (int)c;
  p->systems = count;
  p->nnz = (long long)ia[n] - ia[0];
  p->smem = (size_t)p->max_nnz * (sizeof(double) + sizeof(int));
  if (p->smem > kTeamMaxSmem || resident(rows, p->smem) < p->ctas) {
    p->smem = 0;
    if (resident(rows, 0) < p->ctas) return GB_OK;
  }
  GB_TRY(to_device(&p->cta_sys, cta_sys));
  cta0.push_back(cta0.back());
  GB_TRY(to_device(&p->cta0, cta0));
  GB_TRY(to_device(&p->mail0, mail0));
  GB_CUDA_TRY(cudaMalloc(&p->mail, sizeof(double) * p->mail_len));
  p->on = true;
  return GB_OK;
}

void team_plan_free(TeamPlan* p) {
  for (void* q : {(void*)p->cta_sys, (void*)p->cta0, (void*)p->mail, (void*)p->mail0})
    if (q) cudaFree(q);
  *p = TeamPlan();
}

int team_debug_silent(TeamPlan* p, int block, PcgState* states) {
  if (!p->on || block >= p->ctas) return GB_BAD_INPUT;
  if (p->debug_block >= 0)
    GB_CUDA_TRY(cudaMemcpy(p->cta_sys + p->debug_block, &p->debug_sys, sizeof(int), cudaMemcpyHostToDevice));
  p->debug_block = -1;
  if (block < 0) return GB_OK;
  const int one = 1;
  GB_CUDA_TRY(cudaMemcpy(&states[p->systems].done, &one, sizeof(int), cudaMemcpyHostToDevice));
  GB_CUDA_TRY(cudaMemcpy(&p->debug_sys, p->cta_sys + block, sizeof(int), cudaMemcpyDeviceToHost));
  GB_CUDA_TRY(cudaMemcpy(p->cta_sys + block, &p->systems, sizeof(int), cudaMemcpyHostToDevice));
  p->debug_block = block;
  return GB_OK;
}

template <typename T, typename TA>
int team_loop(const TeamPlan& p, const TeamData<T, TA>& d, cudaStream_t s) {
  if (!team_runs<T, TA>(p, d.hist == nullptr)) return GB_NOT_SUPPORTED;
  GB_TRY(fill_sentinel_dev((int)p.mail_len, p.mail, s));
  TeamArgs<T, TA> A;
  A.d = d;
  A.cta_sys = p.cta_sys;
  A.cta0 = p.cta0;
  A.mail = p.mail;
  A.mail0 = p.mail0;
  A.cached = p.smem ? p.max_nnz : 0;
  void* args[] = {&A};
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)team_kernel<T, TA>(p.rows), dim3(p.ctas),
                                                    dim3(kTeamThreads + 32), args, std::max(p.smem, p.debug_smem), s);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported) {
    cudaGetLastError();
    return GB_NOT_SUPPORTED;
  }
  GB_CUDA_TRY(e);
  return GB_OK;
}
template int team_loop<double, double>(const TeamPlan&, const TeamData<double, double>&, cudaStream_t);
template int team_loop<float, float>(const TeamPlan&, const TeamData<float, float>&, cudaStream_t);
template int team_loop<double, float>(const TeamPlan&, const TeamData<double, float>&, cudaStream_t);

}  // namespace gb
