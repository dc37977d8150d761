// Domain-restricted two-external products of a local deck (pair domains) over the common virtuals, as the
// reference takes them (two_int_seg_com_lmo_res, three_and_four_seg_mod_2.f90:7137-8005, GEMMs at :7718-7751).
// Source head mu's pair matrix is zero outside D_mu x D_mu and the target head lambda needs only
// D_lambda x D_lambda, so a term reaches only the columns in both domains:
//   R_lambda[a][b] += alpha sum_{c in D_mu} X[a][c] D_mu[c][b]      (a in D_lambda, b in D_lambda and D_mu)
// m_lambda x |common| x m_mu per term instead of m_lambda x m_lambda x m_mu.
//
// A block owns up to 64 rows of one target and walks its jobs (term, at most 48 common columns) in table order: 16-deep
// slices of both operands by cp.async two ahead, the products on the FP64 matrix instruction (a chain of fmas in
// ascending k: the sums of a scalar kernel), alpha times a finished job's sums added at its columns to the tile's
// sums in shared memory (one writer each between two barriers), those added into the padded matrix at the end: every
// sum in a fixed order, no pass over global accumulators.  A job is short (five to ten slices), so the next job's
// record and column lists are loaded during the current one.  Bound by the latency of the gathered slices (about half
// of the FP64 pipe); the scalar kernel it replaces added each job's sums to global memory and ran at 6 TFLOP/s.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "../../include/tigerci_sigma.h"
#include "local_com.h"

namespace {

using tci_com::COLS;
using tci_com::Job;
using tci_com::Task;

constexpr int NT = 256, BK = 16, STG = 3, BP = COLS + 4, SLOTS = 4;

__device__ __forceinline__ void cp_async8(unsigned s, const void* g, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(g), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(unsigned s, const void* g, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
// rows of 16 k as eight 16-byte chunks, chunk c at place c ^ swz(row): as in gemm_mma_f64.cu
__device__ __forceinline__ int swz(int r) { return ((r & 3) << 1) | ((r >> 2) & 1); }
__device__ __forceinline__ unsigned place(int r, int k) {  // bytes
  return 8u * (unsigned)(r * BK + 2 * ((k >> 1) ^ swz(r)) + (k & 1));
}

template <int ROWS>
constexpr int stage_doubles() { return ROWS * BK + BK * BP; }
template <int ROWS>
constexpr size_t smem_bytes(int m) { return sizeof(double) * ((size_t)STG * stage_doubles<ROWS>() + (size_t)m * (ROWS + 4)); }

template <int ROWS>
__global__ void __launch_bounds__(NT, 2) com_products(const Task* __restrict__ tasks, const Job* __restrict__ jobs,
                                                      long long ld) {
  constexpr int STAGE = stage_doubles<ROWS>(), YP = ROWS + 4;
  extern __shared__ __align__(128) double sm[];
  __shared__ double s_alpha[SLOTS];
  __shared__ int s_cnt[SLOTS], s_nsl[SLOTS], s_ct[SLOTS][COLS];
  double* Y = sm + STG * STAGE;  // [position in the target's domain - c0][row]
  const Task T = tasks[blockIdx.x];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  // four row shares of the tile, rotated over the schedulers, two column shares
  const int wm = (warp + (int)blockIdx.x) & 3, wn = warp >> 2;
  const int mblk = (T.rows + 7) >> 3, i0 = mblk * wm >> 2, mb = (mblk * (wm + 1) >> 2) - i0;  // 0 .. 2 8-row blocks
  for (int i = tid; i < T.m * YP; i += NT) Y[i] = 0.0;
  const unsigned sbase = static_cast<unsigned>(__cvta_generic_to_shared(sm));
  // producer cursor: job pj (record J, this thread's column), slice ps; the next job's record and column ahead
  const int bj = tid & 63, bk0 = tid >> 6;     // B: column, first k (+ 4 u)
  const int ac = tid & 7, ar = tid >> 3;       // A: 16-byte chunk, row (+ 32 u)
  const int gk = tid & 15, gr = tid >> 4;      // gathered A: k, row (+ 16 u)
  int pj = T.job0, ps = 0, pslot = 0;
  Job J{}, N{};
  int ncs = 0, nct = 0;
  const double *pa = nullptr, *pb = nullptr;
  if (pj < T.job1) {
    N = jobs[pj];
    if (bj < N.cnt) ncs = N.cs[bj], nct = N.ct[bj];
  }
  auto open = [&]() {
    J = N;
    pslot = (pj - T.job0) % SLOTS;
    pa = J.A + (long long)(T.r0 + ar) * J.pitch_a + 2 * ac;
    pb = J.B + (long long)bk0 * J.pitch_b + ncs;
    if (tid == 0) {
      s_alpha[pslot] = J.alpha;
      s_cnt[pslot] = J.cnt;
      s_nsl[pslot] = (J.m + BK - 1) / BK;
    }
    if (tid < J.cnt) s_ct[pslot][tid] = nct - T.c0;
    if (pj + 1 < T.job1) N = jobs[pj + 1];
  };
  if (pj < T.job1) open();
  auto produce = [&](int st) {
    if (pj < T.job1) {
      const unsigned s = sbase + 8u * (unsigned)(st * STAGE), sb = s + 8u * (unsigned)(ROWS * BK);
      const int krem = J.m - ps * BK;
      if (J.compact) {
        const int bytes = max(0, min(16, 8 * (krem - 2 * ac)));
#pragma unroll
        for (int u = 0; u < (ROWS + 31) / 32; ++u) {
          const int r = ar + 32 * u;
          if (r < T.rows) cp_async16(s + place(r, 2 * ac), bytes ? pa + (long long)(32 * u) * J.pitch_a : J.A, bytes);
        }
        pa += BK;
      } else {
        const bool ok = gk < krem;
        const int col = ok ? J.dom[ps * BK + gk] : 0;
#pragma unroll
        for (int u = 0; u < (ROWS + 15) / 16; ++u) {
          const int r = gr + 16 * u;
          if (r < T.rows) cp_async8(s + place(r, gk), J.A + (long long)T.dom[T.r0 + r] * ld + col, ok ? 8 : 0);
        }
      }
      if (bj < J.cnt) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool ok = bk0 + 4 * u < krem;
          cp_async8(sb + 8u * (unsigned)((bk0 + 4 * u) * BP + bj), ok ? pb : J.B, ok ? 8 : 0);
          pb += 4ll * J.pitch_b;
        }
      }
      if (++ps * BK >= J.m) {  // the job's last slice: on to the next
        if (ps == 1 && pj + 1 < T.job1 && bj < N.cnt) ncs = N.cs[bj], nct = N.ct[bj];
        ps = 0;
        if (++pj < T.job1) open();
      } else if (ps == 1 && pj + 1 < T.job1 && bj < N.cnt) {
        ncs = N.cs[bj], nct = N.ct[bj];  // the record came during the first slice
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  for (int st = 0; st < STG - 1; ++st) produce(st);
  const int f0 = g * BK + 2 * ((tq >> 1) ^ swz(g)) + (tq & 1);  // step s: ^ (s << 2)
  int st = 0;
  for (int j = T.job0; j < T.job1; ++j) {
    const int slot = (j - T.job0) % SLOTS;
    double acc[2][3][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int q = 0; q < 3; ++q) acc[i][q][0] = acc[i][q][1] = 0.0;
    int nsl = 1, cnt = 0, j0 = 0, nb = 0;
    for (int sl = 0; sl < nsl; ++sl) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(STG - 2) : "memory");
      __syncthreads();  // the slice is there, and the stage refilled below is no longer read
      if (sl == 0) {    // the job's record was written before this barrier
        nsl = s_nsl[slot];
        cnt = s_cnt[slot];
        const int nbk = (cnt + 7) >> 3, h0 = (nbk + 1) >> 1;  // column blocks, the first share's
        j0 = wn ? h0 : 0;
        nb = wn ? nbk - h0 : h0;
      }
      produce(st == 0 ? STG - 1 : st - 1);
      const double* as = sm + st * STAGE + 8 * i0 * BK;
      const double* bs = sm + st * STAGE + ROWS * BK + tq * BP + 8 * j0 + g;
      // one body per shape: a matrix instruction whose predicate is off still takes its pipe slot
      auto body = [&](auto rr, auto nn) {
        constexpr int R = decltype(rr)::value, NB = decltype(nn)::value;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int fo = f0 ^ (s << 2);
          double x[R];
#pragma unroll
          for (int i = 0; i < R; ++i) x[i] = as[i * 8 * BK + fo];
#pragma unroll
          for (int q = 0; q < NB; ++q) {
            const double b = bs[4 * s * BP + 8 * q];
#pragma unroll
            for (int i = 0; i < R; ++i) mma884(acc[i][q][0], acc[i][q][1], x[i], b);
          }
        }
      };
      auto bodies = [&](auto rr) {
        if (nb == 3) body(rr, std::integral_constant<int, 3>());
        else if (nb == 2) body(rr, std::integral_constant<int, 2>());
        else if (nb == 1) body(rr, std::integral_constant<int, 1>());
      };
      if (mb == 2) bodies(std::integral_constant<int, 2>());
      else if (mb == 1) bodies(std::integral_constant<int, 1>());
      st = st == STG - 1 ? 0 : st + 1;
    }
    // into the tile's sums: the next job's writer of a column is at least one barrier later
    const double alpha = s_alpha[slot];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int x = 8 * (j0 + q) + 2 * tq + e;
        if (q >= nb || x >= cnt) continue;
        double* y = Y + s_ct[slot][x] * YP + 8 * i0 + g;
        if (mb > 0) y[0] = fma(alpha, acc[0][q][e], y[0]);
        if (mb > 1) y[8] = fma(alpha, acc[1][q][e], y[8]);
      }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  for (int r = warp; r < T.rows; r += NT / 32) {
    double* row = T.R + (long long)T.dom[T.r0 + r] * ld;
    for (int c = lane; c < T.m; c += 32) row[T.dom[T.c0 + c]] += Y[c * YP + r];
  }
}

template <int ROWS>
cudaError_t go(const Task* tasks, int ntasks, int mmax, const Job* jobs, long long ld, cudaStream_t st) {
  const size_t smem = smem_bytes<ROWS>(mmax);
  const cudaError_t e = cudaFuncSetAttribute(com_products<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
  if (e != cudaSuccess) return e;
  com_products<ROWS><<<(unsigned)ntasks, NT, smem, st>>>(tasks, jobs, ld);
  return cudaGetLastError();
}

}  // namespace

namespace tci_com {

// 64 and 32 rows leave room for two blocks per SM (113 KB each); larger domains take what one block can hold, and above
// that their columns are cut in even windows of the 16-row class.
static int task_class(int m) { return m <= 126 ? 0 : m <= 280 ? 1 : m <= 1200 ? 2 : 3; }
constexpr int MAX_COLS = 2100, WINDOW = 1200;

void HostPlan::add(double* R, const int* dom, int m, const std::vector<Term>& terms) {
  const int nwin = m <= MAX_COLS ? 1 : (m + WINDOW - 1) / WINDOW;
  for (int w = 0; w < nwin; ++w) {
    const int c0 = (int)((long long)m * w / nwin), c1 = (int)((long long)m * (w + 1) / nwin);
    const int cls = task_class(c1 - c0), job0 = (int)jobs.size();
    double work = 0;
    for (const Term& x : terms) {
      // the term's columns in the window, COLS at a time
      const int f0 = (int)(std::lower_bound(x.host_ct, x.host_ct + x.job.cnt, c0) - x.host_ct);
      const int n = (int)(std::lower_bound(x.host_ct + f0, x.host_ct + x.job.cnt, c1) - x.host_ct) - f0;
      const int parts = (n + COLS - 1) / COLS;
      for (int q = 0; q < parts; ++q) {
        const int f = f0 + (int)((long long)n * q / parts), e = f0 + (int)((long long)n * (q + 1) / parts);
        Job j = x.job;
        j.cs += f;
        j.ct += f;
        j.cnt = e - f;
        jobs.push_back(j);
        work += (double)((j.m + 15) / 16) * (double)(8 + j.cnt);
      }
    }
    if (job0 == (int)jobs.size()) continue;
    const int rows = 64 >> cls, nt = (m + rows - 1) / rows;  // even row tiles
    for (int t = 0; t < nt; ++t) {
      const int f = (int)((long long)m * t / nt), e = (int)((long long)m * (t + 1) / nt);
      tasks[cls].push_back(HostTask{work, Task{R, dom, c1 - c0, f, e - f, job0, (int)jobs.size(), c0}});
    }
  }
}

std::vector<Task> HostPlan::sorted(int cls) {
  std::stable_sort(tasks[cls].begin(), tasks[cls].end(), [](const HostTask& x, const HostTask& y) { return x.work > y.work; });
  std::vector<Task> v;
  for (const auto& x : tasks[cls]) v.push_back(x.t);
  return v;
}

cudaError_t launch(const Tables& t, long long ld, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  if (t.ntasks[0] > 0) e = go<64>(t.tasks[0], t.ntasks[0], t.mmax[0], t.jobs, ld, st);
  if (e == cudaSuccess && t.ntasks[1] > 0) e = go<32>(t.tasks[1], t.ntasks[1], t.mmax[1], t.jobs, ld, st);
  if (e == cudaSuccess && t.ntasks[2] > 0) e = go<16>(t.tasks[2], t.ntasks[2], t.mmax[2], t.jobs, ld, st);
  if (e == cudaSuccess && t.ntasks[3] > 0) e = go<8>(t.tasks[3], t.ntasks[3], t.mmax[3], t.jobs, ld, st);
  return e;
}

}  // namespace tci_com

// Test entry on host arrays: one target with m externals dom of n, nsrc sources with ms[s] externals (sdom, one after the
// other), A (nsrc x n x n) and D (nsrc x n x n, read on the sources' domains): R (n x n) += the terms' products on the
// common columns.
extern "C" int tci_selftest_com(int64_t device, int64_t n, int64_t m, const int64_t* dom, int64_t nsrc, const int64_t* ms,
                                const int64_t* sdom, const double* alpha, const double* A, const double* D, int64_t compact,
                                double* R) {
  if (n < 1 || m < 1 || m > n || nsrc < 1 || !dom || !ms || !sdom || !alpha || !A || !D || !R) return TCI_ERR_ARG;
  std::vector<void*> owned;
  int rc = TCI_OK;
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess && rc == TCI_OK) rc = TCI_ERR_CUDA;
    return rc == TCI_OK;
  };
  auto up = [&](const auto& v) {
    using V = typename std::decay<decltype(v[0])>::type;
    void* p = nullptr;
    if (ok(cudaMalloc(&p, sizeof(V) * std::max<size_t>(1, v.size())))) {
      owned.push_back(p);
      if (!v.empty()) ok(cudaMemcpy(p, v.data(), sizeof(V) * v.size(), cudaMemcpyHostToDevice));
    }
    return static_cast<V*>(p);
  };
  try {
    const auto sorted_in = [&](const int64_t* d, int64_t c) {
      for (int64_t i = 0; i < c; ++i)
        if (d[i] < 0 || d[i] >= n || (i > 0 && d[i] <= d[i - 1])) return false;
      return true;
    };
    if (!sorted_in(dom, m)) return TCI_ERR_ARG;
    for (int64_t s = 0, o = 0; s < nsrc; o += ms[s++])
      if (ms[s] < 1 || ms[s] > n || !sorted_in(sdom + o, ms[s])) return TCI_ERR_ARG;
    ok(cudaSetDevice((int)device));
    std::vector<std::vector<int>> cts;
    std::vector<tci_com::Term> terms;
    const int* d_dom = up(std::vector<int>(dom, dom + m));
    for (int64_t s = 0, o = 0; s < nsrc && rc == TCI_OK; o += ms[s++]) {
      const int64_t k = ms[s], p = k + (k & 1), *sd = sdom + o;
      std::vector<int> cs, ct;
      for (int64_t x = 0; x < k; ++x) {
        const int64_t* y = std::lower_bound(dom, dom + m, sd[x]);
        if (y < dom + m && *y == sd[x]) cs.push_back((int)x), ct.push_back((int)(y - dom));
      }
      if (cs.empty()) continue;
      std::vector<double> sq((size_t)(k * p)), a;
      const double *As = A + s * n * n, *Ds = D + s * n * n;
      for (int64_t r = 0; r < k; ++r)
        for (int64_t c = 0; c < k; ++c) sq[(size_t)(r * p + c)] = Ds[sd[r] * n + sd[c]];
      if (compact) {
        a.resize((size_t)(m * p));
        for (int64_t r = 0; r < m; ++r)
          for (int64_t c = 0; c < k; ++c) a[(size_t)(r * p + c)] = As[dom[r] * n + sd[c]];
      } else {
        a.assign(As, As + n * n);
      }
      cts.push_back(ct);
      const double *da = up(a), *db = up(sq);
      const int *dd = up(std::vector<int>(sd, sd + k)), *dcs = up(cs), *dct = up(ct);
      terms.push_back({Job{da, db, dd, dcs, dct, (int)k, (int)cs.size(), (int)p, (int)p, alpha[s], compact ? 1 : 0, 0}, nullptr});
    }
    for (size_t i = 0; i < terms.size(); ++i) terms[i].host_ct = cts[i].data();
    double* d_R = up(std::vector<double>(R, R + n * n));
    tci_com::HostPlan plan;
    plan.add(d_R, d_dom, (int)m, terms);
    tci_com::Tables t;
    for (int c = 0; c < tci_com::CLASSES; ++c) {
      const std::vector<Task> v = plan.sorted(c);
      for (const Task& x : v) t.mmax[c] = std::max(t.mmax[c], x.m);
      t.tasks[c] = up(v);
      t.ntasks[c] = (int)v.size();
    }
    t.jobs = up(plan.jobs);
    if (rc == TCI_OK) ok(tci_com::launch(t, n, 0));
    ok(cudaDeviceSynchronize());
    if (rc == TCI_OK) ok(cudaMemcpy(R, d_R, sizeof(double) * (size_t)(n * n), cudaMemcpyDeviceToHost));
  } catch (...) {
    rc = TCI_ERR_INTERNAL;
  }
  for (void* p : owned) cudaFree(p);
  return rc;
}
