// All-external term over pair domains from the packed integrals, FP64:
//   S_h[a][b] = sum_{c,d in D_h} (ac|bd) C_h[c][d],   a >= b in D_h,
// for every head h with its own domain D_h (the reference's local loops take the same products,
// ext_3_4_seg_loops_vec_lmo_res_2, three_and_four_seg_mod_1.f90:3240-3518).
//
// For one a and one c the integral row (ac) is an n x n symmetric matrix over (b, d), and the blocks whose domains hold
// both a and c (a twelfth of them where a domain is 28 % of the externals) are its right-hand sides: C_h[c][:] with
// zeros outside D_h.  A thread block owns one a and up to 64 rows b, walks the c that occur, multiplies the row's part
// by its right-hand sides on the FP64 matrix instruction (up to 48 columns at a time, 16-deep slices of d staged by
// cp.async two ahead) and adds the products to per-column sums in shared memory; b <= a is half of the matrix.  Four
// warps copy and four multiply, a stage handed over by named barriers: the index arithmetic of the copies (triangular
// rows, three cases) is most of the instructions, and in the warps that multiply it held the products back (15.4 ms at
// 150 pairs of 20-150 of 300 externals with eight warps doing both, 13.8 with eight multiplying, 13.5 with four; four
// stages, or two of 32 k, are no faster: 13.7, 14.4).  The zero
// padding inside a column costs 1 / density in d and b, but nothing is gathered: the index arithmetic of a
// gathering kernel (lanes over the domain, integrals from shared memory) cost more than the padding (30 ms against
// 15.4 for the form with eight warps doing both), and n^2 sum n_h^2 flops replace the Cholesky form's 4 nchol sum n_h^3.
// Bound by the copies (9.9 ms alone) and the products of half-filled tiles (11.4 alone) together.  Every sum in a fixed order.
#include <algorithm>
#include <limits>
#include <mutex>
#include <type_traits>

#include "../../include/tigerci_sigma.h"
#include "local_integral.h"

namespace {

using tci_lint::Block;
using tci_lint::Job;
using tci_lint::Task;

constexpr int NC = 128, NP = 128, NT = NC + NP;  // four warps of up to 16 rows x all columns each, four that copy
constexpr int ROWS = 64, COLS = 48, BK = 16, STG = 3;
constexpr int ACC_COLS = 128, YP = ROWS + 4;  // accumulators of a task: columns, pitch
constexpr int STAGE = (ROWS + COLS) * BK;     // doubles
constexpr size_t SMEM = sizeof(double) * (size_t)(STG * STAGE + ACC_COLS * YP);

__device__ __forceinline__ int tri(int a, int b) { return a >= b ? a * (a + 1) / 2 + b : b * (b + 1) / 2 + a; }
__device__ __forceinline__ void cp_async8(unsigned s, const void* g, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(g), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(unsigned s, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(g) : "memory");
}
__device__ __forceinline__ void mma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
// named barriers: a stage is full (the copying warps arrive, the others wait) or free again (the other way round)
__device__ __forceinline__ void bar_sync(int id) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(NT) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(NT) : "memory"); }
constexpr int FULL = 1, FREE = FULL + STG;
// rows of 16 k as eight 16-byte chunks, chunk c at place c ^ swz(row): as in gemm_mma_f64.cu
__device__ __forceinline__ int swz(int r) { return ((r & 3) << 1) | ((r >> 2) & 1); }
__device__ __forceinline__ unsigned place(int r, int k) {  // bytes
  return 8u * (unsigned)(r * BK + 2 * ((k >> 1) ^ swz(r)) + (k & 1));
}

__global__ void __launch_bounds__(NT, 2) local_integral(const Task* __restrict__ tasks, const Job* __restrict__ jobs,
                                                        const int* __restrict__ cblk, const int* __restrict__ jcol,
                                                        const Block* __restrict__ blocks, const short* __restrict__ pos,
                                                        const double* __restrict__ X, long long npv,
                                                        const double* __restrict__ C, int nv, int ldc,
                                                        double* __restrict__ sigma, long long total) {
  extern __shared__ __align__(128) double sm[];
  double* Y = sm + STG * STAGE;  // [column][row]
  const Task T = tasks[blockIdx.x];
  const int tid = threadIdx.x;
  for (int i = tid; i < T.ncol * YP; i += NT) Y[i] = 0.0;
  __syncthreads();
  const int nsl = (nv + BK - 1) / BK, total_sl = (T.job1 - T.job0) * nsl;
  if (tid >= NC) {
    // copying warps: job by job, slice by slice
    const int pt = tid - NC, b1 = T.b0 + T.rows;
    const unsigned sbase = static_cast<unsigned>(__cvta_generic_to_shared(sm));
    // this thread's copies of a slice: rows r0, r0 + 8, ... at one k where the integrals of a row b lie along d <= b,
    // row ru at k0, k0 + 2, ... where those of one d lie along b; 16 bytes of up to three columns of the job
    const int kl = pt & 15, r0 = pt >> 4, ru = pt & 63, k0 = pt >> 6, bj = pt >> 3, bk = 2 * (pt & 7);
    int offl[8];
    unsigned pl[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      offl[u] = tri(T.b0 + r0 + 8 * u, 0) + kl;
      pl[u] = place(ru, k0 + 2 * u);
    }
    const unsigned pk = place(r0, kl), pb = place(bj, bk);
    int st = 0, i = 0;
    for (int j = T.job0; j < T.job1; ++j) {
      const Job J = jobs[j];
      const double* prow = X + (long long)tri(T.a, J.c) * npv;
      const double* pc[3];
#pragma unroll
      for (int u = 0; u < 3; ++u)
        if (bj + 16 * u < J.cnt) pc[u] = C + ((long long)cblk[T.col0 + jcol[J.off + bj + 16 * u]] * nv + J.c) * ldc + bk;
      for (int d0 = 0; d0 < nsl * BK; d0 += BK, ++i) {
        if (i >= STG) bar_sync(FREE + st);
        const unsigned s = sbase + 8u * (unsigned)(st * STAGE), sb = s + 8u * (unsigned)(ROWS * BK);
        if (d0 + BK <= T.b0 + 1) {  // d <= b throughout
          const double* q = prow + d0;
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (r0 + 8 * u < T.rows) cp_async8(s + pk + 8u * (8 * u * BK), q + offl[u], 8);
        } else if (d0 >= b1) {  // d above every b
          if (ru < T.rows) {
            const int d = d0 + k0;
            int o = d * (d + 1) / 2 + T.b0 + ru;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const bool ok = d + 2 * u < nv;
              cp_async8(s + pl[u], prow + (ok ? o : 0), ok ? 8 : 0);
              o += 2 * (d + 2 * u) + 3;
            }
          }
        } else {
          const int d = d0 + kl;
          const bool ok = d < nv;
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (r0 + 8 * u < T.rows)
              cp_async8(s + pk + 8u * (8 * u * BK), prow + (ok ? tri(T.b0 + r0 + 8 * u, d) : 0), ok ? 8 : 0);
        }
#pragma unroll
        for (int u = 0; u < 3; ++u)
          if (bj + 16 * u < J.cnt) cp_async16(sb + pb + 8u * (16 * u * BK), pc[u] + d0);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (i > 0) {
          asm volatile("cp.async.wait_group 1;\n" ::: "memory");
          bar_arrive(FULL + (st == 0 ? STG - 1 : st - 1));  // the slice before
        }
        st = st == STG - 1 ? 0 : st + 1;
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (total_sl > 0) bar_arrive(FULL + (st == 0 ? STG - 1 : st - 1));
  } else {
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    // the four row shares of the tile, rotated so that the uneven ones fall on every scheduler in turn; two column shares
    const int wm = (warp + (int)blockIdx.x) & 3;
    const int mblk = (T.rows + 7) >> 3, i0 = mblk * wm >> 2, mb = (mblk * (wm + 1) >> 2) - i0;  // its 8-row blocks: 0 .. 2
    const int f0 = g * BK + 2 * ((tq >> 1) ^ swz(g)) + (tq & 1);  // step s: ^ (s << 2)
    int st = 0, i = 0;
    Job next = jobs[T.job0];
    for (int j = T.job0; j < T.job1; ++j) {
      const Job J = next;
      if (j + 1 < T.job1) next = jobs[j + 1];
      const int nb = (J.cnt + 7) >> 3;  // column blocks
      int col[6][2];  // accumulator columns of this lane's sums
#pragma unroll
      for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int x = 8 * q + 2 * tq + e;
          col[q][e] = x < J.cnt ? jcol[J.off + x] : -1;
        }
      double acc[2][6][2];
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int q = 0; q < 6; ++q) acc[r][q][0] = acc[r][q][1] = 0.0;
      for (int sl = 0; sl < nsl; ++sl, ++i) {
        bar_sync(FULL + st);
        const double* as = sm + st * STAGE + 8 * i0 * BK;
        const double* bs = sm + st * STAGE + ROWS * BK;
        // one body per number of column blocks: a matrix instruction whose predicate is off still takes its pipe slot
        auto body = [&](auto rr, auto nn) {
          constexpr int R = decltype(rr)::value, N = decltype(nn)::value;
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const int fo = f0 ^ (s << 2);
            double x[R];
#pragma unroll
            for (int r = 0; r < R; ++r) x[r] = as[r * 8 * BK + fo];
#pragma unroll
            for (int q = 0; q < N; ++q) {
              const double b = bs[q * 8 * BK + fo];
#pragma unroll
              for (int r = 0; r < R; ++r) mma884(acc[r][q][0], acc[r][q][1], x[r], b);
            }
          }
        };
        auto bodies = [&](auto rr) {
          if (nb == 3) body(rr, std::integral_constant<int, 3>());
          else if (nb == 4) body(rr, std::integral_constant<int, 4>());
          else if (nb == 5) body(rr, std::integral_constant<int, 5>());
          else if (nb == 6) body(rr, std::integral_constant<int, 6>());
          else if (nb == 2) body(rr, std::integral_constant<int, 2>());
          else if (nb == 1) body(rr, std::integral_constant<int, 1>());
        };
        if (mb == 2) bodies(std::integral_constant<int, 2>());
        else if (mb == 1) bodies(std::integral_constant<int, 1>());
        if (i + STG < total_sl) bar_arrive(FREE + st);
        st = st == STG - 1 ? 0 : st + 1;
      }
      // into the columns' sums: the next job's writer of a column is at least one barrier later
#pragma unroll
      for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (col[q][e] >= 0) {
            double* y = Y + col[q][e] * YP + 8 * i0 + g;
            if (mb > 0) y[0] += acc[0][q][e];
            if (mb > 1) y[8] += acc[1][q][e];
          }
    }
  }
  __syncthreads();
  double* out = sigma + T.part * total;
  for (int e = tid; e < T.ncol * ROWS; e += NT) {
    const int cidx = e / ROWS, r = e % ROWS;
    if (r >= T.rows) continue;
    const Block B = blocks[cblk[T.col0 + cidx]];
    const short* ph = pos + (long long)B.head * nv;
    const int i = ph[T.a], j = ph[T.b0 + r];
    if (j < 0) continue;
    const double v = Y[cidx * YP + r];
    if (j < i) {
      if (B.ab >= 0) out[B.ab + (long long)i * (i - 1) / 2 + j] = B.p * v;
    } else if (j == i && B.aa >= 0) {
      out[B.aa + i] = 0.70710678118654757 * v;
    }
  }
}

// Padded pair matrices C[block][c][d] (n x n, row pitch ldc, zero outside the domain): sqrt2 C_aa on the diagonal,
// x and p x off it.
__global__ void __launch_bounds__(256) pad_blocks(const Block* __restrict__ blocks, const int* __restrict__ dom,
                                                  const double* __restrict__ c, int nv, int ldc, double* __restrict__ C) {
  const Block B = blocks[blockIdx.x];
  const int* d = dom + B.dom;
  double* M = C + (long long)blockIdx.x * nv * ldc;
  for (int e = threadIdx.x; e < B.n * B.n; e += blockDim.x) {
    const int r = e / B.n, s = e - r * B.n;
    double v = 0.0;
    if (r == s) {
      if (B.aa >= 0) v = 1.4142135623730951 * c[B.aa + r];
    } else if (B.ab >= 0) {
      const int i = max(r, s), j = min(r, s);
      const double x = c[B.ab + (long long)i * (i - 1) / 2 + j];
      v = r < s ? x : B.p * x;
    }
    M[(long long)d[r] * ldc + d[s]] = v;
  }
}

__global__ void __launch_bounds__(256) sum_parts(const double* __restrict__ part, int parts, long long n,
                                                 double* __restrict__ out) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double v = 0.0;
    for (int p = 0; p < parts; ++p) v += part[p * n + i];
    out[i] = v;
  }
}

// X[i][j] = X[j][i] for j > i
__global__ void __launch_bounds__(256) mirror_lower(double* __restrict__ X, long long n) {
  __shared__ double t[32][33];
  if (blockIdx.x > blockIdx.y) return;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const long long r0 = 32ll * blockIdx.y, c0 = 32ll * blockIdx.x;  // source tile, c0 <= r0
  for (int i = y; i < 32; i += 8)
    if (r0 + i < n && c0 + x < n) t[i][x] = X[(r0 + i) * n + c0 + x];
  __syncthreads();
  for (int i = y; i < 32; i += 8) {
    const long long r = c0 + i, c = r0 + x;
    if (c > r && r < n && c < n) X[r * n + c] = t[x][i];
  }
}

}  // namespace

namespace tci_lint {

bool fits(const std::vector<Block>& blocks) {
  double entries = 0;  // of jcol; the other lists are no longer
  for (const Block& b : blocks) entries += (double)b.n * (double)b.n;
  return entries <= (double)std::numeric_limits<int>::max();
}

void make_plan(int nv, int nheads, const std::vector<int>& dom, std::vector<Block> blocks, int sms, Plan& P) {
  P.nv = nv;
  P.dom = dom;
  P.blocks = std::move(blocks);
  P.pos.assign((size_t)nheads * nv, -1);
  std::vector<std::vector<int>> of((size_t)nv);  // the blocks whose domains hold an external
  for (size_t i = 0; i < P.blocks.size(); ++i) {
    const Block& B = P.blocks[i];
    for (int x = 0; x < B.n; ++x) {
      P.pos[(size_t)B.head * nv + dom[(size_t)(B.dom + x)]] = (short)x;
      of[(size_t)dom[(size_t)(B.dom + x)]].push_back((int)i);
    }
  }
  struct Batch {
    int a, col0, ncol, job0, job1;
  };
  std::vector<Batch> batches;
  std::vector<std::vector<int>> by_c((size_t)nv);
  double rows_total = 0;
  for (int a = nv - 1; a >= 0; --a) {  // the longest rows first
    const auto& L = of[(size_t)a];
    const size_t nbt = (L.size() + ACC_COLS - 1) / ACC_COLS;  // batches of even width
    for (size_t x = 0; x < nbt; ++x) {
      const size_t l0 = L.size() * x / nbt;
      const int ncol = (int)(L.size() * (x + 1) / nbt - l0);
      Batch bt{a, (int)P.cblk.size(), ncol, (int)P.jobs.size(), 0};
      for (auto& v : by_c) v.clear();
      for (int k = 0; k < ncol; ++k) {
        const int i = L[l0 + (size_t)k];
        P.cblk.push_back(i);
        const Block& B = P.blocks[(size_t)i];
        for (int x = 0; x < B.n; ++x) by_c[(size_t)dom[(size_t)(B.dom + x)]].push_back(k);
      }
      for (int c = 0; c < nv; ++c) {
        const auto& v = by_c[(size_t)c];
        const int np = ((int)v.size() + COLS - 1) / COLS;  // passes of even width
        for (int q = 0; q < np; ++q) {
          const int f = (int)(v.size() * (size_t)q / (size_t)np), t = (int)(v.size() * (size_t)(q + 1) / (size_t)np);
          P.jobs.push_back(Job{c, (int)P.jcol.size(), t - f, 0});
          P.jcol.insert(P.jcol.end(), v.begin() + f, v.begin() + t);
          P.flops += 2.0 * ((t - f + 7) / 8 * 8) * (double)(a + 1) * (double)nv;
        }
      }
      bt.job1 = (int)P.jobs.size();
      batches.push_back(bt);
      rows_total += (a + ROWS) / ROWS;
    }
  }
  // tasks: even row tiles; where they are too few for the chip the jobs are split and the parts added afterwards
  P.parts = 1;
  while (P.parts < 8 && rows_total * P.parts < 6.0 * sms) P.parts *= 2;
  for (const auto& b : batches) {
    const int tiles = (b.a + ROWS) / ROWS;
    for (int t = 0; t < tiles; ++t) {
      const int r0 = (b.a + 1) * t / tiles, r1 = (b.a + 1) * (t + 1) / tiles;
      for (int p = 0; p < P.parts; ++p) {
        const int nj = b.job1 - b.job0, f = b.job0 + (int)((long long)nj * p / P.parts),
                  e = b.job0 + (int)((long long)nj * (p + 1) / P.parts);
        if (e > f) P.tasks.push_back(Task{b.a, r0, r1 - r0, b.col0, b.ncol, f, e, p});
      }
    }
  }
}

cudaError_t mirror(double* X, int64_t npv, cudaStream_t st) {
  const unsigned t = (unsigned)((npv + 31) / 32);
  mirror_lower<<<dim3(t, t), 256, 0, st>>>(X, npv);
  return cudaGetLastError();
}

cudaError_t launch(const Device& d, const double* X, int64_t npv, const double* c, double* sigma, int64_t total,
                   cudaStream_t st) {
  if (d.ntasks <= 0) return cudaSuccess;
  static std::once_flag once[64];  // the attribute, once per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::call_once(once[dev],
                 [] { cudaFuncSetAttribute(local_integral, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM); });
  const int ldc = (int)pitch(d.nv);
  pad_blocks<<<(unsigned)d.nblocks, 256, 0, st>>>(d.blocks, d.dom, c, d.nv, ldc, d.C);
  double* out = d.parts > 1 ? d.part : sigma;
  if (d.parts > 1) {
    e = cudaMemsetAsync(d.part, 0, sizeof(double) * (size_t)d.parts * (size_t)total, st);
    if (e != cudaSuccess) return e;
  }
  local_integral<<<(unsigned)d.ntasks, NT, SMEM, st>>>(d.tasks, d.jobs, d.cblk, d.jcol, d.blocks, d.pos, X, npv, d.C, d.nv,
                                                       ldc, out, total);
  if (d.parts > 1)
    sum_parts<<<(unsigned)std::min<int64_t>((total + 255) / 256, 4096), 256, 0, st>>>(d.part, d.parts, total, sigma);
  return cudaGetLastError();
}

}  // namespace tci_lint

// Test entry, host only: the plan of nblocks singlet-coupled blocks with the domains dom_idx[dom_off .. + dom_len) for sms
// multiprocessors. out: {the lists fit (0: nothing else is set), parts, tasks, jobs, entries of the columns' list}.
extern "C" int tci_selftest_integral_plan(int64_t num_external, int64_t nblocks, const int64_t* dom_off, const int64_t* dom_len,
                                          const int64_t* dom_idx, int64_t ndom, int64_t sms, int64_t* out) {
  if (num_external < 1 || num_external > tci_lint::MAX_NV || nblocks < 1 || ndom < 1 || sms < 1 || !dom_off || !dom_len ||
      !dom_idx || !out)
    return TCI_ERR_ARG;
  try {
    std::vector<int> dom;
    for (int64_t i = 0; i < ndom; ++i) {
      if (dom_idx[i] < 0 || dom_idx[i] >= num_external) return TCI_ERR_ARG;
      dom.push_back((int)dom_idx[i]);
    }
    std::vector<Block> bl;
    for (int64_t b = 0; b < nblocks; ++b) {
      if (dom_off[b] < 0 || dom_len[b] < 1 || dom_off[b] + dom_len[b] > ndom) return TCI_ERR_ARG;
      bl.push_back(Block{0, 0, 1.0, (int)dom_len[b], (int)dom_off[b], (int)b, 0});
    }
    for (int k = 0; k < 5; ++k) out[k] = 0;
    if (!tci_lint::fits(bl)) return TCI_OK;
    tci_lint::Plan P;
    tci_lint::make_plan((int)num_external, (int)nblocks, dom, std::move(bl), (int)sms, P);
    out[0] = 1;
    out[1] = P.parts;
    out[2] = (int64_t)P.tasks.size();
    out[3] = (int64_t)P.jobs.size();
    out[4] = (int64_t)P.jcol.size();
    return TCI_OK;
  } catch (...) {
    return TCI_ERR_INTERNAL;
  }
}
