// FP64 grouped GEMM on the double-precision matrix instruction (mma.sync m8n8k4 f64; tcgen05 has no FP64 kind):
// C (M x N) = beta C + sum over a problem's segments of alpha op(A) op(B), any leading dimension and 8-byte
// alignment, the problem / segment tables of gemm_tables.h. The instruction is a chain of four fmas in ascending k and every
// element is one chain, so every sum is the one a scalar kernel makes, whatever tile and work split a launch takes: segments
// in table order, k ascending, alpha on op(B) (on op(A) where the operands change places). Mixed-precision solves need that:
// a last bit of an integral or a vector flips roundings of the TF32 splits, which moves a converged vector by 1e-8.
//
// Bound by the FP64 pipe: the instruction runs at 37 TFLOP/s on this part, the same as scalar fma, but one operand
// word read from shared memory feeds eight products instead of four or eight registers' worth of broadcasts, so the
// pipe, not shared memory or issue slots, sets the rate (the scalar tiled kernels it replaced ran at 10-24 TFLOP/s).
// Four warps own a 64 x 128 tile, each 64 x 32 of it in 128 accumulator registers, two blocks per SM so that one's
// copies and barriers run under the other's products; four 16-deep slices in flight by cp.async. Tiles of up to 40 rows
// (48 with odd leading dimensions) leave room for a third block with three slices each: 36 x 28920 x 28920 2.56 -> 2.30
// ms. Measured on a B200: 592 problems of 256 x 256 x (40 x 256) 31 TFLOP/s, 576 of 173 x 173 x (40 x 173) 24.5 (6 % of
// the blocks padding, uneven column shares; 20 with one body for all shapes and predicates for the missing blocks).
// Against the scalar kernels: two-external step at 24 pairs x 173 virtuals 102 -> 32 ms, all-external at 240 virtuals
// 6.8 -> 4.5 ms. Tried and slower: the left-over column blocks of a tile dealt by rows,
// as a second phase (6-10 %), four blocks per SM on 64 x 64 tiles (21-25), a fifth warp that only copies (registers
// spill at two blocks per SM), the copies dealt between the products (the loop outgrows the instruction cache: 9-17).
//
// A launch of few tiles is bound by the latency of a slice (copy, barrier, products: 1.3 us), one after another: there the
// 8 x 8 blocks of tiles down to 16 x 16 are dealt to eight warps, with 64-deep slices. A sigma build of 33,055 CSFs (mixed,
// its FP64 steps) takes 329 us with four warps and 16-deep slices alone, 264 so; eight warps sharing k, their sums added at
// the end, took 262, but their sums were not the other form's.
#include <algorithm>
#include <array>
#include <cmath>
#include <map>
#include <mutex>
#include <stdexcept>
#include <type_traits>
#include <utility>

#include "../../include/tigerci_sigma.h"
#include "device_info.h"
#include "gemm_mma_f64.h"

namespace {

using tci_dev::DGemmProblem;
using tci_dev::DGemmSeg;

// Threads of a block by work split (WS): four warps side by side on a tile's columns (1), or its 8 x 8 blocks dealt to
// eight (8).
constexpr int threads(int wk) { return wk == 1 ? 128 : 256; }

__device__ __forceinline__ void cp_async16(unsigned s, const void* g, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async8(unsigned s, const void* g, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(g), "r"(bytes) : "memory");
}
struct CpAsync {
  __device__ __forceinline__ void copy16(unsigned s, const void* g, int bytes) const { cp_async16(s, g, bytes); }
  __device__ __forceinline__ void copy8(unsigned s, const void* g, int bytes) const { cp_async8(s, g, bytes); }
};
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void mma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Shared-memory layout of an operand slice whose k are contiguous in a row: row r (of the tile) holds BK
// consecutive k as 16-byte chunks, chunk c at place c ^ swz(r) (within groups of 8).  A fragment read (four rows x
// four k per half warp) is free of bank conflicts, a transposing copy (consecutive rows, one k) spreads over eight
// places.  swz moves bits only, so swz(r0 + r1) = swz(r0) ^ swz(r1) where r0 and r1 share no bits.
__host__ __device__ constexpr int swz(int r) { return ((r & 3) << 1) | ((r >> 2) & 1); }
// byte offset of chunk c0 + c1 (no common bits, c1 a constant) of a row with swizzle sw
__host__ __device__ __forceinline__ unsigned chunk(int c0, int c1, int sw) {
  return 16u * (unsigned)(((c0 & ~7) + (c1 & ~7)) | ((c0 & 7) ^ (c1 & 7) ^ sw));
}

// The copies of Operand::issue go to the device (CpAsync) or to a host check of their addresses.
#pragma nv_diag_suppress 20011, 20014

// How an operand reaches shared memory: rows of the tile with k contiguous by 16-byte (K16) or 8-byte (K8) copies,
// or with the tile rows contiguous: transposed into the row layout by 8-byte copies (RT8, the row operand), or kept
// as BK rows of the tile rows, pitch R + 4 (R16, the column operand; reads of two k and eight rows spread over the
// banks).  K16 wants a 16-byte aligned operand with an even leading dimension; R16 copies the 16-byte words a row lies
// in, so that a row may start one place into its shared-memory row.
enum Mode { K16, K8, RT8, R16 };

template <int R, int BK, Mode M, int NT>
struct Operand {
  static constexpr int RP = R <= 8 ? 8 : R <= 16 ? 16 : R <= 32 ? 32 : R <= 64 ? 64 : 128;
  static constexpr bool KROWS = M == R16, KC = M == K16 || M == K8;
  static constexpr int PITCH = R + 4;
  static_assert(!(M == R16) || PITCH % 16 == 4 || PITCH % 16 == 12, "bank spread");
  static constexpr int SIZE = KROWS ? BK * PITCH : BK * R;  // doubles of a slice
  // lanes along the contiguous index, rows (of tile or k) a pass, passes
  static constexpr int LANES = M == K16 ? BK / 2 : M == K8 ? BK : M == R16 ? RP / 2 : RP;
  static constexpr int PER = NT / LANES, U = KC ? (R + PER - 1) / PER : BK / PER;
  const double* p;   // this thread's next element
  long long ustep;   // from one pass to the next
  int sh = 0;        // R16: the places this thread's rows are shifted by (0 or 1; PER is even)
  // returns, for R16, the shifts of even (bit 0) and odd (bit 1) k
  __host__ __device__ __forceinline__ int open(int tid, const double* X, long long ld, long long row0) {
    const int x = tid % LANES, y = tid / LANES;
    p = X + (KC ? row0 * ld : row0) + (long long)y * ld + (M == K16 || M == R16 ? 2 * x : x);
    ustep = PER * ld;
    if constexpr (M == R16) {
      static_assert(PER % 2 == 0, "a thread's rows have one parity");
      const int s0 = (int)((reinterpret_cast<uintptr_t>(X + row0) >> 3) & 1), s1 = s0 ^ (int)(ld & 1);
      sh = (y & 1) ? s1 : s0;
      p -= sh;
      return s0 | (s1 << 1);
    }
    return 0;
  }
  // the slice with min(krem, BK) valid k (zeros past them) into shared memory at s, and on to the next; rows past nr
  // are left alone: they reach only outputs that are not stored.  A copy of no bytes keeps to its instruction's
  // alignment and to the operand as well.
  template <class Copy>
  __host__ __device__ __forceinline__ void issue(int tid, unsigned s, int nr, int krem, Copy&& to) {
    const int x = tid % LANES, y = tid / LANES;
    if constexpr (KC) {
      const int k = M == K16 ? 2 * x : x, sw = swz(y);
      const int bytes = max(0, min(M == K16 ? 16 : 8, 8 * (krem - k)));
      if (!bytes) p -= k;  // where nothing is read: an address inside the row (the segment ends here)
      const unsigned d = s + 8u * (unsigned)(y * BK + (k & 1));
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned o = d + 8u * (u * PER * BK) + chunk(k >> 1, 0, sw ^ swz(u * PER));
        if (y + u * PER < nr) {
          if (M == K16) to.copy16(o, p, bytes);
          else to.copy8(o, p, bytes);
        }
        p += ustep;
      }
      p += BK - U * ustep;
    } else {
      const int r = M == R16 ? 2 * x - sh : x, sw = swz(r);
      const unsigned d = s + 8u * (unsigned)(KROWS ? y * PITCH + 2 * x : r * BK + (PER > 1 ? (y & 1) : 0));
      const int bytes = M == RT8 || r + 1 >= nr ? 8 : 16;
      auto copy = [&](int u, const double* q, int n) {
        unsigned o;
        if constexpr (KROWS) o = d + 8u * (u * PER * PITCH);
        else o = d + (PER > 1 ? chunk(y >> 1, (u * PER) >> 1, sw) : chunk(0, u >> 1, sw) + 8u * (u & 1));
        if (M == R16) to.copy16(o, q, n);
        else to.copy8(o, q, n);
      };
      if (krem >= BK) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (r < nr) copy(u, p, bytes);
          p += ustep;
        }
      } else {
        // where nothing is read: row 0's place at the slice's first k (R16: the 16-byte word that holds it)
        const double* z = p - y * (ustep / PER) - r;
        if constexpr (M == R16) z -= (reinterpret_cast<uintptr_t>(z) >> 3) & 1;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool ok = y + u * PER < krem;
          if (r < nr) copy(u, ok ? p : z, ok ? bytes : 0);
          p += ustep;
        }
      }
    }
  }
};

// MB: 8-row blocks of a tile.  WS = 1: the four warps share a tile's columns (up to 16 blocks of 8, dealt evenly),
// 16-deep k slices; WS = 8: the 8 x 8 blocks of a tile (up to 4 columns of them) are dealt to eight warps, 64-deep slices.
// Tiles are cut evenly in 8-row / 8-column blocks (a 173-row problem gives 64 + 56 + 56 rows, not 64 + 64 + 45); blocks
// past the edge are not computed.
constexpr int NB = 4;  // column blocks of a warp (WS = 8: of a tile) at most
template <int MB, int WS, Mode AM, Mode BM_>
struct Shape {
  static constexpr int NT = threads(WS), BK = WS == 1 ? 16 : 64;
  static constexpr int BM = 8 * MB, BN = 8 * NB * (WS == 1 ? 4 : 1);
  using A = Operand<BM, BK, AM, NT>;
  using B = Operand<(WS > 1 && BM_ == R16 ? BN + 8 : BN), BK, BM_, NT>;  // room for a shifted row
  static constexpr int STAGE = A::SIZE + B::SIZE;  // doubles
  static constexpr int BLOCKS = WS > 1 ? 1 : MB <= 5 || (MB == 6 && AM == K8 && BM_ == R16) ? 3 : 2;  // per SM
  static constexpr int STG = BLOCKS == 3 ? 3 : 4;
  static constexpr size_t smem = sizeof(double) * (size_t)STAGE * STG;
};

// ANY: tiles of 1 to MB row blocks in one launch, else of MB or MB - 1.
template <int MB, int WS, Mode AM, Mode BM_, bool ANY>
__global__ void __launch_bounds__(threads(WS), (Shape<MB, WS, AM, BM_>::BLOCKS)) gemm_mma_f64(const DGemmProblem* __restrict__ probs, int nprob,
                                                      const DGemmSeg* __restrict__ segs) {
  using Sh = Shape<MB, WS, AM, BM_>;
  constexpr int NT = Sh::NT, BK = Sh::BK, STG = Sh::STG;
  constexpr bool KB = Sh::B::KROWS;
  extern __shared__ __align__(128) double sm[];
  __shared__ double meta_alpha[STG];
  __shared__ int meta_k[STG];  // valid k of the slice; + 256: alpha is not 1; + 512, 1024: shifts of even, odd k
  const int lane = threadIdx.x & 31;
  // rotated: the uneven shares fall on every scheduler in turn
  const int role = WS == 1 ? ((threadIdx.x >> 5) + blockIdx.x) & 3 : threadIdx.x >> 5;
  // the problem of this tile (the last with tile_begin <= tile), 32 probes at a time
  const long long tile = blockIdx.x;
  int lo = 0, cnt = nprob;
  while (cnt > 1) {
    const int step = (cnt + 31) >> 5, off = lane * step;
    const bool ok = off < cnt && probs[lo + off].tile_begin <= tile;
    const int c = 31 - __clz(__ballot_sync(0xffffffffu, ok));
    lo += c * step;
    cnt = min(step, cnt - c * step);
  }
  const DGemmProblem P = probs[lo];
  const bool tr = (P.trans_c & 1) != 0;
  const long long rows = tr ? P.N : P.M, cols = tr ? P.M : P.N;
  const int tn = (int)P.tiles_n, t = (int)(tile - P.tile_begin), ti = t / tn, tj = t % tn;
  const int mblk = (int)((rows + 7) >> 3), nblk = (int)((cols + 7) >> 3), tm = (int)(P.trans_c >> 1);
  const int mq = mblk / tm, mr = mblk % tm, nw = nblk / tn, nr = nblk % tn;
  const long long m0 = 8ll * (ti * mq + min(ti, mr)), n0 = 8ll * (tj * nw + min(tj, nr));
  const int mb = mq + (ti < mr ? 1 : 0), nbt = nw + (tj < nr ? 1 : 0);  // mb: MB or MB - 1, ANY: 1 .. MB
  const int mrows = (int)min((long long)(8 * mb), rows - m0), ncols = (int)min((long long)(8 * nbt), cols - n0);
  // this warp's column blocks of the tile
  const int j0 = WS == 1 ? (nbt * role) >> 2 : 0, nb = WS == 1 ? ((nbt * (role + 1)) >> 2) - j0 : nbt;
  const int g = lane >> 2, tq = lane & 3;

  // WS = 8: block e = role + 8 q of the tile, row by row, in acc[q][0]
  constexpr int AR = WS == 1 ? MB : (MB * NB + 7) / 8, AC = WS == 1 ? NB : 1;
  double acc[AR][AC][2];
#pragma unroll
  for (int i = 0; i < AR; ++i)
#pragma unroll
    for (int j = 0; j < AC; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int nq = WS == 1 ? 0 : max(0, (mb * nbt - role + 7) >> 3);

  // the slices of all segments in table order, copied STG - 1 ahead
  const unsigned sbase = static_cast<unsigned>(__cvta_generic_to_shared(sm));
  int sg = (int)P.seg_begin;
  const int sge = (int)P.seg_end;
  int krem = 0, flags = 0;
  double alpha = 1.0;
  typename Sh::A oa;
  typename Sh::B ob;
  // the segment records, RING ahead, by cp.async with the slices (a record loaded at its use cost a short segment's
  // slice its latency again)
  constexpr int RING = 16, WORDS = sizeof(DGemmSeg) / 8;
  static_assert(sizeof(DGemmSeg) == 8 * WORDS && RING * WORDS <= NT, "records by 8-byte words");
  __shared__ __align__(8) double ring[RING * WORDS];
  if ((int)threadIdx.x < RING * WORDS && sg + (int)threadIdx.x / WORDS < sge)
    ring[threadIdx.x] = reinterpret_cast<const double*>(segs + sg)[threadIdx.x];
  __syncthreads();
  const unsigned rbase = static_cast<unsigned>(__cvta_generic_to_shared(ring));
  int rs = 0;  // the place of segment sg
  auto open = [&]() {
    const DGemmSeg& S = *reinterpret_cast<const DGemmSeg*>(ring + rs * WORDS);
    krem = (int)S.K;
    alpha = S.alpha;
    oa.open(threadIdx.x, tr ? S.B : S.A, tr ? S.ldb : S.lda, m0);
    flags = 512 * ob.open(threadIdx.x, tr ? S.A : S.B, tr ? S.lda : S.ldb, n0) + (alpha != 1.0 ? 256 : 0);
    // the record RING - 1 ahead takes the place of the one before this, which everyone has left
    const int ahead = sg + RING - 1, pl = rs == 0 ? RING - 1 : rs - 1;
    if (sg > (int)P.seg_begin && ahead < sge && (int)threadIdx.x < WORDS)
      cp_async8(rbase + 8u * (unsigned)(pl * WORDS + threadIdx.x), reinterpret_cast<const double*>(segs + ahead) + threadIdx.x, 8);
    rs = rs == RING - 1 ? 0 : rs + 1;
  };
  if (sg < sge) open();
  auto produce = [&](int st) {
    if (krem > 0) {
      const unsigned s = sbase + 8u * (unsigned)(st * Sh::STAGE);
      oa.issue(threadIdx.x, s, mrows, krem, CpAsync());
      ob.issue(threadIdx.x, s + 8u * (unsigned)Sh::A::SIZE, ncols, krem, CpAsync());
      if (threadIdx.x == 0) {
        meta_alpha[st] = alpha;
        meta_k[st] = min(BK, krem) + flags;
      }
      krem -= BK;
      if (krem <= 0 && ++sg < sge) open();
    } else if (threadIdx.x == 0) {
      meta_k[st] = 0;
    }
    cp_commit();
  };
#pragma unroll 1
  for (int st = 0; st < STG - 1; ++st) {
    __syncthreads();  // a record's place is refilled one segment after its use
    produce(st);
  }
  // fragment addresses: lane (g, tq) holds row g of a block at k = 4 s + tq of step s; with k contiguous, step s's
  // chunks 2 s, 2 s + 1 of a row's 8
  const int f0 = g * BK + 2 * ((tq >> 1) ^ swz(g)) + (tq & 1);
  const int bo = Sh::A::SIZE + (KB ? j0 * 8 + tq * Sh::B::PITCH + g : j0 * 8 * BK);
  int ao[AR], bq[AR];  // WS = 8: a block's rows and columns in a stage
#pragma unroll
  for (int q = 0; q < AR; ++q) {
    const int e = role + 8 * q;
    ao[q] = WS == 1 ? 0 : e / nbt * 8 * BK;
    bq[q] = WS == 1 ? 0 : e % nbt * (KB ? 8 : 8 * BK);
  }
  int st = 0;
  for (;;) {
    cp_wait<STG - 2>();  // this thread's copies of the slice have landed
    __syncthreads();     // everyone's have, and the stage refilled below is no longer read
    const int mk = meta_k[st];
    if (mk == 0) break;
    const int kc = mk & 255;
    const double al = meta_alpha[st];
    produce(st == 0 ? STG - 1 : st - 1);
    const double* as = sm + st * Sh::STAGE;
    const double* bs = as + bo + (KB ? (mk >> (9 + (tq & 1))) & 1 : 0);
    // The warp's R x N blocks of the slice.  One body per shape: a matrix instruction whose predicate is off still
    // takes its slot of the pipe.
    auto body = [&](auto rr, auto nn) {
      constexpr int R = decltype(rr)::value, N = decltype(nn)::value;
      auto step = [&](int s4) {  // four k
        const int fo = (f0 ^ ((s4 & 3) << 2)) + (s4 >> 2) * 16;
        double a[R > 0 ? R : 1];
#pragma unroll
        for (int i = 0; i < R; ++i) a[i] = as[i * 8 * BK + fo];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          double b = KB ? bs[s4 * 4 * Sh::B::PITCH + j * 8] : bs[j * 8 * BK + fo];
          if (mk & 256) b *= al;
#pragma unroll
          for (int i = 0; i < R; ++i) mma884(acc[i][j][0], acc[i][j][1], a[i], b);
        }
      };
#pragma unroll
      for (int s4 = 0; s4 < BK / 4; ++s4)
        if (4 * s4 < kc) step(s4);
    };
    auto bodies = [&](auto rr) {
      if (nb == 4) body(rr, std::integral_constant<int, 4>());
      else if (nb == 3) body(rr, std::integral_constant<int, 3>());
      else if (nb == 2) body(rr, std::integral_constant<int, 2>());
      else if (nb == 1) body(rr, std::integral_constant<int, 1>());
    };
    if constexpr (WS == 8) {
      // one chain of fmas per block, four steps' fragments loaded ahead of it (the zeros past the last k add nothing)
      auto blocks = [&](auto nn) {
        constexpr int N = decltype(nn)::value;
#pragma unroll
        for (int s0 = 0; s0 < BK / 4; s0 += 4) {
          if (4 * s0 >= kc) break;
          double a[N][4], b[N][4];
#pragma unroll
          for (int q = 0; q < N; ++q)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int fo = (f0 ^ (u << 2)) + (s0 >> 2) * 16;
              a[q][u] = as[ao[q] + fo];
              b[q][u] = KB ? bs[(s0 + u) * 4 * Sh::B::PITCH + bq[q]] : bs[bq[q] + fo];
              if (mk & 256) b[q][u] *= al;
            }
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int q = 0; q < N; ++q) mma884(acc[q][0][0], acc[q][0][1], a[q][u], b[q][u]);
        }
      };
      if (AR >= 4 && nq >= 4) blocks(std::integral_constant<int, (AR < 4 ? AR : 4)>());
      else if (AR >= 3 && nq == 3) blocks(std::integral_constant<int, (AR < 3 ? AR : 3)>());
      else if (AR >= 2 && nq == 2) blocks(std::integral_constant<int, (AR < 2 ? AR : 2)>());
      else if (nq >= 1) blocks(std::integral_constant<int, 1>());
    } else if (mb == MB) {
      bodies(std::integral_constant<int, MB>());
    } else if constexpr (ANY) {
      static_assert(MB == 8, "every height has its body");
      if (mb == 7) bodies(std::integral_constant<int, 7>());
      else if (mb == 6) bodies(std::integral_constant<int, 6>());
      else if (mb == 5) bodies(std::integral_constant<int, 5>());
      else if (mb == 4) bodies(std::integral_constant<int, 4>());
      else if (mb == 3) bodies(std::integral_constant<int, 3>());
      else if (mb == 2) bodies(std::integral_constant<int, 2>());
      else bodies(std::integral_constant<int, 1>());
    } else {
      bodies(std::integral_constant<int, MB - 1>());
    }
    st = st == STG - 1 ? 0 : st + 1;
  }
  cp_wait<0>();
  auto store = [&](int i, int j, double v0, double v1) {
    const long long r = m0 + 8 * i + g, c = n0 + 8 * (j0 + j) + 2 * tq;
    if (r >= rows) return;
    double* x = P.C + (tr ? c * P.ldc + r : r * P.ldc + c);
    const long long d = tr ? P.ldc : 1;
    if (c < cols) x[0] = P.beta == 0.0 ? v0 : fma(P.beta, x[0], v0);
    if (c + 1 < cols) x[d] = P.beta == 0.0 ? v1 : fma(P.beta, x[d], v1);
  };
  if constexpr (WS == 1) {
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (j < nb) {
#pragma unroll
        for (int i = 0; i < MB; ++i)
          if (i < mb) store(i, j, acc[i][j][0], acc[i][j][1]);
      }
  } else {
#pragma unroll
    for (int q = 0; q < AR; ++q)
      if (q < nq) store((role + 8 * q) / nbt, (role + 8 * q) % nbt, acc[q][0][0], acc[q][0][1]);
  }
}

template <int MB, int WS, Mode AM, Mode BM_, bool ANY = false>
cudaError_t go(const DGemmProblem* probs, int nprob, const DGemmSeg* segs, long long ntiles, cudaStream_t st) {
  constexpr size_t smem = Shape<MB, WS, AM, BM_>::smem;
  static std::once_flag once[64];  // the attribute, once per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [&] {
    cudaFuncSetAttribute(gemm_mma_f64<MB, WS, AM, BM_, ANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  gemm_mma_f64<MB, WS, AM, BM_, ANY><<<(unsigned)ntiles, threads(WS), smem, st>>>(probs, nprob, segs);
  return cudaGetLastError();
}

using Go = cudaError_t (*)(const DGemmProblem*, int, const DGemmSeg*, long long, cudaStream_t);
// one F per row class
#define TCI_ROWS(F, WS, A, B) \
  F<1, WS, A, B>, F<2, WS, A, B>, F<3, WS, A, B>, F<4, WS, A, B>, F<5, WS, A, B>, F<6, WS, A, B>, F<7, WS, A, B>, F<8, WS, A, B>
#define TCI_PAIR(F, A, B) TCI_ROWS(F, 1, A, B), TCI_ROWS(F, 8, A, B)
#define TCI_CLASSES(F) \
  TCI_PAIR(F, K16, K16), TCI_PAIR(F, K16, R16), TCI_PAIR(F, K8, K8), TCI_PAIR(F, K8, R16), TCI_PAIR(F, RT8, K8), TCI_PAIR(F, RT8, R16)
constexpr Go kGo[tci_dmma::CLASSES] = {TCI_CLASSES(go),
                                       go<8, 1, K16, K16, true>,
                                       go<8, 1, K16, R16, true>,
                                       go<8, 1, K8, K8, true>,
                                       go<8, 1, K8, R16, true>,
                                       go<8, 1, RT8, K8, true>,
                                       go<8, 1, RT8, R16, true>};

// Tile counts of a problem of rows x cols: at most bmb row blocks x bnb column blocks.
struct Cut {
  long long tm, tn;
  int mb, nb;   // blocks of its largest tile
  double cost;  // 8 x 8 blocks computed, each tile's slowest warp times four
};
Cut cut(long long rows, long long cols, int bmb, int bnb) {
  const long long mblk = (rows + 7) / 8, nblk = (cols + 7) / 8;
  Cut c;
  c.tm = (mblk + bmb - 1) / bmb;
  c.tn = (nblk + bnb - 1) / bnb;
  c.mb = (int)((mblk + c.tm - 1) / c.tm);
  c.nb = (int)((nblk + c.tn - 1) / c.tn);
  c.cost = (double)mblk * (double)c.tn * (double)(bnb <= NB ? c.nb : (c.nb + 3) / 4 * 4);
  return c;
}

// What the segments of a problem have in common, of either operand: storage order, room for 16-byte copies.
struct Form {
  bool a_k = true, a_r = true, b_k = true, b_r = true, a_even = true, b_even = true;
  double k = 0;
};
Form form(const DGemmProblem& g, const std::vector<DGemmSeg>& segs) {
  Form f;
  for (long long q = g.seg_begin; q < g.seg_end; ++q) {
    const DGemmSeg& y = segs[(size_t)q];
    f.a_k = f.a_k && y.tA == 0;
    f.a_r = f.a_r && y.tA != 0;
    f.b_k = f.b_k && y.tB != 0;
    f.b_r = f.b_r && y.tB == 0;
    f.a_even = f.a_even && (y.lda & 1) == 0 && (reinterpret_cast<uintptr_t>(y.A) & 15) == 0;
    f.b_even = f.b_even && (y.ldb & 1) == 0 && (reinterpret_cast<uintptr_t>(y.B) & 15) == 0;
    f.k += (double)y.K;
  }
  if ((!f.a_k && !f.a_r) || (!f.b_k && !f.b_r))
    throw std::invalid_argument("a GEMM problem whose segments differ in storage order");
  return f;
}

// Tiles and class of a problem at a largest tile of bmb x bnb blocks; bnb <= NB: the blocks are dealt to eight warps.
struct Place {
  bool swapped;
  Cut c;
  int cls;
  double work;  // its largest tile's blocks x its k (eight warps: four blocks' worth for what a slice costs besides)
};
Place place(const DGemmProblem& g, const Form& f, int bmb, int bnb) {
  Place x;
  x.swapped = cut(g.N, g.M, bmb, bnb).cost < 0.8 * cut(g.M, g.N, bmb, bnb).cost;
  // rows and columns of the tiles, in terms of C^T = B^T A^T when the operands change places
  const bool row_k = x.swapped ? f.b_k : f.a_k, col_k = x.swapped ? f.a_k : f.b_k;
  const bool row_even = x.swapped ? f.b_even : f.a_even, col_even = x.swapped ? f.a_even : f.b_even;
  const int modes = !row_k ? (col_k ? 4 : 5) : col_k ? (row_even && col_even ? 0 : 2) : (row_even ? 1 : 3);
  if (!col_k && !col_even && bnb > NB) bnb = std::min(bnb, 15);  // room for shifted rows
  // odd leading dimensions, more rows than one tile: six blocks high, three blocks per SM (8-byte copies and uneven
  // shares leave gaps in the pipe that a third block fills: 173 x 173 x (40 x 173) 10.4 -> 9.7 ms; even ones lose 3-5 %)
  if (modes == 3 && bnb > NB && (x.swapped ? g.N : g.M) > 64) bmb = std::min(bmb, 6);
  x.c = x.swapped ? cut(g.N, g.M, bmb, bnb) : cut(g.M, g.N, bmb, bnb);
  x.cls = x.c.mb - 1 + (bnb <= NB ? 8 : 0) + 16 * modes;
  x.work = (bnb <= NB ? (double)x.c.mb * x.c.nb + 4 : (double)x.c.mb * ((x.c.nb + 3) / 4 * 4)) * f.k;
  return x;
}

}  // namespace

namespace tci_dmma {

Tiles tile(const std::vector<DGemmProblem>& pr, const std::vector<DGemmSeg>& segs) {
  // the longest problems first: the short ones fill the last wave
  std::vector<Form> forms;
  std::vector<size_t> order, kind;
  // problems of one shape and form are placed alike: looked at once, with the longest k (a plan has hundreds of them)
  struct Kind {
    DGemmProblem g;
    Form f;
    double count;
  };
  std::vector<Kind> kinds;
  std::map<std::array<long long, 3>, size_t> seen;
  for (size_t i = 0; i < pr.size(); ++i) {
    const Form f = form(pr[i], segs);
    const long long flags = f.a_k | f.a_r << 1 | f.b_k << 2 | f.b_r << 3 | f.a_even << 4 | f.b_even << 5;
    const auto at = seen.insert({{pr[i].M, pr[i].N, flags}, kinds.size()});
    if (at.second) kinds.push_back(Kind{pr[i], f, 0});
    Kind& x = kinds[at.first->second];
    x.count += 1;
    x.f.k = std::max(x.f.k, f.k);
    kind.push_back(at.first->second);
    forms.push_back(f);
    order.push_back(i);
  }
  std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) { return forms[a].k > forms[b].k; });
  // Tile width by the time the fullest SM would need: waves of tiles x the largest tile, the narrower ones at the
  // rate they were measured at (28 TFLOP/s for 12 blocks, 24 for 8 and 19 for the eight warps' 4 against 30 for 16 on
  // a launch that fills the chip).  Wide tiles win once there are several waves, narrow and dealt ones where a
  // launch would leave SMs idle.
  const double sms = (double)tci_dev::device_sms();
  struct Try {
    int bmb, bnb;
    double slow;
  };
  Try best{8, 16, 1.0};
  double best_time = 0;
  for (const Try& y : {best, Try{8, 12, 1.12}, Try{8, 8, 1.25}, Try{8, NB, 1.6}, Try{4, NB, 1.6}, Try{3, 3, 1.6}, Try{2, 2, 1.6}}) {
    double work = 0, n = 0;
    for (const Kind& q : kinds) {
      const Place x = place(q.g, q.f, y.bmb, y.bnb);
      n += q.count * (double)(x.c.tm * x.c.tn);
      work = std::max(work, x.work);
    }
    const double time = std::ceil(n / sms) * work * y.slow;
    if (y.bnb == 16 || time < 0.97 * best_time) {
      best = y;
      best_time = time;
    }
    if (n > 16 * sms) break;
  }
  std::vector<Place> places;
  for (const Kind& q : kinds) places.push_back(place(q.g, q.f, best.bmb, best.bnb));
  // The heights of a mode pair run one after another, a launch each. Where those launches are short (problems of many sizes,
  // few tiles of each, a long k: the second product of 30 pair domains of 60-150 externals, 18 + 28 + 74 + 27 tiles, 16.5 ms
  // in four launches, 5.6 in one; the scalar kernel's one launch 10) one launch for all of them: its time by the same rule,
  // with a margin for the two blocks per SM and registers of the highest tile that all its tiles have.
  for (int m = 0; m < 6; ++m) {
    double n[8] = {}, work[8] = {}, all = 0, longest = 0, apart = 0;
    for (size_t i = 0; i < kinds.size(); ++i) {
      const Place& x = places[i];
      if (x.cls / 8 != 2 * m) continue;  // blocks dealt to eight warps, or another pair
      const double tiles = kinds[i].count * (double)(x.c.tm * x.c.tn);
      n[x.cls % 8] += tiles;
      work[x.cls % 8] = std::max(work[x.cls % 8], x.work);
      all += tiles;
      longest = std::max(longest, x.work);
    }
    for (int c = 0; c < 8; ++c) apart += std::ceil(n[c] / sms) * work[c];
    if (std::ceil(all / sms) * longest < 0.8 * apart)
      for (Place& x : places)
        if (x.cls < ROW_CLASSES && x.cls / 8 == 2 * m) x.cls = ROW_CLASSES + m;
  }
  Tiles t;
  for (size_t i : order) {
    const Place& x = places[kind[i]];
    DGemmProblem g = pr[i];
    g.trans_c = (x.swapped ? 1 : 0) | 2 * x.c.tm;
    g.tiles_n = x.c.tn;
    g.tile_begin = t.ntiles[x.cls];
    t.ntiles[x.cls] += x.c.tm * x.c.tn;
    t.probs[x.cls].push_back(g);
  }
  return t;
}

cudaError_t launch(const Tables& t, const DGemmSeg* segs, cudaStream_t st) {
  for (int c = 0; c < CLASSES; ++c) {
    if (t.ntiles[c] <= 0) continue;
    const cudaError_t e = kGo[c](t.probs[c], t.nprob[c], segs, t.ntiles[c], st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace tci_dmma

// Test entry, host only: the copies that a block of class cls makes of a segment's operand (which 0: the row operand, 1:
// the column operand): nr rows of the tile x K, leading dimension ld, from element off of an allocation of len doubles.
// out: {copies, copies with an address not aligned to the instruction's size, copies from outside the allocation or to
// outside the slice}.
namespace {
template <int MB, int WS, Mode AM, Mode BM_>
void copies_of(int which, int nr, long long K, long long ld, long long off, long long len, int64_t* out) {
  using Sh = Shape<MB, WS, AM, BM_>;
  double* const base = reinterpret_cast<double*>((uintptr_t)1 << 40);  // an allocation's alignment; never read
  struct Count {
    int64_t* out;
    uintptr_t lo, hi;
    unsigned size;
    void see(unsigned s, const void* g, int bytes, unsigned unit) const {
      const uintptr_t a = reinterpret_cast<uintptr_t>(g);
      out[0] += 1;
      out[1] += a % unit || s % unit;
      out[2] += a < lo || a + (uintptr_t)std::max(bytes, 1) > hi || s + unit > size || bytes < 0 || bytes > (int)unit;
    }
    void copy16(unsigned s, const void* g, int bytes) const { see(s, g, bytes, 16); }
    void copy8(unsigned s, const void* g, int bytes) const { see(s, g, bytes, 8); }
  };
  auto all = [&](auto op) {
    using Op = decltype(op);
    const Count c{out, reinterpret_cast<uintptr_t>(base), reinterpret_cast<uintptr_t>(base + len), 8u * (unsigned)Op::SIZE};
    for (int tid = 0; tid < Sh::NT; ++tid) {
      Op o;
      o.open(tid, base + off, ld, 0);
      for (long long k = K; k > 0; k -= Sh::BK) o.issue(tid, 0, nr, (int)k, c);
    }
  };
  if (which == 0) all(typename Sh::A());
  else all(typename Sh::B());
}
using CopiesOf = void (*)(int, int, long long, long long, long long, long long, int64_t*);
constexpr CopiesOf kCopies[tci_dmma::ROW_CLASSES] = {TCI_CLASSES(copies_of)};
}  // namespace
extern "C" int tci_selftest_gemm_f64_copies(int64_t cls, int64_t which, int64_t nr, int64_t K, int64_t ld, int64_t off,
                                            int64_t len, int64_t* out) {
  if (!out || cls < 0 || cls >= tci_dmma::ROW_CLASSES || which < 0 || which > 1 || nr < 1 || K < 1 || ld < 1 || off < 0)
    return TCI_ERR_ARG;
  out[0] = out[1] = out[2] = 0;
  kCopies[cls]((int)which, (int)nr, K, ld, off, len, out);
  return TCI_OK;
}

// Test entry: C (M x N) = beta C + alpha sum_s op(A_s) op(B_s) on host arrays, nseg matrices a_step / b_step apart
// from element a_off / b_off on.
extern "C" int tci_selftest_gemm_f64(int64_t device, int64_t M, int64_t N, int64_t K, int64_t nseg, int64_t tA, int64_t tB,
                                     int64_t lda, int64_t ldb, int64_t ldc, int64_t a_off, int64_t b_off, int64_t a_step,
                                     int64_t b_step, double alpha, double beta, const double* A, int64_t na,
                                     const double* B, int64_t nb, double* C) {
  if (!A || !B || !C || M < 1 || N < 1 || K < 1 || nseg < 0 || a_off < 0 || b_off < 0 || a_step < 0 || b_step < 0 ||
      lda < (tA ? M : K) || ldb < (tB ? K : N) || ldc < N)
    return TCI_ERR_ARG;
  const int64_t ea = ((tA ? K : M) - 1) * lda + (tA ? M : K), eb = ((tB ? N : K) - 1) * ldb + (tB ? K : N);
  if (nseg > 0 && (a_off + (nseg - 1) * a_step + ea > na || b_off + (nseg - 1) * b_step + eb > nb)) return TCI_ERR_ARG;
  double *dA = nullptr, *dB = nullptr, *dC = nullptr;
  DGemmSeg* ds = nullptr;
  DGemmProblem* dp = nullptr;
  int rc = TCI_OK;
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess && rc == TCI_OK) rc = TCI_ERR_CUDA;
    return rc == TCI_OK;
  };
  try {
    const size_t cb = sizeof(double) * (size_t)((M - 1) * ldc + N);
    if (ok(cudaSetDevice((int)device)) && ok(cudaMalloc(&dA, sizeof(double) * (size_t)na)) &&
        ok(cudaMalloc(&dB, sizeof(double) * (size_t)nb)) && ok(cudaMalloc(&dC, cb)) &&
        ok(cudaMalloc(&ds, sizeof(DGemmSeg) * (size_t)std::max<int64_t>(1, nseg))) && ok(cudaMalloc(&dp, sizeof(DGemmProblem)))) {
      std::vector<DGemmSeg> segs;
      for (int64_t q = 0; q < nseg; ++q)
        segs.push_back(DGemmSeg{dA + a_off + q * a_step, dB + b_off + q * b_step, lda, ldb, K, tA ? 1 : 0, tB ? 1 : 0, alpha});
      const tci_dmma::Tiles t = tci_dmma::tile({DGemmProblem{dC, ldc, M, N, 0, 0, beta, 0, nseg, 0}}, segs);
      ok(cudaMemcpy(dA, A, sizeof(double) * (size_t)na, cudaMemcpyHostToDevice));
      ok(cudaMemcpy(dB, B, sizeof(double) * (size_t)nb, cudaMemcpyHostToDevice));
      ok(cudaMemcpy(dC, C, cb, cudaMemcpyHostToDevice));
      if (nseg > 0) ok(cudaMemcpy(ds, segs.data(), sizeof(DGemmSeg) * segs.size(), cudaMemcpyHostToDevice));
      tci_dmma::Tables d;
      for (int c = 0; c < tci_dmma::CLASSES; ++c)
        if (t.ntiles[c] > 0) {
          ok(cudaMemcpy(dp, t.probs[c].data(), sizeof(DGemmProblem), cudaMemcpyHostToDevice));
          d.probs[c] = dp;
          d.nprob[c] = 1;
          d.ntiles[c] = t.ntiles[c];
        }
      if (rc == TCI_OK) ok(tci_dmma::launch(d, ds, 0));
      ok(cudaDeviceSynchronize());
      ok(cudaMemcpy(C, dC, cb, cudaMemcpyDeviceToHost));
    }
  } catch (...) {
    rc = TCI_ERR_INTERNAL;
  }
  for (void* p : {(void*)dA, (void*)dB, (void*)dC, (void*)ds, (void*)dp}) cudaFree(p);
  return rc;
}

// Test entry: nprob products C_p (M x N) = op(A_p) op(B_p) of one launch, the matrices one after the other from 16-byte
// aligned places, leading dimensions pad above the rows' lengths. tiles[CLASSES]: the tiles of each class; device < 0: only
// these.
extern "C" int tci_selftest_gemm_f64_group(int64_t device, int64_t nprob, const int64_t* M, const int64_t* N, const int64_t* K,
                                           int64_t tA, int64_t tB, int64_t pad, const double* A, int64_t na, const double* B,
                                           int64_t nb, double* C, int64_t nc, int64_t* tiles) {
  if (nprob < 1 || !M || !N || !K || pad < 0 || !tiles || (device >= 0 && (!A || !B || !C))) return TCI_ERR_ARG;
  double *dA = nullptr, *dB = nullptr, *dC = nullptr;
  DGemmSeg* ds = nullptr;
  DGemmProblem* dp = nullptr;
  int rc = TCI_OK;
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess && rc == TCI_OK) rc = TCI_ERR_CUDA;
    return rc == TCI_OK;
  };
  try {
    int64_t ea = 0, eb = 0, ec = 0;
    auto take = [](int64_t& at, int64_t rows, int64_t ld) {
      const int64_t o = at;
      at += (rows * ld + 1) / 2 * 2;
      return o;
    };
    std::vector<int64_t> oa, ob, oc;
    for (int64_t p = 0; p < nprob; ++p) {
      if (M[p] < 1 || N[p] < 1 || K[p] < 1) return TCI_ERR_ARG;
      oa.push_back(take(ea, tA ? K[p] : M[p], (tA ? M[p] : K[p]) + pad));
      ob.push_back(take(eb, tB ? N[p] : K[p], (tB ? K[p] : N[p]) + pad));
      oc.push_back(take(ec, M[p], N[p]));
    }
    if (device >= 0) {
      if (ea > na || eb > nb || ec > nc) return TCI_ERR_ARG;
      if (ok(cudaSetDevice((int)device)) && ok(cudaMalloc(&dA, sizeof(double) * (size_t)ea)) &&
          ok(cudaMalloc(&dB, sizeof(double) * (size_t)eb)) && ok(cudaMalloc(&dC, sizeof(double) * (size_t)ec)) &&
          ok(cudaMalloc(&ds, sizeof(DGemmSeg) * (size_t)nprob)))
        ok(cudaMalloc(&dp, sizeof(DGemmProblem) * (size_t)nprob));
    }
    if (rc == TCI_OK) {
      std::vector<DGemmProblem> pr;
      std::vector<DGemmSeg> sg;
      for (int64_t p = 0; p < nprob; ++p) {
        pr.push_back(DGemmProblem{dC + oc[p], N[p], M[p], N[p], 0, 0, 0.0, p, p + 1, 0});
        sg.push_back(DGemmSeg{dA + oa[p], dB + ob[p], (tA ? M[p] : K[p]) + pad, (tB ? K[p] : N[p]) + pad, K[p], tA ? 1 : 0,
                              tB ? 1 : 0, 1.0});
      }
      const tci_dmma::Tiles t = tci_dmma::tile(pr, sg);
      for (int c = 0; c < tci_dmma::CLASSES; ++c) tiles[c] = t.ntiles[c];
      if (device >= 0) {
        const tci_dmma::Tables d = tci_dmma::tables(t, [&](const std::vector<DGemmProblem>& v) {
          ok(cudaMemcpy(dp, v.data(), sizeof(DGemmProblem) * v.size(), cudaMemcpyHostToDevice));
          return dp;
        });
        ok(cudaMemcpy(ds, sg.data(), sizeof(DGemmSeg) * sg.size(), cudaMemcpyHostToDevice));
        ok(cudaMemcpy(dA, A, sizeof(double) * (size_t)ea, cudaMemcpyHostToDevice));
        ok(cudaMemcpy(dB, B, sizeof(double) * (size_t)eb, cudaMemcpyHostToDevice));
        ok(cudaMemcpy(dC, C, sizeof(double) * (size_t)ec, cudaMemcpyHostToDevice));  // the gaps between the products
        if (rc == TCI_OK) ok(tci_dmma::launch(d, ds, 0));
        ok(cudaDeviceSynchronize());
        if (rc == TCI_OK) ok(cudaMemcpy(C, dC, sizeof(double) * (size_t)ec, cudaMemcpyDeviceToHost));
      }
    }
  } catch (...) {
    rc = TCI_ERR_INTERNAL;
  }
  for (void* p : {(void*)dA, (void*)dB, (void*)dC, (void*)ds, (void*)dp}) cudaFree(p);
  return rc;
}
