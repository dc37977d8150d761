// FP64 grouped GEMM on the double-precision matrix instruction (gemm_mma_f64.cu): host side.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "gemm_tables.h"

namespace tci_dmma {

// Problems sorted into the kernel's tile classes: six pairs of operand modes (storage order and copy width of the row and
// the column operand) x two work splits (four warps share a tile's columns, or eight its 8 x 8 blocks where a launch has
// too few tiles) x one to eight 8-row blocks of a tile; six more for tiles of any height on shared columns, one launch where the
// heights' own launches would be short.
constexpr int ROW_CLASSES = 96, CLASSES = ROW_CLASSES + 6;
struct Tiles {
  std::vector<tci_dev::DGemmProblem> probs[CLASSES];
  long long ntiles[CLASSES] = {};
};
// Sorts a launch's problems (their tiles_n, tile_begin and trans_c are set here).
Tiles tile(const std::vector<tci_dev::DGemmProblem>& pr, const std::vector<tci_dev::DGemmSeg>& segs);
// The device copies of a Tiles.
struct Tables {
  tci_dev::DGemmProblem* probs[CLASSES] = {};
  int nprob[CLASSES] = {};
  long long ntiles[CLASSES] = {};
  int launches() const {
    int k = 0;
    for (long long t : ntiles) k += t > 0 ? 1 : 0;
    return k;
  }
};
// The device copies of a launch's problems, all classes in one table; up: uploads a vector of problems.
template <class Upload>
Tables tables(const Tiles& t, Upload&& up) {
  std::vector<tci_dev::DGemmProblem> all;
  for (const auto& p : t.probs) all.insert(all.end(), p.begin(), p.end());
  tci_dev::DGemmProblem* d = up(all);
  Tables x;
  for (int c = 0; c < CLASSES; ++c) {
    x.probs[c] = d;
    x.nprob[c] = (int)t.probs[c].size();
    x.ntiles[c] = t.ntiles[c];
    d += t.probs[c].size();
  }
  return x;
}
// All classes of a launch, segs the table its problems index.
cudaError_t launch(const Tables& t, const tci_dev::DGemmSeg* segs, cudaStream_t st);

}  // namespace tci_dmma
