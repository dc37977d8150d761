// The all-external term over pair domains in the integral form (local_integral.cu): host side.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

namespace tci_lint {

// One spin-function block of a head: the CI offsets of its ab / aa entries (-1: none), its domain (a slice of dom)
// and p = +1 singlet-coupled, -1 triplet-coupled.
struct Block {
  long long ab, aa;
  double p;
  int n, dom, head, pad;
};
// The rows (a, b) of sigma, b in [b0, b0 + rows), of the blocks cblk[col0 .. col0 + ncol) (accumulator columns), over
// the jobs [job0, job1); the sums go to copy `part` of sigma.
struct Task {
  int a, b0, rows, col0, ncol, job0, job1, part;
};
// The columns jcol[off .. off + cnt) (places in the task's accumulators) that share the external c with a.
struct Job {
  int c, off, cnt, pad;
};
struct Plan {
  std::vector<Block> blocks;
  std::vector<Task> tasks;
  std::vector<Job> jobs;
  std::vector<int> cblk, jcol, dom;
  std::vector<short> pos;  // heads x nv: position of an external in the head's domain, -1 outside
  int nv = 0, parts = 1;
  double flops = 0;  // products computed, times two (padding counted)
};
struct Device {
  Block* blocks = nullptr;
  Task* tasks = nullptr;
  Job* jobs = nullptr;
  int *cblk = nullptr, *jcol = nullptr, *dom = nullptr;
  short* pos = nullptr;
  double *C = nullptr, *part = nullptr;  // padded pair matrices; copies of sigma (parts > 1)
  int nblocks = 0, ntasks = 0, nv = 0, parts = 1;
};
// Row pitch of the padded pair matrices.
inline int64_t pitch(int64_t nv) { return (nv + 15) / 16 * 16; }
constexpr int64_t MAX_NV = 2000;
// The tables index their lists (the longest holds n_h^2 entries per block) in 32 bits: do these blocks' fit?
bool fits(const std::vector<Block>& blocks);
// sms: multiprocessors to fill. The blocks fit.
void make_plan(int nv, int nheads, const std::vector<int>& dom, std::vector<Block> blocks, int sms, Plan& out);
// X (npv x npv) from its lower triangle.
cudaError_t mirror(double* X, int64_t npv, cudaStream_t st);
// sigma entries of every block = the all-external term of the CI vector c; X[(ac)][(bd)] = (ac|bd), packed pairs, full
// rows; sigma (total entries) is zero on entry.
cudaError_t launch(const Device& d, const double* X, int64_t npv, const double* c, double* sigma, int64_t total,
                   cudaStream_t st);

}  // namespace tci_lint
