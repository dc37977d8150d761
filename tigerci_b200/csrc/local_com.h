// The two-external products of a local deck on the common virtuals (local_com.cu): host side.
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace tci_com {

constexpr int COLS = 48;  // common columns of a job at most

// One term's columns [.., + cnt): R[a][ct[j]] += alpha sum_k A[a][k] B[k][cs[j]] over the rows a of the task.
struct Job {
  const double* A;   // compact: A[D_target][D_source], row pitch pitch_a (even, 16-byte aligned); else the n x n matrix
  const double* B;   // the source's compact pair matrix, row pitch pitch_b
  const int* dom;    // the source's domain (gathered A only)
  const int* cs;     // the common columns: positions in the source's domain ...
  const int* ct;     // ... and in the target's
  int m, cnt, pitch_a, pitch_b;  // m: the source's domain size (the k range)
  double alpha;
  int compact, pad;
};
// Rows [r0, r0 + rows) and columns [c0, c0 + m) of the target's domain, added into its padded pair matrix R at the end;
// the jobs' ct lie in the columns.
struct Task {
  double* R;
  const int* dom;
  int m, r0, rows, job0, job1, c0;
};
// Row tiles by number of columns: the tile's sums (columns x rows) live in shared memory.
constexpr int CLASSES = 4;
// One term of a target: the operands as in Job, all its common columns, their positions in the target's domain also on
// the host (ascending).
struct Term {
  Job job;
  const int* host_ct;
};
// The tasks and jobs of a launch.
struct HostPlan {
  struct HostTask {
    double work;
    Task t;
  };
  std::vector<Job> jobs;
  std::vector<HostTask> tasks[CLASSES];
  // one target: its padded pair matrix, domain (device) and terms
  void add(double* R, const int* dom, int m, const std::vector<Term>& terms);
  // a class's tasks, the longest first
  std::vector<Task> sorted(int cls);
};
struct Tables {
  Task* tasks[CLASSES] = {};
  int ntasks[CLASSES] = {}, mmax[CLASSES] = {};
  Job* jobs = nullptr;
  int launches() const {
    int k = 0;
    for (int t : ntasks) k += t > 0 ? 1 : 0;
    return k;
  }
};
cudaError_t launch(const Tables& t, long long ld, cudaStream_t st);

}  // namespace tci_com
