// Screened quartet task lists, built on the device (tasks.cu).
#pragma once
#include <cuda_runtime.h>

#include "engine.cuh"

namespace iqcp {

constexpr int kNumRanges = kNumPairClasses * (kNumPairClasses + 1) / 2;
__host__ __device__ constexpr int range_of(int X, int Y) { return X * (X + 1) / 2 + Y; }

// Ket lists as the task kernels see them (device arrays).  Segment li = molecule
// * 6 + class holds positions seg[li] .. seg[li + 1] - 1 of the ket list.
struct TaskLists {
  int n;                    // positions
  int n_seg;                // segments
  const int* ket_list;      // pair of a position
  const int* pos_seg;       // segment of a position
  const int* seg;           // n_seg + 1
  const int* seg_rank;      // pairs of the segment's class in the molecules before
  const int* bucket0;       // n_seg + 1: first bucket of a segment
  const int4* bucket;       // {first position, length, np, -}
  const int4* i0;           // ket tables: .z = np
  const double* Q;          // Schwarz bound by position
  double thr;
  long long entry0[kNumRanges + 1];  // first entry of a range: an entry is (range, bra), up to six per position
};

// Primitive quartets and quartets of every range: sums[2 r], sums[2 r + 1]
cudaError_t launch_task_work(const TaskLists& t, unsigned long long* sums, cudaStream_t st);
// Tasks of every entry, then their exclusive sum in place (offset[entries] = total);
// part: scratch of entries / 1024 + 2 words.  first[r]: first task of range r, first[kNumRanges] the total,
// or -1 where it does not fit an int.
struct PerLane {
  double v[kNumRanges];  // primitive quartets a lane should serve
};
cudaError_t launch_task_offsets(const TaskLists& t, const PerLane& p, int* offset, long long* part, int* first,
                                cudaStream_t st);
cudaError_t launch_task_fill(const TaskLists& t, const PerLane& p, const int* offset, QuartetTask* tasks,
                             cudaStream_t st);

}  // namespace iqcp
