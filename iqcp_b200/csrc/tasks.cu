// Quartet tasks from the Schwarz bounds, built on the device.
//
// A task is one bra against up to 32 kets of a bucket prefix (equal primitive
// count, Q descending) that passes Q_bra Q_ket >= thr; see QuartetTask.  A thread
// per bra walks the ket classes Y <= X of its molecule and their buckets with one
// binary search each: once for the work per class pair, which sets the lanes per
// quartet, once to count its tasks, and once to write them behind an exclusive
// sum.  Tasks lie class pair by class pair, then molecule, bra, bucket.  Building
// them on the host and copying 24 bytes each was most of what a context cost:
// 40 atoms in 6-31G* 41 -> 10 ms with this and the pooled memory.
#include "tasks.h"

namespace iqcp {
namespace {

// Kets of bucket bk that pass with bra position b: a prefix; with a ket list of the
// bra's own class only positions up to b (unique quartets)
__device__ __forceinline__ int bucket_kets(const TaskLists& t, int4 bk, int b, double qb, bool same) {
  int lo = 0, hi = bk.y;
  if (same && b + 1 - bk.x < hi) hi = b + 1 - bk.x;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (qb * t.Q[bk.x + mid] < t.thr) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// f(Y, bucket, kets) for the non-empty buckets of bra position b
template <typename F>
__device__ __forceinline__ void for_buckets(const TaskLists& t, int b, F&& f) {
  const int li = t.pos_seg[b], X = li % kNumPairClasses, l0 = li - X;
  const double qb = t.Q[b];
  for (int Y = 0; Y <= X; ++Y)
    for (int k = t.bucket0[l0 + Y]; k < t.bucket0[l0 + Y + 1]; ++k) {
      const int4 bk = t.bucket[k];
      if (X == Y && bk.x > b) break;
      const int nk = bucket_kets(t, bk, b, qb, X == Y);
      if (nk > 0) f(Y, bk, nk);
    }
}

__device__ __forceinline__ long long entry_of(const TaskLists& t, int b, int X, int Y) {
  const int li = t.pos_seg[b];
  return t.entry0[range_of(X, Y)] + t.seg_rank[li] + b - t.seg[li];
}

// lanes per quartet (log2) of quartets with `prims` primitive quartets
__device__ __forceinline__ int lanes_log2(double prims, double per_lane) {
  int lg = 0;
  while (lg < 5 && prims > per_lane * double(1 << lg)) ++lg;
  return lg;
}

__global__ void __launch_bounds__(128) task_work_kernel(TaskLists t, unsigned long long* sums) {
  __shared__ unsigned long long sh[2 * kNumRanges];
  for (int i = threadIdx.x; i < 2 * kNumRanges; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < t.n) {
    const int X = t.pos_seg[b] % kNumPairClasses;
    const unsigned long long nb = t.i0[b].z;
    unsigned long long w[kNumPairClasses] = {0}, q[kNumPairClasses] = {0};
    for_buckets(t, b, [&](int Y, int4 bk, int nk) {
#pragma unroll
      for (int y = 0; y < kNumPairClasses; ++y)
        if (y == Y) {
          w[y] += nb * bk.z * nk;
          q[y] += nk;
        }
    });
#pragma unroll
    for (int y = 0; y < kNumPairClasses; ++y)
      if (q[y]) {
        atomicAdd(sh + 2 * range_of(X, y), w[y]);
        atomicAdd(sh + 2 * range_of(X, y) + 1, q[y]);
      }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * kNumRanges; i += blockDim.x)
    if (sh[i]) atomicAdd(sums + i, sh[i]);
}

__global__ void __launch_bounds__(128) task_count_kernel(TaskLists t, PerLane p, int* count) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= t.n) return;
  const int X = t.pos_seg[b] % kNumPairClasses;
  const double nb = t.i0[b].z;
  int c[kNumPairClasses] = {0};
  for_buckets(t, b, [&](int Y, int4 bk, int nk) {
    const int per = 32 >> lanes_log2(nb * bk.z, p.v[range_of(X, Y)]);
#pragma unroll
    for (int y = 0; y < kNumPairClasses; ++y)
      if (y == Y) c[y] += (nk + per - 1) / per;
  });
#pragma unroll
  for (int y = 0; y < kNumPairClasses; ++y)
    if (y <= X) count[entry_of(t, b, X, y)] = c[y];
}

__global__ void __launch_bounds__(128) task_fill_kernel(TaskLists t, PerLane p, const int* offset, QuartetTask* tasks) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= t.n) return;
  const int X = t.pos_seg[b] % kNumPairClasses, bra = t.ket_list[b];
  const double nb = t.i0[b].z;
  int lastY = -1;
  long long at = 0;
  for_buckets(t, b, [&](int Y, int4 bk, int nk) {
    if (Y != lastY) {
      lastY = Y;
      at = offset[entry_of(t, b, X, Y)];
    }
    const double prims = nb * bk.z;
    const int lg = lanes_log2(prims, p.v[range_of(X, Y)]);
    for (int k0 = 0; k0 < nk;) {
      QuartetTask q;
      q.bra = bra;
      q.ket0 = bk.x + k0;
      q.nket = nk - k0 < (32 >> lg) ? nk - k0 : 32 >> lg;
      q.diag = X == Y ? 1 : 0;
      q.bra_pos = b;
      q.lg = lg;
      // a bucket's last kets: spread over the lanes left, two primitive quartets a lane at least
      while (q.lg < 5 && (q.nket << (q.lg + 1)) <= 32 && prims >= double(4 << q.lg)) ++q.lg;
      k0 += q.nket;
      tasks[at++] = q;
    }
  });
}

// Exclusive sums of 1024-element chunks in place; part[chunk] = the chunk's total,
// in 64 bits: 1024 bras of a large molecule may have more than 2^31 tasks, and a
// total that wraps would pass for a small one
__global__ void __launch_bounds__(1024) scan_chunks_kernel(long long n, int* v, long long* part) {
  __shared__ long long sh[32];
  const long long i = blockIdx.x * 1024LL + threadIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long x = i < n ? v[i] : 0;
  long long s = x;
  for (int o = 1; o < 32; o <<= 1) {
    const long long u = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += u;
  }
  if (lane == 31) sh[w] = s;
  __syncthreads();
  if (w == 0) {
    long long u = sh[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const long long z = __shfl_up_sync(0xffffffffu, u, o);
      if (lane >= o) u += z;
    }
    sh[lane] = u;
  }
  __syncthreads();
  s += w > 0 ? sh[w - 1] : 0;
  if (i < n) v[i] = int(s - x);
  if (threadIdx.x == 1023) part[blockIdx.x] = s;
}

// Exclusive sum of the chunk totals (one block; n chunks, total behind them; -1 if it passes 2^31 - 1)
__global__ void __launch_bounds__(1024) scan_parts_kernel(int n, long long* part) {
  __shared__ long long sh[32];
  __shared__ long long carry;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int c0 = 0; c0 < n; c0 += 1024) {
    const int i = c0 + threadIdx.x;
    const long long x = i < n ? part[i] : 0;
    long long s = x;
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    if (lane == 31) sh[w] = s;
    __syncthreads();
    if (w == 0) {
      long long u = sh[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const long long z = __shfl_up_sync(0xffffffffu, u, o);
        if (lane >= o) u += z;
      }
      sh[lane] = u;
    }
    __syncthreads();
    s += carry + (w > 0 ? sh[w - 1] : 0);
    if (i < n) part[i] = s - x;
    __syncthreads();
    if (threadIdx.x == 1023) carry = s;
    __syncthreads();
  }
  if (threadIdx.x == 0) part[n] = carry > 0x7fffffffLL ? -1 : carry;
}

__global__ void __launch_bounds__(1024) scan_add_kernel(long long n, int chunks, int* v, const long long* part) {
  const long long i = blockIdx.x * 1024LL + threadIdx.x;
  if (i < n) v[i] += int(part[blockIdx.x]);
  if (i == 0) v[n] = int(part[chunks]);
}

__global__ void range_first_kernel(TaskLists t, const int* offset, int* first) {
  if (threadIdx.x <= kNumRanges) first[threadIdx.x] = offset[t.entry0[threadIdx.x]];
}

}  // namespace

cudaError_t launch_task_work(const TaskLists& t, unsigned long long* sums, cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(sums, 0, sizeof(unsigned long long) * 2 * kNumRanges, st);
  if (e != cudaSuccess || t.n == 0) return e;
  task_work_kernel<<<(t.n + 127) / 128, 128, 0, st>>>(t, sums);
  return cudaGetLastError();
}

cudaError_t launch_task_offsets(const TaskLists& t, const PerLane& p, int* offset, long long* part, int* first,
                                cudaStream_t st) {
  const long long n = t.entry0[kNumRanges];
  const int chunks = int((n + 1023) / 1024);
  if (n == 0) return cudaMemsetAsync(first, 0, sizeof(int) * (kNumRanges + 1), st);
  task_count_kernel<<<(t.n + 127) / 128, 128, 0, st>>>(t, p, offset);
  scan_chunks_kernel<<<chunks, 1024, 0, st>>>(n, offset, part);
  scan_parts_kernel<<<1, 1024, 0, st>>>(chunks, part);
  scan_add_kernel<<<chunks, 1024, 0, st>>>(n, chunks, offset, part);
  range_first_kernel<<<1, 32, 0, st>>>(t, offset, first);
  return cudaGetLastError();
}

cudaError_t launch_task_fill(const TaskLists& t, const PerLane& p, const int* offset, QuartetTask* tasks,
                             cudaStream_t st) {
  if (t.n == 0) return cudaSuccess;
  task_fill_kernel<<<(t.n + 127) / 128, 128, 0, st>>>(t, p, offset, tasks);
  return cudaGetLastError();
}

}  // namespace iqcp
