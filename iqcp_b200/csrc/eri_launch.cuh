// Launchers for one bra class (LA, LB) against every ket class Y <= X.
// Classes with many components use the warp-cooperative kernels
// (eri_team.cuh); the small ones take a group of lanes per quartet.
#pragma once
#include <atomic>

#include "device_pool.h"
#include "eri_md.cuh"
#include "eri_team.cuh"

namespace iqcp {


// Device limits that every launch needs, asked once per device.
struct DeviceLimits {
  int sms = 0, smem_optin = 0;
};
inline DeviceLimits device_limits(int dev) {
  static std::atomic<unsigned long long> known[64];  // SMs << 32 | opt-in shared memory; 0: not asked yet
  const int slot = dev >= 0 && dev < 64 ? dev : -1;
  unsigned long long v = slot >= 0 ? known[slot].load(std::memory_order_relaxed) : 0;
  if (!v) {
    int sms = 0, optin = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 1;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) optin = 0;
    v = ((unsigned long long)sms << 32) | (unsigned)optin;
    if (slot >= 0) known[slot].store(v, std::memory_order_relaxed);
  }
  DeviceLimits d;
  d.sms = int(v >> 32);
  d.smem_optin = int(v & 0xffffffffu);
  return d;
}
inline size_t max_smem_optin() {
  int dev = 0;
  cudaGetDevice(&dev);
  return (size_t)device_limits(dev).smem_optin;
}

// Resident blocks of one kernel at one block size and shared-memory size, per
// device.  The occupancy query and the shared-memory attribute cost as much
// host time as the launch itself, 21 times per call; a kernel's answer for the
// size last asked about is kept (a race between threads only asks again) until
// the device is reset.  The attribute is set to the device's limit, the same
// from every thread.
struct LaunchCache {
  std::atomic<unsigned long long> slot[64];  // epoch << 40 | (smem + 1) << 16 | blocks per SM; 0: not asked yet

  template <typename K>
  cudaError_t resident(K kernel, size_t smem, int threads, int* per_sm, int* sms) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const DeviceLimits lim = device_limits(dev);
    *sms = lim.sms;
    const unsigned long long key = (unsigned long long)device_epoch(dev) << 40 | (unsigned long long)(smem + 1) << 16;
    if (dev < 64) {
      const unsigned long long v = slot[dev].load(std::memory_order_relaxed);
      if ((v >> 16 << 16) == key) {
        *per_sm = int(v & 0xffff);
        return cudaSuccess;
      }
    }
    if (smem > 48 * 1024) {
      if (smem > (size_t)lim.smem_optin) return cudaErrorInvalidValue;
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lim.smem_optin);
      if (e != cudaSuccess) return e;
    }
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    *per_sm = n > 0 ? n : 1;
    if (dev < 64) slot[dev].store(key | (unsigned)*per_sm, std::memory_order_relaxed);
    return cudaSuccess;
  }
};

// Persistent grid: as many blocks as are resident at once (capped by the
// work), each looping over tasks; per-block set-up (the staged tables, the
// gradient accumulator) is then paid once per resident block.
inline int persistent_blocks(int per_sm, int sms, int ntasks, int threads) {
  const int wpb = threads / 32;
  const int need = (ntasks + wpb - 1) / wpb;
  const int cap = per_sm * sms;
  return need < cap ? need : cap;
}

// Launch with the shared memory of an SM cut to what the resident blocks use, which
// leaves the rest to L1 for the pair, density and spill loads: the driver's own
// choice leaves them less.  40 atoms in 6-31G*, J/K (dp|ds) 0.63 -> 0.57 ms, (dd|ps) 0.35 ->
// 0.31, all 9.76 -> 9.41, gradient 26.8 -> 26.5; with all of it for the blocks J/K 10.38.
// An SM changes its split only when idle, and short launches run beside each
// other: those of fewer tasks per resident warp than kFullRounds keep the driver's
// choice (12 atoms, J/K: 0.465 ms with 8, 0.473 with 2, 0.493 with none; 40 atoms 9.41, 9.34,
// 9.34; with 32 9.74).  The warp-per-quartet kernels gain nothing.
constexpr int kFullRounds = 8;

template <typename A>
cudaError_t launch_split(void (*kernel)(A), int blocks, int threads, size_t smem, int per_sm, bool full, const A& args,
                         cudaStream_t st) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(blocks);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at = {};
  if (full) {
    const size_t need = per_sm * (smem + 1024), all = 228 * 1024;  // 1 KB reserved per block
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = need < all ? unsigned((need * 100 + all - 1) / all) : 100;
    c.attrs = &at;
    c.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&c, kernel, args);
}

#define IQCP_LAUNCH_T(KERNEL, THREADS, SMEM, ARGS, ST)                                           \
  do {                                                                                           \
    static LaunchCache cache_;                                                                   \
    int per_sm_ = 0, sms_ = 0;                                                                   \
    cudaError_t e_ = cache_.resident(KERNEL, SMEM, THREADS, &per_sm_, &sms_);                    \
    if (e_ != cudaSuccess) return e_;                                                            \
    e_ = launch_split(KERNEL, persistent_blocks(per_sm_, sms_, (ARGS).ntasks, THREADS), THREADS, SMEM, per_sm_, \
                      (ARGS).ntasks >= kFullRounds * per_sm_ * sms_ * (THREADS / 32), ARGS, ST);              \
    if (e_ != cudaSuccess) return e_;                                                            \
  } while (0)
#define IQCP_LAUNCH(KERNEL, SMEM, ARGS, ST) IQCP_LAUNCH_T(KERNEL, 128, SMEM, ARGS, ST)

// Team kernels walk a task's kets in one warp, one after the other: 32 quartets of
// (dp|dp) are 0.4 ms of one warp, and a launch ends on its longest work item.
// Tasks are therefore split into up to 32 slices of kets, each a work item of its
// own, until there are eight items per resident warp.  Against two, 40 atoms in
// 6-31G*: J/K (dp|dp) 0.55 -> 0.48 ms, (dd|pp) 0.32 -> 0.25; gradient (dp|dp) 2.29 ->
// 1.84, (dd|pp) 1.19 -> 0.88, (dp|pp) 3.35 -> 3.11, all 27.7 -> 27.2; 30 in cc-pVDZ,
// gradient (dp|dp) 2.14 -> 1.23.  Sixteen: 27.2, J/K 9.78 -> 9.85.
inline int team_ket_split(int per_sm, int sms, int ntasks, int threads) {
  const long long warps = (long long)per_sm * sms * (threads / 32);
  int s = 1;
  while (s < 32 && (long long)ntasks * s < 8 * warps) s *= 2;
  return s;
}

#define IQCP_LAUNCH_TEAM(KERNEL, THREADS, SMEM, ARGS, ST)                                                     \
  do {                                                                                                        \
    static LaunchCache cache_;                                                                                \
    int per_sm_ = 0, sms_ = 0;                                                                                \
    cudaError_t e_ = cache_.resident(KERNEL, SMEM, THREADS, &per_sm_, &sms_);                                 \
    if (e_ != cudaSuccess) return e_;                                                                         \
    (ARGS).ket_split = team_ket_split(per_sm_, sms_, (ARGS).ntasks, THREADS);                                 \
    KERNEL<<<persistent_blocks(per_sm_, sms_, (ARGS).ntasks * (ARGS).ket_split, THREADS), THREADS, SMEM, ST>>>( \
        ARGS);                                                                                                \
  } while (0)

// J/K variants (kernel_variant): 1 warp-cooperative (eri_team.cuh), 0 a group of
// lanes per quartet, as wide as the task says (build_tasks).
template <typename R, int LA, int LB, int LC, int LD>
cudaError_t launch_jk_variant(const JKArgs& a, cudaStream_t st) {
  using C = Cls<LA, LB, LC, LD>;
  constexpr bool F32 = sizeof(R) == 4;
  const size_t tb = sizeof(double) * rys_tab_doubles<C::NR>();
  constexpr int X = pair_class(LA, LB), Y = pair_class(LC, LD);
  if (kernel_variant(X, Y, a.mode, F32) == 1) {
    const size_t bytes = sizeof(double) * 4 * TeamJK<LA, LB, LC, LD>::PER_WARP + tb;
    JKArgs b = a;
    if (a.K) IQCP_LAUNCH_TEAM((jk_team_kernel<R, LA, LB, LC, LD, true>), 128, bytes, b, st);
    else IQCP_LAUNCH_TEAM((jk_team_kernel<R, LA, LB, LC, LD, false>), 128, bytes, b, st);
  } else if constexpr (C::NCOMP <= (F32 ? kMaxThreadComp32 : kMaxThreadComp)) {
    if (a.K) IQCP_LAUNCH((jk_kernel<R, LA, LB, LC, LD, true>), tb, a, st);
    else IQCP_LAUNCH((jk_kernel<R, LA, LB, LC, LD, false>), tb, a, st);
  }
  return cudaGetLastError();
}

template <int LA, int LB, int LC, int LD>
cudaError_t launch_jk_class(const JKArgs& a, cudaStream_t st) {
  if (a.mx.pass == 2) return launch_jk_variant<float, LA, LB, LC, LD>(a, st);
  return launch_jk_variant<double, LA, LB, LC, LD>(a, st);
}

// Gradient variants (kernel_variant): 1 warp-cooperative; 0 a group of lanes per
// quartet, by Hermite expansions for FP64 classes with an ss or ps ket, by Rys
// quadrature with the weights in shared memory for the other FP64 classes and
// in registers for the FP32 share.
template <int LA, int LB, int LC>
cudaError_t launch_grad_md(const GradArgs& args, cudaStream_t st) {
  using G = GradMD<LA, LB, LC>;
  GradArgs a = args;
  // the per-block gradient accumulator only when it fits beside the tables
  if (a.gsmem && sizeof(double) * (G::FIXED + 3 * a.natoms) > max_smem_optin()) a.gsmem = 0;
  const size_t bytes = sizeof(double) * (G::FIXED + (a.gsmem ? 3 * a.natoms : 0));
  IQCP_LAUNCH_T((grad_md_kernel<LA, LB, LC>), G::THREADS, bytes, a, st);
  return cudaGetLastError();
}

template <typename R, int LA, int LB, int LC, int LD>
cudaError_t launch_grad_variant(const GradArgs& args, cudaStream_t st) {
  using C = Cls<LA, LB, LC, LD>;
  constexpr bool F32 = sizeof(R) == 4;
  constexpr int X = pair_class(LA, LB), Y = pair_class(LC, LD);
  constexpr int NRG = grad_nroots(LA + LB + LC + LD);
  constexpr bool MD = !F32 && LC + LD <= 1;
  constexpr bool THREAD = !MD && C::NCOMP <= (F32 ? kMaxThreadComp32 : kMaxThreadComp);
  using TG = TeamGrad2<LA, LB, LC, LD>;
  const int variant = kernel_variant(X, Y, args.mode, F32);
  if constexpr (MD)
    if (variant == 0) return launch_grad_md<LA, LB, LC>(args, st);
  // the team variant reads the Rys coefficients through L1 (no staged table)
  size_t fixed = sizeof(double) * rys_tab_doubles<NRG>();
  if (variant == 1) fixed = sizeof(double) * TG::WPB * TG::PER_WARP;
  else if (!F32)
    fixed = sizeof(double) * (grad_stages_rys<LA, LB, LC, LD, true>() ? rys_tab_doubles<NRG>() : 0) +
            sizeof(R) * grad_wsh_doubles<LA, LB, LC, LD>();
  // the per-block gradient accumulator only when it fits beside the tables
  GradArgs a = args;
  if (a.gsmem && fixed + sizeof(double) * 3 * a.natoms > max_smem_optin()) a.gsmem = 0;
  const size_t gacc = a.gsmem ? sizeof(double) * 3 * a.natoms : 0;
  const size_t bytes = fixed + gacc;
  if (variant == 1) {
    IQCP_LAUNCH_TEAM((grad_team2_kernel<R, LA, LB, LC, LD>), 32 * TG::WPB, bytes, a, st);
  } else if constexpr (THREAD) {
    IQCP_LAUNCH((grad_kernel<R, LA, LB, LC, LD, !F32>), bytes, a, st);
  }
  return cudaGetLastError();
}

template <int LA, int LB, int LC, int LD>
cudaError_t launch_grad_class(const GradArgs& a, cudaStream_t st) {
  if (a.mx.pass == 2) return launch_grad_variant<float, LA, LB, LC, LD>(a, st);
  return launch_grad_variant<double, LA, LB, LC, LD>(a, st);
}

#define IQCP_KET_DISPATCH(X, Y, MACRO)                \
  switch (Y) {                                        \
    case 0: MACRO(0, 0); break;                       \
    case 1: if (X >= 1) { MACRO(1, 0); } break;       \
    case 2: if (X >= 2) { MACRO(1, 1); } break;       \
    case 3: if (X >= 3) { MACRO(2, 0); } break;       \
    case 4: if (X >= 4) { MACRO(2, 1); } break;       \
    case 5: if (X >= 5) { MACRO(2, 2); } break;       \
    default: return cudaErrorInvalidValue;            \
  }

template <int LA, int LB>
cudaError_t launch_jk_bra(int Y, const JKArgs& a, cudaStream_t st) {
  constexpr int X = pair_class(LA, LB);
#define LJK(lc, ld) \
  if constexpr (pair_class(lc, ld) <= X) { return launch_jk_class<LA, LB, lc, ld>(a, st); }
  IQCP_KET_DISPATCH(X, Y, LJK)
#undef LJK
  return cudaErrorInvalidValue;
}

template <int LA, int LB>
cudaError_t launch_store_bra(int Y, const StoreArgs& a, cudaStream_t st) {
  constexpr int X = pair_class(LA, LB);
  const int blocks = (a.ntasks + 3) / 4;
#define LST(lc, ld) \
  if constexpr (pair_class(lc, ld) <= X) { store_kernel<LA, LB, lc, ld><<<blocks, 128, 0, st>>>(a); }
  IQCP_KET_DISPATCH(X, Y, LST)
#undef LST
  return cudaGetLastError();
}

template <int LA, int LB>
cudaError_t launch_grad_bra(int Y, const GradArgs& a, cudaStream_t st) {
  constexpr int X = pair_class(LA, LB);
#define LGR(lc, ld) \
  if constexpr (pair_class(lc, ld) <= X) { return launch_grad_class<LA, LB, lc, ld>(a, st); }
  IQCP_KET_DISPATCH(X, Y, LGR)
#undef LGR
  return cudaErrorInvalidValue;
}

}  // namespace iqcp
