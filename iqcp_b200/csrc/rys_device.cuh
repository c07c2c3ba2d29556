// Device Boys function and Rys quadrature.
//
// Rys rule (roots as t^2 in [0,1), weights) for n roots at argument T: the
// same quantities rys_roots returns in the reference (rys/mod.rs:253), which
// computes them per call from moments with Schmidt orthogonalisation and a
// companion-matrix QR (rys/mod.rs:468-790).  On the device a per-call
// eigen-solve diverges across lanes, so the rule is read from tables instead:
// polynomials on intervals of T up to Tasym(n) (degree 9 on half-unit intervals
// for n <= 2, 11 on unit intervals above), and the large-T Hermite limit
// (roots y_i/T, weights W_i/sqrt(T)) beyond it.  The
// tables (rys_tables.inc, made by gen_rys_tables.cpp in binary128) are exact
// to ~3e-16 relative, i.e. closer to the true rule than the reference's own
// FP64 moment method.
//
// Boys F_0..F_m(T): the reference's regime split (boys/mod.rs:587-618: series
// at the highest order plus downward recurrence below the m_max turnover,
// erf + upward recurrence above it), with CUDA's erf/exp.
#pragma once
#include <cuda_runtime.h>

#define RYS_TAB_QUAL __device__ const
#define RYS_TAB_ALIGN __align__(16)
#include "rys_tables.inc"
#undef RYS_TAB_QUAL
#undef RYS_TAB_ALIGN

namespace iqcp {

// Tasym(n), polynomial coefficients per function, intervals per unit of T
__host__ __device__ constexpr int rys_tasym(int n) {
  constexpr int t[RYS_TAB_MAXN + 1] = RYS_TAB_TASYM;
  return t[n];
}
__host__ __device__ constexpr int rys_ncoef(int n) {
  constexpr int t[RYS_TAB_MAXN + 1] = RYS_TAB_NCOEF;
  return t[n];
}
__host__ __device__ constexpr int rys_per_unit(int n) {
  constexpr int t[RYS_TAB_MAXN + 1] = RYS_TAB_PER_UNIT;
  return t[n];
}
// Shared-memory copy of the order-N table: [interval][root 0..N-1, weight
// 0..N-1][coefficient].  Coefficients are read in 16-byte pairs; the interval
// stride is padded to an odd number of pairs so that lanes reading different
// intervals fall on different banks.
template <int N>
__host__ __device__ constexpr int rys_tab_width() { return 2 * N * rys_ncoef(N); }
template <int N>
__host__ __device__ constexpr int rys_tab_stride() { return rys_tab_width<N>() + 2; }
template <int N>
__host__ __device__ constexpr int rys_nint() { return rys_tasym(N) * rys_per_unit(N); }
template <int N>
__host__ __device__ constexpr int rys_tab_doubles() { return rys_nint<N>() * rys_tab_stride<N>(); }

// Asynchronous copy of 16 bytes from global to shared memory.  A block's table of
// 12 to 61 KB is 6 to 30 such copies per thread: issued back to back they cost one
// trip to L2, as loads followed by stores one trip each, 5 to 10 us at the start of
// a kernel that has little else to do in a small molecule.
__device__ __forceinline__ void copy16_async(void* s, const void* g) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(s);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(g) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Copy the order-N table into shared memory (all threads of the block; a barrier
// has to follow).  Each lane reads the interval of its own T, so table reads are
// scattered: from shared memory they cost a few bank wavefronts, from L1 one
// cache line per lane.
template <int N>
__device__ __forceinline__ void rys_stage_table(double* __restrict__ s) {
  constexpr int W = rys_tab_width<N>() / 2;
  const double2* g = reinterpret_cast<const double2*>(kRysPoly + kRysOffset[N]);
  double2* d = reinterpret_cast<double2*>(s);
  for (int i = threadIdx.x; i < rys_nint<N>() * W; i += blockDim.x) {
    const int k = i / W;
    copy16_async(d + k * (rys_tab_stride<N>() / 2) + (i - k * W), g + i);
  }
  copy_async_wait();
}

// Polynomial of NC coefficients (16-byte aligned) at x in [-1, 1]; LDG: through
// the read-only path instead of shared memory.
template <int NC, bool LDG>
__device__ __forceinline__ double rys_poly(const double* __restrict__ c, double x) {
  const double2* p = reinterpret_cast<const double2*>(c);
  double v = 0.0;
#pragma unroll
  for (int j = NC / 2 - 1; j >= 0; --j) {
    const double2 u = LDG ? __ldg(p + j) : p[j];
    v = j == NC / 2 - 1 ? u.y : fma(v, x, u.y);
    v = fma(v, x, u.x);
  }
  return v;
}

// Interval of T < Tasym(N) and the position x in [-1, 1] inside it.
template <int N>
__device__ __forceinline__ int rys_interval(double T, double* x) {
  const double t = T * rys_per_unit(N);
  const int k = int(t);
  *x = 2.0 * (t - double(k)) - 1.0;
  return k;
}

// c / T for T > 0 from it, 1/T to a few roundings: one Newton step on q T = c, whose
// remainder one FMA forms exactly, leaves the rounding of the quotient (2^-53).
// The bare product with 1/T = rsqrt(T)^2 left the roots of the large-T limit off by
// up to 4.4e-16 instead of 2.9e-16; a division of each root costs the J/K builds 2 to
// 4 % (40 atoms in 6-31G* 9.47 -> 9.75 ms), the step 0.2 to 2.4 % (9.45 -> 9.47; 32 atoms
// in 6-31G, s and p shells only, 2.40 -> 2.46).
__device__ __forceinline__ double quotient(double c, double T, double it) {
  const double q = c * it;
  return fma(it, fma(-q, T, c), q);
}
// Arguments of the limit (positive) are cut at 2^996, where its roots no longer
// matter: an infinite one would make the remainder 0 times infinity.  One integer
// minimum on the high word; fmin is six instructions.
__device__ __forceinline__ double rys_cut(double T) {
  return __hiloint2double(min(__double2hiint(T), 0x7e300000), __double2loint(T));
}

// The n-point rule at T.  s: the order-N table staged in shared memory, or
// null to read it through L1.
template <int N, bool LDG = false>
__device__ __forceinline__ void rys_rule_tab(double T, const double* s, double* __restrict__ r,
                                             double* __restrict__ w) {
  static_assert(N >= 1 && N <= RYS_TAB_MAXN, "unsupported Rys order");
  if (T >= double(rys_tasym(N))) {
    const double Tc = rys_cut(T), is = rsqrt(Tc), it = is * is;
    const int base = (N * (N - 1)) / 2;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      r[i] = quotient(__ldg(kRysAsymRoot + base + i), Tc, it);
      w[i] = __ldg(kRysAsymWeight + base + i) * is;
    }
    return;
  }
  constexpr int NC = rys_ncoef(N);
  double x;
  const int k = rys_interval<N>(T, &x);
  const double* c = LDG ? kRysPoly + kRysOffset[N] + k * rys_tab_width<N>() : s + k * rys_tab_stride<N>();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    r[i] = rys_poly<NC, LDG>(c + i * NC, x);
    w[i] = rys_poly<NC, LDG>(c + (N + i) * NC, x);
  }
}

template <int N>
__device__ __forceinline__ void rys_rule(double T, double* __restrict__ r, double* __restrict__ w) {
  rys_rule_tab<N, true>(T, nullptr, r, w);
}

// Root and weight r of the N-point rule alone (kernels whose lanes each take one root)
template <int N, bool LDG = false>
__device__ __forceinline__ void rys_rule_one(double T, int r, const double* s, double* t2, double* w) {
  if (T >= double(rys_tasym(N))) {
    const double Tc = rys_cut(T), is = rsqrt(Tc);
    const int base = (N * (N - 1)) / 2;
    *t2 = quotient(__ldg(kRysAsymRoot + base + r), Tc, is * is);
    *w = __ldg(kRysAsymWeight + base + r) * is;
    return;
  }
  constexpr int NC = rys_ncoef(N);
  double x;
  const int k = rys_interval<N>(T, &x);
  const double* c = LDG ? kRysPoly + kRysOffset[N] + k * rys_tab_width<N>() : s + k * rys_tab_stride<N>();
  *t2 = rys_poly<NC, LDG>(c + r * NC, x);
  *w = rys_poly<NC, LDG>(c + (N + r) * NC, x);
}

// Runtime-order dispatch (tests / batch entry point)
__device__ inline void rys_rule_n(int n, double T, double* r, double* w) {
  switch (n) {
    case 1: rys_rule<1>(T, r, w); break;
    case 2: rys_rule<2>(T, r, w); break;
    case 3: rys_rule<3>(T, r, w); break;
    case 4: rys_rule<4>(T, r, w); break;
    case 5: rys_rule<5>(T, r, w); break;
    case 6: rys_rule<6>(T, r, w); break;
    case 7: rys_rule<7>(T, r, w); break;
    default: break;
  }
}

__device__ __forceinline__ double boys_turnover(int m) {
  // boys/mod.rs:67-108 (m-dependent series/recurrence switch)
  const double tab[16] = {0.0, 0.0, 0.866025403784, 1.295010032056, 1.705493613097,
                          2.106432965305, 2.501471934009, 2.892473348218, 3.280525047072,
                          3.666320693281, 4.05033123037, 4.432891808508, 4.814249856864,
                          5.194593501454, 5.574069276051, 5.952793645111};
  return m < 16 ? tab[m] : 5.952793645111 + 0.372 * double(m - 15);
}

// F_0..F_m(T) into f[0..m] (m <= 31)
__device__ inline void boys_all_dev(int m, double T, double* f) {
  if (T < 1e-14) {
    for (int i = 0; i <= m; ++i) f[i] = 1.0 / (2.0 * i + 1.0);
    return;
  }
  if (T < boys_turnover(m)) {
    const double b = m + 0.5;
    const double e = 0.5 * exp(-T);
    double term = e, sum = e, den = b + 1.0;
    const double tol = 1.1102230246251565e-16 * e;
    for (int it = 0; it < 200 && term > tol; ++it) {
      term *= T / den;
      sum += term;
      den += 1.0;
    }
    f[m] = sum / b;
    double bc = b;
    for (int i = m; i >= 1; --i) {
      bc -= 1.0;
      f[i - 1] = (e + T * f[i]) / bc;
    }
  } else {
    const double st = sqrt(T);
    f[0] = 0.88622692545275801365 / st * erf(st);
    const double e = exp(-T);
    const double h = 0.5 / T;
    for (int i = 1; i <= m; ++i) f[i] = h * ((2 * i - 1) * f[i - 1] - e);
  }
}

}  // namespace iqcp
