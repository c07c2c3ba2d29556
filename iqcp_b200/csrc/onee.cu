// One-electron integrals on the device: overlap S, kinetic T and nuclear
// attraction V over the same normalised Cartesian primitives as the ERIs.
// They stand in for overlap_matrix (integrals/overlap.rs:647), the kinetic
// and nuclear builders behind hcore_matrix (integrals/hcore.rs:103,
// nuclear.rs:68-305): H = T + V.  one_electron_grad_kernel contracts their
// nuclear derivatives with D and W.
//
// One warp per shell pair, all molecules of the context and all angular
// classes in one launch.  The warp stages up to 32 primitive pairs in shared
// memory (one per lane), then its lanes share the (primitive pair, atom) items
// of the nuclear attraction; S and T take one primitive pair per lane.  The
// 1D integrals follow one two-centre recurrence (pair_table): with (PA, PB, 1/2p)
// they are the Gaussian moments of S and T, and a point charge is the q ->
// infinity limit of a Rys ket, (PA - t^2 PC, PB - t^2 PC, (1 - t^2) / 2p), with at
// most three roots.  The second index is not taken by horizontal transfer: for
// a tight shell on B that forms moments of order 1/p as differences of AB^2,
// which the kinetic energy then multiplies by 4 b^2.  Tables and
// sums stay in registers.  What bounds it is latency at small sizes and the FP64
// pipe at large ones; both were far off with a thread per shell pair, Hermite
// arrays in local memory and primitives and atoms in series: the RHF gradient of
// a 30-atom cc-pVDZ molecule 77.6 -> 45.9 ms (this part 29 ms -> under 1 ms), a
// batched SCF of six small molecules 120 -> 79 ms.
#include <cuda_runtime.h>

#include "eri_templates.cuh"
#include "smem_limit.cuh"

namespace iqcp {

namespace {

constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ double rad_norm_dev(double a, int l) {
  const double tap = 2.0 * a / kPi;
  double v = sqrt(sqrt(tap * tap * tap));
  const double fa = 4.0 * a;
  if (l == 1) v *= sqrt(fa);
  else if (l == 2) v *= fa;
  return v;
}

// One primitive pair; ea is the exponent on A
struct Prim1 {
  double p, inv_p, P[3], c, ea, eb;
};

// Shell pair seen from one side: A is the shell that is differentiated
struct Side {
  double A[3], B[3];
  int sa, sb, oa, ob, atom_a, mol;
};

__device__ __forceinline__ Side side_of(const ShellPair& s, bool swap) {
  Side r;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    r.A[d] = swap ? s.B[d] : s.A[d];
    r.B[d] = swap ? s.A[d] : s.B[d];
  }
  r.sa = swap ? s.sb : s.sa;
  r.sb = swap ? s.sa : s.sb;
  r.oa = swap ? s.ob : s.oa;
  r.ob = swap ? s.oa : s.ob;
  r.atom_a = swap ? s.atom_b : s.atom_a;
  r.mol = s.mol;
  return r;
}

// Primitive pair `k` (ip = k / npb, jp = k % npb) of a shell pair
__device__ __forceinline__ Prim1 prim_pair(const OneEArgs& a, const Side& s, int la, int lb, int npb, int k) {
  const int ip = k / npb, jp = k - ip * npb;
  const int pa = a.pstart[s.sa] + ip, pb = a.pstart[s.sb] + jp;
  Prim1 q;
  q.ea = a.exps[pa];
  q.eb = a.exps[pb];
  q.p = q.ea + q.eb;
  q.inv_p = 1.0 / q.p;
  double r2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    q.P[d] = (q.ea * s.A[d] + q.eb * s.B[d]) * q.inv_p;
    r2 += (s.A[d] - s.B[d]) * (s.A[d] - s.B[d]);
  }
  q.c = a.coefs[pa] * rad_norm_dev(q.ea, la) * a.coefs[pb] * rad_norm_dev(q.eb, lb) *
        exp(-q.ea * q.eb * q.inv_p * r2);
  return q;
}

// The warp's staged primitive pairs, one array per field
constexpr int kStage = 32;
struct Stage {
  double f[7][kStage];  // p, 1/p, P, c, ea
};

__device__ __forceinline__ void stage_store(Stage& st, int lane, const Prim1& q) {
  st.f[0][lane] = q.p;
  st.f[1][lane] = q.inv_p;
  st.f[2][lane] = q.P[0];
  st.f[3][lane] = q.P[1];
  st.f[4][lane] = q.P[2];
  st.f[5][lane] = q.c;
  st.f[6][lane] = q.ea;
}

// 1D integrals I(i, j), i <= IA, j <= IB, at I[i (IB+1) + j]:
// I(i, j+1) = cb I(i, j) + b [i I(i-1, j) + j I(i, j-1)], likewise i + 1 with ca
template <int IA, int IB>
__device__ __forceinline__ void pair_table(double ca, double cb, double b, double g00, double* I) {
  constexpr int W = IB + 1;
  I[0] = g00;
#pragma unroll
  for (int j = 0; j < IB; ++j) {
    double v = cb * I[j];
    if (j > 0) v = fma(double(j) * b, I[j > 0 ? j - 1 : 0], v);
    I[j + 1] = v;
  }
#pragma unroll
  for (int i = 0; i < IA; ++i)
#pragma unroll
    for (int j = 0; j <= IB; ++j) {
      double v = ca * I[i * W + j];
      if (i > 0) v = fma(double(i) * b, I[(i > 0 ? i - 1 : 0) * W + j], v);
      if (j > 0) v = fma(double(j) * b, I[i * W + (j > 0 ? j - 1 : 0)], v);
      I[(i + 1) * W + j] = v;
    }
}

// kinetic 1D integral from overlaps I(i, j) with row length LBX: -1/2 d^2/dx^2 on j
template <int LBX>
__device__ __forceinline__ double kinetic_1d(const double* I, int i, int j, double eb) {
  double k = -2.0 * eb * double(2 * j + 1) * I[i * LBX + j] + 4.0 * eb * eb * I[i * LBX + j + 2];
  if (j >= 2) k += double(j * (j - 1)) * I[i * LBX + (j >= 2 ? j - 2 : 0)];
  return -0.5 * k;
}

// ---------------------------------------------------------------------------
template <int LA, int LB>
__device__ __forceinline__ void pair_integrals(const OneEArgs& a, const ShellPair& sp, Stage& st, int lane) {
  constexpr int NA = ncart(LA), NB = ncart(LB), NC = NA * NB, NR = (LA + LB) / 2 + 1;
  const Side s = side_of(sp, false);
  const int npb = a.nprim[s.sb], np = a.nprim[s.sa] * npb, n = a.mol_n[s.mol];
  const long long mb = a.mol_base[s.mol];
  auto put = [&](double* M, const double* v) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double x = warp_sum(v[c]) * ang_factor(LA, c / NB) * ang_factor(LB, c % NB);
      if (lane == (c & 31)) {
        const long long i = s.oa + c / NB, j = s.ob + c % NB;
        M[mb + i * n + j] = x;
        if (s.sa != s.sb) M[mb + j * n + i] = x;
      }
    }
  };
  if (a.V) {
    const int a0 = a.mol_atom0[s.mol], na = a.mol_atom0[s.mol + 1] - a0;
    double v[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = 0.0;
    for (int k0 = 0; k0 < np; k0 += kStage) {
      const int nk = np - k0 < kStage ? np - k0 : kStage;
      __syncwarp();
      if (lane < nk) stage_store(st, lane, prim_pair(a, s, LA, LB, npb, k0 + lane));
      __syncwarp();
      for (int it = lane; it < nk * na; it += 32) {
        const int k = it / na, c = a0 + it - k * na;
        const double p = st.f[0][k], inv_p = st.f[1][k];
        double PA[3], PB[3], PC[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          PA[d] = st.f[2 + d][k] - s.A[d];
          PB[d] = st.f[2 + d][k] - s.B[d];
          PC[d] = st.f[2 + d][k] - a.atom_xyz[3 * c + d];
        }
        double rt[NR], wt[NR];
        rys_rule<NR>(p * (PC[0] * PC[0] + PC[1] * PC[1] + PC[2] * PC[2]), rt, wt);
        const double pre = -double(a.z[c]) * 2.0 * kPi * inv_p * st.f[5][k];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const double b10 = (0.5 - 0.5 * rt[r]) * inv_p;
          double I[3][(LA + 1) * (LB + 1)];
#pragma unroll
          for (int d = 0; d < 3; ++d)
            pair_table<LA, LB>(PA[d] - rt[r] * PC[d], PB[d] - rt[r] * PC[d], b10, d == 2 ? wt[r] * pre : 1.0, I[d]);
#pragma unroll
          for (int q = 0; q < NC; ++q) {
            const int i = q / NB, j = q % NB;
            v[q] = fma(I[0][cart_pow(LA, i, 0) * (LB + 1) + cart_pow(LB, j, 0)] *
                           I[1][cart_pow(LA, i, 1) * (LB + 1) + cart_pow(LB, j, 1)],
                       I[2][cart_pow(LA, i, 2) * (LB + 1) + cart_pow(LB, j, 2)], v[q]);
          }
        }
      }
    }
    put(a.V, v);
  }
  if (a.S || a.T) {
    double sv[NC], tv[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) sv[c] = tv[c] = 0.0;
    for (int k = lane; k < np; k += 32) {
      const Prim1 q = prim_pair(a, s, LA, LB, npb, k);
      const double sp1 = sqrt(kPi * q.inv_p), cc = q.c * sp1 * sp1 * sp1;
      double I[3][(LA + 1) * (LB + 3)];
#pragma unroll
      for (int d = 0; d < 3; ++d)
        pair_table<LA, LB + 2>(q.P[d] - s.A[d], q.P[d] - s.B[d], 0.5 * q.inv_p, 1.0, I[d]);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        double s1[3], t1[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int i = cart_pow(LA, c / NB, d), j = cart_pow(LB, c % NB, d);
          s1[d] = I[d][i * (LB + 3) + j];
          t1[d] = kinetic_1d<LB + 3>(I[d], i, j, q.eb);
        }
        sv[c] = fma(cc * s1[0], s1[1] * s1[2], sv[c]);
        tv[c] = fma(cc, t1[0] * s1[1] * s1[2] + s1[0] * t1[1] * s1[2] + s1[0] * s1[1] * t1[2], tv[c]);
      }
    }
    if (a.S) put(a.S, sv);
    if (a.T) put(a.T, tv);
  }
}

constexpr int kWarps = 4;

// Class of position i of the class-sorted pair list
__device__ __forceinline__ int class_of(const OneEArgs& a, int i) {
  int c = 0;
  while (i >= a.first[c + 1]) ++c;
  return c;
}

}  // namespace

__global__ void __launch_bounds__(32 * kWarps) one_electron_kernel(OneEArgs a) {
  __shared__ Stage stage[kWarps];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = blockIdx.x * kWarps + wib; i < a.first[kNumPairClasses]; i += gridDim.x * kWarps) {
    const ShellPair sp = a.pairs[a.list[i]];
    switch (class_of(a, i)) {
      case 0: pair_integrals<0, 0>(a, sp, stage[wib], lane); break;
      case 1: pair_integrals<1, 0>(a, sp, stage[wib], lane); break;
      case 2: pair_integrals<1, 1>(a, sp, stage[wib], lane); break;
      case 3: pair_integrals<2, 0>(a, sp, stage[wib], lane); break;
      case 4: pair_integrals<2, 1>(a, sp, stage[wib], lane); break;
      default: pair_integrals<2, 2>(a, sp, stage[wib], lane); break;
    }
  }
}

// ---------------------------------------------------------------------------
// Nuclear gradient of the one-electron energy plus the nuclear repulsion
// gradient (the non-ERI terms of rhf_gradient, scf/gradient.rs:900-990, from
// overlap_derivative_matrix / hcore_derivative_matrix, gradient.rs:188,355):
//   g_A += 2 sum_{mu on A, nu} [D_mn d(T+V)_mn/dA - W_mn dS_mn/dA]   (bra derivative;
//          the ket term is equal by symmetry of D and W)
//   g_C += sum_mn D_mn dV^C_mn/dC = -sum_mn (D_mn + D_nm) dV^C_mn/dA   (operator
//          term: V^C depends on differences of A, B and C only)
//   g_A -= sum_{B != A} Z_A Z_B (A - B) / |A - B|^3
// The derivative of a Cartesian Gaussian w.r.t. its centre raises and lowers
// the power: d/dA_x x^i e^{-a x^2} = 2a x^{i+1} e^{..} - i x^{i-1} e^{..}.
// One warp per ordered shell pair; in the nuclear part a group of lanes keeps
// one atom, so that the operator term is one shared-memory atomic per lane and
// pair.  Per-block gradient in shared memory.
namespace {

// weights of the warp's block in shared memory: 2 D_ab, D_ab + D_ba, 2 W_ab with angular factors
struct GradWeights {
  double d2[36], ds[36], w2[36];
};

template <int LA, int LB>
__device__ __forceinline__ void pair_gradient(const OneEArgs& a, const Side& s, Stage& st, GradWeights& w, int lane,
                                              double* gout) {
  constexpr int NA = ncart(LA), NB = ncart(LB), NC = NA * NB, NR = (LA + LB + 1) / 2 + 1;
  const int npb = a.nprim[s.sb], np = a.nprim[s.sa] * npb, n = a.mol_n[s.mol];
  const long long mb = a.mol_base[s.mol];
  const int a0 = a.mol_atom0[s.mol], na = a.mol_atom0[s.mol + 1] - a0;
  __syncwarp();
  for (int c = lane; c < NC; c += 32) {
    const long long i = s.oa + c / NB, j = s.ob + c % NB;
    const double g = ang_factor(LA, c / NB) * ang_factor(LB, c % NB);
    const double dij = a.D[mb + i * n + j], dji = a.D[mb + j * n + i];
    w.d2[c] = 2.0 * g * dij;
    w.ds[c] = g * (dij + dji);
    w.w2[c] = 2.0 * g * a.W[mb + i * n + j];
  }
  double gA[3] = {0, 0, 0};
  // lanes per atom
  int lpa = 1;
  while (2 * lpa * na <= 32) lpa *= 2;
  for (int k0 = 0; k0 < np; k0 += kStage) {
    const int nk = np - k0 < kStage ? np - k0 : kStage;
    __syncwarp();
    if (lane < nk) {
      const Prim1 q = prim_pair(a, s, LA, LB, npb, k0 + lane);
      stage_store(st, lane, q);
      // S and T: this lane's primitive pair
      const double sp1 = sqrt(kPi * q.inv_p), cc = q.c * sp1 * sp1 * sp1;
      double I[3][(LA + 2) * (LB + 3)];
#pragma unroll
      for (int d = 0; d < 3; ++d)
        pair_table<LA + 1, LB + 2>(q.P[d] - s.A[d], q.P[d] - s.B[d], 0.5 * q.inv_p, 1.0, I[d]);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double dmn = cc * w.d2[c], wmn = cc * w.w2[c];
        double s1[3], t1[3], ds[3], dt[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int i = cart_pow(LA, c / NB, d), j = cart_pow(LB, c % NB, d);
          s1[d] = I[d][i * (LB + 3) + j];
          t1[d] = kinetic_1d<LB + 3>(I[d], i, j, q.eb);
          ds[d] = 2.0 * q.ea * I[d][(i + 1) * (LB + 3) + j];
          dt[d] = 2.0 * q.ea * kinetic_1d<LB + 3>(I[d], i + 1, j, q.eb);
          if (i > 0) {
            ds[d] -= double(i) * I[d][(i > 0 ? i - 1 : 0) * (LB + 3) + j];
            dt[d] -= double(i) * kinetic_1d<LB + 3>(I[d], i > 0 ? i - 1 : 0, j, q.eb);
          }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int e1 = (d + 1) % 3, e2 = (d + 2) % 3;
          const double dS = ds[d] * s1[e1] * s1[e2];
          const double dT = dt[d] * s1[e1] * s1[e2] + ds[d] * (t1[e1] * s1[e2] + s1[e1] * t1[e2]);
          gA[d] += dmn * dT - wmn * dS;
        }
      }
    }
    __syncwarp();
    for (int c = lane / lpa; c < na; c += 32 / lpa) {
      const double C[3] = {a.atom_xyz[3 * (a0 + c)], a.atom_xyz[3 * (a0 + c) + 1], a.atom_xyz[3 * (a0 + c) + 2]};
      const double zc = -double(a.z[a0 + c]) * 2.0 * kPi;
      double gC[3] = {0, 0, 0};
      for (int k = lane % lpa; k < nk; k += lpa) {
        const double p = st.f[0][k], inv_p = st.f[1][k], e2 = 2.0 * st.f[6][k];
        double PA[3], PB[3], PC[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          PA[d] = st.f[2 + d][k] - s.A[d];
          PB[d] = st.f[2 + d][k] - s.B[d];
          PC[d] = st.f[2 + d][k] - C[d];
        }
        double rt[NR], wt[NR];
        rys_rule<NR>(p * (PC[0] * PC[0] + PC[1] * PC[1] + PC[2] * PC[2]), rt, wt);
        const double pre = zc * inv_p * st.f[5][k];
#pragma unroll 1
        for (int r = 0; r < NR; ++r) {
          // the rule's entries by selection: an indexed access would put them in local memory
          const double t2 = r == 0 ? rt[0] : (r == 1 ? rt[NR > 1 ? 1 : 0] : rt[NR - 1]);
          const double wr = r == 0 ? wt[0] : (r == 1 ? wt[NR > 1 ? 1 : 0] : wt[NR - 1]);
          const double b10 = (0.5 - 0.5 * t2) * inv_p;
          double I[3][(LA + 2) * (LB + 1)];
#pragma unroll
          for (int d = 0; d < 3; ++d)
            pair_table<LA + 1, LB>(PA[d] - t2 * PC[d], PB[d] - t2 * PC[d], b10, d == 2 ? wr * pre : 1.0, I[d]);
#pragma unroll
          for (int q = 0; q < NC; ++q) {
            double v[3], dv[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const int i = cart_pow(LA, q / NB, d), j = cart_pow(LB, q % NB, d);
              v[d] = I[d][i * (LB + 1) + j];
              dv[d] = e2 * I[d][(i + 1) * (LB + 1) + j];
              if (i > 0) dv[d] -= double(i) * I[d][(i > 0 ? i - 1 : 0) * (LB + 1) + j];
            }
            const double x = dv[0] * (v[1] * v[2]), y = dv[1] * (v[0] * v[2]), z = dv[2] * (v[0] * v[1]);
            const double d2 = w.d2[q], ds = w.ds[q];
            gA[0] = fma(d2, x, gA[0]);
            gA[1] = fma(d2, y, gA[1]);
            gA[2] = fma(d2, z, gA[2]);
            gC[0] = fma(ds, x, gC[0]);
            gC[1] = fma(ds, y, gC[1]);
            gC[2] = fma(ds, z, gC[2]);
          }
        }
      }
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (gC[d] != 0.0) atomicAdd(gout + 3 * (a0 + c - a.atom0) + d, -gC[d]);
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double g = warp_sum(gA[d]);
    if (lane == 0) atomicAdd(gout + 3 * (s.atom_a - a.atom0) + d, g);
  }
}

// Nuclear repulsion gradient of atom i (its molecule's atoms a0 .. a1)
__device__ __forceinline__ void repulsion_gradient(const OneEArgs& a, int i, int a0, int a1, double* gout) {
  double g[3] = {0, 0, 0};
  for (int j = a0; j < a1; ++j) {
    if (j == i) continue;
    double r[3], r2 = 0.0;
    for (int d = 0; d < 3; ++d) {
      r[d] = a.atom_xyz[3 * i + d] - a.atom_xyz[3 * j + d];
      r2 += r[d] * r[d];
    }
    const double rr = sqrt(r2);
    const double f = double(a.z[i]) * double(a.z[j]) / (rr * rr * rr);
    for (int d = 0; d < 3; ++d) g[d] -= f * r[d];
  }
  for (int d = 0; d < 3; ++d) atomicAdd(gout + 3 * (i - a.atom0) + d, g[d]);
}

}  // namespace

__global__ void __launch_bounds__(32 * kWarps) one_electron_grad_kernel(OneEArgs a) {
  __shared__ Stage stage[kWarps];
  __shared__ GradWeights weights[kWarps];
  extern __shared__ double gacc[];
  const int nacc = a.gsmem ? 3 * (a.atom1 - a.atom0) : 0;
  for (int i = threadIdx.x; i < nacc; i += blockDim.x) gacc[i] = 0.0;
  __syncthreads();
  double* gout = a.gsmem ? gacc : a.grad + 3 * a.atom0;  // row 0: atom a.atom0
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // nuclear repulsion: one thread per atom over the grid
  for (int i = a.atom0 + blockIdx.x * blockDim.x + threadIdx.x; i < a.atom1; i += gridDim.x * blockDim.x) {
    int lo = 0, hi = a.n_mol - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (a.mol_atom0[mid] <= i) lo = mid; else hi = mid - 1;
    }
    repulsion_gradient(a, i, a.mol_atom0[lo], a.mol_atom0[lo + 1], gout);
  }
  const int npairs = a.first[kNumPairClasses];
  for (int u = blockIdx.x * kWarps + wib; u < 2 * npairs; u += gridDim.x * kWarps) {
    const int i = u >> 1;
    const bool swap = u & 1;
    const ShellPair sp = a.pairs[a.list[i]];
    if (swap && sp.sa == sp.sb) continue;
    const Side s = side_of(sp, swap);
    Stage& st = stage[wib];
    GradWeights& w = weights[wib];
    switch (2 * class_of(a, i) + (swap ? 1 : 0)) {
      case 0: case 1: pair_gradient<0, 0>(a, s, st, w, lane, gout); break;
      case 2: pair_gradient<1, 0>(a, s, st, w, lane, gout); break;
      case 3: pair_gradient<0, 1>(a, s, st, w, lane, gout); break;
      case 4: case 5: pair_gradient<1, 1>(a, s, st, w, lane, gout); break;
      case 6: pair_gradient<2, 0>(a, s, st, w, lane, gout); break;
      case 7: pair_gradient<0, 2>(a, s, st, w, lane, gout); break;
      case 8: pair_gradient<2, 1>(a, s, st, w, lane, gout); break;
      case 9: pair_gradient<1, 2>(a, s, st, w, lane, gout); break;
      default: pair_gradient<2, 2>(a, s, st, w, lane, gout); break;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nacc; i += blockDim.x)
    if (gacc[i] != 0.0) atomicAdd(a.grad + 3 * a.atom0 + i, gacc[i]);
}

// One resident wave of blocks, fewer for small molecules
static cudaError_t one_e_blocks(const void* kernel, size_t smem, int units, int* blocks) {
  int per_sm = 0, dev = 0, sms = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * kWarps, smem);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int need = (units + kWarps - 1) / kWarps, cap = (per_sm > 0 ? per_sm : 1) * sms;
  *blocks = need < cap ? (need > 0 ? need : 1) : cap;
  return cudaSuccess;
}

cudaError_t launch_one_electron_grad(const OneEArgs& a, cudaStream_t st) {
  const size_t smem = a.gsmem ? sizeof(double) * 3 * (a.atom1 - a.atom0) : 0;
  cudaError_t e = allow_dynamic_smem(one_electron_grad_kernel, smem);
  if (e != cudaSuccess) return e;
  int blocks = 0;
  e = one_e_blocks((const void*)one_electron_grad_kernel, smem, 2 * a.first[kNumPairClasses], &blocks);
  if (e != cudaSuccess) return e;
  one_electron_grad_kernel<<<blocks, 32 * kWarps, smem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_one_electron(const OneEArgs& a, cudaStream_t st) {
  int blocks = 0;
  const cudaError_t e = one_e_blocks((const void*)one_electron_kernel, 0, a.first[kNumPairClasses], &blocks);
  if (e != cudaSuccess) return e;
  one_electron_kernel<<<blocks, 32 * kWarps, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace iqcp
