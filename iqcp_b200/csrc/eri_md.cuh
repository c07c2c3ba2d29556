// Two-electron gradient by Hermite expansions (McMurchie-Davidson) for ss and
// ps kets: the same quantity as grad_kernel (eri_templates.cuh), with fewer
// operations per primitive quartet.
//
// With the D x D weights G_abcd of a contracted quartet fixed, the energy of one
// primitive quartet is e = sum_N L_N R_N, N = (t, u, v), where R_N are the
// Hermite Coulomb integrals (d/dP)^N F_0 at P - Q and L_N the weights expanded
// in the Hermite Gaussians of the two primitive pairs.  Writing a pair's centres
// as P and A - B, the three derivatives that fix all twelve are
//   d/dP_x        sum_N L_N R_{N+x}
//   d/d(A-B)_x    the expansion coefficients' own derivatives: they lower a
//                 power, i E^{i-1,j} (-beta/p) + j E^{i,j-1} (alpha/p), and the
//                 exponential gives -2 mu (A-B)_x e
//   d/d(C-D)_x    the same on the ket
// so  d/dA = (alpha/p) d/dP + d/d(A-B),  d/dB = d/dP - d/dA, and the ket's from
// -d/dP.  Per primitive quartet this takes one Boys function from a table and a
// downward recurrence, the R recursion to L + 1, and a few hundred multiply-adds;
// the Rys form takes 2 n table functions, n x 3 extended 1D tables and 15 n
// operations per component (about 2200 and 4100 FP64 instructions per primitive
// quartet of (pp|ps) and (dp|ps), from the FP64 pipe's activity, against 700 and
// 1400 here).  What bounds it now is latency: 6 to 20 resident warps per SM
// at 96 to 255 registers, FP64 pipe 14-48 %.  40-atom 6-31G*,
// Rys form -> here: (ps|ss) 3.29 -> 2.11 ms, (ps|ps) 2.69 -> 1.45, (pp|ps) 2.75 -> 1.66,
// (ds|ps) 2.55 -> 1.68, (dp|ps) 3.41 -> 2.73, (dd|ps) 2.14 -> 1.54.
//
// The bra's expansion coefficients depend on the bra primitive only: the warp
// stages them in shared memory per task, as products over the axes, and its
// lanes (one quartet each, or a group per quartet: task.lg) read them as
// broadcasts.  The quartet's weights are a shared-memory column per thread.
#pragma once
#include <type_traits>
#include <utility>

#include "eri_templates.cuh"

namespace iqcp {

// f(integral_constant<int, 0>) ... f(integral_constant<int, N - 1>): every index a
// constant, whatever the nesting (a pragma gives up on triangular loops, and an
// array indexed at run time goes to local memory)
template <typename F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl(f, std::make_integer_sequence<int, N>{});
}

// Hermite indices t + u + v <= L in graded order
__host__ __device__ constexpr int hcount(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
__host__ __device__ constexpr int hidx(int t, int u, int v) {
  const int n = t + u + v, r = n - t;  // within degree n: t descending, then u descending
  return n * (n + 1) * (n + 2) / 6 + r * (r + 1) / 2 + (r - u);
}

// powers of Hermite index h
__host__ __device__ constexpr int hdeg(int h) {
  int n = 0;
  while (hcount(n) <= h) ++n;
  return n;
}
__host__ __device__ constexpr int hpow(int h, int axis) {
  const int n = hdeg(h), k = h - n * (n + 1) * (n + 2) / 6;
  int r = 0;
  while ((r + 1) * (r + 2) / 2 <= k) ++r;
  const int u = r - (k - r * (r + 1) / 2);
  return axis == 0 ? n - r : (axis == 1 ? u : r - u);
}

// Expansion coefficients of a pair of shells (I, J): for component (i, j) the
// products of the three axes' E^{ij}_t, t <= i + j, at a fixed stride (the
// longest component's count) so that a lane finds its component's row.
template <int I, int J>
struct Expansion {
  static constexpr int N = I >= 0 && J >= 0 ? ncart(I >= 0 ? I : 0) * ncart(J >= 0 ? J : 0) : 0;
  // most nonzeros of a component: the powers spread evenly over the axes
  static constexpr int S = I + J;
  static constexpr int LEN = S <= 0 ? 1 : (S / 3 + (S % 3 > 0) + 1) * (S / 3 + (S % 3 > 1) + 1) * (S / 3 + 1);
  static constexpr int TOTAL = N * LEN;
};

// Staged coefficients as a kernel reads them: for bras of more than 40 they are
// read through a volatile view, once per use; otherwise the compiler keeps all
// of them in registers across the ket components and spills.
template <int TOTAL>
using StagedPtr = std::conditional_t<(TOTAL > 40), const volatile double*, const double*>;

// Bra-side staging of one warp
template <int LA, int LB>
struct HermiteBra {
  using Main = Expansion<LA, LB>;
  using LowA = Expansion<LA - 1, LB>;   // a power of A lowered by one
  using LowB = Expansion<LA, LB - 1>;
  static constexpr int OA = Main::TOTAL, OB = OA + LowA::TOTAL;
  static constexpr int PER = (OB + LowB::TOTAL) | 1;  // doubles per bra primitive; odd: groups of a warp read different ones
  static constexpr int CHUNK = PER >= 512 ? 1 : 512 / PER;  // bra primitives staged at a time (4 KB per warp)
  static constexpr int NT = (LA + 1) * (LB + 1);            // 1D tables: (i, j), each up to i + j + 1 entries
  static constexpr int TROW = LA + LB + 1;
  static constexpr int WARP = CHUNK * PER + 3 * NT * TROW;  // doubles per warp
};

// One axis: E^{ij}_t for i <= LA, j <= LB at T[(i (LB+1) + j) TROW + t]
template <int LA, int LB>
__device__ __forceinline__ void hermite_axis(double pa, double pb, double o, double* T) {
  constexpr int TROW = HermiteBra<LA, LB>::TROW;
#pragma unroll
  for (int i = 0; i <= LA; ++i)
#pragma unroll
    for (int j = 0; j <= LB; ++j) {
      double* E = T + (i * (LB + 1) + j) * TROW;
      if (i + j == 0) {
        E[0] = 1.0;
        continue;
      }
      const double* L = j > 0 ? E - TROW : E - (LB + 1) * TROW;  // one power less
      const double x = j > 0 ? pb : pa;
#pragma unroll
      for (int t = 0; t <= i + j; ++t) {
        double v = t < i + j ? x * L[t] : 0.0;
        if (t > 0) v = fma(o, L[t - 1], v);
        if (t + 1 < i + j) v = fma(double(t + 1), L[t + 1], v);
        E[t] = v;
      }
    }
}

// Products of the components of shells (I, J) from the 1D tables T (rows of
// TROW entries, (i, j) at i (LB+1) + j), a component per lane
template <int I, int J, int LB, int TROW, int AXIS_STRIDE>
__device__ __forceinline__ void stage_products(int lane, const double* T, double* out) {
  constexpr int NJ = ncart(J);
  for (int c = lane; c < Expansion<I, J>::N; c += 32) {
    const int ci = c / NJ, cj = c % NJ;
    const double* e[3];
    int n[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      const int i = cart_pow(I, ci, ax), j = cart_pow(J, cj, ax);
      e[ax] = T + ax * AXIS_STRIDE + (i * (LB + 1) + j) * TROW;
      n[ax] = i + j;
    }
    double* o = out + c * Expansion<I, J>::LEN;
    for (int t = 0; t <= n[0]; ++t)
      for (int u = 0; u <= n[1]; ++u)
        for (int v = 0; v <= n[2]; ++v) *o++ = e[0][t] * e[1][u] * e[2][v];
  }
}

// Boys function F_M .. F_0 at T: order M from the staged table below T = 36 and
// the downward recurrence; above, F_0 = sqrt(pi / T) / 2 (erf(6) is 1 to rounding)
// and the upward recurrence.
__host__ __device__ constexpr int boys_tab_doubles() { return BOYS_TAB_T * BOYS_TAB_PER_UNIT * (BOYS_TAB_NCOEF + 2); }

template <int M>
__device__ __forceinline__ void boys_stage(double* s) {
  constexpr int W = BOYS_TAB_NCOEF / 2, N = BOYS_TAB_T * BOYS_TAB_PER_UNIT;
  static_assert(M <= BOYS_TAB_MAXM && BOYS_TAB_NCOEF % 2 == 0, "no Boys table of this order");
  const double2* g = reinterpret_cast<const double2*>(kBoysPoly + M * N * BOYS_TAB_NCOEF);
  double2* d = reinterpret_cast<double2*>(s);
  for (int i = threadIdx.x; i < N * W; i += blockDim.x) {
    const int k = i / W;
    copy16_async(d + k * (W + 1) + (i - k * W), g + i);  // rows padded to 6 pairs
  }
  copy_async_wait();
}

template <int M>
__device__ __forceinline__ void boys_tab(double T, const double* s, double* F) {
  const double e = exp(-T);
  if (T < double(BOYS_TAB_T)) {
    const double t = T * BOYS_TAB_PER_UNIT;
    const int k = int(t);
    F[M] = rys_poly<BOYS_TAB_NCOEF, false>(s + k * (BOYS_TAB_NCOEF + 2), 2.0 * (t - double(k)) - 1.0);
    const double T2 = 2.0 * T;
#pragma unroll
    for (int m = M; m > 0; --m) F[m - 1] = fma(T2, F[m], e) * (1.0 / double(2 * m - 1));
  } else {
    const double r = rsqrt(T), h = 0.5 * r * r;
    F[0] = 0.88622692545275801365 * r;
#pragma unroll
    for (int m = 0; m < M; ++m) F[m + 1] = fma(double(2 * m + 1), F[m], -e) * h;
  }
}

// R_N for |N| <= LM at separation (x, y, z) from f[m] = pref (-2 rho)^m F_m; in
// place by levels: R^m_{N+x} = x R^{m+1}_N + N_x R^{m+1}_{N-x}, highest degree first.
template <int LM>
__device__ __forceinline__ void hermite_r(const double* f, double x, double y, double z, double* R) {
  R[0] = f[LM];
  static_for<LM>([&](auto lv) {
    constexpr int m = LM - 1 - lv.value, H1 = hcount(LM - m);  // level m: degrees 1 .. LM - m
    static_for<H1 - 1>([&](auto k) {
      constexpr int h = H1 - 1 - k.value, t = hpow(h, 0), u = hpow(h, 1), v = hpow(h, 2);
      constexpr int ax = t > 0 ? 0 : (u > 0 ? 1 : 2), w = ax == 0 ? t : (ax == 1 ? u : v);
      constexpr int h1 = hidx(t - (ax == 0), u - (ax == 1), v - (ax == 2));
      double r = (ax == 0 ? x : (ax == 1 ? y : z)) * R[h1];
      if constexpr (w > 1) r = fma(double(w - 1), R[hidx(t - 2 * (ax == 0), u - 2 * (ax == 1), v - 2 * (ax == 2))], r);
      R[h] = r;
    });
    R[0] = f[m];
  });
}

// Coefficient o of component (ci, cj) of shells (I, J): f(o, Hermite index), in
// the order stage_products writes them
template <int I, int J, int CI, int CJ, typename F>
__device__ __forceinline__ void for_coefficients(F&& f) {
  constexpr int nt = cart_pow(I, CI, 0) + cart_pow(J, CJ, 0) + 1, nu = cart_pow(I, CI, 1) + cart_pow(J, CJ, 1) + 1,
                nv = cart_pow(I, CI, 2) + cart_pow(J, CJ, 2) + 1;
  static_for<nt * nu * nv>([&](auto o) {
    constexpr int k = o.value;
    f(o, std::integral_constant<int, hidx(k / (nu * nv), (k / nv) % nu, k % nv)>{});
  });
}

// component index of powers (i, j, k), i + j + k = L (cart_pow's order)
__host__ __device__ constexpr int cart_index(int L, int i, int j) {
  const int r = L - i;
  return r * (r + 1) / 2 + (r - j);
}

template <int LA, int LB, int LC>
struct GradMD {
  using C = Cls<LA, LB, LC, 0>;
  static constexpr int L = LA + LB + LC, LM = L + 1;
  static constexpr int TAB = boys_tab_doubles();
  static constexpr int WARP = HermiteBra<LA, LB>::WARP;
  // warps per block: four; six where the weights (110 KB for four warps of
  // (dd|ps)) leave no room for a second block
  static constexpr int WPB = C::NCOMP > 60 ? 6 : 4, THREADS = 32 * WPB;
  // resident blocks asked of the compiler: these kernels wait on their own FP64
  // chains, and warps pay more than the spills of up to 250 bytes that make room
  // for them: 40 atoms in 6-31G*, (ss|ss) 4 -> 5 blocks and (ps|ss), (pp|ss), (ds|ss) 3 -> 4:
  // 1.20 -> 1.01, 2.61 -> 2.11, 0.95 -> 0.86, 0.97 -> 0.81 ms; (dp|ss) 2 -> 3 1.24 -> 1.14.
  // One more costs: (ps|ps) at 4 1.49 against 1.44, (pp|ps) at 3 1.87 against 1.66,
  // (dp|ps) at 3 3.5 against 2.84
  static constexpr int MINB = C::NCOMP > 60 ? 1 : (L == 0 ? 5 : (LC == 1 && L == 2 ? 3 : (L <= 2 ? 4 : (L == 3 && LC == 0 ? 3 : 2))));
  // LOOPC: the ket components in a loop around branches for the part that differs.
  // Unrolled three times, the 18 or 36 bra components' code outruns the instruction
  // cache: (dp|ps) 2.85 -> 2.73 ms, (dd|ps) 1.67 -> 1.54 at 40 atoms in 6-31G*; smaller
  // bras spill with the loop (300 to 600 bytes against 0 to 270).
  static constexpr bool LOOPC = LC == 1 && C::NA * C::NB >= 18;
  // shared memory (doubles) beside the gradient accumulator
  static constexpr int FIXED = TAB + WPB * WARP + THREADS * C::NCOMP;
};

template <int LA, int LB, int LC>
__global__ void __launch_bounds__(GradMD<LA, LB, LC>::THREADS, GradMD<LA, LB, LC>::MINB) grad_md_kernel(GradArgs args) {
  using C = Cls<LA, LB, LC, 0>;
  using G = GradMD<LA, LB, LC>;
  using HB = HermiteBra<LA, LB>;
  constexpr int LBRA = LA + LB, LM = G::LM, NBRA = C::NA * C::NB, NC = C::NC;
  constexpr int HL = hcount(G::L), HB_ = hcount(LBRA), HLOW = LBRA > 0 ? hcount(LBRA > 0 ? LBRA - 1 : 0) : 1;
  extern __shared__ __align__(16) double smem[];
  boys_stage<LM>(smem);
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* Est = smem + G::TAB + wib * G::WARP;
  double* Etab = Est + HB::CHUNK * HB::PER;
  double* Wsh = smem + G::TAB + G::WPB * G::WARP + threadIdx.x;  // weight of component c at Wsh[c * THREADS]
  // blocks of more than nine components: read through a volatile view, so that
  // the weights stay in shared memory instead of being hoisted into registers
  const std::conditional_t<(C::NCOMP > 9), const volatile double*, const double*> Wv = Wsh;
  double* gacc = smem + G::FIXED;
  if (args.gsmem)
    for (int i = threadIdx.x; i < 3 * args.natoms; i += blockDim.x) gacc[i] = 0.0;
  __syncthreads();
  double* gout = args.gsmem ? gacc : args.grad;
  for (int warp = next_task(args.next_task, lane); warp < args.ntasks; warp = next_task(args.next_task, lane)) {
    const QuartetTask task = args.tasks[warp];
    const ShellPair bp = args.pairs[task.bra];
    const int lg = task.lg, NG = 32 >> lg, grp = lane >> lg, sub = lane & ((1 << lg) - 1);
    if (C::NCOMP <= kPrefetchMaxComp && lg > 0) prefetch_bra(args.pp, bp, lane);
    // this task's molecule block (bra and ket pairs always share a molecule)
    const int n = args.mol_n[bp.mol];
    const double* __restrict__ D = args.D + args.mol_base[bp.mol];
    const double xs = args.xscale;
    const bool ij_same = bp.sa == bp.sb;
    double gAt[3] = {0, 0, 0}, gPt[3] = {0, 0, 0};
    const unsigned sel = task_sel(args.mx, warp, task.nket);
    const int nsel = __popc(sel);
    for (int kbase = 0; kbase < nsel; kbase += NG) {
      const int kk = kbase + grp;
      bool active = kk < nsel;
      ShellPair kp = bp;
      KetPrims ket{nullptr, 0};
      int kpos = 0;
      if (active) {
        kpos = task.ket0 + (args.mx.pass ? nth_set_bit(sel, kk) : kk);
        kp = load_ket(args.kets, kpos, bp.mol, &ket);
        if (C::NCOMP <= kPrefetchMaxComp && lg > 0) ket.prefetch(kp.np, sub, 1 << lg);
        // the reference skips when the Schwarz bound of its bra pair (the larger
        // composite index) is below threshold (gradient.rs:1457-1460)
        const double qref = bp.comp >= kp.comp ? bp.Q : kp.Q;
        if (qref < args.schwarz_thr) active = false;
      }
      if (active) {
        const bool kl_same = kp.sa == kp.sb, bk_same = task.diag && kpos == task.bra_pos;
        // not unrolled over the bra components: 54 copies of the weight would be
        // a third of (dp|ps)'s code
#pragma unroll 1
        for (int ab = 0; ab < NBRA; ++ab)
#pragma unroll
          for (int c = 0; c < NC; ++c)
            Wsh[(ab * NC + c) * G::THREADS] =
                grad_weight<LA, LB, LC, 0>(D, n, bp, kp, ab * NC + c, ij_same, kl_same, bk_same, xs);
      }
      const double CD[3] = {kp.A[0] - kp.B[0], kp.A[1] - kp.B[1], kp.A[2] - kp.B[2]};
      double gP[3] = {0, 0, 0}, gC[3] = {0, 0, 0};
      for (int i0 = 0; i0 < bp.np; i0 += HB::CHUNK) {
        const int nb = bp.np - i0 < HB::CHUNK ? bp.np - i0 : HB::CHUNK;
        // the bra's expansion coefficients of primitives i0 .. i0 + nb - 1
        if (bp.np > HB::CHUNK || kbase == 0) {
          for (int i = 0; i < nb; ++i) {
            const PrimPair b = load_pp(args.pp + bp.pstart + i0 + i);
            __syncwarp();
            if (lane < 3) {
              const double P = lane == 0 ? b.P[0] : (lane == 1 ? b.P[1] : b.P[2]);
              const double A = lane == 0 ? bp.A[0] : (lane == 1 ? bp.A[1] : bp.A[2]);
              const double B = lane == 0 ? bp.B[0] : (lane == 1 ? bp.B[1] : bp.B[2]);
              hermite_axis<LA, LB>(P - A, P - B, 0.5 * b.inv_p, Etab + lane * HB::NT * HB::TROW);
            }
            __syncwarp();
            double* E = Est + i * HB::PER;
            constexpr int AXIS = HB::NT * HB::TROW;
            stage_products<LA, LB, LB, HB::TROW, AXIS>(lane, Etab, E);
            if constexpr (LA > 0) stage_products<LA - 1, LB, LB, HB::TROW, AXIS>(lane, Etab, E + HB::OA);
            if constexpr (LB > 0) stage_products<LA, LB - 1, LB, HB::TROW, AXIS>(lane, Etab, E + HB::OB);
          }
          __syncwarp();
        }
        if (!active) continue;
        PrimPair k;
        for (PrimItems it(nb, kp.np, sub, 1 << lg); it.more(); it.next()) {  // ket-major order (see quartet)
          if (it.new_ket()) k = ket(it.j);
          const PrimPair b = load_pp(args.pp + bp.pstart + i0 + it.i);
          if (b.K * k.K < args.prim_thr) continue;
          const StagedPtr<HB::Main::TOTAL> E = Est + it.i * HB::PER;
          const double p = b.p, q = k.p, s = p + q;
          const double PQ[3] = {b.P[0] - k.P[0], b.P[1] - k.P[1], b.P[2] - k.P[2]};
          const double rs = rsqrt(s), inv_s = rs * rs;  // 1/(p+q), 1/sqrt(p+q): one rsqrt
          const double rho = p * q * inv_s;
          double f[LM + 1];
          boys_tab<LM>(rho * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]), smem, f);
          double sc = kTwoPi52 * b.cK * k.cK * b.inv_p * k.inv_p * rs;
#pragma unroll
          for (int m = 0; m <= LM; ++m) {
            f[m] *= sc;
            sc *= -2.0 * rho;
          }
          double R[hcount(LM)];
          hermite_r<LM>(f, PQ[0], PQ[1], PQ[2], R);
          const double ap = b.aa * b.inv_p, bq = 1.0 - ap;  // alpha/p, beta/p
          double Lm[HL];
#pragma unroll
          for (int h = 0; h < HL; ++h) Lm[h] = 0.0;
          double gRa[3] = {0, 0, 0}, gRb[3] = {0, 0, 0}, Tc[3] = {0, 0, 0};
          const double oq = 0.5 * k.inv_p;
          // ket components: s, or p_x, p_y, p_z with E_0 = QC_c and E_{1c} = 1/2q
          // (odd Hermite orders of the ket change sign)
          double S[HLOW];  // R contracted with the ket component, |H| <= LA + LB - 1
          // Lc[h]: the weighted bra expansion of ket component c
          const auto ket_part = [&](auto cc, const double* Lc) {
            constexpr int c = cc.value;
            const double qc = LC == 0 ? 1.0 : k.P[LC == 0 ? 0 : c] - kp.A[LC == 0 ? 0 : c];
            static_for<HB_>([&](auto hc) {
              constexpr int h = hc.value;
              Lm[h] = fma(qc, Lc[h], Lm[h]);
              if constexpr (LC > 0) {
                constexpr int up = hidx(hpow(h, 0) + (c == 0), hpow(h, 1) + (c == 1), hpow(h, 2) + (c == 2));
                Lm[up] = fma(-oq, Lc[h], Lm[up]);
                Tc[c] = fma(Lc[h], R[h], Tc[c]);
                if constexpr (hdeg(h) < LBRA) S[h] = fma(-oq, R[up], qc * R[h]);
              } else if constexpr (hdeg(h) < LBRA) {
                S[h] = R[h];
              }
            });
          };
          const auto component = [&](int c, auto&& ket) {
            double g[NBRA], Lc[HB_];
#pragma unroll
            for (int ab = 0; ab < NBRA; ++ab) g[ab] = Wv[(ab * NC + c) * G::THREADS];
#pragma unroll
            for (int h = 0; h < HB_; ++h) Lc[h] = 0.0;
            static_for<NBRA>([&](auto abc) {
              constexpr int ab = abc.value, ca = ab / C::NB, cb = ab % C::NB;
              const StagedPtr<HB::Main::TOTAL> Ec = E + ab * HB::Main::LEN;
              for_coefficients<LA, LB, ca, cb>([&](auto o, auto h) { Lc[h.value] = fma(g[ab], Ec[o.value], Lc[h.value]); });
            });
            ket(Lc);
            if constexpr (LA > 0) {
              static_for<ncart(LA > 0 ? LA - 1 : 0) * C::NB>([&](auto lc) {
                constexpr int LL = LA > 0 ? LA - 1 : 0, ca = lc.value / C::NB, cb = lc.value % C::NB;
                const StagedPtr<HB::Main::TOTAL> Ec = E + HB::OA + lc.value * HB::LowA::LEN;
                double y = 0.0;
                for_coefficients<LL, LB, ca, cb>([&](auto o, auto h) { y = fma(Ec[o.value], S[h.value], y); });
                constexpr int i = cart_pow(LL, ca, 0), j = cart_pow(LL, ca, 1), l = cart_pow(LL, ca, 2);
                gRa[0] = fma(double(i + 1) * g[cart_index(LA, i + 1, j) * C::NB + cb], y, gRa[0]);
                gRa[1] = fma(double(j + 1) * g[cart_index(LA, i, j + 1) * C::NB + cb], y, gRa[1]);
                gRa[2] = fma(double(l + 1) * g[cart_index(LA, i, j) * C::NB + cb], y, gRa[2]);
              });
            }
            if constexpr (LB > 0) {
              static_for<C::NA * ncart(LB > 0 ? LB - 1 : 0)>([&](auto lc) {
                constexpr int LL = LB > 0 ? LB - 1 : 0, ca = lc.value / ncart(LL), cb = lc.value % ncart(LL);
                const StagedPtr<HB::Main::TOTAL> Ec = E + HB::OB + lc.value * HB::LowB::LEN;
                double y = 0.0;
                for_coefficients<LA, LL, ca, cb>([&](auto o, auto h) { y = fma(Ec[o.value], S[h.value], y); });
                constexpr int i = cart_pow(LL, cb, 0), j = cart_pow(LL, cb, 1), l = cart_pow(LL, cb, 2);
                gRb[0] = fma(double(i + 1) * g[ca * C::NB + cart_index(LB, i + 1, j)], y, gRb[0]);
                gRb[1] = fma(double(j + 1) * g[ca * C::NB + cart_index(LB, i, j + 1)], y, gRb[1]);
                gRb[2] = fma(double(l + 1) * g[ca * C::NB + cart_index(LB, i, j)], y, gRb[2]);
              });
            }
          };
          if constexpr (G::LOOPC) {
#pragma unroll 1
            for (int c = 0; c < NC; ++c)
              component(c, [&](const double* Lc) {
                if (c == 0) ket_part(std::integral_constant<int, 0>{}, Lc);
                else if (c == 1) ket_part(std::integral_constant<int, 1>{}, Lc);
                else ket_part(std::integral_constant<int, 2>{}, Lc);
              });
          } else {
            static_for<NC>([&](auto cc) { component(cc.value, [&](const double* Lc) { ket_part(cc, Lc); }); });
          }
          double e = 0.0, dP[3] = {0, 0, 0};
          static_for<HL>([&](auto hc) {
            constexpr int h = hc.value, t = hpow(h, 0), u = hpow(h, 1), v = hpow(h, 2);
            const double l = Lm[h];
            e = fma(l, R[h], e);
            dP[0] = fma(l, R[hidx(t + 1, u, v)], dP[0]);
            dP[1] = fma(l, R[hidx(t, u + 1, v)], dP[1]);
            dP[2] = fma(l, R[hidx(t, u, v + 1)], dP[2]);
          });
          const double m2 = -2.0 * b.aa * bq * e;                          // -2 mu e
          const double ck = k.aa * k.inv_p, dk = 1.0 - ck;                 // gamma/q, delta/q
          const double n2 = -2.0 * k.aa * dk * e;
#pragma unroll
          for (int x = 0; x < 3; ++x) {
            gAt[x] += fma(ap, dP[x], fma(m2, bp.A[x] - bp.B[x], fma(ap, gRb[x], -bq * gRa[x])));
            gP[x] += dP[x];
            gC[x] += fma(n2, CD[x], fma(-ck, dP[x], -dk * Tc[x]));
          }
        }
      }
      // ket atoms differ per group: segmented reduction, lane 0 of the group adds
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const double c = group_sum(gC[x], lg), t = group_sum(gP[x], lg);
        if (active && sub == 0) {
          atomicAdd(gout + 3 * kp.atom_a + x, c);
          atomicAdd(gout + 3 * kp.atom_b + x, -t - c);  // dC + dD = -dP
        }
        gPt[x] += gP[x];
      }
    }
    // bra atoms are shared by the whole warp: one reduction per task
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const double sa = warp_sum(gAt[x]), sp = warp_sum(gPt[x]);
      if (lane == 0) {
        atomicAdd(gout + 3 * bp.atom_a + x, sa);
        atomicAdd(gout + 3 * bp.atom_b + x, sp - sa);
      }
    }
    __syncwarp();
  }
  if (args.gsmem) {
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * args.natoms; i += blockDim.x)
      if (gacc[i] != 0.0) atomicAdd(args.grad + i, gacc[i]);
  }
}

}  // namespace iqcp
