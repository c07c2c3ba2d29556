// Shared device/host definitions of the ERI engine: shell-pair tables in HBM,
// quartet tasks, Cartesian component tables.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace iqcp {

constexpr int kNumModes = 4;  // quartet-kernel variants per class

// Angular-momentum classes of a shell pair with la >= lb:
// 0 ss, 1 ps, 2 pp, 3 ds, 4 dp, 5 dd  (index la*(la+1)/2 + lb)
constexpr int kNumPairClasses = 6;
constexpr int kMaxL = 2;

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
// Rys roots of the first-derivative integrals.  Every product the gradient
// contracts has one index raised by one, total angular momentum L + 1, i.e. a
// polynomial of degree L + 1 in t^2, which an n-point rule integrates exactly
// once 2n - 1 >= L + 1.  (The reference takes L/2 + 2 for even L,
// integrals/eri/mod.rs:2146-2147, one root more than exactness needs; the
// results agree to rounding.)
__host__ __device__ constexpr int grad_nroots(int L) { return (L + 1) / 2 + 1; }
__host__ __device__ constexpr int pair_class(int la, int lb) { return la * (la + 1) / 2 + lb; }
__host__ __device__ constexpr int class_la(int c) { return c == 0 ? 0 : (c <= 2 ? 1 : 2); }
__host__ __device__ constexpr int class_lb(int c) { return c - class_la(c) * (class_la(c) + 1) / 2; }

// Largest block (components) of the FP64 thread kernels; above, only the
// warp-cooperative ones exist.  Measured on 40 atoms in 6-31G*: at 108
// components ((dp|ds), (dd|ps)) a lane group per quartet takes 0.57 and 0.36 ms
// against a warp's 1.06 and 0.53 (J/K), 1.62 and 1.55 against 2.69 and 1.61
// (gradient); at 162 ((dp|pp)) the block no longer fits the registers and the
// warp wins, 0.86 against 1.60 ms (J/K) and 3.1 against 8.2 (gradient).
constexpr int kMaxThreadComp = 108;
constexpr int kMaxThreadComp32 = 324;      // the same for the FP32 share of a mixed call

__host__ __device__ constexpr int class_comps(int X, int Y) {
  return ncart(class_la(X)) * ncart(class_lb(X)) * ncart(class_la(Y)) * ncart(class_lb(Y));
}
// The variant that a requested mode runs: 1 a warp per quartet, 0 a lane group per
// quartet (also for modes 2 and 3, which had kernels of their own)
__host__ __device__ constexpr int kernel_variant(int X, int Y, int mode, bool f32) {
  return mode == 1 || class_comps(X, Y) > (f32 ? kMaxThreadComp32 : kMaxThreadComp) ? 1 : 0;
}
// Variant before autotuning.  With fewer quartets than one wave of thread-kernel
// lanes (148 SMs x 8 warps at 255 registers) the largest blocks leave most of the
// chip idle behind a few long threads, and a warp per quartet is faster: 12 atoms
// in 6-31G*, gradient (pp|pp) 0.12 against 0.15 ms, (dp|ds) 0.11 / 0.22, (dd|ps) 0.10 /
// 0.24, J/K (dp|ds) 0.05 / 0.07, (dd|ps) 0.04 / 0.05; below those sizes of block the
// thread kernels stay ahead ((ds|pp) J/K 0.06 against 0.04 ms, gradient 0.12 / 0.11).
__host__ __device__ constexpr int default_mode(int X, int Y, int kind, long long quartets) {
  const int n = class_comps(X, Y);
  if (n > kMaxThreadComp) return 1;
  return n >= (kind == 1 ? 81 : 108) && quartets < 148LL * 8 * 32 ? 1 : 0;
}

// Whether a mixed call runs a class twice, FP64 share and FP32 share, before
// autotuning; otherwise the whole class runs in FP64.  Roots, weights, pair data
// and digestion are FP64 in both, so up to 108 components the FP32 share alone
// takes what the class takes in FP64 and the other share comes on top: J/K of 40
// atoms in 6-31G* at cutoff 1e-3 (96 % FP32), (ps|ss) 1.13 ms against 0.37 + 1.10,
// (ds|ps) 0.79 / 0.14 + 0.73, (dd|ps) 0.36 / 0.13 + 0.60; gradient (dp|ps) 2.87 / 0.41 + 2.49,
// (dp|ds) 1.62 / 0.34 + 3.28.  Above, the contraction is most of the work: gradient
// (dp|pp) 3.02 / 0.50 + 1.93, (dd|dp) 1.02 / 0.28 + 0.69; J/K breaks even, (dp|pp) 0.83 /
// 0.20 + 0.63.  The whole mixed Fock build 12.3 -> 9.8 ms.  A context without such
// blocks splits its largest class alone (0.1 ms on (pp|pp)), so that no context's
// mixed form is FP64 only.  largest: components of the context's largest class.
__host__ __device__ constexpr int default_split(int X, int Y, int largest) {
  return class_comps(X, Y) > kMaxThreadComp || class_comps(X, Y) == largest ? 1 : 0;
}

// Cartesian powers, reference order (integrals/cartesian.rs:113-136):
// x exponent descending, then y exponent descending.
__host__ __device__ constexpr int cart_pow(int l, int c, int axis) {
  // l = 0: (000); l = 1: x y z; l = 2: xx xy xz yy yz zz
  return l == 0 ? 0
       : l == 1 ? (c == axis ? 1 : 0)
       : (axis == 0 ? (c == 0 ? 2 : (c <= 2 ? 1 : 0))
          : axis == 1 ? (c == 1 ? 1 : (c == 3 ? 2 : (c == 4 ? 1 : 0)))
                      : (c == 2 ? 1 : (c == 4 ? 1 : (c == 5 ? 2 : 0))));
}

// One primitive pair of a shell pair (A first, la >= lb), 64 bytes.
struct __align__(16) PrimPair {
  double p;       // alpha_a + alpha_b
  double P[3];    // Gaussian product centre
  double K;       // exp(-alpha_a alpha_b / p |AB|^2)  (screening value)
  double cK;      // K * c_a * c_b * Nrad(alpha_a, la) * Nrad(alpha_b, lb)
  double aa;      // alpha_a (alpha_b = p - alpha_a)
  double inv_p;   // 1 / p
};

// One shell pair (la >= lb after the swap), 96 bytes.
struct __align__(16) ShellPair {
  double A[3];
  double B[3];
  double Q;       // Schwarz bound sqrt(max |(ab|ab)|)
  int pstart;     // first PrimPair
  int np;         // number of PrimPairs (K >= prim threshold)
  int oa, ob;     // first basis function of shell a / b
  int sa, sb;     // shell indices (for same-shell degeneracy)
  int atom_a, atom_b;
  int comp;       // reference composite index si(si+1)/2+sj, si>=sj
  int mol;        // molecule of a batched context (0 for a single geometry)
};

// Ket-side tables of the thread kernels, in the order of the ket lists: the lanes
// of a warp take consecutive kets, so every field is an array of its own and a
// warp's loads are contiguous.  The primitives of a bucket (m kets of np
// primitives each) are stored [primitive][field][ket].
struct KetTables {
  const int4* i0;      // oa, ob, np, offset (unsigned) of the ket's first primitive field in prim
  const int4* i1;      // atom_a, atom_b, comp, bucket size m (negative when both shells are the same)
  const double* geom;  // A xyz, B xyz, Q: geom[f * n + position]
  const double* prim;  // field f of primitive j: prim[offset + (8 j + f) m]; fields in PrimPair's order
  int n;               // positions
};

// Field f of a position among n, in geom
__host__ __device__ constexpr unsigned long long ket_geom_offset(int f, int n) {
  return (unsigned long long)(unsigned)f * (unsigned)n;
}
// Kets of one bucket, so that every offset within it is an int: the kernels' index
// arithmetic (64-bit products cost the J/K builds of 40 atoms in 6-31G* 1 %).  A
// longer run of kets with equal primitive counts becomes several buckets (0: not
// even one ket fits, which context creation refuses).
constexpr int max_bucket_kets(int np) { return int(0x7fffffffLL / (8LL * (np > 0 ? np : 1))); }

// Unit of work for one warp: one bra pair against up to 32 consecutive ket
// pairs of a class list.
struct QuartetTask {
  int bra;        // ShellPair index
  int ket0;       // first position in the ket class list
  int nket;       // 1..32
  int diag;       // 1 when bra and ket lists are the same class (position ket0+i == bra_pos => pair with itself)
  int bra_pos;    // position of the bra in its class list
  int lg;         // thread kernels: 2^lg lanes share each ket's primitive quartets (nket <= 32 >> lg)
};

// Dynamic task distribution of the persistent quartet kernels: lane 0 of a
// warp takes the next task index from the launch's counter.
__device__ __forceinline__ int next_task(int* counter, int lane) {
  int t = 0;
  if (lane == 0) t = atomicAdd(counter, 1);
  return __shfl_sync(0xffffffffu, t, 0);
}

// Mixed precision.  A mixed call runs a class either wholly in FP64 or twice
// over the same task list: pass 1 takes the quartets whose bound
// Q_ij Q_kl Dmax is at or above the cutoff (FP64 quadrature), pass 2 the rest
// (FP32 quadrature, FP64 roots, weights and accumulation).  Dmax is the
// largest |D| over the six shell blocks the quartet digests with (J/K) or its
// square (gradient, whose weights are products of two density elements).
// Pass 0 takes every quartet.  The split is fixed once per call as a bit mask
// per task (precision_mask_kernel).
struct Mixed {
  const double* dmax;       // per molecule: max |D| per shell block, ns x ns at dbase[m]
  const long long* dbase;
  const int* shell0;        // per molecule: first global shell
  const int* ns;            // per molecule: shell count
  double cutoff;
  int pass;                 // 0 all, 1 FP64 share, 2 FP32 share
  unsigned long long* fp32_count;  // quartets evaluated in pass 2 (may be null)
  const unsigned* mask;     // per task of the launch: bit k set = ket k runs in FP32 (passes 1, 2)
};

__device__ __forceinline__ double mixed_dbound(const Mixed& mx, const ShellPair& bp, const ShellPair& kp) {
  const int m = bp.mol, s0 = mx.shell0[m], ns = mx.ns[m];
  const double* dm = mx.dmax + mx.dbase[m];
  const int i = bp.sa - s0, j = bp.sb - s0, k = kp.sa - s0, l = kp.sb - s0;
  return fmax(fmax(dm[i * ns + j], dm[k * ns + l]),
              fmax(fmax(dm[i * ns + k], dm[i * ns + l]), fmax(dm[j * ns + k], dm[j * ns + l])));
}

// Bit mask of a task's kets in this launch's pass.
__device__ __forceinline__ unsigned task_sel(const Mixed& mx, int task, int nket) {
  const unsigned all = nket >= 32 ? 0xffffffffu : ((1u << nket) - 1u);
  if (mx.pass == 0) return all;
  const unsigned f32 = __ldg(mx.mask + task);
  return mx.pass == 2 ? (f32 & all) : (all & ~f32);
}

// Position of the (k+1)-th set bit of mask (k < popc(mask)).
__device__ __forceinline__ int nth_set_bit(unsigned mask, int k) {
  for (int i = 0; i < k; ++i) mask &= mask - 1;
  return __ffs(mask) - 1;
}

// Kernel argument blocks (passed by value).
struct JKArgs {
  const ShellPair* pairs;
  const PrimPair* pp;
  const int* ket_list;
  KetTables kets;
  const QuartetTask* tasks;
  int ntasks;
  const double* D;   // angular-scaled density
  int nbf;
  double* J;         // unsymmetrised accumulators (nbf x nbf)
  double* K;         // may be null
  double prim_thr;
  int mode;          // kernel variant: 1 warp-cooperative, else a group of lanes per quartet
  Mixed mx;
  int* next_task;             // work counter (zeroed before the launch)
  int ket_split = 1;          // team kernels: warps per task, each taking a slice of its kets
  const long long* mol_base;  // per molecule: offset of its nbf x nbf block in D, J, K
  const int* mol_n;           // per molecule: nbf (row stride of its block)
  int nset;                   // densities digested per quartet (1, or several response densities)
  long long set_stride;       // elements between consecutive densities in D, J and K
  const int* mol_active;      // per molecule: 0 = skip its tasks (a converged geometry of a batched SCF); may be null
};

// Tasks of molecules flagged inactive are skipped (the same on every lane).
__device__ __forceinline__ bool task_inactive(const int* mol_active, int mol) {
  return mol_active != nullptr && __ldg(mol_active + mol) == 0;
}

struct StoreArgs {
  const ShellPair* pairs;
  const PrimPair* pp;
  const int* ket_list;
  const QuartetTask* tasks;
  int ntasks;
  double* out;
  double prim_thr;
};

struct GradArgs {
  const ShellPair* pairs;
  const PrimPair* pp;
  const int* ket_list;
  KetTables kets;
  const QuartetTask* tasks;
  int ntasks;
  const double* D;   // angular-scaled density
  int nbf;
  double xscale;     // 0.25 * hf_frac
  double* grad;      // natoms x 3
  double prim_thr;
  double schwarz_thr;
  int mode;          // kernel variant: 1 warp-cooperative, else a group of lanes per quartet
  int natoms;        // gradient rows; accumulated per block in shared memory when gsmem
  int gsmem;
  Mixed mx;
  int* next_task;    // work counter (zeroed before the launch)
  int ket_split = 1;  // team kernel: warps per task, each taking a slice of its kets
  const long long* mol_base;  // per molecule: offset of its block in D
  const int* mol_n;           // per molecule: nbf
};

// One launch covers the shell pairs of consecutive molecules (atoms atom0 ..
// atom1 - 1 of the context).
struct OneEArgs {
  const ShellPair* pairs;
  const int* list;                   // the launch's pairs, sorted by class
  int first[kNumPairClasses + 1];    // class c: list[first[c]] .. list[first[c + 1] - 1]
  int n_mol, atom0, atom1;
  const int* mol_atom0;              // per molecule: first atom (n_mol + 1)
  const int* mol_n;                  // per molecule: nbf
  const long long* mol_base;         // per molecule: offset of its block in the packed matrices
  const int* nprim;                  // per shell
  const int* pstart;                 // per shell: first primitive
  const double* exps;
  const double* coefs;
  const double* atom_xyz;
  const int* z;
  double* S;  // may be null
  double* T;  // may be null
  double* V;  // may be null
  // nuclear gradient of the one-electron energy (one_electron_grad_kernel)
  const double* D;     // density, packed
  const double* W;     // energy-weighted density (factor 2 convention), packed
  double* grad;        // atoms of the context x 3, added to
  int gsmem;           // accumulate per block in shared memory (3 doubles per atom of the launch)
};

// Host launchers (eri_aux.cu, onee.cu)
cudaError_t launch_jk(int X, int Y, const JKArgs& a, cudaStream_t st);
cudaError_t launch_store(int X, int Y, const StoreArgs& a, cudaStream_t st);
cudaError_t launch_grad(int X, int Y, const GradArgs& a, cudaStream_t st);
cudaError_t launch_schwarz(int X, ShellPair* pairs, const PrimPair* pp, const int* list, int n,
                           double thr, cudaStream_t st);
// Packed per-molecule matrices: molecule m owns elements [base[m], base[m+1])
// as an n[m] x n[m] row-major block; its basis functions start at bf0[m] in
// the global angular-factor array.
struct Packing {
  const long long* base;  // nmol + 1 offsets (device)
  const int* n;           // nmol (device)
  const int* bf0;         // nmol (device)
  int nmol;
  long long total;
};
cudaError_t launch_scale_density(const double* D, const double* ang, const Packing& P, double* Ds, cudaStream_t st);
cudaError_t launch_symmetrize(const double* X, const double* ang, const Packing& P, double* out, cudaStream_t st);
cudaError_t launch_fock(const double* H, const double* Jt, const double* Kt, const double* ang, const Packing& P,
                        double kscale, double* F, cudaStream_t st);
cudaError_t launch_boys_batch(int m, int n, const double* T, double* F, cudaStream_t st);
cudaError_t launch_rys_batch(int nr, int n, const double* T, double* R, double* W, cudaStream_t st);
cudaError_t launch_one_electron(const OneEArgs& a, cudaStream_t st);
cudaError_t launch_one_electron_grad(const OneEArgs& a, cudaStream_t st);
// max |D| per shell block of every molecule (layout of Mixed::dmax); D packed
cudaError_t launch_shell_dmax(const double* D, const Packing& P, const int* shell_off, const int* shell_l,
                              const Mixed& mx, long long total, double* dmax, cudaStream_t st);
// FP32 masks of the mixed form for every task (GRAD: density bound squared)
cudaError_t launch_precision_masks(const ShellPair* pairs, const int* ket_list, const QuartetTask* tasks,
                                   int ntasks, const Mixed& mx, bool grad, unsigned* mask, cudaStream_t st);
// Fill the ket tables: place[position] = {offset in prim, bucket size}
cudaError_t launch_ket_tables(const ShellPair* pairs, const PrimPair* pp, const int* ket_list, const int2* place,
                              int n, int4* i0, int4* i1, double* geom, double* prim, cudaStream_t st);
cudaError_t launch_count_prim_quartets(const ShellPair* pairs, const PrimPair* pp, const int* ket_list,
                                       const QuartetTask* tasks, int ntasks, double thr,
                                       unsigned long long* out, cudaStream_t st);
// FMA-throughput probe: which = 0 FP64, 1 FP32; returns flops done and device ms
cudaError_t launch_fma_peak(int which, double* flops, float* ms);

}  // namespace iqcp
