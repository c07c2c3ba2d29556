// Offline generator for the device Rys quadrature tables (rys_tables.inc).
//
// For n = 1..kMaxN roots, the n-point Rys rule over x = t^2 on [0, 1) with
// weight  x^{-1/2} exp(-T x) / 2  (moments F_k(T), the Boys function) is
// computed in IEEE binary128 by
//   * moments F_0..F_2n(T) from the convergent Kummer series,
//   * the Chebyshev (modified-moment free) algorithm for the three-term
//     recurrence coefficients (Gautschi, "Orthogonal Polynomials", 2.1.7),
//   * eigenvalues of the Jacobi matrix by Sturm-sequence bisection,
//   * Christoffel numbers w_i = 1 / sum_j p_j(x_i)^2 (orthonormal p_j).
// Roots and weights are then fitted piecewise on T in [0, Tasym(n)): Chebyshev
// interpolation in binary128 on intervals of fixed width, converted to powers
// of x = 2 (T - T0) / width - 1 in [-1, 1] before rounding to double, so that
// the device evaluates them with one FMA per coefficient (Horner).  Their
// coefficients fall by more than a factor of four per order, so the power form
// loses nothing: worst relative error of Horner in double 2.0e-16 (n = 1) to
// 2.9e-16 (n = 5), against 2.8e-16 to 3.6e-16 for the Chebyshev form by Clenshaw's
// recurrence, which needs an add and an FMA per coefficient.  Orders 1 and 2 take half-width intervals and degree 9 (ten
// coefficients; 12 and 28 KB), the others unit intervals and degree 11, whose
// half-width tables (48 KB and more) would cost resident blocks.  Beyond Tasym(n)
// the rule is the large-T limit: roots y_i / T and weights W_i / sqrt(T), with
// (y_i, W_i) the Gauss rule for the weight y^{-1/2} e^{-y} / 2 on [0, inf).
// Tasym(n) is the first integer T from which that limit agrees with the exact
// rule to the target accuracy everywhere in the sampled range.
//
// The Boys functions F_m(T), m = 0..kMaxBoys, are tabulated the same way on
// half-unit intervals of [0, kBoysT): the Hermite gradient kernels read one
// order and recur downwards.  From kBoysT = 36 on erf(sqrt(T)) is 1 to rounding
// and the upward recurrence from F_0 = sqrt(pi/T)/2 loses nothing.
//
// Build/run:  g++ -O2 -o /tmp/gen gen_rys_tables.cpp -lquadmath && /tmp/gen rys_tables.inc
#include <quadmath.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

typedef __float128 q;

static const int kMaxN = 7;
// polynomial degree per interval (odd: an even number of coefficients, read in
// 16-byte pairs) and intervals per unit of T
static int deg_of(int n) { return n <= 2 ? 9 : 11; }
static int per_unit(int n) { return n <= 2 ? 2 : 1; }
static const int kMaxBoys = 6, kBoysT = 36, kBoysDeg = 9, kBoysPerUnit = 2;

// F_k(T) = int_0^1 t^{2k} e^{-T t^2} dt, k = 0..m, by the series of F_m and
// downward recurrence (all terms positive, no cancellation).
static void boys_q(int m, q T, q* F) {
  const q e = expq(-T);
  q term = 1.0Q / (2 * m + 1), sum = term;
  for (int k = 1; k < 100000; ++k) {
    term *= 2 * T / (2 * m + 2 * k + 1);
    sum += term;
    if (term < sum * 1e-40Q) break;
  }
  F[m] = e * sum;
  for (int k = m; k >= 1; --k) F[k - 1] = (2 * T * F[k] + e) / (2 * k - 1);
}

// Gauss rule from moments mu_0..mu_2n via the Chebyshev algorithm.
static void gauss_from_moments(int n, const q* mu, q* x, q* w) {
  // sigma_{k,l} recursion (Gautschi 2004, Alg. 2.1)
  std::vector<q> a(n), b(n);
  const int L = 2 * n;
  std::vector<q> sm1(L + 1, 0), s0(L + 1), s1(L + 1);
  for (int l = 0; l <= L - 1; ++l) s0[l] = mu[l];
  a[0] = mu[1] / mu[0];
  b[0] = mu[0];
  for (int k = 1; k < n; ++k) {
    for (int l = k; l <= L - k - 1; ++l)
      s1[l] = s0[l + 1] - a[k - 1] * s0[l] - b[k - 1] * sm1[l];
    a[k] = s1[k + 1] / s1[k] - s0[k] / s0[k - 1];
    b[k] = s1[k] / s0[k - 1];
    sm1 = s0;
    s0 = s1;
  }
  // eigenvalues of the Jacobi matrix J (diag a, offdiag sqrt(b_k)), bisection
  auto count_below = [&](q lam) {
    int cnt = 0;
    q d = a[0] - lam;
    if (d < 0) ++cnt;
    for (int k = 1; k < n; ++k) {
      if (d == 0) d = 1e-60Q;
      d = a[k] - lam - b[k] / d;
      if (d < 0) ++cnt;
    }
    return cnt;
  };
  // Gershgorin bounds of the Jacobi matrix
  q lo = a[0], hi = a[0];
  for (int k = 0; k < n; ++k) {
    const q r = (k > 0 ? sqrtq(b[k]) : 0) + (k + 1 < n ? sqrtq(b[k + 1]) : 0);
    if (a[k] - r < lo) lo = a[k] - r;
    if (a[k] + r > hi) hi = a[k] + r;
  }
  lo -= 1e-3Q;
  hi += 1e-3Q;
  for (int i = 0; i < n; ++i) {
    q l = lo, h = hi;
    for (int it = 0; it < 240; ++it) {
      q m = 0.5Q * (l + h);
      if (count_below(m) > i) h = m; else l = m;
    }
    x[i] = 0.5Q * (l + h);
  }
  // orthonormal polynomials p_0 = 1/sqrt(b0); sqrt(b_{k+1}) p_{k+1} = (x-a_k) p_k - sqrt(b_k) p_{k-1}
  for (int i = 0; i < n; ++i) {
    q pm1 = 0, p0 = 1 / sqrtq(b[0]), s = p0 * p0;
    for (int k = 0; k < n - 1; ++k) {
      q p1 = ((x[i] - a[k]) * p0 - (k > 0 ? sqrtq(b[k]) * pm1 : 0)) / sqrtq(b[k + 1]);
      s += p1 * p1;
      pm1 = p0;
      p0 = p1;
    }
    w[i] = 1 / s;
  }
}

static void exact_rule(int n, q T, q* x, q* w) {
  q F[2 * kMaxN + 2];
  boys_q(2 * n, T, F);
  gauss_from_moments(n, F, x, w);
}

// Large-T rule: weight y^{-1/2} e^{-y}/2 on [0, inf), moments Gamma(k+1/2)/2
static void asym_base(int n, q* y, q* W) {
  q mu[2 * kMaxN + 2];
  q g = sqrtq(M_PIq);  // Gamma(1/2)
  for (int k = 0; k <= 2 * n; ++k) {
    mu[k] = g / 2;
    g *= (k + 0.5Q);
  }
  gauss_from_moments(n, mu, y, W);
}

static double horner(const double* c, int deg, double x) {
  double v = c[deg];
  for (int j = deg - 1; j >= 0; --j) v = std::fma(v, x, c[j]);
  return v;
}

// powers of x from Chebyshev coefficients c_0..c_deg
static std::vector<q> to_powers(const std::vector<q>& c) {
  const size_t n = c.size();
  std::vector<q> out(n, 0), t0(n, 0), t1(n, 0), t2(n, 0);
  t0[0] = 1;
  t1[1] = 1;
  for (size_t k = 0; k < n; ++k) {
    for (size_t i = 0; i < n; ++i) out[i] += c[k] * t0[i];
    for (size_t i = 0; i < n; ++i) t2[i] = (i ? 2 * t1[i - 1] : 0) - t0[i];
    t0 = t1;
    t1 = t2;
  }
  return out;
}

int main(int argc, char** argv) {
  if (argc < 2) { fprintf(stderr, "usage: gen out.inc\n"); return 1; }
  const double tol = 2e-15;
  int tasym[kMaxN + 1];
  std::vector<double> asy_y, asy_w;
  std::vector<double> coef;       // [n][interval][func 2n][deg+1]
  std::vector<int> offset(kMaxN + 2, 0);
  for (int n = 1; n <= kMaxN; ++n) {
    q y[kMaxN], W[kMaxN], x[kMaxN], w[kMaxN];
    asym_base(n, y, W);
    for (int i = 0; i < n; ++i) { asy_y.push_back((double)y[i]); asy_w.push_back((double)W[i]); }
    // smallest integer Ta with relative agreement for all sampled T >= Ta
    int Ta = 0;
    for (int T0 = 200; T0 >= 1; --T0) {
      bool ok = true;
      for (int s = 0; s < 8 && ok; ++s) {
        q T = T0 + s * 0.125Q;
        exact_rule(n, T, x, w);
        for (int i = 0; i < n; ++i) {
          q xa = y[i] / T, wa = W[i] / sqrtq(T);
          if (fabsq(xa - x[i]) > tol * x[i] || fabsq(wa - w[i]) > tol * w[i]) ok = false;
        }
      }
      if (!ok) { Ta = T0 + 1; break; }
    }
    tasym[n] = Ta;
    const int deg = deg_of(n), np = deg + 1, nint = Ta * per_unit(n);
    const double width = 1.0 / per_unit(n);
    offset[n] = int(coef.size());
    for (int k = 0; k < nint; ++k) {
      const double t0 = k * width;
      // Chebyshev interpolation at deg+1 Chebyshev points of the 1st kind
      std::vector<q> vals(size_t(np) * 2 * n);
      for (int j = 0; j < np; ++j) {
        q th = M_PIq * (j + 0.5Q) / np;
        q xx = cosq(th);
        q T = t0 + (xx + 1) * 0.5Q * width;
        exact_rule(n, T, x, w);
        for (int i = 0; i < n; ++i) {
          vals[size_t(j) * 2 * n + i] = x[i];
          vals[size_t(j) * 2 * n + n + i] = w[i];
        }
      }
      for (int f = 0; f < 2 * n; ++f) {
        std::vector<q> c(np);
        for (int m = 0; m <= deg; ++m) {
          q s = 0;
          for (int j = 0; j < np; ++j)
            s += vals[size_t(j) * 2 * n + f] * cosq(m * M_PIq * (j + 0.5Q) / np);
          c[m] = s * (m == 0 ? 1.0Q : 2.0Q) / np;
        }
        for (q v : to_powers(c)) coef.push_back((double)v);
      }
    }
    // accuracy report on a dense grid
    double worst = 0;
    for (int k = 0; k < nint; ++k)
      for (int s = 0; s < 23; ++s) {
        const double T = k * width + (s + 0.37) / 23.0 * width;
        exact_rule(n, T, x, w);
        const double* c = &coef[offset[n] + size_t(k) * 2 * n * np];
        const double xx = 2 * (T - k * width) / width - 1;
        for (int f = 0; f < 2 * n; ++f) {
          const q ex = f < n ? x[f] : w[f - n];
          worst = std::fmax(worst, (double)fabsq((horner(c + f * np, deg, xx) - ex) / ex));
        }
      }
    fprintf(stderr, "n=%d Tasym=%d intervals=%d degree=%d worst rel err %.3e\n", n, Ta, nint, deg, worst);
  }
  offset[kMaxN + 1] = int(coef.size());
  FILE* f = fopen(argv[1], "w");
  fprintf(f, "// Generated by gen_rys_tables.cpp (binary128 Rys rules, piecewise polynomials). Do not edit.\n");
  fprintf(f, "#define RYS_TAB_MAXN %d\n", kMaxN);
  fprintf(f, "#ifndef RYS_TAB_QUAL\n#define RYS_TAB_QUAL static const\n#endif\n#ifndef RYS_TAB_ALIGN\n#define RYS_TAB_ALIGN\n#endif\n");
  fprintf(f, "#define RYS_TAB_TASYM {0");
  for (int n = 1; n <= kMaxN; ++n) fprintf(f, ", %d", tasym[n]);
  fprintf(f, "}\n#define RYS_TAB_NCOEF {0");
  for (int n = 1; n <= kMaxN; ++n) fprintf(f, ", %d", deg_of(n) + 1);
  fprintf(f, "}\n#define RYS_TAB_PER_UNIT {0");
  for (int n = 1; n <= kMaxN; ++n) fprintf(f, ", %d", per_unit(n));
  fprintf(f, "}\n");
  fprintf(f, "RYS_TAB_QUAL int kRysOffset[%d] = {0", kMaxN + 2);
  for (int n = 1; n <= kMaxN + 1; ++n) fprintf(f, ", %d", offset[n]);
  fprintf(f, "};\n// large-T rule per n (n entries each, n = 1..%d concatenated)\n", kMaxN);
  fprintf(f, "RYS_TAB_QUAL double kRysAsymRoot[%zu] = {\n", asy_y.size());
  for (double v : asy_y) fprintf(f, "  %.17e,\n", v);
  fprintf(f, "};\nRYS_TAB_QUAL double kRysAsymWeight[%zu] = {\n", asy_w.size());
  for (double v : asy_w) fprintf(f, "  %.17e,\n", v);
  fprintf(f, "};\n// [n][interval][root 0..n-1, weight 0..n-1][power of x, 0..NCOEF-1]\n");
  fprintf(f, "RYS_TAB_ALIGN RYS_TAB_QUAL double kRysPoly[%zu] = {\n", coef.size());
  for (size_t i = 0; i < coef.size(); ++i) fprintf(f, "%.17e,%s", coef[i], (i % 4 == 3) ? "\n" : " ");
  fprintf(f, "};\n");
  // Boys functions: [m][interval][power of x]
  std::vector<double> boys;
  double worst = 0;
  for (int m = 0; m <= kMaxBoys; ++m)
    for (int k = 0; k < kBoysT * kBoysPerUnit; ++k) {
      const int np = kBoysDeg + 1;
      const double width = 1.0 / kBoysPerUnit;
      q F[kMaxBoys + 1];
      std::vector<q> v(np), c(np);
      for (int j = 0; j < np; ++j) {
        boys_q(m, k * width + (cosq(M_PIq * (j + 0.5Q) / np) + 1) * 0.5Q * width, F);
        v[j] = F[m];
      }
      for (int i = 0; i < np; ++i) {
        q t = 0;
        for (int j = 0; j < np; ++j) t += v[j] * cosq(i * M_PIq * (j + 0.5Q) / np);
        c[i] = t * (i == 0 ? 1.0Q : 2.0Q) / np;
      }
      for (q t : to_powers(c)) boys.push_back((double)t);
      for (int i = 0; i < 11; ++i) {
        const double T = (k + (i + 0.37) / 11.0) * width, xx = 2 * (T - k * width) / width - 1;
        boys_q(m, T, F);
        worst = std::fmax(worst, (double)fabsq((horner(&boys[boys.size() - np], kBoysDeg, xx) - F[m]) / F[m]));
      }
    }
  fprintf(stderr, "Boys F_0..F_%d: worst rel err %.3e\n", kMaxBoys, worst);
  fprintf(f, "#define BOYS_TAB_MAXM %d\n#define BOYS_TAB_T %d\n#define BOYS_TAB_NCOEF %d\n#define BOYS_TAB_PER_UNIT %d\n",
          kMaxBoys, kBoysT, kBoysDeg + 1, kBoysPerUnit);
  fprintf(f, "// [order m][interval][power of x, 0..NCOEF-1]\n");
  fprintf(f, "RYS_TAB_ALIGN RYS_TAB_QUAL double kBoysPoly[%zu] = {\n", boys.size());
  for (size_t i = 0; i < boys.size(); ++i) fprintf(f, "%.17e,%s", boys[i], (i % 4 == 3) ? "\n" : " ");
  fprintf(f, "};\n");
  fclose(f);
  return 0;
}
