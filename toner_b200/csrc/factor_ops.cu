// Factor engine: inverse p-th roots of damped, trace-normalised input statistics by a coupled Newton
// iteration with minimax scaling, every product on the tcgen05 GEMM in FP32-accurate split precision.
//
//   A   = sym(C) / mean(diag C) + damping * I                 (what the reference factors by eigh)
//   A'  = A - (lambda_1 - c) v v^T                            (dominant direction deflated when power iteration finds it)
//   M_0 = A' / beta,  beta >= lambda_max(A')                  (beta = min(||A'||_F, 1.04 ||A'||_F ||P^2||_F^(1/2)), P = A'/||A'||_F)
//   T_k = a_k I - b_k M_k ;  X_{k+1} = X_k T_k ;  M_{k+1} = T_k^p M_k          (X_0 = I)
//   X_K = X_{K-1} (c0 I + c1 R + c2 R^2 + ... ),  R = I - M_{K-1}               (Chebyshev fit of (1 - r)^(-1/p))
//   X_K ~ M_0^{-1/p}  =>  A^{-1/p} = X_K beta^{-1/p} + (lambda_1^{-1/p} - c^{-1/p}) v v^T
// (a_k, b_k) map the interval [l_k, 1] known to contain the spectrum of M_k onto [l_{k+1}, 1] with
// l_{k+1} as large as a linear T allows (the ends of the interval and the interior maximum of
// mu (a - b mu)^p are levelled, subject to a cap on b/a that bounds the dynamic range of T^p); once
// l_k is close to 1 they become the Newton values ((p+1)/p, 1/p).
// l_0 is the caller's lower bound of the spectrum of M_0 (checked per statistic on the device), or
// damping / (n (1 + damping)), which always holds; the schedule and the iteration count depend only on
// (l_0, p), so they are fixed before anything is launched and stated by toner_inv_roots_iterations[_for].
// Every operand of every product is a pair of FP16 hi/lo planes written by the epilogue of the product that
// made it, scaled by a power of two taken from a norm bound known in advance.
#include <cmath>
#include <cstdlib>
#include <unordered_map>
#include <vector>

#include "root_steps.cuh"
#include "runtime.cuh"

namespace toner {

// Dynamic range allowed for T^p.  The unconstrained minimax step sends the top of the spectrum (mu = 1)
// down to the new lower bound, i.e. T = a I - b M gets an eigenvalue (a - b) << a and T^p spans
// (a / (a - b))^p; a component that small relative to ||T^p|| is lost in operand rounding and can come
// out negative, after which the iteration diverges.  Capping b / a keeps every eigen-component of T^p
// above 1e-3 of its norm, at the price of one more iteration.
constexpr double kMaxPowerRange = 1e3;

// Minimax-scaled schedule; returns the steps and the final lower bound of the spectrum.
static std::vector<NewtonStep> newton_schedule(double l0, int p, int iters, double* lower_out) {
  std::vector<NewtonStep> out;
  const double max_ratio = 1.0 - std::pow(kMaxPowerRange, -1.0 / p);
  double l = l0;
  for (int k = 0; k < iters; ++k) {
    NewtonStep s;
    s.lower = l;
    const double r = std::pow(l, 1.0 / p);
    double ratio = (l < 1.0 - 1e-9) ? (1.0 - r) / (1.0 - r * l) : 0.0;  // b/a levelling f(l) = f(1)
    if (ratio > max_ratio) ratio = max_ratio;
    const double mu_star = ratio > 0 ? 1.0 / (ratio * (p + 1)) : 2.0;   // interior maximum of f
    if (mu_star < 1.0 && mu_star > l) {
      const double fmax = mu_star * std::pow((double)p / (p + 1), p);    // with a = 1
      const double f_low = l * std::pow(1.0 - ratio * l, p), f_top = std::pow(1.0 - ratio, p);
      s.a = std::pow(fmax, -1.0 / p);                                    // rescale so that max f = 1
      s.b = s.a * ratio;
      l = (f_low < f_top ? f_low : f_top) / fmax;
    } else {
      s.a = (p + 1.0) / p;
      s.b = 1.0 / p;
      l = l * std::pow((p + 1.0 - l) / p, p);
    }
    if (l > 1.0) l = 1.0;
    out.push_back(s);
  }
  if (lower_out) *lower_out = l;
  return out;
}

// k-blocks (64 deep) per tensor-core accumulation chain for the products that update M, given the lower
// bound of M's spectrum (0 = one chain over the whole product, the fastest kernel).  Truncation costs about
// 1.2e-7 per k-block on same-sign sums, i.e. up to 1e-5 over a whole product of depth 5632; the damage to the
// result is that divided by the smallest eigenvalue of M.
static int chain_length(double lower) {
  if (lower < 5e-3) return kPromoteAccurate;
  if (lower < 5e-2) return kPromoteLinear;
  return 0;
}

// The same after steps of higher degree.  Fewer products and these chains leave the roots 0.30 to 0.46 times as far from FP64 as linear
// steps do (means of 467 calls, p = 4, 8, 16: rows of 0.1 to 6 a column, log-uniform spectra of condition 30 to 1e6, widths 264 to 2048, bounds
// from the one that always holds to the spectrum's end), 0.97 times in the worst.  Without the rank-deficient ones, of 540 calls: 0.4 in the median
// and 1.06 in the worst; two k-blocks below 5e-3: 1.6 times in the worst, below 5e-4: 1.7; eight from 5e-2 on, as the linear steps have: 1.7.
// (12 products of 3072: 790 us in one chain, 920 in chains of eight k-blocks, 980 of two, 1000 to 1150 of one.)
static int steep_chain_length(double lower) {
  if (lower < 5e-3) return 1;
  if (lower < 0.5) return kPromoteAccurate;
  return 0;
}
// Products with X, and the final squarings, which in one chain would be 8 times as far off in the worst case: their one-sided
// truncation no longer cancels part of the iteration's.
constexpr int kPromoteSteepX = 2, kPromoteSteepSquares = 1;

// Products applied to X (and the final squarings) pass their error on linearly: one chain, about 1e-5.
constexpr int kPromoteX = 0;

constexpr long long kHalfFrom = 4 << 20;   // elements of a stack of statistics from which operand planes are stored by half

// power-iteration steps spent on the dominant direction (each one pass over the statistic)
constexpr int kPowerSteps = 6;

// The last step does not square the error once more; it finishes with a polynomial q(R) ~ (I - R)^(-1/p), R = I - M:
// X <- X q(R).  The spectrum of R lies in [0, e] with e known from the schedule, so q is fixed in advance: the
// Chebyshev interpolant of (1 - r)^(-1/p) on [kFinishLow, kFinishGrow e + kFinishPad] (the margins cover rounding
// at the lower end and the allowance an estimated bound is verified with at the upper end) of the smallest degree
// whose relative error stays below kFinishTail there.  Spreading the error over the interval takes about half
// the degree of the binomial series, whose error sits at r = e alone (e = 0.5, p = 8: degree 6 instead of 12).
// The powers come from single-pass products of FP16 planes (a third of a split-precision product each; R is small, so its
// rounding to FP16 costs about 5e-4 c_2 e^2), m - 1 in Horner form and about half as many in steps of R (R + beta I) where
// quadratic_steps() allows them.  Either is cheaper than the log2(p) + 2 split-precision products of one more Newton step; the
// step count is the one with the fewest plane passes in total, Horner's counted.
constexpr double kFinishRadius = 0.6;
constexpr int kMaxFinishOrder = 12;
constexpr double kFinishTail = 3e-6;
constexpr double kFinishLow = -0.02, kFinishGrow = 1.15, kFinishPad = 1e-3;

struct FinishPoly {
  int order = 0;                       // 0: no degree up to the cap reaches the bound at this distance
  double c[kMaxFinishOrder + 1] = {};  // q(r) = sum_j c[j] r^j
  double reach = 0.0;                  // upper end of the interval it is fitted to (0: not fitted)
};
// Entries of I - M above this before the finish: not converged.  No entry of a symmetric matrix exceeds its norm, and up to where the
// finish is fitted to, the schedule's e with its margin, the root is right; a hundredth more for rounding.  At least 0.5, which M that
// diverges goes far beyond.  (0.5 whatever e flagged right roots: 768 columns in plane order, p = 4, nothing known, end at e = 0.527.)
static float converged_within(const FinishPoly& f) { return (float)std::max(0.5, f.reach + 0.01); }

// (1 - r)^(1/p) at the points where a fit is checked; a point is evaluated when a fit first gets that far.
struct FitSamples {
  static constexpr int kPoints = 257;
  double g[kPoints];
  int known = 0;
  double at(int i, int p, double lo, double hi) {
    for (; known <= i; ++known) g[known] = std::pow(1.0 - (lo + (hi - lo) * known / (kPoints - 1)), 1.0 / p);
    return g[i];
  }
};

// Degree-m Chebyshev interpolant of (1 - r)^(-1/p) on [lo, hi] as monomial coefficients; whether its largest relative
// error on the interval is below `tail`.
static bool finish_fit(int p, double lo, double hi, int m, double tail, FitSamples& samples, double* c) {
  const double kPi = 3.14159265358979323846;
  double cheb[kMaxFinishOrder + 1] = {};
  for (int k = 0; k <= m; ++k) {
    const double th = kPi * (k + 0.5) / (m + 1);
    const double r = lo + (hi - lo) * (std::cos(th) + 1.0) * 0.5;
    const double f = std::pow(1.0 - r, -1.0 / p);
    for (int j = 0; j <= m; ++j) cheb[j] += f * std::cos(j * th);
  }
  for (int j = 0; j <= m; ++j) cheb[j] *= (j == 0 ? 1.0 : 2.0) / (m + 1);
  // sum_j cheb[j] T_j(x) in powers of x (T_{j+1} = 2 x T_j - T_{j-1}) ...
  double t0[kMaxFinishOrder + 1] = {1.0}, t1[kMaxFinishOrder + 1] = {0.0, 1.0}, px[kMaxFinishOrder + 1] = {};
  px[0] = cheb[0];
  for (int i = 0; i <= m; ++i) px[i] += (m >= 1 ? cheb[1] : 0.0) * t1[i];
  for (int j = 2; j <= m; ++j) {
    double t2[kMaxFinishOrder + 1] = {};
    for (int i = 0; i <= m; ++i) t2[i] = (i > 0 ? 2.0 * t1[i - 1] : 0.0) - t0[i];
    for (int i = 0; i <= m; ++i) {
      px[i] += cheb[j] * t2[i];
      t0[i] = t1[i];
      t1[i] = t2[i];
    }
  }
  // ... then in powers of r, x = alpha r + beta (Horner over the polynomial in x)
  const double alpha = 2.0 / (hi - lo), beta = -(hi + lo) / (hi - lo);
  for (int i = 0; i <= m; ++i) c[i] = 0.0;
  for (int j = m; j >= 0; --j) {
    for (int i = m; i >= 1; --i) c[i] = c[i] * beta + c[i - 1] * alpha;
    c[0] = c[0] * beta + px[j];
  }
  for (int i = 0; i < FitSamples::kPoints; ++i) {
    const double r = lo + (hi - lo) * i / (FitSamples::kPoints - 1);
    double q = 0.0;
    for (int j = m; j >= 0; --j) q = q * r + c[j];
    if (!(std::fabs(q * samples.at(i, p, lo, hi) - 1.0) < tail)) return false;
  }
  return true;
}

// q(r) of degree m in half of Horner's m - 1 products, and about one: repeated division of an even-degree polynomial by
// y = r (r + beta) leaves (..(w y + l_1(r)) y + ..) y + l_k(r) with linear l_i, which cost no product (they enter it in FP32);
// beta is chosen so that the innermost quotient is affine in y itself, top y + top0.  m = 6: q itself, three products for five.
// m odd: q = c_0 + c_1 r + r v(r) with v of degree m - 1 divided so (m = 7: four products for six).  What the single planes
// (11 bits) of the products lose shows in the roots as follows, short form against Horner's, error against FP64 of statistics
// of width 768 and 1024 (Marchenko-Pastur spectra of 1.2 to 36 rows a column, log-uniform ones of condition 10 to 1e3): m = 6
// 0.92 to 1.02 for p = 4 and 8 but up to 1.25 for p = 2, which keeps Horner's rule; m = 7 0.83 to 1.00; m = 5 1.00 from p = 8
// on, 1.05 below, where it keeps Horner's rule too.  m = 8 (rare: p = 8, a lower bound near 5e-4, 6.5e-3, 0.069) reaches 1.18 and
// keeps it as well, like any other even degree; q itself divided with m = 7, or m = 4, reaches 1.7: near r = 0, where most
// eigenvalues are, an error must fall with r^2 as Horner's does.  32 statistics of width 2048, m = 7: two products of 350 us
// each go.
struct QuadraticSteps {
  double beta = 0.0, top = 0.0, top0 = 0.0;
  bool by_r = false;                            // a last step by r (m odd)
  std::vector<std::pair<double, double>> lin;   // (linear, constant) of every division, the outermost first
};
static bool quadratic_steps(const FinishPoly& fin, int p, QuadraticSteps& out) {
  const int m = fin.order;
  if ((m & 1) != 0 ? (m < 5 || (m == 5 && p < 8)) : (m != 6 || p < 4)) return false;
  out.by_r = (m & 1) != 0;
  int deg = out.by_r ? m - 1 : m;
  double q[kMaxFinishOrder + 1];
  for (int j = 0; j <= deg; ++j) q[j] = !out.by_r ? fin.c[j] : (j == 0 ? 0.0 : fin.c[j + 1]);
  const double beta = q[deg - 1] / ((deg / 2) * q[deg]);
  if (!(q[deg] > 0.0 && std::fabs(beta) < 1.0)) return false;
  out.beta = beta;
  for (; deg > 2; deg -= 2) {
    for (int j = deg; j >= 2; --j) q[j - 1] -= beta * q[j];   // q[j] is now the quotient's coefficient of r^(j-2)
    out.lin.emplace_back(q[1], q[0]);
    for (int j = 0; j <= deg - 2; ++j) q[j] = q[j + 2];
  }
  out.top = q[2];
  out.top0 = q[0];
  return true;
}

// In powers of r the fit's coefficients grow as the interval approaches the singularity at r = 1 (sooner for small p):
// sums with cancellation, which single-pass FP16 products would not survive and whose Horner intermediates
// W_j = sum_{k >= j} c_k r^(k-j+1) would leave the range the operand planes are scaled for.  Such a fit is not used.
constexpr double kFinishMaxCond = 2.5;   // sum_k |c_k| hi^k, against q(r) <= 1.8
constexpr double kFinishMaxTerm = 3.5;   // bound of every W_j (planes hold |x| <= 4)

static bool finish_usable(const FinishPoly& f, double hi) {
  double cond = 0.0;
  for (int k = f.order; k >= 0; --k) cond = cond * hi + std::fabs(f.c[k]);   // Horner of sum |c_k| hi^k
  if (cond > kFinishMaxCond) return false;
  double w = 0.0;
  for (int j = f.order; j >= 1; --j) {
    w = (w + std::fabs(f.c[j])) * hi;
    if (w > kFinishMaxTerm) return false;
  }
  return true;
}

static FinishPoly finish_poly(int p, double e, double grow = kFinishGrow, double radius = kFinishRadius) {
  FinishPoly f;
  if (!(e < radius)) return f;
  const double hi = grow * e + kFinishPad;
  FitSamples samples;
  for (int m = 2; m <= kMaxFinishOrder; ++m) {
    if (finish_fit(p, kFinishLow, hi, m, kFinishTail, samples, f.c)) {
      f.order = m;
      if (!finish_usable(f, hi)) return FinishPoly();
      f.reach = hi;
      return f;
    }
  }
  return f;
}
static int finish_order_or_zero(int p, double e) { return finish_poly(p, e).order; }
// A caller's own (too small) step count leaves M too far from I for a usable fit: the binomial series of
// (1 - r)^(-1/p) at the cap (all coefficients positive and below 1); status reports the statistic.
static FinishPoly finish_poly_or_best(int p, double e) {
  FinishPoly f = finish_poly(p, e);
  if (f.order) return f;
  f.order = kMaxFinishOrder;
  f.c[0] = 1.0;
  for (int j = 1; j <= kMaxFinishOrder; ++j) f.c[j] = f.c[j - 1] * (1.0 / p + j - 1) / j;
  return f;
}
static int default_iterations(double l0, int p) {
  // k steps of M, then the finishing step on X alone: the k with the fewest plane passes,
  // 3 (log2 p + 2) per step of M and order - 1 for the series, among those the series can finish
  int log2p = 0;
  while ((1 << log2p) < p) ++log2p;
  int best = 0;
  long best_cost = 0;
  for (int k = 1; k < 64; ++k) {
    double l;
    newton_schedule(l0, p, k, &l);
    const double e = 1.0 - l;
    const int m = finish_order_or_zero(p, e);
    if (m) {
      const long cost = 3L * k * (log2p + 2) + (m - 1);
      if (!best || cost < best_cost) {
        best = k + 1;
        best_cost = cost;
      }
      if (m == 2) break;  // further steps only add cost
    }
  }
  return best ? best : 64;
}

// The graded finish: where the spectrum of M reaches further down than a polynomial in R = I - M can follow, q(M) ~ M^(-1/p) is
// written in Z, M mapped from [lo, hi] onto [-1, 1], and U = 2 Z^2 - I = T_2(Z):  a Chebyshev interpolant of odd degree
// m = 2 K + 1 is  sum_j (alpha_j I + beta_j Z) U^j,  Horner's rule in U takes K products, and the coefficients fall like the
// square of the interpolant's rate (1/6 a power and less), so only what is near the front needs both planes: U itself and
// the last product or two, three plane products each; those before are single passes.  An M that reaches down to 0.1 takes
// K = 7 and no Newton step, where each is five split products and more.  It is used on M_0 alone, where the lower bound is an
// estimate that is verified afterwards (Marchenko-Pastur spectra of three rows a column and more): after Newton steps it was
// less accurate than another step (two steps, 3328 wide, A^(-1/8) 4.8e-6 -> 2.3e-5 against FP64; one, 2048 wide, 3.3e-6 -> 9.5e-6),
// because what the steps have left in M is divided by the smallest eigenvalue the finish starts from.
// Error against FP64, Newton's finish / graded, of A^(-1/8) and A^(-1/2), means of nine:
//   384 wide, 3073 rows 3.6e-6 / 1.6e-6, 4.0e-6 / 3.7e-6;   768, 4609 rows 6.5e-6 / 0.6e-6, 6.1e-6 / 3.2e-6;
//   768, 18433 rows 8.3e-6 / 0.7e-6, 1.2e-5 / 3.6e-6;   2048, 12289 rows 1.7e-5 / 1.0e-6, 1.3e-5 / 5.0e-6;   3072, 73216 rows
//   2.4e-5 / 0.7e-6, 2.0e-5 / 3.4e-6.  24 statistics of 2048, condition 2 / 3 / 5: 6150 / 6310 / 6530 -> 5040 / 5570 / 6120 us.
constexpr int kMaxGraded = 12;    // K
// How much of A^(-1/p) the finish may lose, by width: Newton's finish loses less on narrow statistics (A^(-1/2) 2.7e-6 at 264
// columns, 6e-6 at 768, 1.1e-5 at 1280), and so may this one.
//   single: W_(j+1) at most this part of W_0, and W_j is a single pass (11 bits of it).  1.5 % at every width: A^(-1/2) up to 1.4
//           times as far from FP64 as after Newton's finish at 512 columns, 1.16 at 1024, at most 0.95 from 1288 on.  0.5 % at
//           every width: 24 statistics of 2048, condition 2 and 3, 5040 and 5570 -> 5280 and 5890 us.
//   tail:   the interpolant's remainder.  3e-6 at 264 columns, squarings in chains of two: A^(-1/2) up to 2.3 times as far as after
//           Newton's finish, with 1e-6 and chains of one 0.8 to 1.02 times.  The product that it takes is 0 to 1 % of a call at 264
//           and 512 columns, 5 % from 768 on.
struct GradedCare {
  double single, tail;
};
static GradedCare graded_care(int n) {
  if (n < 640) return {0.005, 1e-6};
  if (n < 1280) return {0.005, 3e-6};
  return {0.015, 3e-6};
}
constexpr double kGradedTail = 3e-6;   // (at any width)
// Allowed of I - A^(-1/2) A A^(-1/2) where a bound was an estimate, beside p times the interpolant's remainder: p = 8 accepts 3.4e-5
// of A^(-1/8) on one eigenvector, as large as Newton's finish left by itself (1e-5 to 1e-4), and an eigenvalue down to 0.85
// of the bound; 9e-5 is the most that was seen of statistics the bound held for.
constexpr double kGradedResidual = 2.5e-4;
constexpr double kGradedHigh = 1.02, kGradedLow = 0.97;   // margins for rounding
struct GradedPoly {
  int products = 0;               // K; 0: none
  int split = 0;                  // W_j with 1 <= j <= split are split products as well
  double lo = 0.0;
  double za = 0.0, zb = 0.0;      // Z = zb I + za M
  double alpha[kMaxGraded + 1] = {}, beta[kMaxGraded + 1] = {};
  double bound[kMaxGraded + 1] = {};   // of W_j = sum_{i >= j} (alpha_i + beta_i z) U^(i-j)
};

// (A tracked call asks for this with a new lower end every step: one expansion of the function, 64 powers, serves every
// degree, and nothing is fitted again.)
static GradedPoly graded_poly(int p, double lo, const GradedCare& care) {
  constexpr int kNodes = 64, kTerms = 40, kPoints = 65;
  struct Cosines {
    double at[kTerms][kNodes];       // T_j at the Chebyshev nodes
    double z[kPoints];               // where the sums are bounded
    Cosines() {
      const double kPi = 3.14159265358979323846;
      for (int j = 0; j < kTerms; ++j)
        for (int k = 0; k < kNodes; ++k) at[j][k] = std::cos(j * kPi * (k + 0.5) / kNodes);
      for (int i = 0; i < kPoints; ++i) z[i] = std::cos(kPi * i / (kPoints - 1));
    }
  };
  static const Cosines cosines;
  const double hi = kGradedHigh;
  double f[kNodes], c[kTerms], tail = 0.0;
  for (int k = 0; k < kNodes; ++k) f[k] = std::pow(0.5 * (hi + lo) + 0.5 * (hi - lo) * cosines.at[1][k], -1.0 / p);
  for (int j = 0; j < kTerms; ++j) {
    c[j] = 0.0;
    for (int k = 0; k < kNodes; ++k) c[j] += f[k] * cosines.at[j][k];
    c[j] *= (j == 0 ? 1.0 : 2.0) / kNodes;
  }
  // the smallest odd degree 2 K + 1 whose remainder stays below the bound; the function is above hi^(-1/p) everywhere
  GradedPoly g;
  int K = kTerms / 2;
  const double most = care.tail * std::pow(hi, -1.0 / p);
  for (; K > 2; --K) {
    const double more = tail + (2 * K + 1 < kTerms ? std::fabs(c[2 * K + 1]) : 0.0) + (2 * K < kTerms ? std::fabs(c[2 * K]) : 0.0);
    if (more > most) break;
    tail = more;
  }
  if (K > kMaxGraded) return g;
  // T_{2j}(z) = T_j(U),  T_{2j+1}(z) = z V_j(U) with V_0 = 1, V_1 = 2 U - 1, V_{j+1} = 2 U V_j - V_{j-1}
  double t0[kMaxGraded + 1] = {1.0}, t1[kMaxGraded + 1] = {0.0, 1.0}, v0[kMaxGraded + 1] = {1.0}, v1[kMaxGraded + 1] = {-1.0, 2.0};
  for (int j = 0; j <= K; ++j) {
    for (int i = 0; i <= K; ++i) {
      g.alpha[i] += c[2 * j] * t0[i];
      g.beta[i] += c[2 * j + 1] * v0[i];
    }
    for (int i = K; i >= 0; --i) {   // (t0, t1) <- (t1, 2 U t1 - t0), and v likewise; from above, so that t1[i - 1] is still old
      const double t2 = (i > 0 ? 2.0 * t1[i - 1] : 0.0) - t0[i], v2 = (i > 0 ? 2.0 * v1[i - 1] : 0.0) - v0[i];
      t0[i] = t1[i];
      v0[i] = v1[i];
      t1[i] = t2;
      v1[i] = v2;
    }
  }
  for (int i = 0; i < kPoints; ++i) {
    const double z = cosines.z[i], u = 2.0 * z * z - 1.0;
    double w = 0.0;
    for (int j = K; j >= 0; --j) {
      w = g.alpha[j] + g.beta[j] * z + u * w;
      g.bound[j] = std::max(g.bound[j], 1.1 * std::fabs(w));
    }
  }
  while (g.split < K && g.bound[std::min(g.split + 2, K)] > care.single * g.bound[0]) ++g.split;
  if (g.split > K - 2 || !(std::fabs(g.beta[K]) > 1e-12)) return GradedPoly();   // (W_K has one plane)
  g.products = K;
  g.lo = lo;
  g.za = 2.0 / (hi - lo);
  g.zb = -(hi + lo) / (hi - lo);
  return g;
}

// Cost of a single pass in split products: 0.43 of one at width 3072, 0.5 at 2048, 0.77 at 768, where writing the results is most
// of it (interleaved products in batches; C and operand planes as the finish has them).
static double single_pass(int n) { return 0.35 + 320.0 / n; }

// What steps of higher degree are weighed with against linear ones: times in products of one chain of accumulations.  Products in
// chains of 8 / 2 / 1 k-blocks take 1.15 / 1.3 / 1.42 of one around 1000 columns (1.14 to 1.22, 1.18 to 1.43, 1.15 to 1.7 with 4 to 36 statistics),
// less below 800, where a launch is ever more of it (1.05 / 1.1 / 1.11 at 264), and on wide statistics (1.10 / 1.24 / 1.34 at 2048, 1.05 / 1.19 / 1.25 at 3072), a single
// pass at most 0.85, the FP32 matrix of a linear term 0.15: 1080 calls, each with steps and with linear ones.
struct StepCosts {
  double single, chained[3];   // (of chains of 8, of 2, of 1)
  explicit StepCosts(int n) : single(std::min(0.85, single_pass(n))) {
    const double share = std::min(1.0, n / 800.0) * std::min(1.0, std::sqrt(1280.0 / n));
    chained[0] = 1.0 + 0.15 * share;
    chained[1] = 1.0 + 0.3 * share;
    chained[2] = 1.0 + 0.42 * share;
  }
  double product(int chain) const { return chain == 0 ? 1.0 : chain == 1 ? chained[2] : chain == 2 ? chained[1] : chained[0]; }
};

// Newton steps of degree 1, 2 and 4 (root_steps.cuh) in the order that costs least.  Between steps the bound of M's spectrum is
// rounded down to an eighth of an octave: every schedule is then a path through 256 bounds, whose steps (0.1 ms of host
// time a bound to find) and finishing polynomials a thread keeps, and a bound that moves a little from call to call costs nothing.  Against
// exact bounds a step loses 4 % of l' on average.
// The last product of the finish is a split one: single passes lose 2^-12 e^2 of it, which linear steps' own errors cover and these
// would not (p = 8, e = 0.59: A^(-1/2) 2.5 times as far off as after linear steps without, 0.94 times with it).
constexpr int kBoundsPerOctave = 8, kBounds = 32 * kBoundsPerOctave;
// A certified bound needs no margin for an estimate's allowance, only for rounding (M_0's planes resolve 2^-25: 4e-4 of the smallest
// eigenvalue at a norm of 16, damping 1e-3), and so may end further from I.
constexpr double kCertifiedGrow = 1.04, kCertifiedRadius = 0.66;
// Products with T^p lose 2^-22 of its largest eigenvalue.  Where T is smallest, on the large eigenvalues of M, that is as much more
// of T^p as its range, and it mixes their eigenvectors with those of the small ones: errors that the Frobenius norm of an inverse
// root hardly shows and its norm weighted by the statistic itself does.  So weighted, A^(-q/p) was 1.55 times as far off as after
// linear steps in the worst (p = 8; 1.9 for p = 4, 4.4 for p = 2) with a range of 1e3, of 135 calls: rank-deficient statistics of 0.1 to
// 0.9 rows a column, full ones of 1.5 and 4, log-uniform ones of condition 1e2 to 1e6, 256 to 2048 wide, three bounds each.  With
// these 1.02, 0.58 and 0.84, and 0.6, 0.3 and 0.45 in the mean (p = 8, 4, 16); l' is a sixth smaller.  Narrower still for p = 8: 0.94 with
// 300, but a fourth step where nothing is known (roots of four 2048 columns wide 2.38 -> 3.44 ms; with 1e3 2.34).  Square roots keep linear
// steps: rank-deficient statistics' were 1.18 times as far off with 50.
static double step_range(int p) { return std::min(400.0, 6.25 * p * p); }
constexpr int kSteepFromPower = 4;
constexpr int kSteepFrom = 256;   // columns: on narrower statistics linear steps can be closer (by 2.8 times, of 8e-7, 8 wide)
struct BoundNode {
  bool ok[3] = {};
  NewtonStep step[3];
  FinishPoly fin[2][3];       // after that step, under an estimated and a certified bound; order 0: M is too far from I
  int fin_products[2][3] = {};
};
static double bound_of(int j) { return std::exp2(-(double)j / kBoundsPerOctave); }
static int bound_below(double l) { return std::max(1, (int)std::ceil(-kBoundsPerOctave * std::log2(l) - 1e-6)); }

static const BoundNode& bound_node(int p, int j) {
  static thread_local std::unordered_map<int, BoundNode> known;   // (at most kBounds for each of six p)
  const auto found = known.find(p * kBounds + j);
  if (found != known.end()) return found->second;
  BoundNode& node = known[p * kBounds + j];
  for (int i = 0; i < 3; ++i) {
    node.ok[i] = best_step(p, bound_of(j), kStepDegrees[i], i ? step_range(p) : kMaxPowerRange, node.step[i]);
    if (!node.ok[i]) continue;
    for (int c = 0; c < 2; ++c) {
      FinishPoly& fin = node.fin[c][i];
      fin = c ? finish_poly(p, 1.0 - node.step[i].next, kCertifiedGrow, kCertifiedRadius) : finish_poly(p, 1.0 - node.step[i].next);
      QuadraticSteps q;
      if (fin.order) node.fin_products[c][i] = quadratic_steps(fin, p, q) ? 1 + (int)q.lin.size() + (q.by_r ? 1 : 0) : fin.order - 1;
    }
  }
  return node;
}

struct StepPlan {
  double cost = 1e9;                // in split products, the finish and its product with X counted
  std::vector<std::pair<int, int>> path;   // (bound, degree's index)
};
// A step from bound j on: T's own products, its powers and M, and the next product with X; with a linear term an FP32 matrix is written
// and read more.
static double step_cost(const NewtonStep& s, int j, int log2p, const StepCosts& costs) {
  return (log2p + 1 + (s.degree == 4 ? 2 : s.degree - 1)) * costs.product(steep_chain_length(bound_of(j))) + (s.lin != 0.0 ? 0.15 : 0.0) +
         costs.product(kPromoteSteepX);
}
static const StepPlan& cheapest(int p, int j, bool certified, const StepCosts& costs, std::unordered_map<int, StepPlan>& memo, bool linear);
// Cheapest steps from bound j on, the first of degree two or four unless `linear`; `memo` is the call's own.
// Where the bound is an estimate so may the norm be, and M_0 may reach above 1.  A T of degree two or four sends what lies there
// further up, to where a linear T is negative; T^p is not, so M could come back to I with the sign of X turned and no check to see it
// (p = 8: degrees 4, 1 from a reach of 1.12).  So after a step of even degree, whose T is positive everywhere, only such steps follow:
// 0.5 split products more for 4 bounds in 400 at p = 4, none at p = 8 to 32.  Linear steps before them leave what linear ones alone leave
// (verified vectors below).
static StepPlan cheapest_first(int p, int j, bool certified, const StepCosts& costs, std::unordered_map<int, StepPlan>& memo, bool linear) {
  StepPlan best;
  const BoundNode& node = bound_node(p, j);
  int log2p = 0;
  while ((1 << log2p) < p) ++log2p;
  for (int i = 2; i >= (linear ? 0 : 1); --i) {
    if (!node.ok[i]) continue;
    const double own = step_cost(node.step[i], j, log2p, costs);
    const double end = costs.single * (node.fin_products[certified][i] - 1) + 1.0;
    if (node.fin[certified][i].order && own + end < best.cost) {
      best.cost = own + end;
      best.path = {{j, i}};
    }
    const int next = bound_below(node.step[i].next);
    if (next >= j || node.step[i].next > 0.9 || own + log2p + 2 >= best.cost) continue;
    const StepPlan& rest = cheapest(p, next, certified, costs, memo, certified || i == 0);
    if (own + rest.cost < best.cost) {
      best.cost = own + rest.cost;
      best.path = {{j, i}};
      best.path.insert(best.path.end(), rest.path.begin(), rest.path.end());
    }
  }
  return best;
}
static const StepPlan& cheapest(int p, int j, bool certified, const StepCosts& costs, std::unordered_map<int, StepPlan>& memo, bool linear) {
  const int key = linear ? j : -j;
  const auto found = memo.find(key);
  if (found != memo.end()) return found->second;
  return memo[key] = cheapest_first(p, j, certified, costs, memo, linear);
}

// Everything a call runs for a lower bound l0: the steps, the distance of the last M from I, the finishing polynomial.
// Working it out takes tens of microseconds of host time and is asked for several times per factorisation (the call itself,
// the step count and the degree it states), so a thread keeps the last few.
struct Schedule {
  double l0 = 0.0;
  int p = 0, asked = 0;   // asked: the caller's step count, 0 = the one with the fewest plane passes; -n: graded
                          // finishes considered as well, for statistics of width n
  int steep_n = 0;        // > 0: steps of higher degree considered as well, for statistics of that width
  int kind = 0;           // for these: the bound is an estimate (0), certified (1), the one that always holds (2)
  bool steep = false;     // ... and taken: cheaper than linear ones
  double late = 0.0;      // > 0: a statistic whose spectrum is above this starts with the second step
  int iters = 0;
  std::vector<NewtonStep> steps;
  double l_last = 0.0;    // lower bound of the spectrum of the last M, i.e. after iters - 1 updates
  FinishPoly fin;
  GradedPoly graded;      // graded.products > 0: this finish, of M_0 itself (iters == 1)
};

static const Schedule& schedule_for(double l0, int p, int iters, int grade_n = 0, int steep_n = 0,
                                    int kind = 0) {
  constexpr int kKept = 8;
  static thread_local Schedule kept[kKept];
  static thread_local int oldest = 0;
  iters = iters > 0 ? iters : -grade_n;
  for (const Schedule& s : kept)
    if (s.p == p && s.l0 == l0 && s.asked == iters && s.steep_n == steep_n && s.kind == kind) return s;
  Schedule& s = kept[oldest];
  oldest = (oldest + 1) % kKept;
  s.p = 0;   // (not a match until it is complete)
  s.l0 = l0;
  s.asked = iters;
  s.steep_n = steep_n;
  s.kind = kind;
  s.steep = false;
  s.late = 0.0;
  s.iters = iters > 0 ? iters : default_iterations(l0, p);
  if (s.iters >= 2) {
    s.steps = newton_schedule(l0, p, s.iters, nullptr);
    newton_schedule(l0, p, s.iters - 1, &s.l_last);
    s.fin = finish_poly_or_best(p, 1.0 - s.l_last);
  }
  s.graded = GradedPoly();
  if (iters < 0) {
    const int n = grade_n;
    // Costs in split products.  The final squarings, in short chains after a graded finish, take a tenth more at width 3072 and a
    // third at 768.  k linear updates of M are k (log2 p + 1) split products and k - 1 products with X; Newton's finish ends in one
    // with X, the graded one makes U and the root.  (Against steps of higher degree, which take fewer products, the graded finish
    // stays where it is the cheaper one of these two: it is ten times closer to the root.)
    int log2p = 0;
    while ((1 << log2p) < p) ++log2p;
    const double single = single_pass(n), squarings = (log2p - 1) * (0.05 + 250.0 / n);
    QuadraticSteps q;
    const double newton = (s.iters - 1) * (log2p + 2) +
                          single * (quadratic_steps(s.fin, p, q) ? 1 + (int)q.lin.size() + (q.by_r ? 1 : 0) : s.fin.order - 1);
    const GradedPoly g = graded_poly(p, kGradedLow * l0, graded_care(n));
    if (g.products && 2 + squarings + g.split + single * (g.products - 1 - g.split) < newton) {
      s.graded = g;
      s.iters = 1;
      s.steps = newton_schedule(l0, p, 1, nullptr);
      s.l_last = l0;
    }
  }
  const int first = steep_n >= kSteepFrom && iters <= 0 && !s.graded.products && p >= kSteepFromPower ? bound_below(l0) : kBounds;
  if (first < kBounds) {
    int log2p = 0;
    while ((1 << log2p) < p) ++log2p;
    const StepCosts costs(steep_n);
    QuadraticSteps q;
    double linear = costs.single * (quadratic_steps(s.fin, p, q) ? 1 + (int)q.lin.size() + (q.by_r ? 1 : 0) : s.fin.order - 1);
    for (int k = 0; k < s.iters - 1; ++k) linear += (log2p + 1) * costs.product(chain_length(s.steps[k].lower)) + 1.0;
    // (the squarings that follow, of 2 q = p: in one chain after linear steps)
    const double squarings = (p > 4 ? log2p - 1 : 0) * (costs.product(kPromoteSteepSquares) - 1.0);
    std::unordered_map<int, StepPlan> memo;
    StepPlan plan = cheapest(p, first, kind > 0, costs, memo, true);
    if (kind == 2) {
      // The bound that always holds, damping / n, is a norm of n; statistics have one of 1.4 to 16 (rows of synthetic.py, 512 to 5632
      // columns, up to four outliers deflated; 24 where 752 rows of 3072 columns are log-uniform to 1e6; more outliers than the block
      // holds leave hundreds), which the device knows before the first product.  So the first step goes from this bound to that of a norm of 16, damping / 16, or as far as it gets, and is
      // left out for every statistic whose norm allows it; the others follow as they would from there.
      const BoundNode& node = bound_node(p, first);
      const int norm16 = bound_below(l0 * steep_n / 16.0);
      for (int i = 1; i < 3 && norm16 < first - 2 * kBoundsPerOctave; ++i) {
        if (!node.ok[i]) continue;
        const int from = std::max(norm16, bound_below(node.step[i].next));
        if (from > norm16 && i < 2) continue;   // (degree four gets further)
        const StepPlan rest = cheapest_first(p, from, true, costs, memo, false);   // (a first T of degree one is no product's result)
        if (rest.path.empty()) break;
        // (What is left out is launched all the same, hence a tenth less at least.  Statistics of which none starts late pay for all: 0.80 to
        // 0.99 of the linear steps' time with norms of 95 to 1025, 264 to 3072 wide, p = 4 to 16, those that do 0.60 to 0.83; hence 5 % more allowed.)
        const double all = step_cost(node.step[i], first, log2p, costs) + rest.cost;
        if (rest.cost < 0.9 * plan.cost && all + squarings < 1.05 * linear) {
          s.late = bound_of(from);
          plan.cost = all;
          plan.path = {{first, i}};
          plan.path.insert(plan.path.end(), rest.path.begin(), rest.path.end());
        }
        break;
      }
    }
    // (Of 731 such calls -- p = 4, 8, 16, widths 264 to 3072, bounds from 5e-5 to 0.3 -- 44 then took more than 1 % longer than with linear
    // steps: 25 times a single statistic of 3072 columns, whose 78 tiles are two waves, by 16 % at most, the others by 7 %.  By product counts, 0.3
    // fewer wanted, 188 of 951 did, by 19 %.)
    if (!plan.path.empty() && (s.late > 0.0 || plan.cost + squarings < 0.98 * linear)) {
      s.steep = true;
      s.steps.clear();
      for (const auto& at : plan.path) s.steps.push_back(bound_node(p, at.first).step[at.second]);
      const auto& end = plan.path.back();
      s.l_last = s.steps.back().next;
      s.fin = bound_node(p, end.first).fin[kind > 0][end.second];
      s.iters = (int)s.steps.size() + 1;
      s.steps.push_back(s.steps.back());   // (the finish multiplies by none of them)
    }
  }
  s.p = p;
  return s;
}

// Directions that are deflated at most: four numbers a statistic and direction (Ritz value, residual, coefficients) lie this far apart.
constexpr int kMaxDeflate = 12;

// ------------------------------------------------------------------ elementwise helpers
__global__ void __launch_bounds__(256) trace_kernel(const float* __restrict__ c, int n, float* __restrict__ trace) {
  ptx::pdl_begin();
  const int b = blockIdx.x;
  const float* C = c + (long long)b * n * n;
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += C[(long long)i * n + i];
  __shared__ float red[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < 8; ++w) t += red[w];
    trace[b] = t;
  }
}

// A = sym(C) / max(trace/n, 1e-30) + damping I, written to `a`.
// 64 x 64 tile pairs, so that C and C^T are both read along rows, by 16-byte accesses with the whole pair (32 KB a block) on its
// way at once; blocks are numbered over the tiles of the upper triangle.  HBM bounds it: 32 statistics of width 2048 and 96 of 512
// 366 -> 227 us (with 32 x 32 tiles, 4-byte accesses and a block per tile of the square).  A statistic that does not start on 16
// bytes (a view into a larger buffer) is read by floats.
constexpr int kDampTile = 64;
template <bool kAligned>
__global__ void __launch_bounds__(256) damp_kernel(const float* __restrict__ c, float* __restrict__ a, int n, float damping,
                                                   const float* __restrict__ trace) {
  ptx::pdl_begin();
  __shared__ float up[kDampTile][kDampTile + 1], lo[kDampTile][kDampTile + 1];
  int ti = 0, rest = blockIdx.x;
  for (int row = (n + kDampTile - 1) / kDampTile; rest >= row; --row) {
    rest -= row;
    ++ti;
  }
  const int tj = ti + rest;
  const long long b = blockIdx.y;
  const float* C = c + b * (long long)n * n;
  float* A = a + b * (long long)n * n;
  const float inv = 1.f / fmaxf(trace[b] / n, 1e-30f);
  const int tx = (threadIdx.x & 15) * 4, ty = threadIdx.x >> 4;   // 16 bytes of a row, 16 rows at a time
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto four = [](const float* p) {
    if constexpr (kAligned) return *reinterpret_cast<const float4*>(p);
    else return make_float4(p[0], p[1], p[2], p[3]);
  };
  float4 u[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int lr = ty + 16 * i, r = ti * kDampTile + lr, cc = tj * kDampTile + tx;
    const int r2 = tj * kDampTile + lr, c2 = ti * kDampTile + tx;
    u[i] = (r < n && cc < n) ? four(C + (long long)r * n + cc) : zero;    // (n is a multiple of 8)
    l[i] = (r2 < n && c2 < n) ? four(C + (long long)r2 * n + c2) : zero;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int lr = ty + 16 * i;
    up[lr][tx] = u[i].x; up[lr][tx + 1] = u[i].y; up[lr][tx + 2] = u[i].z; up[lr][tx + 3] = u[i].w;
    lo[lr][tx] = l[i].x; lo[lr][tx + 1] = l[i].y; lo[lr][tx + 2] = l[i].z; lo[lr][tx + 3] = l[i].w;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int lr = ty + 16 * i;
    {
      const int r = ti * kDampTile + lr, cc = tj * kDampTile + tx;
      const float v[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
      float o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = 0.5f * (v[e] + lo[tx + e][lr]) * inv + (r == cc + e ? damping : 0.f);
      if (r < n && cc < n) *reinterpret_cast<float4*>(A + (long long)r * n + cc) = make_float4(o[0], o[1], o[2], o[3]);
    }
    if (ti != tj) {
      const int r = tj * kDampTile + lr, cc = ti * kDampTile + tx;
      const float v[4] = {l[i].x, l[i].y, l[i].z, l[i].w};
      float o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = 0.5f * (v[e] + up[tx + e][lr]) * inv;
      if (r < n && cc < n) *reinterpret_cast<float4*>(A + (long long)r * n + cc) = make_float4(o[0], o[1], o[2], o[3]);
    }
  }
}

// FP16 hi/lo planes of the two operands the iteration starts from, from A (FP32, damped and normalised):
//   M_0 = A / ||A||_F  (scaled by s_m)      T_0 = a I - b M_0  (scaled by s_t), which is also X_1
// planes layout [2][batch][n][n], hi plane first.  With t_planes == nullptr only the hi plane of M_0 is written (all
// that the single-pass squarings of the norm bound read).
// With defl_v the input is A and the deflation A' = A + sum_j coef[j] v_j v_j^T is applied on the way (the terms of
// rankr_update_kernel, in its order), so that A' is never written.
// With m32 M_0 is written there in FP32 (the graded finish, steps with a term linear in M).  With hi_only (the graded finish) its
// planes -- the hi plane alone -- are those of M_0 + m_diag I.
// half: of every output only the blocks of 256 x 256 on and above the diagonal are written (and of A read).
// late (per statistic, optional): where it is not zero the iteration starts with the second step, whose operands l gives.
struct InitLate {
  float a, b;
  __half* m_planes;
  __half* t_planes;
  float* m32;
};
__global__ void __launch_bounds__(256) init_planes_kernel(const float* a32, int n, int batch,
                                                          const float* __restrict__ sumsq, float a, float b, float s_m,
                                                          float s_t, __half* __restrict__ m_planes,
                                                          __half* __restrict__ t_planes,
                                                          const float* __restrict__ defl_v,
                                                          const float* __restrict__ defl_coef, int defl_r,
                                                          int vstride, float* m32, float m_diag, bool hi_only,
                                                          const int* __restrict__ late, InitLate second, bool half) {
  ptx::pdl_begin();
  const int bi = blockIdx.y;
  if (late && late[bi]) {   // (second.m32 may be a32 itself: every element is read before it is written, by one thread)
    a = second.a;
    b = second.b;
    m_planes = second.m_planes;
    t_planes = second.t_planes;
    m32 = second.m32;
  }
  float cf[kMaxDeflate];
  bool any = false;
#pragma unroll
  for (int j = 0; j < kMaxDeflate; ++j) {
    cf[j] = (defl_v != nullptr && j < defl_r) ? defl_coef[bi * kMaxDeflate + j] : 0.f;
    any = any || cf[j] != 0.f;
  }
  const float* DV = defl_v ? defl_v + (long long)bi * vstride * n : nullptr;
  const long long nn = (long long)n * n;
  const float4* A = reinterpret_cast<const float4*>(a32 + bi * nn);
  const float f = rsqrtf(fmaxf(sumsq[bi], 1e-60f));
  __half* mh = m_planes + bi * nn;
  __half* ml = m_planes + ((long long)batch + bi) * nn;
  __half* th = t_planes + bi * nn;
  __half* tl = t_planes + ((long long)batch + bi) * nn;
  const int n4 = n / 4;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nn / 4; i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / n4), c = (int)(i - (long long)r * n4) * 4;
    if (half && (c >> kHalfShift) < (r >> kHalfShift)) continue;
    float4 v = A[i];
    if (any) {
#pragma unroll
      for (int j = 0; j < kMaxDeflate; ++j) {
        if (cf[j] != 0.f) {
          const float vr = DV[(long long)j * n + r];
          const float4 vc = *reinterpret_cast<const float4*>(DV + (long long)j * n + c);
          v.x = fmaf(cf[j], vr * vc.x, v.x); v.y = fmaf(cf[j], vr * vc.y, v.y);
          v.z = fmaf(cf[j], vr * vc.z, v.z); v.w = fmaf(cf[j], vr * vc.w, v.w);
        }
      }
    }
    const float m[4] = {v.x * f, v.y * f, v.z * f, v.w * f};
    __half h[4], l[4], g[4], k[4];
    if (t_planes == nullptr) {
#pragma unroll
      for (int e = 0; e < 4; ++e) h[e] = __float2half_rn(m[e] * s_m);
      *reinterpret_cast<uint2*>(mh + i * 4) = *reinterpret_cast<uint2*>(h);
      continue;
    }
    if (m32) *reinterpret_cast<float4*>(m32 + bi * nn + i * 4) = make_float4(m[0], m[1], m[2], m[3]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = ((c + e) == r ? m[e] + m_diag : m[e]) * s_m;
      h[e] = __float2half_rn(x);
      l[e] = __float2half_rn(x - __half2float(h[e]));
      const float t = (((c + e) == r ? a : 0.f) - b * m[e]) * s_t;
      g[e] = __float2half_rn(t);
      k[e] = __float2half_rn(t - __half2float(g[e]));
    }
    *reinterpret_cast<uint2*>(mh + i * 4) = *reinterpret_cast<uint2*>(h);
    if (!hi_only) *reinterpret_cast<uint2*>(ml + i * 4) = *reinterpret_cast<uint2*>(l);
    *reinterpret_cast<uint2*>(th + i * 4) = *reinterpret_cast<uint2*>(g);
    *reinterpret_cast<uint2*>(tl + i * 4) = *reinterpret_cast<uint2*>(k);
  }
}

// ------------------------------------------------------------------ deflation of a dominant direction
// Activation statistics usually have one eigenvalue far above the rest (the mean activation).  It sets ||A||
// and with it the spectrum's lower bound after normalisation, i.e. the number of Newton steps and the
// attainable accuracy.  A few power-iteration steps find that eigenpair (lambda_1, v) to working accuracy when
// the gap is large; then  A' = A - (lambda_1 - c) v v^T  (c = mean of the remaining eigenvalues) has the same
// eigenvectors, and  A^{-s} = A'^{-s} + (lambda_1^{-s} - c^{-s}) v v^T.  When the iteration has not converged
// (no dominant direction) nothing is deflated.

// v_0: a fixed pattern of +-1 / sqrt(n)
__global__ void power_start_kernel(float* __restrict__ v, int n) {
  ptx::pdl_begin();
  const int b = blockIdx.y;
  const float s = rsqrtf((float)n);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    v[(long long)b * n + i] = (((unsigned)i * 2654435761u) >> 15) & 1u ? s : -s;
}

// y = A v, one warp per row, FP64 accumulation
__global__ void __launch_bounds__(256) gemv_kernel(const float* __restrict__ a, const float* __restrict__ v,
                                                   float* __restrict__ y, int n) {
  ptx::pdl_begin();
  const int b = blockIdx.y;
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n) return;
  const float* A = a + ((long long)b * n + row) * n;
  const float* X = v + (long long)b * n;
  // Four products at a time are summed in FP32 (their rounding, 6e-8 of the partial sum, is that of the FP32 result
  // itself) and the partial sums in FP64: one conversion per four elements instead of eight -- conversions to FP64 run
  // at a quarter of the FP64 rate and were what bound this kernel.
  double acc = 0.0;
  for (int c = lane * 4; c < n; c += 128) {
    const float4 av = *reinterpret_cast<const float4*>(A + c);
    const float4 xv = *reinterpret_cast<const float4*>(X + c);
    acc += (double)fmaf(av.x, xv.x, fmaf(av.y, xv.y, fmaf(av.z, xv.z, av.w * xv.w)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) y[(long long)b * n + row] = (float)acc;
}

// lambda = v.y / v.v (Rayleigh quotient), res = ||y - lambda v|| / ||lambda v||, then v <- y / ||y||.
// The residual is summed term by term: the shortcut ||y||^2 - lambda^2 cancels catastrophically.
__global__ void __launch_bounds__(256) power_norm_kernel(float* __restrict__ v, const float* __restrict__ y, int n,
                                                         float* __restrict__ lam, float* __restrict__ res) {
  ptx::pdl_begin();
  const int b = blockIdx.x;
  float* V = v + (long long)b * n;
  const float* Y = y + (long long)b * n;
  __shared__ double red[3][8];
  __shared__ double tot[3];
  auto block_sum3 = [&](double a0, double a1, double a2) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a0 += __shfl_xor_sync(0xffffffffu, a0, o);
      a1 += __shfl_xor_sync(0xffffffffu, a1, o);
      a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    __syncthreads();  // the previous round's totals have been read
    if ((threadIdx.x & 31) == 0) {
      red[0][threadIdx.x >> 5] = a0;
      red[1][threadIdx.x >> 5] = a1;
      red[2][threadIdx.x >> 5] = a2;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
      double t = 0.0;
      for (int w = 0; w < 8; ++w) t += red[threadIdx.x][w];
      tot[threadIdx.x] = t;
    }
    __syncthreads();
  };
  double yy = 0.0, vy = 0.0, vv = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double t = Y[i], u = V[i];
    yy += t * t;
    vy += t * u;
    vv += u * u;
  }
  block_sum3(yy, vy, vv);
  yy = tot[0];
  vy = tot[1];
  vv = tot[2];
  const double l = vv > 0.0 ? vy / vv : 0.0;
  double rr = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double d = (double)Y[i] - l * (double)V[i];
    rr += d * d;
  }
  block_sum3(rr, 0.0, 0.0);
  rr = tot[0];
  const double inv = yy > 0.0 ? 1.0 / sqrt(yy) : 0.0;
  // (Y of a root that overflowed -- a norm taken too low, status 1 -- says nothing: V, which the next call starts from, stays)
  if (isfinite(yy)) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) V[i] = (float)(Y[i] * inv);
  }
  if (threadIdx.x == 0) {
    lam[b] = (float)l;
    res[b] = (l > 0.0 && vv > 0.0) ? (float)(sqrt(rr) / (l * sqrt(vv))) : INFINITY;
  }
}

// sigma = lambda_1 - c if the pair converged and stands well above the rest, else 0;  corr = lambda_1^{-1/p} - c^{-1/p}
__global__ void deflate_decide_kernel(const float* __restrict__ lam, const float* __restrict__ res, int k, int n,
                                      float damping, int p, float* __restrict__ neg_sigma, float* __restrict__ corr) {
  ptx::pdl_begin();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= k) return;
  const float l1 = lam[b];
  const float tr = (float)n * (1.f + damping);  // A has unit mean diagonal plus the damping
  const float c = (tr - l1) / (float)(n - 1);
  const bool ok = n > 1 && isfinite(l1) && isfinite(res[b]) && res[b] < 1e-5f && c > 0.f && l1 > 8.f * c;
  neg_sigma[b] = ok ? -(l1 - c) : 0.f;
  corr[b] = ok ? powf(l1, -1.f / p) - powf(c, -1.f / p) : 0.f;
}

// A_b += coef[b] v_b v_b^T  (skipped where coef is zero)
__global__ void __launch_bounds__(256) rank1_update_kernel(float* __restrict__ a, const float* __restrict__ v,
                                                           const float* __restrict__ coef, int n) {
  ptx::pdl_begin();
  const int b = blockIdx.y;
  const float cf = coef[b];
  if (cf == 0.f) return;
  float* A = a + (long long)b * n * n;
  const float* V = v + (long long)b * n;
  const int n4 = n / 4;
  const long long total = (long long)n * n4;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / n4), c = (int)(i - (long long)r * n4) * 4;
    const float vr = V[r];
    const float4 vc = *reinterpret_cast<const float4*>(V + c);
    float4 x = *reinterpret_cast<float4*>(A + (long long)r * n + c);
    // cf * (v_r v_c): the product v_r v_c is the same bits at (r, c) and (c, r), so symmetry is kept exactly
    x.x = fmaf(cf, vr * vc.x, x.x); x.y = fmaf(cf, vr * vc.y, x.y); x.z = fmaf(cf, vr * vc.z, x.z); x.w = fmaf(cf, vr * vc.w, x.w);
    *reinterpret_cast<float4*>(A + (long long)r * n + c) = x;
  }
}


// ------------------------------------------------------------------ deflation of several dominant directions
// Statistics of real activations often have a handful of directions far above the rest (outlier features), not just
// the mean.  Block power iteration with Rayleigh-Ritz finds r <= kMaxDeflate of them at the cost of one pass over the
// statistic per sweep, whatever r is, and converges with the ratio of the (r+1)-th eigenvalue to the wanted one, so
// close pairs among the dominant ones do not slow it down; the vectors are kept by the caller between calls.
// Vectors are stored vector-major: v[(b * vstride + j) * n + c].
// Eight slots a statistic, or twelve.
constexpr int kSlots = 8, kMoreSlots = kMaxDeflate;

// Y_j = A v_j, j < R: one pass over A.  A block takes 32 rows (four per warp; 16 and two from six vectors on) and walks the columns 256 at a time; the
// 256-column slice of the vectors is staged in shared memory once per block, so the vectors are read from L2 once per
// 32 rows instead of once per row pair (that traffic, not the pass over A, bounded the first version of this kernel).
// The products of four slices (32 per lane) are summed in FP32 before they join the FP64 sums: conversions and FP64
// additions run at a fraction of the FP32 rate, and with one per eight products they, not the pass over A, set the
// pace.  R (the number of vectors, rounded up to even) is a template argument so that absent vectors cost nothing.
// What bounds the rest is how much of A is on its way: slices come by asynchronous copies into shared memory ahead of the one
// being multiplied, with two blocks on an SM 128 KB of A up to four vectors (two slices of 32 rows) and 96 KB from six on (three of
// 16).  With the next slice in registers it was 64 KB, and 32 with the one block that eight vectors' sums for four rows leave room
// for, hence two rows a warp there: 32
// statistics of width 2048 and 96 of 512, four vectors, 104 -> 70 us a pass, two vectors 79 -> 60; eight vectors on 12 of
// width 1280 and four of 3328 128 -> 102.
template <int R>
struct BlockGemv {
  static constexpr int kWarpRows = R <= 4 ? 4 : 2;
  static constexpr int kRows = 8 * kWarpRows;
  static constexpr int kStages = R <= 4 || R > 10 ? 3 : 4;
  static constexpr int kStageFloat4 = (kRows + R) * 64;   // 256 columns of the block's rows and of the vectors
  static constexpr int kBytes = kStages * kStageFloat4 * 16;
};
template <int R>
__global__ void __launch_bounds__(256, 2) block_gemv_kernel(const float* __restrict__ a, const float* __restrict__ v,
                                                            float* __restrict__ y, int n, int r, int vstride) {
  ptx::pdl_begin();
  using B = BlockGemv<R>;
  constexpr int kWarpRows = B::kWarpRows;
  extern __shared__ float4 gemv_smem[];
  const int b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.x * B::kRows + warp * kWarpRows;
  const float* V = v + (long long)b * vstride * n;
  const float* A = a + (long long)b * n * n;
  double acc[kWarpRows][R];
  float part[kWarpRows][R];
#pragma unroll
  for (int i = 0; i < kWarpRows; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) {
      acc[i][j] = 0.0;
      part[i][j] = 0.f;
    }
  // slice `k`, 256 columns: a warp's rows, two 16-byte pieces a lane and row; zeros outside the matrix
  auto fetch = [&](int k) {
    float4* const stage = gemv_smem + (k % B::kStages) * B::kStageFloat4;
    const int c0 = k * 256;
    if (c0 < n) {
#pragma unroll
      for (int q = 0; q < (R * 64 + 255) / 256; ++q) {
        const int i = threadIdx.x + 256 * q, j = i >> 6, col = c0 + (i & 63) * 4;
        if (i < R * 64) {
          const bool in = j < r && col < n;
          ptx::cp_async16(ptx::smem_u32(stage + B::kRows * 64 + i), in ? V + (long long)j * n + col : V, in);
        }
      }
#pragma unroll
      for (int i = 0; i < kWarpRows; ++i) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = c0 + (lane + 32 * h) * 4;
          const bool in = row0 + i < n && col < n;
          ptx::cp_async16(ptx::smem_u32(stage + (warp * kWarpRows + i) * 64 + lane + 32 * h),
                          in ? A + (long long)(row0 + i) * n + col : A, in);
        }
      }
    }
    ptx::cp_async_commit();
  };
#pragma unroll
  for (int k = 0; k < B::kStages - 1; ++k) fetch(k);
  int slice = 0;
  for (int c0 = 0; c0 < n; c0 += 256, ++slice) {
    ptx::cp_async_wait<B::kStages - 2>();
    __syncthreads();                     // the slice is there for everyone, and the stage filled next has been read by everyone
    fetch(slice + B::kStages - 1);
    const float4* const stage = gemv_smem + (slice % B::kStages) * B::kStageFloat4;
    float4 a0[kWarpRows], a1[kWarpRows];
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i) {
      a0[i] = stage[(warp * kWarpRows + i) * 64 + lane];
      a1[i] = stage[(warp * kWarpRows + i) * 64 + lane + 32];
    }
    // a lane's eight columns of a vector are read from shared memory once for the warp's rows (read per row, the
    // shared-memory traffic is R times the traffic of A and sets the pace from four vectors on)
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const float4 x0 = stage[(B::kRows + j) * 64 + lane], x1 = stage[(B::kRows + j) * 64 + lane + 32];
#pragma unroll
      for (int i = 0; i < kWarpRows; ++i) {
        const float s0 = fmaf(a0[i].x, x0.x, fmaf(a0[i].y, x0.y, fmaf(a0[i].z, x0.z, a0[i].w * x0.w)));
        const float s1 = fmaf(a1[i].x, x1.x, fmaf(a1[i].y, x1.y, fmaf(a1[i].z, x1.z, a1[i].w * x1.w)));
        part[i][j] += s0 + s1;
      }
    }
    if ((slice & 3) == 3) {
#pragma unroll
      for (int i = 0; i < kWarpRows; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) {
          acc[i][j] += (double)part[i][j];
          part[i][j] = 0.f;
        }
    }
  }
#pragma unroll
  for (int i = 0; i < kWarpRows; ++i) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      double t = acc[i][j] + (double)part[i][j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0 && j < r && row0 + i < n) y[((long long)b * vstride + j) * n + row0 + i] = (float)t;
    }
  }
}
template <int R>
static cudaError_t launch_block_gemv(int k, cudaStream_t stream, const float* a, const float* v, float* y, int n, int r, int vstride) {
  return launch(block_gemv_kernel<R>, dim3((n + BlockGemv<R>::kRows - 1) / BlockGemv<R>::kRows, k), 256, BlockGemv<R>::kBytes, stream, 0,
                a, v, y, n, r, vstride);
}
bool allow_factor_kernels() {
  auto allow = [](auto kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
  };
  return allow(block_gemv_kernel<2>, BlockGemv<2>::kBytes) && allow(block_gemv_kernel<4>, BlockGemv<4>::kBytes) &&
         allow(block_gemv_kernel<6>, BlockGemv<6>::kBytes) && allow(block_gemv_kernel<8>, BlockGemv<8>::kBytes) &&
         allow(block_gemv_kernel<10>, BlockGemv<10>::kBytes) && allow(block_gemv_kernel<12>, BlockGemv<12>::kBytes);
}

// Sum over the block of one double per thread; every thread gets the total.  256 threads.
__device__ __forceinline__ double block_sum(double x, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();  // the previous total has been read by everyone
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < 8; ++w) t += red[w];
  return t;
}
__device__ __forceinline__ double block_dot(const float* x, const float* y, int n, double* red) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += (double)x[i] * (double)y[i];
  return block_sum(s, red);
}

// Sums over the warp of K doubles per lane: at every step of the butterfly a lane keeps the half of its values that its bit of the
// lane index names and hands over the other, so that K + 31 shuffles do what 5 K did (the same pairs are added, and so the bits).
// Value i ends up with the lanes whose bits, the highest first, are those of i's place in the halvings; store(i, sum) is called by one.
template <int kHalf, int kBit, int P>
__device__ __forceinline__ void warp_fold(double (&v)[P], int lane, int& at) {
  const bool upper = (lane & kBit) != 0;
#pragma unroll
  for (int i = 0; i < kHalf; ++i) {
    const double keep = upper ? v[i + kHalf] : v[i], give = upper ? v[i] : v[i + kHalf];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, kBit);
  }
  at += upper ? kHalf : 0;
  if constexpr (kBit > 1) warp_fold<kHalf / 2, kBit / 2>(v, lane, at);
}
template <int K, typename Store>
__device__ __forceinline__ void warp_sum_many(const double (&acc)[K], Store store) {
  constexpr int kPadded = (K + 31) / 32 * 32;
  const int lane = threadIdx.x & 31;
  double v[kPadded];
#pragma unroll
  for (int i = 0; i < kPadded; ++i) v[i] = i < K ? acc[i] : 0.0;
  int at = 0;
  warp_fold<kPadded / 2, 16>(v, lane, at);
#pragma unroll
  for (int i = 0; i < kPadded / 32; ++i)
    if (at + i < K) store(at + i, v[i]);
}

// Sums over the block of K doubles per thread (256 threads): out[i] holds the total of acc[i] afterwards (shared
// memory, valid for every thread after the call).  `part` is 8 * K doubles of shared scratch.
template <int K>
__device__ __forceinline__ void block_sum_many(const double (&acc)[K], double* part, double* out) {
  __syncthreads();  // earlier readers of part / out are done
  warp_sum_many<K>(acc, [&](int i, double x) { part[(threadIdx.x >> 5) * K + i] = x; });
  __syncthreads();
  if (threadIdx.x < K) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += part[w * K + threadIdx.x];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// entry (i, j), j <= i, of a symmetric matrix's lower triangle
__device__ __forceinline__ int pair_index(int i, int j) { return i * (i + 1) / 2 + j; }

// Cholesky-QR of the r vectors held in Y (r x n, vector-major; a thread's columns from `first` on): G = Y Y^T = L L^T (FP64), V = L^-1 Y.  `gram` holds G's
// lower triangle (pair_index order) on entry.  A vector that is (numerically) a combination of the earlier ones comes out as
// zero; its slot is seeded afresh by the next call.  L's columns are formed one after the other by the lanes of one warp (row
// i of a column by lane i); the diagonal of `L` holds its reciprocal (zero for a dropped vector), the diagonal itself where
// `divide` asks for divisions by it (see ritz_kernel).
template <int R>
__device__ void cholesky_orthonormalise(const float* Y, float* V, int n, int r, const double* gram, double (*L)[kMaxDeflate],
                                        bool divide, int first, int step) {
  if (threadIdx.x < 32) {
    const int i = threadIdx.x;
    double row[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const bool on = i < r && j <= i && j < r;
      double sum = on ? gram[pair_index(i, j)] : 0.0;
#pragma unroll
      for (int k = 0; k < R; ++k)
        if (k < j) sum -= row[k] * __shfl_sync(0xffffffffu, row[k], j);
      // lane j holds the pivot
      const double pivot = __shfl_sync(0xffffffffu, sum, j);
      const double floor = j < r ? 1e-24 * gram[pair_index(j, j)] : 0.0;
      const bool kept = j < r && pivot > floor && pivot > 0.0;
      if (divide) {
        const double diag = kept ? sqrt(pivot) : 0.0;
        row[j] = i == j ? diag : (kept ? sum / diag : 0.0);
        if (on) L[i][j] = row[j];
      } else {
        const double inv = kept ? rsqrt(pivot) : 0.0;
        row[j] = i == j ? pivot * inv : sum * inv;
        if (on) L[i][j] = i == j ? inv : row[j];
      }
    }
  }
  __syncthreads();
  for (int c = first; c < n; c += step) {
    double out[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (j < r) {
        double sum = (double)Y[(long long)j * n + c];
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (i < j) sum -= L[j][i] * out[i];
        out[j] = !divide ? sum * L[j][j] : (L[j][j] > 0.0 ? sum / L[j][j] : 0.0);
      } else {
        out[j] = 0.0;
      }
    }
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (j < r) V[(long long)j * n + c] = (float)out[j];
  }
  __syncthreads();
}

// Eigenpairs of the symmetric r x r matrix H (shared memory, FP64) by Jacobi rotations, zeros from r to R (even).  One warp: each of
// the R - 1 rounds of a sweep rotates R / 2 disjoint pairs at once (round-robin order), the lanes of a pair taking its rows and
// columns in turn.  A single thread doing the rotations one by one took 20 us of a 23 us launch at r = 4 and most of 160 us at r = 8;
// eight seats whatever R, seven rounds for three at R = 4.
template <int R>
__device__ void jacobi_warp(double (*H)[kMaxDeflate], double (*Q)[kMaxDeflate]) {
  constexpr int kPairs = R / 2, kLanes = 32 / kPairs;
  const int lane = threadIdx.x, pair = lane / kLanes, k0 = lane % kLanes;
  const bool on = pair < kPairs;
  for (int sweep = 0; sweep < 12; ++sweep) {
    double off = 0.0, diag = 0.0;
    for (int e = lane; e < R * R; e += 32) {
      const int i = e / R, j = e - i * R;
      const double h = H[i][j];
      if (i == j) diag += h * h;
      else if (j > i) off += h * h;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      diag += __shfl_xor_sync(0xffffffffu, diag, o);
    }
    if (!(off > 1e-28 * diag)) break;   // off-diagonal part 1e-14 of the largest: far below what FP32 vectors hold
    for (int round = 0; round < R - 1; ++round) {
      // the last seat stays, the others rotate
      const int a = pair == 0 ? R - 1 : (round + pair) % (R - 1), b = pair == 0 ? round : (round + R - 1 - pair) % (R - 1);
      const int pp = on ? min(a, b) : 0, qq = on ? max(a, b) : 0;
      const double apq = on ? H[pp][qq] : 0.0;
      double cs = 1.0, sn = 0.0;
      // (The angle in FP32, which leaves 1e-7 of the entry for the next sweep; the rotation itself is orthogonal to FP64.  FP64
      // divisions and a square root were half of a round's time.)
      const float twice = 2.f * (float)apq;
      if (on && twice != 0.f) {
        const float tau = (float)(H[qq][qq] - H[pp][pp]) / twice;
        const double t = (double)((tau >= 0.f ? 1.f : -1.f) / (fabsf(tau) + sqrtf(1.f + tau * tau)));
        cs = rsqrt(1.0 + t * t);
        sn = t * cs;
      }
      __syncwarp();   // every pair has its rotation before any entry changes
      if (on) {
        for (int k = k0; k < R; k += kLanes) {
          const double hp = H[k][pp], hq = H[k][qq], qp = Q[k][pp], qv = Q[k][qq];   // columns pp, qq of H and Q
          H[k][pp] = cs * hp - sn * hq;
          H[k][qq] = sn * hp + cs * hq;
          Q[k][pp] = cs * qp - sn * qv;
          Q[k][qq] = sn * qp + cs * qv;
        }
      }
      __syncwarp();
      if (on) {
        for (int k = k0; k < R; k += kLanes) {
          const double rp = H[pp][k], rq = H[qq][k];                                 // rows pp, qq of H
          H[pp][k] = cs * rp - sn * rq;
          H[qq][k] = sn * rp + cs * rq;
        }
      }
      __syncwarp();
    }
  }
}

// The same with one rotation after the other, row by row of the upper triangle, and rounded as a single thread doing so would
// (lane k takes column / row k; every lane adds up the same sums in the same order).
__device__ void jacobi_in_order(double (*H)[kMaxDeflate], double (*Q)[kMaxDeflate], int r) {
  const int k = threadIdx.x & 7;
  const bool on = threadIdx.x < r;
  for (int sweep = 0; sweep < 12; ++sweep) {
    double off = 0.0, diag = 0.0;
    for (int pp = 0; pp < r; ++pp)
      for (int qq = pp + 1; qq < r; ++qq) off += H[pp][qq] * H[pp][qq];
    for (int pp = 0; pp < r; ++pp) diag += H[pp][pp] * H[pp][pp];
    if (!(off > 1e-30 * diag)) break;
    for (int pp = 0; pp < r; ++pp) {
      for (int qq = pp + 1; qq < r; ++qq) {
        const double apq = H[pp][qq];
        if (apq == 0.0) continue;
        const double tau = (H[qq][qq] - H[pp][pp]) / (2.0 * apq);
        const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
        const double cs = 1.0 / sqrt(1.0 + t * t), sn = t * cs;
        __syncwarp();   // every lane has the rotation before an entry changes
        if (on) {
          const double hp = H[k][pp], hq = H[k][qq], qp = Q[k][pp], qv = Q[k][qq];
          H[k][pp] = cs * hp - sn * hq;
          H[k][qq] = sn * hp + cs * hq;
          Q[k][pp] = cs * qp - sn * qv;
          Q[k][qq] = sn * qp + cs * qv;
        }
        __syncwarp();
        if (on) {
          const double hp = H[pp][k], hq = H[qq][k];
          H[pp][k] = cs * hp - sn * hq;
          H[qq][k] = sn * hp + cs * hq;
        }
        __syncwarp();
      }
    }
  }
}

// start vectors: the caller's vectors (warm), or r different fixed +-1 patterns (cold, and for a slot that holds
// nothing yet because the rank grew since the last call), orthonormalised
template <int R>
__global__ void __launch_bounds__(256) block_start_kernel(float* __restrict__ v, int n, int r, int vstride, int cold, int in_order) {
  ptx::pdl_begin();
  __shared__ double red[8];
  constexpr int kPairs = R * (R + 1) / 2;
  __shared__ double part[8 * kPairs], gram[kPairs];
  __shared__ double L[kMaxDeflate][kMaxDeflate];
  const int b = blockIdx.x;
  float* V = v + (long long)b * vstride * n;
  const float s = rsqrtf((float)n);
  for (int j = 0; j < r; ++j) {
    float* vj = V + (long long)j * n;
    const bool seed = cold || !(block_dot(vj, vj, n, red) > 0.0);
    if (seed)
      for (int c = threadIdx.x; c < n; c += blockDim.x)
        vj[c] = ((((unsigned)c + 977u * (unsigned)j) * 2654435761u) >> (15 + (j & 7))) & 1u ? s : -s;
    __syncthreads();
  }
  double acc[kPairs];
#pragma unroll
  for (int i = 0; i < kPairs; ++i) acc[i] = 0.0;
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    double x[R];
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = i < r ? (double)V[(long long)i * n + c] : 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) acc[i * (i + 1) / 2 + j] += x[i] * x[j];
  }
  block_sum_many<kPairs>(acc, part, gram);
  cholesky_orthonormalise<R>(V, V, n, r, gram, L, in_order != 0, threadIdx.x, blockDim.x);
}

// Sums over a cluster's CTAs, as block_sum_many's over one block: `mine` is K doubles of shared memory that the others read.
template <int K>
__device__ __forceinline__ void cluster_sum_many(double (&acc)[K], double* part, double* mine, double* out, int ctas) {
  block_sum_many<K>(acc, part, ctas > 1 ? mine : out);
  if (ctas > 1) {
    ptx::cluster_sync();   // every CTA's sums are there
    if (threadIdx.x < K) {
      double t = 0.0;
      for (int rank = 0; rank < ctas; ++rank) t += ptx::ld_cluster_f64(ptx::mapa(ptx::smem_u32(mine + threadIdx.x), rank));
      out[threadIdx.x] = t;
    }
    ptx::cluster_sync();   // ... and have been read
  }
}

// Rayleigh-Ritz on span(V) with Y = A V (V orthonormal): H = V Y^T, H = Q diag(theta) Q^T (Jacobi, FP64), V <- Q^T V,
// Y <- Q^T Y (Ritz vectors, descending theta), res_j = ||Y_j - theta_j V_j|| / |theta_j|.  Unless this is the last sweep, V is
// then replaced by the orthonormalised Y - sigma V, one more step of the power iteration on A - sigma I: with sigma = 0.8 c, c the
// mean of the eigenvalues that do not stand out, what lies below 1.6 c shrinks as if it were 0.8 c (a bulk up to 1.8 under a
// direction of 10: by 0.11 a sweep where A itself gives 0.18; four sweeps then reach the residual that deflation asks for, with
// which the fifth direction of spiked:4 was left in one call of four).  Where no trace is given sigma is 0: the last step takes A itself,
// which leaves nothing of the smallest eigenvalues' directions in V, where their inverse roots are largest; after a shifted one the Ritz
// rotation took that from the block's other vectors and rounded the top vector once more (4.3e-8 off for 3.5e-8; A^(-1/2) weighted by the
// statistic, columns that decay exponentially: 1.08 times as far off as without shifts in the mean of 40 calls and 1.31 in the worst,
// now 0.93 and 1.02).
// Three passes over the two blocks of vectors (five from ten vectors on, whose sums are taken for half of the rows at a time);
// every reduction is taken for all pairs at once.  R: r rounded up to even, as in block_gemv_kernel -- with eight
// vectors' sums (64 and 44 doubles to reduce) whatever r, a launch took 42 us on 12 statistics of width 3072 and r = 2, with r's 17.
// A cluster shares a statistic's columns (a few statistics are a few blocks on 148 SMs, and a pass of one block over 3328 columns is
// thirteen round trips to L2): every CTA factors the small matrix for itself, from the same sums.
// in_order (one CTA, no sigma): a caller that keeps its order of additions (the plane-by-plane products) has the small
// factorisations keep theirs too: Jacobi's rotations one after the other and divisions by Cholesky's diagonal.  The vectors are no
// better for it, but a deflated eigenvalue hundreds of times the rest turns their last bits into 1e-5 of what remains.
template <int R>
__global__ void __launch_bounds__(256) ritz_kernel(float* __restrict__ v, float* __restrict__ y, int n, int r, int vstride,
                                                   int last, float* __restrict__ theta, float* __restrict__ res, int in_order,
                                                   float trace) {
  ptx::pdl_begin();
  constexpr int kPairs = R * (R + 1) / 2, kMost = kMaxDeflate;
  constexpr bool kHalves = R > 8;
  constexpr int kRows = kHalves ? R / 2 : R;                            // of the rows whose sums are taken at a time
  constexpr int kFirst = kRows * R, kSecond = kHalves ? kRows * R + kRows : kPairs + R;
  constexpr int kSums = kFirst > kSecond ? kFirst : kSecond;
  __shared__ double part[8 * kSums], mine[kSums], sums[kSums], gram[kPairs], resid[R];
  __shared__ double H[kMost][kMost], Q[kMost][kMost], lam[kMost], L[kMost][kMost], shift;
  const int ctas = (int)ptx::cluster_nctarank(), rank = (int)ptx::cluster_ctarank();
  const int b = blockIdx.y;
  const int first = rank * blockDim.x + threadIdx.x, step = ctas * blockDim.x;
  float* V = v + (long long)b * vstride * n;
  float* Y = y + (long long)b * vstride * n;
  for (int e = threadIdx.x; e < kMost * kMost; e += blockDim.x) {
    const int i = e / kMost, j = e - i * kMost;
    H[i][j] = 0.0;
    Q[i][j] = i == j ? 1.0 : 0.0;
  }
  // V Y^T, kept in L until it is whole
#pragma unroll
  for (int half = 0; half < R / kRows; ++half) {
    double acc[kFirst];
#pragma unroll
    for (int i = 0; i < kFirst; ++i) acc[i] = 0.0;
    for (int c = first; c < n; c += step) {
      double vv[kRows], yy[R];
#pragma unroll
      for (int i = 0; i < kRows; ++i) vv[i] = half * kRows + i < r ? (double)V[(long long)(half * kRows + i) * n + c] : 0.0;
#pragma unroll
      for (int i = 0; i < R; ++i) yy[i] = i < r ? (double)Y[(long long)i * n + c] : 0.0;
#pragma unroll
      for (int i = 0; i < kRows; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[i * R + j] += vv[i] * yy[j];
    }
    cluster_sum_many<kFirst>(acc, part, mine, sums, ctas);
    for (int e = threadIdx.x; e < kFirst; e += blockDim.x) L[half * kRows + e / R][e % R] = sums[e];
    __syncthreads();
  }
  for (int e = threadIdx.x; e < R * R; e += blockDim.x) {
    const int i = e / R, j = e % R;
    if (i < r && j < r) H[i][j] = 0.5 * (L[i][j] + L[j][i]);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    if (in_order) jacobi_in_order(H, Q, r);
    else jacobi_warp<R>(H, Q);
    // descending order: lane i's place is the number of values before it; the columns of Q follow
    const int i = threadIdx.x % kMost;
    const double own = H[i][i];
    int place = 0;
    for (int j = 0; j < r; ++j) {
      const double o = H[j][j];
      if (o > own || (o == own && j < i)) ++place;
    }
    double col[kMost];
#pragma unroll
    for (int k = 0; k < kMost; ++k) col[k] = Q[k][i];
    __syncwarp();
    if (threadIdx.x < r) {
      lam[place] = own;
#pragma unroll
      for (int k = 0; k < kMost; ++k) Q[k][place] = col[k];
    }
    __syncwarp();
    if (threadIdx.x == 0) {
      // the mean of what does not stand above eight times it, as block_decide_kernel has it
      double sum = 0.0;
      int m = 0;
      for (; m < r && n - (m + 1) > 0; ++m) {
        const double rest = ((double)trace - sum - lam[m]) / (double)(n - (m + 1));
        if (!(rest > 0.0 && lam[m] > 8.0 * rest)) break;
        sum += lam[m];
      }
      const double rest = ((double)trace - sum) / (double)(n - m);
      shift = in_order || last || !(rest > 0.0) ? 0.0 : 0.8 * rest;
    }
  }
  __syncthreads();
  const double sigma = shift;
  {
    // rotate both blocks (new vector j = sum_i Q[i][j] old vector i); on the way: the squared residuals and the Gram
    // matrix of the rotated Y (for its orthonormalisation)
    double acc[kHalves ? 1 : kSecond];
    if constexpr (!kHalves) {
#pragma unroll
      for (int i = 0; i < kSecond; ++i) acc[i] = 0.0;
    }
    for (int c = first; c < n; c += step) {
      double vv[R], yy[R], nv[R], ny[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        vv[i] = i < r ? (double)V[(long long)i * n + c] : 0.0;
        yy[i] = i < r ? (double)Y[(long long)i * n + c] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < R; ++j) {
        double sv = 0.0, sy = 0.0;
        if (j < r) {
#pragma unroll
          for (int i = 0; i < R; ++i) {
            if (i < r) {
              sv += Q[i][j] * vv[i];
              sy += Q[i][j] * yy[i];
            }
          }
          // what is stored is what later passes read: round before the sums
          const float fv = (float)sv;
          sv = fv;
          if (sigma != 0.0) sy -= sigma * sv;
          const float fy = (float)sy;
          V[(long long)j * n + c] = fv;
          Y[(long long)j * n + c] = fy;
          sy = fy;
        }
        nv[j] = sv;
        ny[j] = sy;
      }
      if constexpr (!kHalves) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (i < r) {
#pragma unroll
            for (int j = 0; j <= i; ++j) acc[i * (i + 1) / 2 + j] += ny[i] * ny[j];
            const double d = ny[i] - (lam[i] - sigma) * nv[i];
            acc[kPairs + i] += d * d;
          }
        }
      }
    }
    if constexpr (!kHalves) {
      cluster_sum_many<kSecond>(acc, part, mine, sums, ctas);
      for (int e = threadIdx.x; e < kPairs + R; e += blockDim.x) (e < kPairs ? gram[e] : resid[e - kPairs]) = sums[e];
    }
  }
  if constexpr (kHalves) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      double acc[kSecond];
#pragma unroll
      for (int i = 0; i < kSecond; ++i) acc[i] = 0.0;
      for (int c = first; c < n; c += step) {   // (columns this thread has just written)
        double ny[R];
#pragma unroll
        for (int i = 0; i < R; ++i) ny[i] = i < r ? (double)Y[(long long)i * n + c] : 0.0;
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const int row = half * kRows + i;
          if (row < r) {
#pragma unroll
            for (int j = 0; j < R; ++j) acc[i * R + j] += ny[half * kRows + i] * ny[j];
            const double d = ny[half * kRows + i] - (lam[row] - sigma) * (double)V[(long long)row * n + c];
            acc[kRows * R + i] += d * d;
          }
        }
      }
      cluster_sum_many<kSecond>(acc, part, mine, sums, ctas);
      for (int e = threadIdx.x; e < kRows * R; e += blockDim.x) {
        const int i = half * kRows + e / R, j = e % R;
        if (j <= i) gram[pair_index(i, j)] = sums[e];
      }
      if (threadIdx.x < kRows) resid[half * kRows + threadIdx.x] = sums[kRows * R + threadIdx.x];
      __syncthreads();
    }
  }
  __syncthreads();
  if (rank == 0 && threadIdx.x < r) {
    const double l = lam[threadIdx.x];
    theta[b * kMost + threadIdx.x] = (float)l;
    res[b * kMost + threadIdx.x] = l > 0.0 ? (float)(sqrt(resid[threadIdx.x]) / l) : INFINITY;
  }
  if (!last) cholesky_orthonormalise<R>(Y, V, n, r, gram, L, in_order != 0, first, step);
}
// CTAs that share a statistic.  A launch, four statistics of width 768 / 1280 / 3328 / 5632 without a gap in their spectrum, us:  r = 4
// 15 / 19 / 34 / 52 by one, 13 / 13 / 16 / 23 by eight;  r = 8  42 / 50 / 94 / 171, 31 / 31 / 37 / 49;  r = 11  107 / 129 / 235 / 434,
// 79 / 80 / 92 / 117.  (Before the sums were folded and the angles taken in FP32, by one: r = 4  17 / 20 / 31 / 61, r = 8  43 / 53 / 91 / 182.)
// By one / two / four / eight, us:  384 columns, 12 statistics, r = 8  36 / 32 / 28 / 28, 264 and 24 of them 32 / 30 / 31 / 55;  512, 24, r = 4
// 15.5 / 15.3 / 15.5 / 15.6;  768, 12, r = 4  22 / 16 / 15 / 14;  1024, 4, r = 4  58 / 56 / 43 / 33;  2048, 12, r = 8  78 / 56 / 43 / 36.
// No more blocks than find a place at once: the wide kernels (r > 4) take an SM each, and clusters fill the GPU's groups of SMs unevenly.
// r = 8, 768 columns:  24 statistics 43 / 37 / 32 / 56, 36  43 / 38 / 59 / 82, 96  44 / 70 / 86 / 188;  r = 4:  48  21 / 21 / 18 / 29, 96  21 / 20 / 30 / 51.
static int ritz_ctas(int n, int k, int width) {
  int ctas = n >= 1024 ? 8 : n >= 512 ? 4 : 1;
  while (ctas > 1 && (long long)k * ctas > (width > 4 ? 96 : 192)) ctas /= 2;
  return ctas;
}
template <int R>
static cudaError_t launch_ritz(int k, cudaStream_t stream, float* v, float* y, int n, int r, int vstride, int last, float* theta, float* res,
                               int in_order, float trace) {
  const int ctas = in_order ? 1 : ritz_ctas(n, k, R);
  return launch(ritz_kernel<R>, dim3(ctas, k), 256, 0, stream, ctas > 1 ? ctas : 0, v, y, n, r, vstride, last, theta, res, in_order, trace);
}

// Which of the r Ritz pairs are deflated: in descending order, as long as each has converged and stands above eight
// times the mean c of everything that would remain, at most `most` of them (one fewer than r where the norm is to come from
// the largest one that stays); all accepted directions are moved to that common c.
//   coef[b][j] = -(theta_j - c)  (0 where not deflated)      corr[b][j] = theta_j^(-1/p) - c^(-1/p)
// rest_top[b] / rest_idx[b]: the largest Ritz value that stays in A' and its vector's index (0 / -1 when every vector of
// the block was deflated: nothing is known about the remainder then).
__global__ void block_decide_kernel(const float* __restrict__ theta, const float* __restrict__ res, int k, int n, int r,
                                    float damping, int p, int most, float* __restrict__ coef, float* __restrict__ corr,
                                    int* __restrict__ count, float* __restrict__ rest_top, int* __restrict__ rest_idx,
                                    float* __restrict__ rest_trace) {
  ptx::pdl_begin();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= k) return;
  const double tr = (double)n * (1.0 + (double)damping);  // A has unit mean diagonal plus the damping
  double sum = 0.0;
  int m = 0;
  for (int j = 0; j < most && n - (j + 1) > 0; ++j) {
    const double t = theta[b * kMaxDeflate + j];
    const double e = res[b * kMaxDeflate + j];
    const double c = (tr - sum - t) / (double)(n - (m + 1));
    if (!(isfinite(t) && isfinite(e) && e < 1e-5 && c > 0.0 && t > 8.0 * c)) break;
    sum += t;
    ++m;
  }
  const double c = (tr - sum) / (double)(n - m);
  for (int j = 0; j < kMaxDeflate; ++j) {
    const bool on = j < m;
    const double t = on ? (double)theta[b * kMaxDeflate + j] : 0.0;
    coef[b * kMaxDeflate + j] = on ? (float)-(t - c) : 0.f;
    corr[b * kMaxDeflate + j] = on ? (float)(pow(t, -1.0 / p) - pow(c, -1.0 / p)) : 0.f;
  }
  // also reported (bits 8..15): how many Ritz values stand above 8x the rest whether converged or not -- directions
  // that look like outliers; a caller that iterates fewer vectors than there are of those widens its block
  int cand = 0;
  for (int j = 0; j < r; ++j)
    if ((double)theta[b * kMaxDeflate + j] > 8.0 * c) ++cand;
  if (count) count[b] = m | (cand << 8);
  const float rest = m < r ? theta[b * kMaxDeflate + m] : 0.f;
  const bool known = m < r && isfinite(rest) && rest > 0.f;
  rest_top[b] = known ? rest : 0.f;
  rest_idx[b] = known ? m : -1;
  rest_trace[b] = (float)(c * (double)n);   // trace of A' (every deflated direction moved to c): above its Frobenius norm
}

// An ESTIMATE of lambda_max(A') in place of the certified bound: kRitzGrow times the largest Ritz value that was not
// deflated, never above the trace of A' (which bounds its Frobenius norm).  A Rayleigh quotient errs low, and at the dense upper
// edge of an activation statistic's bulk it stays low however long the block has followed the statistic: 17-20 % on
// the benchmark's statistics (Marchenko-Pastur edges 1.36 and 1.63, Ritz values 1.08 and 1.30).  The factor leaves
// ten percent above that.  Three squarings give n^(1/16) = 1.7 times lambda_max for a flat spectrum and cost three
// passes; what the estimate risks -- eigenvalues of M_0 above 1, which the first Newton step sends BELOW the new lower
// bound -- is looked for after the chain (see the verification).
constexpr float kRitzGrow = 1.4f;
__global__ void ritz_norm_kernel(float* __restrict__ bound2, const float* __restrict__ rest_top,
                                 const float* __restrict__ rest_trace, int k) {
  ptx::pdl_begin();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= k) return;
  const float cap = rest_trace[b];      // ||A'||_F <= trace(A') for a positive matrix: costs no pass over A'
  const float t = kRitzGrow * rest_top[b];
  bound2[b] = (t > 0.f && t < cap) ? t * t : cap * cap;
}

// out[b][0] = first[b] (the tracked direction), out[b][1] = the Ritz vector rest_idx[b] of statistic b (zero where there
// is none): the two starting vectors of the verification, side by side for the two-vector passes.  `spread` > 0 adds fixed signs
// of norm `spread` to both: a share of about 1 / sqrt(n) of every direction.  With y = A v the second vector is that Ritz vector's
// residual y - theta v.
__global__ void __launch_bounds__(256) pick_vector_kernel(const float* __restrict__ first, const float* __restrict__ v,
                                                          const int* __restrict__ idx, float* __restrict__ out, int n,
                                                          int vstride, float spread, const float* __restrict__ y,
                                                          const float* __restrict__ theta) {
  ptx::pdl_begin();
  const int b = blockIdx.y;
  const int j = idx[b];
  const float value = y && j >= 0 ? theta[b * kMaxDeflate + j] : 0.f;
  const float amount = spread * rsqrtf((float)n);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned h = (unsigned)i * (unsigned)i * 2654435761u;   // (signs of two quadratic sequences)
    const float s0 = (h >> 31) ? amount : -amount, s1 = ((h + (unsigned)i * 1013904223u) >> 31) ? amount : -amount;
    const float x0 = first[(long long)b * n + i];
    float x1 = j >= 0 ? v[((long long)b * vstride + j) * n + i] : 0.f;
    if (y && j >= 0) x1 = y[((long long)b * vstride + j) * n + i] - value * x1;
    out[((long long)b * 2) * n + i] = spread > 0.f ? x0 + s0 : x0;
    out[((long long)b * 2 + 1) * n + i] = spread > 0.f ? x1 + s1 : x1;
  }
}

// A_b += sum_j coef[b][j] v_bj v_bj^T  (terms with a zero coefficient are skipped; exact symmetry is kept: the
// product v_r v_c has the same bits at (r, c) and (c, r) and the terms are added in the same order)
__global__ void __launch_bounds__(256) rankr_update_kernel(float* __restrict__ a, const float* __restrict__ v,
                                                           const float* __restrict__ coef, int n, int r, int vstride) {
  ptx::pdl_begin();
  const int b = blockIdx.y;
  float cf[kMaxDeflate];
  bool any = false;
#pragma unroll
  for (int j = 0; j < kMaxDeflate; ++j) {
    cf[j] = j < r ? coef[b * kMaxDeflate + j] : 0.f;
    any = any || cf[j] != 0.f;
  }
  if (!any) return;
  float* A = a + (long long)b * n * n;
  const float* V = v + (long long)b * vstride * n;
  const int n4 = n / 4;
  const long long total = (long long)n * n4;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(i / n4), c = (int)(i - (long long)row * n4) * 4;
    float4 x = *reinterpret_cast<float4*>(A + (long long)row * n + c);
#pragma unroll
    for (int j = 0; j < kMaxDeflate; ++j) {
      if (cf[j] != 0.f) {
        const float vr = V[(long long)j * n + row];
        const float4 vc = *reinterpret_cast<const float4*>(V + (long long)j * n + c);
        x.x = fmaf(cf[j], vr * vc.x, x.x); x.y = fmaf(cf[j], vr * vc.y, x.y);
        x.z = fmaf(cf[j], vr * vc.z, x.z); x.w = fmaf(cf[j], vr * vc.w, x.w);
      }
    }
    *reinterpret_cast<float4*>(A + (long long)row * n + c) = x;
  }
}

// The last pass over the roots: R_b += sum_j coef[b][j] v_bj v_bj^T as above, the partial sums of its squares (the grid, the
// order of the additions and so the bits are sumsq_det's), and its FP16 hi/lo planes scaled by s (a power of two; planes ==
// nullptr: none), the lo plane lo_step matrices behind the hi plane.  One read and two writes of the stack where the three
// passes took four reads and two writes.  inv[b] <- 1 / s, inv2[b] <- 1 / s2.
__global__ void __launch_bounds__(256) root_finish_kernel(float* __restrict__ a, const float* __restrict__ v,
                                                          const float* __restrict__ coef, int n, int r, int vstride, int cstride,
                                                          float s, __half* __restrict__ planes, int lo_step,
                                                          float* __restrict__ inv, float s2, float* __restrict__ inv2,
                                                          float* __restrict__ partial, const float* __restrict__ diag_scale,
                                                          float diag) {
  ptx::pdl_begin();
  const int b = blockIdx.y;
  float cf[kMaxDeflate];
  const float dg = diag_scale ? diag * diag_scale[b] : 0.f;   // added to the diagonal
  bool any = dg != 0.f;
#pragma unroll
  for (int j = 0; j < kMaxDeflate; ++j) {
    cf[j] = j < r ? coef[b * cstride + j] : 0.f;
    any = any || cf[j] != 0.f;
  }
  const long long nn = (long long)n * n;
  float4* A = reinterpret_cast<float4*>(a + b * nn);
  const float* V = v + (long long)b * vstride * n;
  uint2* hi = reinterpret_cast<uint2*>(planes + b * nn);
  uint2* lo = reinterpret_cast<uint2*>(planes + ((long long)lo_step + b) * nn);
  const unsigned n4 = n / 4, total4 = (unsigned)(nn / 4);   // (n <= 65536)
  const unsigned per = (total4 + gridDim.x - 1) / gridDim.x;
  const unsigned first = per * blockIdx.x, last = min(first + per, total4);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (inv) inv[b] = 1.f / s;
    if (inv2) inv2[b] = 1.f / s2;
  }
  auto finished = [&](unsigned i, float4 x) {
    if (any) {
      const unsigned row = i / n4, c = (i - row * n4) * 4;
      if (row - c < 4u) {
        if (row == c) x.x += dg;
        else if (row == c + 1) x.y += dg;
        else if (row == c + 2) x.z += dg;
        else x.w += dg;
      }
#pragma unroll
      for (int j = 0; j < kMaxDeflate; ++j) {
        if (cf[j] != 0.f) {
          const float vr = V[(long long)j * n + row];
          const float4 vc = *reinterpret_cast<const float4*>(V + (long long)j * n + c);
          x.x = fmaf(cf[j], vr * vc.x, x.x); x.y = fmaf(cf[j], vr * vc.y, x.y);
          x.z = fmaf(cf[j], vr * vc.z, x.z); x.w = fmaf(cf[j], vr * vc.w, x.w);
        }
      }
      A[i] = x;
    }
    if (planes) {
      const __half2 h0 = __floats2half2_rn(s * x.x, s * x.y), h1 = __floats2half2_rn(s * x.z, s * x.w);
      const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
      const __half2 l0 = __floats2half2_rn(s * x.x - f0.x, s * x.y - f0.y), l1 = __floats2half2_rn(s * x.z - f1.x, s * x.w - f1.y);
      hi[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
      lo[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
    }
    return x;
  };
  float s0 = 0.f, s1 = 0.f, s2q = 0.f, s3 = 0.f;
  auto square = [&](const float4 x) {
    s0 = fmaf(x.x, x.x, s0); s1 = fmaf(x.y, x.y, s1); s2q = fmaf(x.z, x.z, s2q); s3 = fmaf(x.w, x.w, s3);
  };
  unsigned i = first + threadIdx.x;
  for (; i + 768 < last; i += 1024) {
    const float4 x0 = A[i], x1 = A[i + 256], x2 = A[i + 512], x3 = A[i + 768];
    square(finished(i, x0)); square(finished(i + 256, x1)); square(finished(i + 512, x2)); square(finished(i + 768, x3));
  }
  for (; i < last; i += 256) square(finished(i, A[i]));
  float t = (s0 + s1) + (s2q + s3);
  __shared__ float red[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    float sum = 0.f;
    for (int w = 0; w < 8; ++w) sum += red[w];
    partial[(long long)b * gridDim.x + blockIdx.x] = sum;
  }
}
__global__ void __launch_bounds__(32) root_norm_kernel(const float* __restrict__ partial, float* __restrict__ out) {
  ptx::pdl_begin();
  const float t = sumsq_total(partial + (long long)blockIdx.x * kSumsqBlocks, threadIdx.x);
  if (threadIdx.x == 0) out[blockIdx.x] = t;
}

// With P = A' / ||A'||_F:  lambda_max(P) <= ||P^(2^j)||_F^(1 / 2^j) = (sum lambda^(2^(j+1)))^(1 / 2^(j+1))  for every j, and
// the bound tightens with j (for a flat spectrum it is n^(-1/2) times n^(1/4), n^(1/8), n^(1/16) for j = 1, 2, 3).
// bound^2 <- bound^2 * t^2 with t the smallest of the three, 3 % above it for the single-pass products' rounding.
// late (optional): 1 where the norm puts the spectrum's lower end, damping / norm at least, above late_from.
__global__ void tighten_bound_kernel(float* __restrict__ bound2, const float* __restrict__ ss2, const float* __restrict__ ss4,
                                     const float* __restrict__ ss8, int k, int* __restrict__ late, float late_from, float damping) {
  ptx::pdl_begin();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= k) return;
  float t = 1.f;
  const float t2 = powf(fmaxf(ss2[b], 0.f), 0.25f);
  if (isfinite(t2) && t2 > 0.f) t = fminf(t, 1.03f * t2);
  if (ss4) {
    const float t4 = powf(fmaxf(ss4[b], 0.f), 0.125f);
    if (isfinite(t4) && t4 > 0.f) t = fminf(t, 1.03f * t4);
  }
  if (ss8) {
    const float t8 = powf(fmaxf(ss8[b], 0.f), 0.0625f);
    if (isfinite(t8) && t8 > 0.f) t = fminf(t, 1.03f * t8);
  }
  if (t < 1.f) bound2[b] *= t * t;
  if (late) late[b] = damping > late_from * sqrtf(bound2[b]) ? 1 : 0;   // (not for a NaN)
}

// x <- x - sum_i (v_i . x) v_i over the deflated directions v_i of one statistic (coef[i] != 0).  By a block of 256 threads.
__device__ __forceinline__ void project_out(float* __restrict__ x, const float* __restrict__ v, const float* __restrict__ coef, int n,
                                            int r, double* red) {
  for (int i = 0; i < r; ++i) {
    if (coef[i] == 0.f) continue;
    const float* V = v + (long long)i * n;
    const float dot = (float)block_dot(V, x, n, red);
    for (int j = threadIdx.x; j < n; j += blockDim.x) x[j] = fmaf(-dot, V[j], x[j]);
  }
}
__global__ void __launch_bounds__(256) project_kernel(float* __restrict__ x, const float* __restrict__ v, const float* __restrict__ coef,
                                                      int n, int r, int vstride) {
  ptx::pdl_begin();
  __shared__ double red[8];
  const int b = blockIdx.x;
  project_out(x + ((long long)b * 2 + blockIdx.y) * n, v + (long long)b * vstride * n, coef + b * kMaxDeflate, n, r, red);
}

// v <- (v - y) / ||v - y||  with y = M v:  one power-iteration step on R = I - M;  e[b] = the Rayleigh quotient of R at
// the incoming v, 1 - v.y / v.v (0 where v is zero: nothing is known).
// Vector j = blockIdx.y of statistic b sits at (b * vs + j) * n; its quotient goes to e[j * e_stride + b].
// With defl_v the new v is kept orthogonal to the deflated directions.
// The step of vector 1 is one on (1 - shift) I - M, and lowest[b] (optional, zero at first) keeps the least of its quotients.
__global__ void __launch_bounds__(256) power_shift_kernel(float* __restrict__ v, const float* __restrict__ y, int n,
                                                          float* __restrict__ e, int vs, long long e_stride,
                                                          const float* __restrict__ defl_v, const float* __restrict__ defl_coef,
                                                          int defl_r, int vstride, float shift, float* __restrict__ lowest) {
  ptx::pdl_begin();
  const int b = blockIdx.x;
  const double keep = blockIdx.y == 1 ? 1.0 - (double)shift : 1.0;
  float* V = v + ((long long)b * vs + blockIdx.y) * n;
  const float* Y = y + ((long long)b * vs + blockIdx.y) * n;
  e += (long long)blockIdx.y * e_stride;
  __shared__ double red[3][8];
  __shared__ double tot[3];
  double vy = 0.0, vv = 0.0, tt = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double yi = Y[i], vi = V[i], d = keep * vi - yi;
    vy += vi * yi;
    vv += vi * vi;
    tt += d * d;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vy += __shfl_xor_sync(0xffffffffu, vy, o);
    vv += __shfl_xor_sync(0xffffffffu, vv, o);
    tt += __shfl_xor_sync(0xffffffffu, tt, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = vy;
    red[1][threadIdx.x >> 5] = vv;
    red[2][threadIdx.x >> 5] = tt;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[threadIdx.x][w];
    tot[threadIdx.x] = t;
  }
  __syncthreads();
  const double inv = tot[2] > 0.0 ? 1.0 / sqrt(tot[2]) : 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) V[i] = (float)((keep * (double)V[i] - (double)Y[i]) * inv);
  if (threadIdx.x == 0) {
    const float quotient = tot[1] == 0.0 ? 0.f : (float)(1.0 - tot[0] / tot[1]);   // (NaN stays NaN)
    e[b] = quotient;
    if (lowest && blockIdx.y == 1) lowest[b] = fminf(lowest[b], quotient);
  }
  if (defl_v) project_out(V, defl_v + (long long)b * vstride * n, defl_coef + b * kMaxDeflate, n, defl_r, red[0]);
}

// status 4 where the distance of the last M from the identity, estimated by power iteration on I - M, exceeds what the
// schedule was built for: the caller's estimate of the spectrum's lower end was too high for this statistic.  With theta and
// rest_trace (a graded finish) e may have either sign, and the rounding of A's entries is allowed for as well: where one
// eigenvalue theta_1 is far above the mean c of the rest, 2^-24 theta_1 |v_i v_j| of them, is 2^-24 theta_1 / (c sqrt(n)) of R
// (a mean of 20 standard deviations, 1000 wide: 1e-4 to 3.5e-4 seen, 7.6e-4 allowed for).
__global__ void verify_kernel(const float* __restrict__ e_est, const float* __restrict__ e_top, float e_allowed, float e_below,
                              int* __restrict__ status, float* __restrict__ e_out, int k, const float* __restrict__ theta,
                              const float* __restrict__ rest_trace, int n, const float* __restrict__ lowest) {
  ptx::pdl_begin();
  const bool both_signs = theta != nullptr;
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= k) return;
  // (an even T sends what lies above the norm above 1: R negative there, past what the finish was fitted to)
  auto size = [&](float x) { return both_signs ? fabsf(x) : (x < -e_below ? 1.f - x : x); };
  float e = size(e_est[b]);
  if (e_top && isfinite(e)) {   // (fmaxf would pass over a NaN)
    const float t = size(e_top[b]);
    e = isfinite(t) ? fmaxf(e, t) : t;
    if (lowest && isfinite(e)) e = fmaxf(e, size(lowest[b]));
  }
  if (e_out) e_out[b] = e;
  if (theta) e_allowed += 5.96e-8f * sqrtf((float)n) * theta[b * kMaxDeflate] / rest_trace[b];
  if (status && status[b] == 0 && (!isfinite(e) || e > e_allowed)) status[b] = 4;
}

// After steps of higher degree R may reach this far below zero: the finish is fitted to kFinishLow, and a Rayleigh quotient of
// four power steps sits inside the spectrum.
constexpr float kSteepBelow = 0.03f;

// lmin[b] = theta^(-power): the smallest eigenvalue of A from the largest eigenvalue theta (a Rayleigh quotient, so a
// lower estimate) of its computed inverse root A^(-1/power).
__global__ void lmin_from_root_kernel(const float* __restrict__ theta, float power, float* __restrict__ lmin, int k) {
  ptx::pdl_begin();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= k) return;
  const float t = theta[b];
  lmin[b] = (isfinite(t) && t > 0.f) ? powf(t, -power) : 0.f;
}

// Per statistic: the scale that turns M_0^{-1/p} into A^{-1/p}, and the convergence status from the
// distance max|I - M| gathered when the last M was produced (0 converged, 1 above tol, 2 non-finite).
// 3: the statistic's spectrum reaches below the lower bound the schedule was built for (caller's bound too high).
// Also the bound of the finished root's entries for its operand planes: a symmetric positive matrix has no entry above
// its largest eigenvalue, and A >= damping I by construction, so |A^(-1/p)|_ij <= damping^(-1/p) -- known without a
// pass over the result.
// With `ritz` (steps of higher degree under an estimated norm: the Ritz values of A, the largest of which is finite only where A
// is) a residual that is not finite is 2 only where A is not finite: T of degree four, raised to the p-th power, overflows where
// the norm was far too low, as a linear T does not.
__global__ void finish_kernel(const unsigned int* __restrict__ resid, const float* __restrict__ sumsq_a,
                              float* root_scale_lo, int* status, float* norm_out, int k, int p, float tol, float damping,
                              float lower_used, const float* __restrict__ ritz) {
  ptx::pdl_begin();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= k) return;
  const float ub = sqrtf(fmaxf(sumsq_a[b], 1e-60f));
  root_scale_lo[b] = powf(ub, -1.f / p);
  if (norm_out) norm_out[b] = ub;
  const float r = __uint_as_float(resid[b]);
  int st = !isfinite(r) ? (ritz && isfinite(ritz[b * kMaxDeflate]) ? 1 : 2) : (r > tol ? 1 : 0);
  // lower_used < 0: the bound is an estimate, verified after the chain instead (verify_kernel)
  if (st == 0 && lower_used > 0.f && damping / ub < lower_used * 0.999f) st = 3;
  if (status) status[b] = st;
}

// What the host reads after a factorisation, written straight to its pinned memory: status, norms, lmin, deflated (k words
// each) and the status word of the kernels' bounded waits.  One launch instead of five copies of a few bytes.
__global__ void report_kernel(const int* __restrict__ status, const float* __restrict__ norms, const float* __restrict__ lmin,
                              const int* __restrict__ deflated, const int* __restrict__ word, int* __restrict__ host, int k) {
  ptx::pdl_begin();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b == 0) host[4 * k] = *word;
  if (b >= k) return;
  host[b] = status[b];
  host[k + b] = __float_as_int(norms[b]);
  host[2 * k + b] = __float_as_int(lmin[b]);
  host[3 * k + b] = deflated[b];
}

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

static size_t per_statistic_bytes(int n) {
  // A (FP32) + seven FP16 hi/lo plane pairs (T, M x2, X x2, two powers of T) = 8 FP32-sized matrices
  return align_up((size_t)n * n * 4, 256) * 8;
}
static size_t small_bytes(int chunk, int n) {
  // twenty per-statistic scalars, four blocks of kMaxDeflate scalars per statistic (Ritz values, residuals, deflation
  // coefficients, root corrections), the reduction scratch, and two blocks of as many n-vectors per statistic
  // (block power iteration: V and A V)
  return align_up((size_t)chunk * 4, 256) * 20 + 4 * align_up((size_t)chunk * kMaxDeflate * 4, 256) +
         align_up(sumsq_scratch_bytes(chunk), 256) + 2 * align_up((size_t)chunk * kMaxDeflate * n * 4, 256);
}

// Largest power of two s with s * bound <= 2^14: FP16 planes of s * x then stay a factor four below overflow
// for |x| <= bound, and elements down to 2^-16 of the bound keep all 22 bits of the hi/lo pair.
static float plane_scale(double bound) {
  return (float)std::ldexp(1.0, (int)std::floor(std::log2(16384.0 / bound)));
}
// The scale toner_split16 gives a matrix whose largest entry is `bound`.
static float root_plane_scale(double bound) {
  int e;
  std::frexp((float)bound, &e);
  return (float)std::ldexp(1.0, 14 - e);
}

}  // namespace toner

extern "C" {

size_t toner_inv_roots_workspace_bytes(int32_t chunk, int32_t n) {
  if (chunk <= 0 || n <= 0) return 0;
  return toner::per_statistic_bytes(n) * (size_t)chunk + toner::small_bytes(chunk, n);
}

int toner_inv_roots_iterations(int32_t n, float damping, int32_t p) {
  if (n <= 0 || !(damping > 0) || p < 1) return 0;
  return toner::schedule_for((double)damping / ((double)n * (1.0 + damping)), p, 0).iters;
}

int toner_inv_roots_iterations_for(float lower, int32_t p) {
  if (!(lower > 0.f) || !(lower < 1.f) || p < 1) return 0;
  return toner::schedule_for((double)lower, p, 0).iters;
}

int toner_inv_roots_finish_order_for(float lower, int32_t p, int32_t iters) {
  if (!(lower > 0.f) || !(lower < 1.f) || p < 1) return 0;
  const toner::Schedule& s = toner::schedule_for((double)lower, p, iters);
  return s.iters < 2 ? 0 : s.fin.order;
}

int toner_inv_roots_finish_products_for(float lower, int32_t p, int32_t iters, int32_t plane_order) {
  if (!(lower > 0.f) || !(lower < 1.f) || p < 1) return 0;
  const toner::Schedule& s = toner::schedule_for((double)lower, p, iters);
  if (s.iters < 2) return 0;
  toner::QuadraticSteps q;
  if (plane_order || p == 1 || !toner::quadratic_steps(s.fin, p, q)) return s.fin.order - 1;
  return 1 + (int)q.lin.size() + (q.by_r ? 1 : 0);
}

int toner_inv_roots_schedule(float lower, int32_t p, int32_t iters, double* ab_out, int32_t ab_capacity, double* coef_out,
                             int32_t coef_capacity, int32_t* order_out, double* e_out) {
  if (!(lower > 0.f) || !(lower < 1.f) || p < 1) return 0;
  const toner::Schedule& s = toner::schedule_for((double)lower, p, iters);
  if (s.iters < 2) return 0;
  if (ab_out) {
    for (int k = 0; k < s.iters - 1 && 2 * k + 1 < ab_capacity; ++k) {
      ab_out[2 * k] = s.steps[k].a;
      ab_out[2 * k + 1] = s.steps[k].b;
    }
  }
  if (coef_out)
    for (int j = 0; j <= s.fin.order && j < coef_capacity; ++j) coef_out[j] = s.fin.c[j];
  if (order_out) *order_out = s.fin.order;
  if (e_out) *e_out = 1.0 - s.l_last;
  return s.iters;
}

int toner_inv_roots_graded_for(float lower, int32_t p, int32_t n, int32_t* steps_out, int32_t* split_out, double* coef_out,
                               int32_t coef_capacity) {
  if (!(lower > 0.f) || !(lower < 1.f) || p < 2 || n <= 0) return 0;
  const toner::Schedule& s = toner::schedule_for((double)lower, p, 0, n);
  const toner::GradedPoly& g = s.graded;
  if (!g.products) return 0;
  if (steps_out) *steps_out = 0;
  if (split_out) *split_out = g.split;
  if (coef_out) {
    if (coef_capacity > 0) coef_out[0] = g.zb;
    if (coef_capacity > 1) coef_out[1] = g.za;
    for (int j = 0; j <= g.products && 2 * j + 3 < coef_capacity; ++j) {
      coef_out[2 * j + 2] = g.alpha[j];
      coef_out[2 * j + 3] = g.beta[j];
    }
  }
  return g.products;
}

int toner_inv_roots_steps_for(float lower, int32_t p, int32_t n, int32_t kind, double* step_out, int32_t step_capacity,
                              double* coef_out, int32_t coef_capacity, int32_t* order_out, int32_t* products_out, double* e_out,
                              double* late_out) {
  if (!(lower > 0.f) || !(lower < 1.f) || p < 2 || (p & (p - 1)) || p > 32 || n <= 0 || kind < 0 || kind > 2) return 0;
  const toner::Schedule& s = toner::schedule_for((double)lower, p, 0, 0, n, kind);
  if (!s.steep) return 0;
  if (late_out) *late_out = s.late;
  int log2p = 0, split = 0;
  while ((1 << log2p) < p) ++log2p;
  for (int k = 0; k < s.iters - 1; ++k) {
    const toner::NewtonStep& st = s.steps[k];
    split += log2p + 2 + (st.degree == 4 ? 2 : st.degree - 1);
    if (!step_out || 7 * k + 6 >= step_capacity) continue;
    const double out[7] = {(double)st.degree, st.zb, st.za, st.kappa, st.top, st.degree == 1 ? -st.b : st.lin, st.degree == 1 ? st.a : st.con};
    for (int j = 0; j < 7; ++j) step_out[7 * k + j] = out[j];
  }
  toner::QuadraticSteps q;
  if (coef_out)
    for (int j = 0; j <= s.fin.order && j < coef_capacity; ++j) coef_out[j] = s.fin.c[j];
  if (order_out) *order_out = s.fin.order;
  if (products_out) {
    products_out[0] = split + 1;
    products_out[1] = toner::quadratic_steps(s.fin, p, q) ? (int)q.lin.size() + (q.by_r ? 1 : 0) : s.fin.order - 2;
  }
  if (e_out) *e_out = 1.0 - s.l_last;
  return s.iters - 1;
}

int toner_factor_report(const int32_t* status, const float* norms, const float* lmin, const int32_t* deflated, int32_t k,
                        int32_t* host_out, void* stream) {
  using namespace toner;
  Context* ctx = context();
  if (!ctx) return kErrCuda;
  if (!status || !norms || !lmin || !deflated || !host_out || k <= 0) return fail(kErrArg, "factor_report: bad arguments");
  TONER_LAUNCH(report_kernel, (k + 127) / 128, 128, static_cast<cudaStream_t>(stream), status, norms, lmin, deflated, ctx->status_dev,
               host_out, k);
  return 0;
}

int toner_inv_roots(const float* ema, int32_t k, int32_t n, float damping, int32_t p, int32_t q, int32_t iters,
                    float* root_lo, float* root_hi, float* fro2_lo, int32_t* status, void* workspace,
                    size_t workspace_bytes, void* stream_) {
  return toner_inv_roots_ex(ema, k, n, damping, p, q, iters, 0.f, root_lo, root_hi, fro2_lo, status, nullptr, workspace,
                            workspace_bytes, stream_);
}

int toner_inv_roots_ex(const float* ema, int32_t k, int32_t n, float damping, int32_t p, int32_t q, int32_t iters,
                       float lower, float* root_lo, float* root_hi, float* fro2_lo, int32_t* status, float* norm_out,
                       void* workspace, size_t workspace_bytes, void* stream_) {
  return toner_inv_roots_tracked(ema, k, n, damping, p, q, iters, lower, 0, root_lo, root_hi, fro2_lo, status, norm_out,
                                 nullptr, nullptr, nullptr, 0, nullptr, 0, nullptr, workspace, workspace_bytes, stream_);
}

int toner_inv_roots_tracked(const float* ema, int32_t k, int32_t n, float damping, int32_t p, int32_t q, int32_t iters,
                            float lower, int32_t lower_is_estimate, float* root_lo, float* root_hi, float* fro2_lo,
                            int32_t* status, float* norm_out, float* track, float* lmin_out, float* resid_out,
                            int32_t track_sweeps, float* deflate, int32_t deflate_rank, int32_t* deflated_out,
                            void* workspace, size_t workspace_bytes, void* stream_) {
  return toner_inv_roots_planes(ema, k, n, damping, p, q, iters, lower, lower_is_estimate, root_lo, root_hi, fro2_lo, status, norm_out,
                                track, lmin_out, resid_out, track_sweeps, deflate, deflate_rank, deflated_out, nullptr, nullptr,
                                nullptr, nullptr, workspace, workspace_bytes, stream_);
}

int toner_inv_roots_planes(const float* ema, int32_t k, int32_t n, float damping, int32_t p, int32_t q, int32_t iters,
                           float lower, int32_t lower_is_estimate, float* root_lo, float* root_hi, float* fro2_lo,
                           int32_t* status, float* norm_out, float* track, float* lmin_out, float* resid_out,
                           int32_t track_sweeps, float* deflate, int32_t deflate_rank, int32_t* deflated_out,
                           void* lo_planes, float* lo_inv, void* hi_planes, float* hi_inv,
                           void* workspace, size_t workspace_bytes, void* stream_) {
  using namespace toner;
  if (!ema || !root_lo || !workspace) return fail(kErrArg, "inv_roots: null pointer");
  if (k <= 0 || n <= 0) return fail(kErrArg, "inv_roots: sizes must be positive");
  if (!lo_planes != !lo_inv || !hi_planes != !hi_inv || (hi_planes && q == 1))
    return fail(kErrArg, "inv_roots: planes come with their inverse scales, the second root's only where there is one");
  if ((reinterpret_cast<uintptr_t>(lo_planes) | reinterpret_cast<uintptr_t>(hi_planes)) & 15u)
    return fail(kErrArg, "inv_roots: operand planes must be 16-byte aligned");
  // (`ema` may start anywhere; root_hi is read by 16 bytes only where its smallest direction is tracked)
  if ((reinterpret_cast<uintptr_t>(root_lo) | reinterpret_cast<uintptr_t>(workspace) | reinterpret_cast<uintptr_t>(deflate)) & 15u)
    return fail(kErrArg, "inv_roots: root_lo, deflate and workspace must be 16-byte aligned");
  if (track && (track_sweeps & 63) != 0 && ((reinterpret_cast<uintptr_t>(track) | reinterpret_cast<uintptr_t>(root_hi)) & 15u))
    return fail(kErrArg, "inv_roots: track and root_hi must be 16-byte aligned where the smallest direction is tracked");
  Context* ctx = context();
  if (!ctx) return kErrCuda;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (n % 8 != 0) return fail(kErrUnsupported, "inv_roots: n must be a multiple of 8");
  if (!(damping > 0.f)) return fail(kErrArg, "inv_roots: damping must be positive");
  if (p < 1 || p > 32 || (p & (p - 1))) return fail(kErrUnsupported, "inv_roots: root order p must be a power of two <= 32");
  if (q < 1 || q > p || (q & (q - 1))) return fail(kErrUnsupported, "inv_roots: q must be a power of two <= p");
  if (q > 1 && !root_hi) return fail(kErrArg, "inv_roots: root_hi is required when q > 1");
  // Lower bound of the normalised spectrum the schedule is built for: the caller's (checked per statistic, status 3
  // where it does not hold), else the bound that holds for every statistic, damping / (n (1 + damping)).
  const double l_worst = (double)damping / ((double)n * (1.0 + damping));
  if (lower != 0.f && !(lower > 0.f && lower < 1.f)) return fail(kErrArg, "inv_roots: lower must be 0 or inside (0, 1)");
  const double l0 = (lower > 0.f && (double)lower > l_worst) ? (double)lower : l_worst;
  const bool estimated = lower_is_estimate != 0 && l0 > l_worst;
  if (estimated && !track) return fail(kErrArg, "inv_roots: an estimated bound needs the tracking vectors to verify it");
  if (track_sweeps < 0 || (track_sweeps & ~(63 | 256 | 512)))
    return fail(kErrArg, "inv_roots: track_sweeps is 0..63, plus 256 to start afresh, plus 512 for plane-by-plane products");
  const int defl_r = deflate ? (deflate_rank & 15) : 0;      // directions the block iteration looks for (0: one, the old way)
  const bool defl_cold = deflate && (deflate_rank & 256);
  const int slots = (deflate_rank & 1024) ? kMoreSlots : kSlots;
  const bool ritz_norm = deflate && (deflate_rank & 512);   // norm from the block iteration instead of three squarings
  if (deflate && (defl_r < 1 || defl_r > slots || (deflate_rank & ~(15 | 256 | 512 | 1024))))
    return fail(kErrArg, "inv_roots: deflate_rank is 1..8, plus 256 to start from fixed vectors, plus 512 to take the "
                         "norm from the block iteration; 1..12 with 1024, twelve slots a statistic");
  if (deflate && defl_r > kSlots && (track_sweeps & 512))
    return fail(kErrUnsupported, "inv_roots: calls in plane order look for eight directions at most");
  if (ritz_norm && (defl_cold || !estimated))
    return fail(kErrArg, "inv_roots: the norm estimate needs vectors from an earlier call and an estimated lower bound "
                         "(both are verified together after the chain)");
  // > 0: certified bound, checked against damping / norm per statistic; < 0: estimate, verified after the chain
  const float lower_used = l0 > l_worst ? (estimated ? -(float)l0 : (float)l0) : 0.f;
  // (verifying the estimate after a graded finish takes A^(-1/2) and the deflated vectors)
  const bool may_grade = estimated && iters <= 0 && (track_sweeps & 512) == 0 && p > 1 && 2 * q == p && defl_r > 0 &&
                         (reinterpret_cast<uintptr_t>(root_hi) & 15u) == 0;
  // (steps of higher degree: other roundings, so not where the plane-by-plane order is asked for, nor where the count is)
  const Schedule plan = schedule_for(l0, p, iters, may_grade ? n : 0, iters <= 0 && (track_sweeps & 512) == 0 ? n : 0,
                                     estimated ? 0 : (l0 > l_worst ? 1 : 2));
  iters = plan.iters;
  const GradedPoly& graded = plan.graded;
  if (iters < 2 && !graded.products) return fail(kErrArg, "inv_roots: at least two iterations are required");
  const std::vector<NewtonStep>& sched = plan.steps;
  const double l_last = plan.l_last;
  const FinishPoly& fin = plan.fin;
  const int order = fin.order;
  int log2p = 0;
  while ((1 << log2p) < p) ++log2p;

  const size_t per = per_statistic_bytes(n);
  long long chunk_cap = 0;
  for (long long c = k; c >= 1; --c) {
    if (per * (size_t)c + small_bytes((int)c, n) <= workspace_bytes) {
      chunk_cap = c;
      break;
    }
  }
  if (chunk_cap < 1) return fail(kErrWorkspace, "inv_roots: workspace holds less than one statistic");
  const long long nn = (long long)n * n;
  const size_t mat = align_up((size_t)nn * 4, 256);
  const int ew_blocks = (int)std::min<long long>((nn / 4 + 255) / 256, 8LL * ctx->num_sms / (k < 8 ? k : 8) + 1);

  // Plane scales from norm bounds known in advance (no pass over the data is needed to find them):
  // ||M_k|| <= 1, ||T_k|| <= a_k, ||T_k^(2^j)|| <= a_k^(2^j), ||X_k|| <= min(prod_{j<k} a_j, l0^(-1/p)),
  // ||A^(-1/p)|| <= damping^(-1/p).
  const float s_m = plane_scale(1.0);
  const double x_cap = 1.01 * std::pow(l0, -1.0 / p);
  const double root_bound = 1.01 * std::pow((double)damping, -1.0 / p);

  for (int k0 = 0; k0 < k; k0 += (int)chunk_cap) {
    const int kc = (int)std::min<long long>(chunk_cap, k - k0);
    char* w = static_cast<char*>(workspace);
    float* A32 = reinterpret_cast<float*>(w); w += mat * kc;
    __half* Tb[2];
    __half* Mb[2];
    __half* Xb[2];
    __half* Pb[2];
    Tb[0] = reinterpret_cast<__half*>(w); w += mat * kc;
    Mb[0] = reinterpret_cast<__half*>(w); w += mat * kc;
    Mb[1] = reinterpret_cast<__half*>(w); w += mat * kc;
    Xb[0] = reinterpret_cast<__half*>(w); w += mat * kc;
    Xb[1] = reinterpret_cast<__half*>(w); w += mat * kc;
    Pb[0] = reinterpret_cast<__half*>(w); w += mat * kc;
    Pb[1] = reinterpret_cast<__half*>(w); w += mat * kc;
    Tb[1] = Pb[0];  // p == 1 has no powers of T to store: the next T is written beside the current one
    const size_t sm = align_up((size_t)kc * 4, 256);
    auto small = [&](int i) { return reinterpret_cast<float*>(w + sm * i); };
    float* trace = small(0);
    float* sumsq_a = small(1);
    unsigned int* resid = reinterpret_cast<unsigned int*>(small(2));
    float* scale_lo = small(3);
    float* fro_tmp = small(4);
    float* lam = small(5);
    float* pres = small(6);
    float* neg_sigma = small(7);
    float* corr = small(8);
    float* inv_r = small(9);
    float* ss2 = small(11);
    float* ss4 = small(12);
    float* ss8 = small(13);
    float* e_est = small(14);
    float* theta = small(15);
    float* rest_top = small(16);
    int* rest_idx = reinterpret_cast<int*>(small(17));
    float* e_top = small(18);
    float* rest_trace = small(10);
    float* const lowest = plan.steep && ritz_norm ? small(19) : nullptr;   // (`late` is for calls that certify the norm)
    const size_t sm8 = align_up((size_t)kc * kMaxDeflate * 4, 256);
    char* wp = w + sm * 20;
    float* th8 = reinterpret_cast<float*>(wp); wp += sm8;     // Ritz values, residuals, deflation coefficients and
    float* res8 = reinterpret_cast<float*>(wp); wp += sm8;    // root corrections of the block deflation
    float* coef8 = reinterpret_cast<float*>(wp); wp += sm8;
    float* corr8 = reinterpret_cast<float*>(wp); wp += sm8;
    float* partials = reinterpret_cast<float*>(wp); wp += align_up(sumsq_scratch_bytes(kc), 256);
    const size_t vec = align_up((size_t)kc * kMaxDeflate * n * 4, 256);
    float* pv = reinterpret_cast<float*>(wp);
    float* py = reinterpret_cast<float*>(wp + vec);
    float* dv = deflate ? deflate + (long long)k0 * slots * n : nullptr;
    TONER_CUDA(cudaMemsetAsync(w, 0, sm * 20 + 4 * sm8, stream));

    const float* C = ema + (long long)k0 * nn;
    const int damp_tiles = (n + kDampTile - 1) / kDampTile;
    TONER_LAUNCH(trace_kernel, kc, 256, stream, C, n, trace);
    TONER_LAUNCH((reinterpret_cast<uintptr_t>(C) & 15u) == 0 ? damp_kernel<true> : damp_kernel<false>,
                 dim3(damp_tiles * (damp_tiles + 1) / 2, kc), 256, stream, C, A32, n, damping, trace);
    if (defl_r > 0) {
      // dominant directions: block power iteration with Rayleigh-Ritz on the caller's vectors (eight sweeps from fixed
      // vectors -- the first three or four only find the subspace --, four from last call's), then deflate those that
      // converged and stand above the rest
      const int sweeps = defl_cold ? 8 : 4, in_order = (track_sweeps & 512) ? 1 : 0;
      auto iterate = [&](auto width) -> int {   // (R as a type: every kernel of the iteration is specialised for it)
        constexpr int R = decltype(width)::value;
        TONER_LAUNCH(block_start_kernel<R>, kc, 256, stream, dv, n, defl_r, slots, defl_cold ? 1 : 0, in_order);
        for (int sw = 0; sw < sweeps; ++sw) {
          TONER_CUDA(launch_block_gemv<R>(kc, stream, A32, dv, py, n, defl_r, slots));
          // (the last step of the power iteration is one on A itself, see ritz_kernel)
          const float trace = sw < sweeps - 2 ? (float)((double)n * (1.0 + (double)damping)) : 0.f;
          TONER_CUDA(launch_ritz<R>(kc, stream, dv, py, n, defl_r, slots, sw == sweeps - 1 ? 1 : 0, th8, res8, in_order, trace));
        }
        return 0;
      };
      int rcd;
      if (defl_r <= 2) rcd = iterate(std::integral_constant<int, 2>());
      else if (defl_r <= 4) rcd = iterate(std::integral_constant<int, 4>());
      else if (defl_r <= 6) rcd = iterate(std::integral_constant<int, 6>());
      else if (defl_r <= 8) rcd = iterate(std::integral_constant<int, 8>());
      else if (defl_r <= 10) rcd = iterate(std::integral_constant<int, 10>());
      else rcd = iterate(std::integral_constant<int, 12>());
      if (rcd) return rcd;
      TONER_LAUNCH(block_decide_kernel, (kc + 127) / 128, 128, stream, th8, res8, kc, n, defl_r, damping, p, ritz_norm ? defl_r - 1 : defl_r, coef8, corr8, deflated_out ? deflated_out + k0 : nullptr, rest_top, rest_idx, rest_trace);
      if (!ritz_norm) {   // (with the norm estimate the deflation is applied where the operand planes are formed)
        TONER_LAUNCH(rankr_update_kernel, dim3(ew_blocks, kc), 256, stream, A32, dv, coef8, n, defl_r, slots);
      }
    } else {
      // dominant direction: six power-iteration steps, then deflate where they converged
      TONER_LAUNCH(power_start_kernel, dim3(8, kc), 256, stream, pv, n);
      for (int pi = 0; pi < kPowerSteps; ++pi) {
        TONER_LAUNCH(gemv_kernel, dim3((n + 7) / 8, kc), 256, stream, A32, pv, py, n);
        TONER_LAUNCH(power_norm_kernel, kc, 256, stream, pv, py, n, lam, pres);
      }
      TONER_LAUNCH(deflate_decide_kernel, (kc + 127) / 128, 128, stream, lam, pres, kc, n, damping, p, neg_sigma, corr);
      TONER_LAUNCH(rank1_update_kernel, dim3(ew_blocks, kc), 256, stream, A32, pv, neg_sigma, n);
    }
    TONER_CUDA(cudaGetLastError());
    if (!ritz_norm) {
      int rc0 = sumsq_det(A32, kc, n, n, n, nn, partials, sumsq_a, stream);
      if (rc0) return rc0;
    }
    // What the engine starts from: planes of M_0 and of T_0 = a I - b M_0; for a graded finish those of Z
    // in T_0's place, and M_0 in FP32 with the hi plane of M_0 + g I, of which W_K is a multiple
    const bool graded_finish = graded.products > 0;
    // plane products interleaved (toner_gemm_desc::interleave), and the finish in its short form: unless the caller asked for
    // the plane-by-plane order of additions
    const bool interleave = (track_sweeps & 512) == 0;
    // Operand planes between products are stored by half: writing the mirror images took 4 to 10 % of a product (12 x 3072 in chains
    // of two, one / two pairs of planes: 948 -> 906 and 1055 -> 958 us; 36 x 768 81 -> 76 and 98 -> 90; a product of the finish, with C,
    // 12 x 3072 390 -> 348).  On the few matrices of a small step a map more per operand costs the host what it saves.
    // Half storage takes tiles of CTA pairs, and narrow statistics are faster on others: whole over half, a call on 4 Mi / 12 Mi elements,
    // 0.60 at 64 columns, 0.74 at 128, 0.96 / 0.80 at 256, 0.87 / 0.91 at 264, 0.83 at 320, 0.98 / 0.91 at 384, 1.00 / 1.04 at 440, 1.03 at 504, 1.04 /
    // 1.06 at 512, 1.01 / 0.98 at 576, 1.04 / 1.09 at 768.  (Interleaved linear steps in long chains also round by the tile: square roots of
    // 64 x 264 were 2.45e-5 off on pairs and 2.08e-5 on theirs.)
    const bool half = (long long)kc * nn >= kHalfFrom && n >= (plan.steep || graded_finish || !interleave ? 440 : 512);
    const double top_gain = graded.products ? graded.beta[graded.products] * graded.za : 1.0;
    const double top_diag =
        graded.products ? (graded.alpha[graded.products] + graded.beta[graded.products] * graded.zb) / top_gain : 0.0;
    const bool first_z = graded_finish || sched[0].degree > 1;   // planes of Z instead of T_0's
    float* const m32 = graded_finish || sched[0].lin != 0.0 ? reinterpret_cast<float*>(Xb[0]) : nullptr;   // M_0
    __half* const first_planes = first_z && !graded_finish ? Tb[0] : Xb[1];
    double most_z = graded_finish ? 1.2 : 0.0;   // (one scale for all steps: statistics that start late have the second Z in the first one's planes)
    for (int i = 0; !graded_finish && i < iters - 1; ++i) most_z = std::max(most_z, sched[i].most_z);
    const float s_z = plane_scale(most_z > 0.0 ? most_z : 1.0), s_top = plane_scale(1.1 * (1.0 + std::fabs(top_diag)));
    const float init_a = (float)(graded_finish ? graded.zb : first_z ? sched[0].zb : sched[0].a);
    const float init_b = (float)(graded_finish ? -graded.za : first_z ? -sched[0].za : sched[0].b);
    const float init_sm = graded_finish ? s_top : s_m, init_diag = graded_finish ? (float)top_diag : 0.f;
    float s_t = first_z ? s_z : plane_scale(sched[0].a);
    // Statistics that start with the second step: M_0 where the first one leaves M, planes of the second Z, and the first step's
    // products left out; T_1 is their X_2 (the product with X is left out too).
    int* const late = plan.late > 0.0 ? reinterpret_cast<int*>(small(19)) : nullptr;
    InitLate second = {};
    if (late) second = {(float)sched[1].zb, (float)-sched[1].za, Mb[1], Tb[0], sched[1].lin != 0.0 ? A32 : nullptr};
    if (ritz_norm) {
      // Neither A' nor its Frobenius norm is formed: the norm is the estimate (capped by the trace), and the planes of
      // M_0 and T_0 are made from A with the deflation applied on the way.
      TONER_LAUNCH(ritz_norm_kernel, (kc + 127) / 128, 128, stream, sumsq_a, rest_top, rest_trace, kc);
      TONER_LAUNCH(init_planes_kernel, dim3(ew_blocks, kc), 256, stream, A32, n, kc, sumsq_a, init_a, init_b, init_sm, s_t, Mb[0], first_planes, dv, coef8, defl_r, slots, m32, init_diag, graded_finish, nullptr, InitLate(), half);
      TONER_CUDA(cudaGetLastError());
    } else {
    TONER_LAUNCH(init_planes_kernel, dim3(ew_blocks, kc), 256, stream, A32, n, kc, sumsq_a, 0.f, 0.f, s_m, s_t, Mb[0], nullptr, nullptr, nullptr, 0, 0, nullptr, 0.f, false, nullptr, InitLate(), half);
    TONER_CUDA(cudaGetLastError());
    {
      // A tighter bound of the largest eigenvalue than ||A'||_F: with P = A' / ||A'||_F, lambda_max(P) <= ||P^2||_F^(1/2)
      // = (sum lambda^4)^(1/4), and likewise ||P^4||_F^(1/4), ||P^8||_F^(1/8).  For a flat spectrum these are n^(-1/4),
      // n^(-3/8), n^(-7/16) instead of 1, which raises the spectrum's lower bound after normalisation by the same factor
      // and saves Newton steps (each costs fifteen plane passes; these three squarings cost one pass each).  Single-pass
      // products of hi planes are accurate enough for a bound (3 % is added); the FP32 results and the planes of P^2
      // and P^4 (written by the epilogues, entries at most 1) go to buffers that are free here.
      float* P2 = reinterpret_cast<float*>(Pb[0]);
      const float s_w = plane_scale(1.0);
      toner_gemm_desc g = {};
      toner_operand op = {};
      op.base = Mb[0];
      op.rows = n; op.cols = n; op.ld = n; op.z_stride = nn; op.nz = 2 * kc; op.z_step = 1;
      g.a = op; g.b = op;
      g.m = n; g.n = n; g.k = n; g.batch = kc; g.segs = 1; g.fmt = 0;
      g.tri = 1; g.mirror = 1;
      g.alpha = (float)(1.0 / ((double)s_m * (double)s_m));
      g.d = P2; g.ldd = n; g.d_bs = nn;
      g.split0 = Pb[1]; g.split0_scale = s_w; g.split_ld = n; g.split_bs = nn; g.split_plane = (long long)kc * nn;
      GemmMore planes;
      planes.half_in = planes.half_out = half;
      int rc1 = launch_gemm(g, stream, planes);
      if (rc1) return rc1;
      rc1 = sumsq_det(P2, kc, n, n, n, nn, partials, ss2, stream);
      if (rc1) return rc1;
      float* P4 = reinterpret_cast<float*>(Xb[0]);
      toner_gemm_desc g4 = g;
      g4.a.base = Pb[1]; g4.b.base = Pb[1];
      g4.alpha = (float)(1.0 / ((double)s_w * (double)s_w));
      g4.d = P4; g4.split0 = Mb[1];
      rc1 = launch_gemm(g4, stream, planes);
      if (rc1) return rc1;
      rc1 = sumsq_det(P4, kc, n, n, n, nn, partials, ss4, stream);
      if (rc1) return rc1;
      toner_gemm_desc g8 = g4;
      g8.a.base = Mb[1]; g8.b.base = Mb[1];
      g8.d = P2; g8.split0 = nullptr;
      rc1 = launch_gemm(g8, stream, planes);
      if (rc1) return rc1;
      rc1 = sumsq_det(P2, kc, n, n, n, nn, partials, ss8, stream);
      if (rc1) return rc1;
      TONER_LAUNCH(tighten_bound_kernel, (kc + 127) / 128, 128, stream, sumsq_a, ss2, ss4, ss8, kc, late, (float)(1.0001 * plan.late), damping);
      TONER_LAUNCH(init_planes_kernel, dim3(ew_blocks, kc), 256, stream, A32, n, kc, sumsq_a, init_a, init_b, init_sm, s_t, Mb[0], first_planes, nullptr, nullptr, 0, 0, m32, init_diag, graded_finish, late, second, half);
      TONER_CUDA(cudaGetLastError());
    }
    }

    // D = (A planes) * (B planes)^T / (sa * sb): symmetric result, FP32-accurate; outputs as requested
    struct Out {
      float* d = nullptr;           // FP32 result
      const float* alpha_a = nullptr;  // optional per-statistic factors of the result
      const float* alpha_b = nullptr;
      __half* s0 = nullptr; float s0_scale = 0.f, s0_a = 0.f;
      __half* s1 = nullptr; float s1_scale = 0.f, s1_a = 0.f, s1_b = 0.f;
      unsigned int* maxres = nullptr;
      int lo_step = 0;              // s0: matrices between its hi and lo planes (0: the chunk's)
      const float* c = nullptr; float beta = 0.f;  // result = gain * product + beta * c (c symmetric, FP32)
      const float* beta_v = nullptr;               // per-statistic factors of beta
      double gain = 1.0;
      int segs = 3;                                // 1: hi planes only (a single pass)
      bool upper_d = false;                        // d is read as a product's C alone, which takes its upper triangle
      bool whole_in = false, whole_out = false;    // operands, planes of the result that are stored whole
    };
    // (in_step: matrices between the hi and lo planes of the operands; 0: the chunk's)
    auto sym_product = [&](const __half* ap, float sa, const __half* bp, float sb, const Out& o, int promote, int in_step = 0, const int* skip = nullptr) -> int {
      toner_gemm_desc g = {};
      toner_operand op = {};
      const int lo = in_step ? in_step : kc;
      op.rows = n; op.cols = n; op.ld = n; op.z_stride = nn; op.nz = lo + kc; op.z_step = 1;
      g.a = op; g.a.base = ap;
      g.b = op; g.b.base = bp;
      g.a.seg_z[0] = 0; g.a.seg_z[1] = 0; g.a.seg_z[2] = lo;   // Ah Ah Al
      g.b.seg_z[0] = 0; g.b.seg_z[1] = lo; g.b.seg_z[2] = 0;   // Bh Bl Bh
      g.m = n; g.n = n; g.k = n; g.batch = kc; g.segs = o.segs; g.fmt = 0;
      g.tri = 1; g.mirror = 1;
      g.alpha = (float)(o.gain / ((double)sa * (double)sb));
      g.c = o.c; g.ldc = n; g.c_bs = nn; g.beta = o.beta; g.beta_v = o.beta_v;
      g.alpha_a = o.alpha_a;
      g.alpha_b = o.alpha_b;
      g.d = o.d; g.ldd = n; g.d_bs = nn; g.upper_d = o.upper_d ? 1 : 0;
      g.split0 = o.s0; g.split0_scale = o.s0_scale; g.split0_aff_a = o.s0_a;
      g.split1 = o.s1; g.split1_scale = o.s1_scale; g.split1_aff_a = o.s1_a; g.split1_aff_b = o.s1_b;
      g.split_ld = n; g.split_bs = nn; g.split_plane = (long long)(o.lo_step ? o.lo_step : kc) * nn;
      g.maxres = o.maxres;
      g.promote = promote;
      g.interleave = interleave ? 1 : 0;
      GemmMore more;
      more.skip = skip;
      more.half_in = half && !o.whole_in;
      more.half_out = half && !o.whole_out;
      return launch_gemm(g, stream, more);
    };
    int rc = 0;
    // the finish in steps of Y; its planes of R + beta I go where the powers of T leave room (p = 1 has no such buffer)
    QuadraticSteps fast;
    const bool shorten = interleave && log2p > 0 && !graded_finish && quadratic_steps(fin, p, fast);
    __half* const shifted_planes = Pb[log2p & 1];
    __half* root_planes = nullptr;   // of A^{-1/p}, root_step matrices between hi and lo
    int root_step = 0;
    const float s_root = root_plane_scale(root_bound);
    const float s_hi = root_plane_scale(1.01 * std::pow((double)damping, -(double)q / p));
    // X_1 = T_0, read by both chains until the first product with X; the next T goes to T's own buffer
    const __half* Xcur = Xb[1];
    const __half* Tcur = first_planes;   // (before a step of higher degree has formed T, planes of Z)
    float s_x = s_t;
    double x_bound = sched[0].a;
    int xi = 0, mi = 0, ti = 1;   // ti: which T buffer was written last

    const float* root_diag_scale = nullptr;
    float root_diag = 0.f;
    for (int it = 0; it < iters; ++it) {
      const bool last = (it == iters - 1);
      const int* const skip = it == 0 ? late : nullptr;
      if (!last && sched[it].degree > 1) {
        // T from planes of Z (Tcur), see root_steps.cuh: its square, of degree four the square of that, shifted.  T_0 is X_1 as well.
        // The errors of these products matter as those of the powers of T do.
        const NewtonStep& st = sched[it];
        const int chain = steep_chain_length(st.lower);
        const __half* from = Tcur;
        float s_from = s_t;
        if (st.degree == 4) {
          Out y;
          y.s0 = Pb[1]; y.s0_scale = plane_scale(st.most_y);
          y.s0_a = (float)st.kappa;
          rc = sym_product(from, s_from, from, s_from, y, chain, 0, skip);
          if (rc) return rc;
          from = y.s0;
          s_from = y.s0_scale;
        }
        Out t;
        t.gain = st.top;
        t.s0 = it == 0 ? Xb[1] : (st.degree == 4 ? Tb[0] : Pb[1]);
        t.s0_scale = plane_scale(st.a);
        t.s0_a = (float)st.con;
        if (st.lin != 0.0) {
          t.c = it == 0 ? m32 : A32; t.beta = (float)st.lin;
        }
        if (it == 1 && late) {
          t.s1 = Xb[xi]; t.s1_scale = plane_scale(std::min(x_bound * st.a, x_cap));
          t.s1_a = (float)st.con; t.s1_b = 1.f;
        }
        rc = sym_product(from, s_from, from, s_from, t, chain, 0, skip);
        if (rc) return rc;
        Tcur = t.s0;
        s_t = t.s0_scale;
        if (it == 0) s_x = s_t;
      }
      if (it > 0 || last) {
        x_bound = std::min(x_bound * sched[it].a, x_cap);
        if (last) {
          // The graded finish starts from planes of Z (Xb[1]), M_0 in FP32 (m32) and the hi plane of M_0 + g I (Mb[0]).
          // U = 2 Z^2 - I; the distance of Z^2 from I, which has no entry above 1, is what a non-finite or divergent statistic
          // is told by
          __half* const up = Pb[1];
          const float s_u = plane_scale(2.0);
          if (graded_finish) {
            Out u;
            u.s1 = up; u.s1_scale = s_u;
            u.s1_a = -1.f; u.s1_b = 2.f;
            u.maxres = resid;
            rc = sym_product(Xb[1], s_t, Xb[1], s_t, u, chain_length(graded.lo));
            if (rc) return rc;
          }
          // fold ||A||_F^{-1/p} into the product; the distance of M from I was gathered when M was produced
          TONER_LAUNCH(finish_kernel, (kc + 127) / 128, 128, stream, resid, sumsq_a, scale_lo, status ? status + k0 : nullptr, norm_out ? norm_out + k0 : nullptr, kc, p, graded_finish ? 1.5f : converged_within(fin), damping, lower_used, plan.steep && ritz_norm ? th8 : nullptr);
          TONER_CUDA(cudaGetLastError());
          // Tcur holds planes of R = I - M and A32 the FP32 M (both from the last update of M).  q(R), one plane per product,
          // into Mb[1]; the terms linear in M enter in FP32 as beta * c.
          const float s_w = plane_scale(1.0), s_f = plane_scale(2.0);
          float* R = root_lo + (long long)k0 * nn;
          if (graded_finish) {
            // W_j = alpha_j I + beta_j Z + U W_(j+1); the FP32 M brings in Z.  W_1 keeps both planes for the last product.
            const int K = graded.products;
            __half* const spare[2] = {Mb[1], Pb[0]};
            const __half* wcur = Mb[0];
            float s_cur = s_top;
            double gain = top_gain;
            for (int j = K - 1; j >= 1; --j) {
              Out w;
              w.segs = j <= graded.split ? 3 : 1;
              w.gain = gain;
              w.c = m32; w.beta = (float)(graded.beta[j] * graded.za);
              w.s1 = spare[j & 1]; w.s1_scale = plane_scale(graded.bound[j]);
              w.s1_a = (float)(graded.alpha[j] + graded.beta[j] * graded.zb); w.s1_b = 1.f;
              rc = sym_product(up, s_u, wcur, s_cur, w, 0);
              if (rc) return rc;
              wcur = w.s1;
              s_cur = w.s1_scale;
              gain = 1.0;
            }
            const double front = graded.alpha[0] + graded.beta[0] * graded.zb;
            Out f;                 // the root, up to `front` on the diagonal, which root_finish_kernel adds
            f.gain = gain;
            f.c = m32; f.beta = (float)(graded.beta[0] * graded.za);
            f.d = R;
            f.alpha_a = f.beta_v = scale_lo;
            root_diag_scale = scale_lo;
            root_diag = (float)front;
            rc = sym_product(up, s_u, wcur, s_cur, f, kPromoteX);
            if (rc) return rc;
          } else if (shorten) {
            // Steps of Y = R (R + beta I), see quadratic_steps: the product that makes Y writes its planes and those of W, an
            // affine function of Y, at once.  (shifted_planes are those of -(R + beta I).)
            __half* const Yp = Pb[(log2p & 1) ^ 1];
            const float s_y = plane_scale(1.0 + std::fabs(fast.beta));
            int left = (int)fast.lin.size() + (fast.by_r ? 1 : 0);   // products after this one; the last writes Mb[1]
            auto target = [&]() { return Mb[(left & 1) ^ 1]; };
            auto scale = [&](double bound) { return left == 0 ? s_f : plane_scale(std::max(1.0, bound)); };
            double bound = std::fabs(fast.top) * (1.0 + std::fabs(fast.beta)) + std::fabs(fast.top0);
            Out y;
            y.segs = plan.steep && left == 0 ? 3 : 1;
            y.gain = -1.0;
            y.s0 = Yp; y.s0_scale = s_y;
            y.s1 = target(); y.s1_scale = scale(bound);
            y.s1_a = (float)fast.top0; y.s1_b = (float)fast.top;
            rc = sym_product(Tcur, s_t, shifted_planes, s_m, y, 0);
            if (rc) return rc;
            const __half* wcur = y.s1;
            float s_cur = y.s1_scale;
            auto step = [&](const __half* by, float s_by, double linear, double constant) {
              --left;
              bound = (1.0 + std::fabs(fast.beta)) * bound + std::fabs(linear) + std::fabs(constant);
              Out w;
              w.segs = plan.steep && left == 0 ? 3 : 1;
              if (linear != 0.0) {
                w.c = A32; w.beta = (float)-linear;
              }
              w.s1 = target(); w.s1_scale = scale(bound);
              w.s1_a = (float)(linear + constant); w.s1_b = 1.f;
              const int err = sym_product(by, s_by, wcur, s_cur, w, 0);
              wcur = w.s1;
              s_cur = w.s1_scale;
              return err;
            };
            for (auto it2 = fast.lin.rbegin(); it2 != fast.lin.rend(); ++it2) {
              rc = step(Yp, s_y, it2->first, it2->second);
              if (rc) return rc;
            }
            if (fast.by_r) {
              rc = step(Tcur, s_t, fin.c[1], fin.c[0]);
              if (rc) return rc;
            }
          } else {
            // Horner steps W_j = c_j R + R W_{j+1} (W_m = c_m R) build q(R) = c_0 I + W_1
            const __half* wcur = Tcur;
            float s_cur = s_t;
            double gain = fin.c[order];
            for (int j = order - 1; j >= 1; --j) {
              const double aj = fin.c[j];
              Out w;
              w.segs = plan.steep && j == 1 ? 3 : 1;
              w.gain = gain;
              w.c = A32; w.beta = (float)-aj;
              w.s1 = Mb[j & 1];
              w.s1_scale = (j == 1) ? s_f : s_w;
              w.s1_a = (float)(j == 1 ? fin.c[0] + aj : aj);
              w.s1_b = 1.f;
              rc = sym_product(Tcur, s_t, wcur, s_cur, w, 0);
              if (rc) return rc;
              wcur = w.s1;
              s_cur = w.s1_scale;
              gain = 1.0;
            }
          }
          if (!graded_finish) {
            Out o;
            o.d = R;
            o.alpha_a = scale_lo;
            rc = sym_product(Xcur, s_x, Mb[1], s_f, o, plan.steep ? kPromoteSteepX : kPromoteX);
            if (rc) return rc;
          }
          // put the deflated directions back: A^{-1/p} = A'^{-1/p} + (lambda_1^{-1/p} - c^{-1/p}) v v^T; with that the root's
          // norm and its operand planes, for the squarings below and for the caller
          if (lo_planes) {
            root_planes = static_cast<__half*>(lo_planes) + (long long)k0 * nn;
            root_step = k;
          } else if (q > 1) {
            root_planes = Xb[xi];
          }
          TONER_LAUNCH(root_finish_kernel, dim3(kSumsqBlocks, kc), 256, stream, R, defl_r > 0 ? dv : pv, defl_r > 0 ? corr8 : corr, n,
                       defl_r > 0 ? defl_r : 1, defl_r > 0 ? slots : 1, defl_r > 0 ? kMaxDeflate : 1, s_root, root_planes,
                       root_step ? root_step : kc, lo_planes ? lo_inv + k0 : inv_r, s_hi, hi_inv ? hi_inv + k0 : nullptr, partials, root_diag_scale, root_diag);
          TONER_LAUNCH(root_norm_kernel, kc, 32, stream, partials, fro_tmp);
          TONER_CUDA(cudaGetLastError());
          break;
        }
        Out o;
        o.s0 = Xb[xi];
        o.s0_scale = plane_scale(x_bound);
        rc = sym_product(Xcur, s_x, Tcur, s_t, o, plan.steep ? kPromoteSteepX : kPromoteX, 0, it == 1 ? late : nullptr);
        if (rc) return rc;
        Xcur = Xb[xi];
        s_x = o.s0_scale;
        xi ^= 1;
      }
      // M_{k+1} = T^p M_k.  The tensor core adds into its accumulator by truncation, a one-sided error that
      // grows with the length of the accumulation chain and, unlike rounding noise, does not average out over
      // the sum; a relative error e of M matters as e / (smallest eigenvalue of M), so the chains are kept
      // short while the spectrum's lower bound is small and lengthened as it approaches 1.
      const int chain = plan.steep ? steep_chain_length(sched[it].lower) : chain_length(sched[it].lower);
      const __half* pw = Tcur;
      float s_pw = s_t;
      double pw_bound = sched[it].a;
      for (int j = 0; j < log2p; ++j) {
        pw_bound *= pw_bound;
        Out o;
        o.s0 = Pb[j & 1];
        o.s0_scale = plane_scale(pw_bound);
        rc = sym_product(pw, s_pw, pw, s_pw, o, chain, 0, skip);
        if (rc) return rc;
        pw = o.s0;
        s_pw = o.s0_scale;
      }
      {
        const float na = (float)sched[it + 1].a, nb = (float)sched[it + 1].b;
        const int tn = (log2p == 0) ? (ti ^ 1) : 0;  // with p == 1 the product reads T itself
        Out o;
        o.s1 = Tb[tn];
        if (it == iters - 2) {
          // the last M: kept in FP32 with planes of R = I - M for the finishing series, and its distance from I
          o.d = A32;
          o.s1_scale = s_m;
          o.s1_a = 1.f;
          o.s1_b = -1.f;
          o.maxres = resid;
          if (shorten) {
            o.s0 = shifted_planes;
            o.s0_scale = s_m;
            o.s0_a = (float)-(1.0 + fast.beta);
          }
        } else {
          o.s0 = Mb[mi ^ 1];
          o.s0_scale = s_m;
          if (sched[it + 1].degree > 1) {   // planes of the next Z, and M in FP32 where T has a term linear in it
            if (sched[it + 1].lin != 0.0) {
              o.d = A32;
              o.upper_d = true;
            }
            o.s1_scale = s_z;
            o.s1_a = (float)sched[it + 1].zb;
            o.s1_b = (float)sched[it + 1].za;
          } else {
            o.s1_scale = plane_scale(na);
            o.s1_a = na;
            o.s1_b = -nb;
          }
        }
        rc = sym_product(pw, s_pw, Mb[mi], s_m, o, chain, 0, skip);
        if (rc) return rc;
        mi ^= 1;
        ti = tn;
        Tcur = Tb[tn];
        s_t = o.s1_scale;
      }
    }
    if (fro2_lo) TONER_CUDA(cudaMemcpyAsync(fro2_lo + k0, fro_tmp, sizeof(float) * kc, cudaMemcpyDeviceToDevice, stream));

    if (q > 1) {
      // A^{-q/p} by repeated squaring of A^{-1/p}
      Xcur = root_planes;
      int have = 1;
      double bound = root_bound;
      int pi = 0;
      s_x = 1.f;  // the root's planes carry per-statistic scales (inv_r), applied below
      while (have < q) {
        const bool first = (have == 1);
        have *= 2;
        bound *= bound;
        Out o;
        if (first) {
          o.alpha_a = o.alpha_b = lo_planes ? lo_inv + k0 : inv_r;
          o.whole_in = true;   // (root_finish_kernel's planes)
        }
        if (have == q) {
          o.whole_out = true;
          o.d = root_hi + (long long)k0 * nn;
          if (hi_planes) {
            o.s0 = static_cast<__half*>(hi_planes) + (long long)k0 * nn;
            o.s0_scale = s_hi;
            o.lo_step = k;
          }
        } else {
          o.s0 = Pb[pi];
          o.s0_scale = plane_scale(bound);
        }
        // (One chain's truncation, 2e-5 at depth 2048 and twice that after the second squaring, makes up for part of the
        // Newton chain's.  A^(-1/p) from a graded finish is ten times closer than that; two squarings in chains of two k-blocks
        // leave 3.5e-6 of A^(-1/2) whatever the width, of one k-block 2e-6, in the same time: 24 statistics of 2048, condition 2
        // and 5, 5570 and 6125 / 5620 and 6080 us a call.)
        rc = sym_product(Xcur, s_x, Xcur, s_x, o, graded_finish ? 1 : plan.steep ? kPromoteSteepSquares : kPromoteX, first ? root_step : 0);
        if (rc) return rc;
        Xcur = Pb[pi];
        s_x = o.s0_scale;
        pi ^= 1;
      }
    }

    if (track) {
      float* vt = track + (long long)k0 * n;
      if (lower_used < 0.f) {
        // The schedule was built for an ESTIMATE of the spectrum's lower end.  If the estimate was too high for a
        // statistic, its smallest eigenvalues have not reached the distance from 1 the finishing series was cut for,
        // and they are the dominant eigenvalues of R = I - M of the last M (kept in FP32): four power-iteration steps
        // on R from the tracked direction (the eigenvector of the smallest eigenvalue, as of the previous call) find
        // them.  The allowance: the assumed distance with 15 % and the noise floor of the estimate.
        if (graded_finish) {
          // After a graded finish the roots themselves are looked at: R = I - A^(-1/2) A A^(-1/2) is p times the relative error of
          // A^(-1/p) on every eigenvector, of either sign, 1e-5 to 9e-5 where the interpolant holds (rounding included, widths to
          // 5632) and growing fast where an eigenvalue lies outside the interval.  One step from the tracked direction and from
          // the largest Ritz vector that stayed in A', each with a share of every other direction, leaves next to nothing but
          // such eigenvectors; the quotients of the second step tell.  R is taken on the complement of the deflated directions:
          // a Ritz vector's residual r couples it to the rest by r (theta / lambda)^(3/2) in R, 2e-2 for a mean of eight standard
          // deviations, where the root it leaves is as good as any.
          const float* root = (q > 1 ? root_hi : root_lo) + (long long)k0 * nn;
          float* const py2 = py + (long long)kc * 2 * n;
          TONER_LAUNCH(pick_vector_kernel, dim3(8, kc), 256, stream, vt, dv, rest_idx, pv, n, slots, 1.f, nullptr, nullptr);
          for (int sw = 0; sw < 2; ++sw) {
            TONER_CUDA(launch_block_gemv<2>(kc, stream, root, pv, py, n, 2, 2));
            TONER_LAUNCH(project_kernel, dim3(kc, 2), 256, stream, py, dv, coef8, n, defl_r, slots);
            TONER_CUDA(launch_block_gemv<2>(kc, stream, A32, py, py2, n, 2, 2));
            TONER_CUDA(launch_block_gemv<2>(kc, stream, root, py2, py, n, 2, 2));
            TONER_LAUNCH(power_shift_kernel, dim3(kc, 2), 256, stream, pv, py, n, e_est, 2, (long long)(e_top - e_est), dv, coef8, defl_r, slots, 0.f, nullptr);
          }
        } else if (ritz_norm) {
          // The norm was an estimate too.  Eigenvalues of M_0 above 1 (the estimate was too low for them) come out of
          // linear steps BELOW the lower bound the schedule continues from -- T = a I - b M is small there -- and lag the same way;
          // they belong to the top of A', so the same four steps from the largest Ritz vector that stayed in A' find them.  Both
          // starting vectors go through M in one pass per step.  (What lies beyond a / b, where T is negative, may come back to I with the
          // sign of X turned, which nothing here sees: from a reach of 1.03 on for p = 2, 1.24 for p = 4, 1.95 for p = 8, none up to 3.4
          // for 16 and 32.  The norm is 1.4 times the Ritz value, so that has to be as much more too low.)
          // Steps of higher degree send them ABOVE 1, where R is negative and small at first beside what it may be on the other side
          // (degree 2 from l = 0.034: R = -0.3 for a reach of 1.2, 0.54 for the lower end).  Steps on R lose such a direction; those on
          // (1 - e / 2) I - M gain it.  And they start from the Ritz vector's residual, which holds what the block has not found yet,
          // the largest eigenvalues first.  (From the Ritz vector itself, on R: A^(-1/8) 6e-2 off, unflagged, where 0.3 % of it were
          // a direction 1.68 times as large.)
          TONER_LAUNCH(pick_vector_kernel, dim3(8, kc), 256, stream, vt, dv, rest_idx, pv, n, slots, 0.f, lowest ? py : nullptr, th8);
          for (int sw = 0; sw < 4; ++sw) {
            TONER_CUDA(launch_block_gemv<2>(kc, stream, A32, pv, py, n, 2, 2));
            TONER_LAUNCH(power_shift_kernel, dim3(kc, 2), 256, stream, pv, py, n, e_est, 2, (long long)(e_top - e_est), nullptr, nullptr, 0, 0, lowest ? (float)(0.5 * (1.0 - l_last)) : 0.f, lowest);
          }
        } else {
          TONER_CUDA(cudaMemcpyAsync(pv, vt, sizeof(float) * (size_t)kc * n, cudaMemcpyDeviceToDevice, stream));
          for (int sw = 0; sw < 4; ++sw) {
            TONER_LAUNCH(gemv_kernel, dim3((n + 7) / 8, kc), 256, stream, A32, pv, py, n);
            TONER_LAUNCH(power_shift_kernel, kc, 256, stream, pv, py, n, e_est, 1, 0, nullptr, nullptr, 0, 0, 0.f, nullptr);
          }
        }
        TONER_LAUNCH(verify_kernel, (kc + 127) / 128, 128, stream, e_est, ritz_norm || graded_finish ? e_top : nullptr, graded_finish ? (float)(kGradedResidual + p * kGradedTail) : (float)(1.15 * (1.0 - l_last) + 1e-3), plan.steep ? kSteepBelow : INFINITY, status ? status + k0 : nullptr, resid_out ? resid_out + k0 : nullptr, kc, graded_finish ? th8 : nullptr, rest_trace, n, lowest);
        TONER_CUDA(cudaGetLastError());
      }
      const int sweeps = track_sweeps & 63;
      if (sweeps > 0) {
        // Track the direction of the smallest eigenvalue of A for the next call: it is the dominant eigenvector of the
        // highest inverse power just computed, where it stands out however small it is next to lambda_max(A).
        const float* top = (q > 1 ? root_hi : root_lo) + (long long)k0 * nn;
        if (track_sweeps & 256) {
          TONER_LAUNCH(power_start_kernel, dim3(8, kc), 256, stream, vt, n);
        }
        for (int sw = 0; sw < sweeps; ++sw) {
          TONER_LAUNCH(gemv_kernel, dim3((n + 7) / 8, kc), 256, stream, top, vt, py, n);
          TONER_LAUNCH(power_norm_kernel, kc, 256, stream, vt, py, n, theta, pres);
        }
        if (lmin_out) {
          TONER_LAUNCH(lmin_from_root_kernel, (kc + 127) / 128, 128, stream, theta, (float)p / (float)q, lmin_out + k0, kc);
        }
        TONER_CUDA(cudaGetLastError());
      }
    }
  }
  return 0;
}

}  // extern "C"
