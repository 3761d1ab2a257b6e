// Newton steps of higher degree (host only): T = q(M) of degree 1, 2 or 4 in the coupled iteration X <- X T, M <- T^p M.
//
// A step takes the spectrum of M from [l, 1] to [l', 1].  With the best linear T l' is 13 l at most (p = 8) and the step takes
// log2 p + 2 products; a T of degree two costs one product more and reaches 34 l, one of degree four two more and 110 l: the
// logarithm gained per product is 0.51, 0.59 and 0.67, and the steps next to I gain likewise (l = 0.013: one step of degree four
// where it took two linear ones).
//
// The q for which l' is largest:  maximise r subject to  r g(mu) <= q(mu) <= mu^(-1/p)  on [l, kStepHigh], with  g = mu^(-1/p)
// or, where that is more, the cap on the dynamic range of T^p (max_range); l' = r^p.  This is a linear Chebyshev problem: at
// the best q the two bounds are touched in turn at degree + 2 points, found by Remez' exchange on a grid.
//
// q is formed as  top z^2 + con  or  top (z^2 + kappa)^2 + lin mu + con  with z = zb + za mu: a square is a product of one pair of
// operand planes by itself and its shifts go into the planes' diagonals, so T takes one or two products that write one pair of
// planes each.  The linear term of degree four needs M in FP32, written by one product and read by another; where q is hardly
// worse without it (l < 1e-3) it is left out.
#pragma once
#include <algorithm>
#include <cmath>

namespace toner {

// q is levelled up to here: rounding lifts the top of M's spectrum above 1, and where the norm is an estimate the top may lie
// above it.  A linear T forgives that (what lies above 1 lags), one of even degree sends it past 1: at 1.05 to 1.8 (degree 4, l =
// 0.013, levelled up to 1.005) and to 0.9 levelled up to 1.06, which costs 2 to 5 % of l'.
constexpr double kStepHigh = 1.06;
constexpr int kStepDegrees[3] = {1, 2, 4};

// One step.  Degree 1: T = a I - b M.  Otherwise a bounds |T| on [0, kStepHigh] and T is formed from Z = zb I + za M.
struct NewtonStep {
  double a = 0.0, b = 0.0, lower = 0.0;
  int degree = 1;
  double za = 0.0, zb = 0.0, kappa = 0.0, top = 0.0, lin = 0.0, con = 0.0;
  double next = 0.0;     // lower end of the spectrum of T^p M
  double most_z = 0.0, most_y = 0.0;   // bounds of |z| and |z^2 + kappa| on [0, kStepHigh], which their operand planes are scaled for
  double at(double mu) const {
    if (degree == 1) return a - b * mu;
    const double z = zb + za * mu, y = degree == 2 ? z : z * z + kappa;
    return top * y * y + lin * mu + con;
  }
};

inline double chebyshev_sum(const double* c, int degree, double z) {
  double b1 = 0.0, b2 = 0.0;
  for (int j = degree; j >= 1; --j) {
    const double b0 = c[j] + 2.0 * z * b1 - b2;
    b2 = b1;
    b1 = b0;
  }
  return c[0] + z * b1 - b2;
}

// q for a spectrum in [lower, kStepHigh], in Chebyshev polynomials of z = (mu - mid) / half.  (Not scaled to its bounds.)
inline bool level(int p, double lower, int degree, double max_range, double* c) {
  constexpr int kGrid = 129, kMost = 6;
  const double kPi = 3.14159265358979323846;
  const double mid = 0.5 * (kStepHigh + lower), half = 0.5 * (kStepHigh - lower);
  const double cap = std::pow(max_range * lower, -1.0 / p);
  double z[kGrid], up[kGrid], lo[kGrid], q[kGrid];
  for (int i = 0; i < kGrid; ++i) {
    z[i] = -std::cos(kPi * i / (kGrid - 1));
    up[i] = std::pow(mid + half * z[i], -1.0 / p);
    lo[i] = std::max(up[i], cap);
  }
  // where it starts from: the extrema for p = 2 and l = 0, sqrt(mu) = cos(k pi / (2 degree + 1)), and the lower end
  const int points = degree + 2;
  int at[kMost];
  at[0] = 0;
  for (int k = 1; k < points; ++k) {
    const double root = std::cos(kPi * (points - 1 - k) / (2 * degree + 1));
    at[k] = std::max(at[k - 1] + 1, (int)std::lround(std::acos(1.0 - 2.0 * root * root) / kPi * (kGrid - 1)));
  }
  at[points - 1] = std::min(at[points - 1], kGrid - 1);
  for (int round = 0; round < 16; ++round) {
    // unknowns c_0 .. c_degree and r:  q = r lo at even points, q = up at odd ones
    double m[kMost][kMost + 1];
    for (int k = 0; k < points; ++k) {
      double t0 = 1.0, t1 = z[at[k]];
      for (int j = 0; j <= degree; ++j) {
        m[k][j] = t0;
        const double t2 = 2.0 * z[at[k]] * t1 - t0;
        t0 = t1;
        t1 = t2;
      }
      m[k][degree + 1] = (k & 1) ? 0.0 : -lo[at[k]];
      m[k][points] = (k & 1) ? up[at[k]] : 0.0;
    }
    for (int col = 0; col < points; ++col) {
      int pivot = col;
      for (int k = col + 1; k < points; ++k)
        if (std::fabs(m[k][col]) > std::fabs(m[pivot][col])) pivot = k;
      if (!(std::fabs(m[pivot][col]) > 1e-14)) return false;
      for (int j = col; j <= points; ++j) std::swap(m[col][j], m[pivot][j]);
      for (int k = col + 1; k < points; ++k) {
        const double f = m[k][col] / m[col][col];
        for (int j = col; j <= points; ++j) m[k][j] -= f * m[col][j];
      }
    }
    double x[kMost];
    for (int k = points - 1; k >= 0; --k) {
      double sum = m[k][points];
      for (int j = k + 1; j < points; ++j) sum -= m[k][j] * x[j];
      x[k] = sum / m[k][k];
    }
    for (int j = 0; j <= degree; ++j) c[j] = x[j];
    for (int i = 0; i < kGrid; ++i) q[i] = chebyshev_sum(c, degree, z[i]);
    // every point moves to the extremum between its neighbours
    bool moved = false;
    for (int k = 0; k < points; ++k) {
      const int first = k == 0 ? 0 : at[k - 1] + 1, last = k == points - 1 ? kGrid - 1 : at[k + 1] - 1;
      int best = at[k];
      for (int i = first; i <= last; ++i)
        if ((k & 1) ? q[i] / up[i] > q[best] / up[best] : q[i] / lo[i] < q[best] / lo[best]) best = i;
      moved = moved || best != at[k];
      at[k] = best;
    }
    if (!moved) break;
  }
  return true;
}

// The step scaled to mu T^p <= 1 on [lower, kStepHigh], by a grid of its own, and what it leaves; false where T is not positive.
inline bool scale_step(int p, NewtonStep& s) {
  constexpr int kCheck = 385;
  constexpr double kMargin = 1e-4;   // of q: what this grid misses of an extremum
  const double kPi = 3.14159265358979323846;
  double most = 0.0, least = 1e300, smallest = 1e300, largest = std::fabs(s.at(0.0));
  for (int i = 0; i < kCheck; ++i) {
    const double mu = 0.5 * (s.lower + kStepHigh) - 0.5 * (kStepHigh - s.lower) * std::cos(kPi * i / (kCheck - 1));
    const double t = s.at(mu), f = t * std::pow(mu, 1.0 / p);
    most = std::max(most, f);
    least = std::min(least, f);
    smallest = std::min(smallest, t);
    largest = std::max(largest, t);
  }
  if (!(smallest > 0.0) || !(most < 1e3)) return false;
  const double scale = 1.0 / (most * (1.0 + kMargin));
  if (s.degree == 1) {
    s.a *= scale;
    s.b *= scale;
  } else {
    s.top *= scale;
    s.lin *= scale;
    s.con *= scale;
    s.a = 1.01 * largest * scale;
  }
  s.next = std::pow(least * scale * (1.0 - kMargin), p);
  const double z0 = std::fabs(s.zb), z1 = std::fabs(s.zb + s.za * kStepHigh);   // (z is linear: largest at an end; z^2 least at 0)
  s.most_z = std::max(z0, z1);
  s.most_y = std::max(std::fabs(s.kappa), std::fabs(s.most_z * s.most_z + s.kappa));
  return true;
}

// The step of this degree for a spectrum in [lower, 1]; false where none was found that gains.
inline bool best_step(int p, double lower, int degree, double max_range, NewtonStep& s) {
  if (!(lower > 0.0 && lower < 0.95)) return false;
  double c[5] = {};
  if (!level(p, lower, degree, max_range, c)) return false;
  const double mid = 0.5 * (kStepHigh + lower), half = 0.5 * (kStepHigh - lower);
  s = NewtonStep();
  s.lower = lower;
  s.degree = degree;
  if (degree == 1) {
    s.a = c[0] - c[1] * mid / half;
    s.b = -c[1] / half;
    if (!(s.b > 0.0)) return false;
  } else {
    // z is (mu - mid) / half + shift
    double shift, rest = 0.0;   // rest: of the linear term, in z
    if (degree == 2) {
      if (!(std::fabs(c[2]) > 1e-6)) return false;
      s.top = 2.0 * c[2];
      shift = c[1] / (4.0 * c[2]);
      s.con = c[0] - c[2] - s.top * shift * shift;
    } else {
      // 8 c4 z^4 + 4 c3 z^3 + (2 c2 - 8 c4) z^2 + (c1 - 3 c3) z + (c0 - c2 + c4)
      if (!(std::fabs(c[4]) > 1e-6)) return false;
      const double b4 = 8.0 * c[4], b3 = 4.0 * c[3], b2 = 2.0 * c[2] - 8.0 * c[4], b1 = c[1] - 3.0 * c[3], b0 = c[0] - c[2] + c[4];
      shift = b3 / (4.0 * b4);
      s.top = b4;
      const double d2 = b2 - 6.0 * b4 * shift * shift;      // of (z + shift)^2
      s.kappa = d2 / (2.0 * b4);
      // top ((z + shift)^2 + kappa)^2 has 4 top shift (shift^2 + kappa) z and top (shift^2 + kappa)^2
      const double k = shift * shift + s.kappa;
      rest = b1 - 4.0 * s.top * shift * k;
      s.con = b0 - s.top * k * k;
    }
    s.za = 1.0 / half;
    s.zb = -mid / half + shift;
    // (operand planes of z and z^2 + kappa: a T much smaller than its terms would lose bits)
    if (!(std::fabs(shift) < 2.0 && std::fabs(s.kappa) < 8.0 && std::fabs(s.con) < 8.0)) return false;
    NewtonStep bare = s;
    s.lin = rest / half;
    s.con -= rest * mid / half;
    if (rest != 0.0 && scale_step(p, bare)) {
      if (!scale_step(p, s)) return false;
      if (bare.next > 0.97 * s.next) s = bare;
      return s.next > 1.5 * lower || s.next > 0.9;
    }
  }
  return scale_step(p, s) && (s.next > 1.5 * lower || s.next > 0.9);
}

}  // namespace toner
