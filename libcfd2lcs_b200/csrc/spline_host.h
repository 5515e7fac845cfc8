// Host set-up of a B-spline interpolation axis (knots, band LU, reciprocal spans).
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

namespace cfd2lcs {

template <typename R>
struct SplineAxisHost {
  int n = 0, k = 0;
  std::vector<R> t;     // n + k knots
  std::vector<R> lu;    // (2k-1) x n band LU, column-major, diagonal in row k (1-based)
  std::vector<R> rinv;  // 6 reciprocal knot spans per interval
  std::vector<R> tu;    // per interval l, pair at 2(l-1): t(l), and 1/h where the knots the basis
                        // depends on are equally spaced by h (else 0)
  // x: strictly increasing abscissae (the padded coordinate line); order k.
  bool build(const std::vector<R> &x, int order);
};

// Band LU of one axis in the pull form the device sweeps read, 8 values per row r (0-based):
// [j-1] the factor of L multiplying y(r-j) in the forward sweep, [3+j-1] the factor of U
// multiplying x(r+j) in the backward sweep (j = 1 .. k-1), [6] 1 / U(r,r).
template <typename R>
std::vector<R> spline_pull_table(const SplineAxisHost<R> &A) {
  const int n = A.n, k = A.k, nr = 2 * k - 1, mid = k;
  auto W = [&](int r, int c) { return A.lu[(size_t)(r - 1) + (size_t)nr * (c - 1)]; };
  std::vector<R> p((size_t)8 * n, R(0));
  for (int i = 1; i <= n; i++) {
    for (int j = 1; j <= k - 1; j++) {
      if (i - j >= 1) p[(size_t)8 * (i - 1) + j - 1] = W(mid + j, i - j);
      if (i + j <= n) p[(size_t)8 * (i - 1) + 3 + j - 1] = W(mid - j, i + j);
    }
    p[(size_t)8 * (i - 1) + 6] = R(1) / W(mid, i);
  }
  return p;
}

// The same factors arranged for the transposed solve (L U)^T f = c, used by the adjoint of a fit:
// U^T z = c forward, z(r) = (c(r) - sum_j U(r-j,r) z(r-j)) / U(r,r), with U(r-j,r) at [j-1] and
// 1/U(r,r) at [6]; then L^T f = z backward, f(r) = z(r) - sum_j L(r+j,r) f(r+j), with L(r+j,r)
// at [3+j-1].
template <typename R>
std::vector<R> spline_pull_table_transposed(const std::vector<R> &p, int n) {
  std::vector<R> t((size_t)8 * n, R(0));
  for (int r = 0; r < n; r++) {
    for (int j = 1; j <= 3; j++) {
      if (r - j >= 0) t[(size_t)8 * r + j - 1] = p[(size_t)8 * (r - j) + 3 + j - 1];
      if (r + j < n) t[(size_t)8 * r + 3 + j - 1] = p[(size_t)8 * (r + j) + j - 1];
    }
    t[(size_t)8 * r + 6] = p[(size_t)8 * r + 6];
  }
  return t;
}

// Elements after which both sweeps of a pull table (either form) have forgotten the window they
// started from: the smallest w such that, from every element of the line, a unit value in any
// entry of the window before it has fallen below tol, in every entry, w elements further on.
// 0 where some start needs more than `most`.  The device starts the sweeps of a line's chunks w
// elements early from a zero window (k_fit_block).
template <typename R>
int spline_fit_warmup(const std::vector<R> &p, int n, int k, bool transposed, double tol, int most) {
  int worst = 1;
  for (int dir = 0; dir < 2; dir++)
    for (int s = 0; s < n; s++)
      for (int b = 0; b < k - 1; b++) {
        double w[3] = {0, 0, 0};
        w[b] = 1;
        int m = 0;
        while (true) {
          double top = 0;
          for (int j = 0; j < k - 1; j++) top = std::max(top, std::fabs(w[j]));
          if (top <= tol || s + m >= n) break;
          if (m >= most) return 0;
          const int r = dir == 0 ? s + m : n - 1 - (s + m);
          const R *c = &p[(size_t)8 * r];
          double v = 0;
          for (int j = 0; j < k - 1; j++) v -= w[j] * (double)c[(dir == 0 ? 0 : 3) + j];
          if ((dir == 1) != transposed) v *= (double)c[6];
          w[2] = w[1];
          w[1] = w[0];
          w[0] = v;
          m++;
        }
        worst = std::max(worst, m);
      }
  return worst;
}

// What k_fit_block reads of an axis' factors, for a fit in type D (Axis: warm, mid0, mid1).
// The warm-up reaches 20 (FP64) or 11 (FP32) binary places below the last one: once the sweeps from
// the zero window and from the whole line differ by less than a last place, each further element
// rounds them to the same value with probability above one half.  Shorter warm-ups repeat more
// lines, longer ones cost every chunk: at 2^-53 alone one chunk in 400 differed, here none of 10^5.
template <typename D, typename R, typename Axis>
void spline_fit_shape(const std::vector<R> &p, int n, int k, bool transposed, int most, Axis &A) {
  A.warm = spline_fit_warmup(p, n, k, transposed, sizeof(D) == 8 ? 0x1p-73 : 0x1p-35, most);
  auto wide = [&](int r) { return p[(size_t)8 * r + 1] != R(0) || p[(size_t)8 * r + 2] != R(0) || p[(size_t)8 * r + 4] != R(0) || p[(size_t)8 * r + 5] != R(0); };
  // the longest run of rows with one factor on either side (the ends of a not-a-knot line have more)
  A.mid0 = A.mid1 = 0;
  for (int r = 0, run = 0; r < n; r++) {
    run = wide(r) ? 0 : run + 1;
    if (run > A.mid1 - A.mid0) A.mid0 = r + 1 - run, A.mid1 = r + 1;
  }
}

}  // namespace cfd2lcs
