// Scalar pieces of the point-wise kernels in forms that cost the device little, each with the value of
// the plain form it stands for in every case (tests/test_scalar_ops.py compares them on the host).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define CFD2LCS_HD __host__ __device__
#else
#define CFD2LCS_HD
#endif

namespace cfd2lcs {

CFD2LCS_HD inline int32_t high_word(double v) {
#ifdef __CUDA_ARCH__
  return __double2hiint(v);
#else
  uint64_t b;
  std::memcpy(&b, &v, 8);
  return (int32_t)(b >> 32);
#endif
}

// max(min(v, 1), 0) with min and max taking the number where the other side is a NaN, so that a NaN
// yields 1 (as the reference's compiled intrinsics do), from the sign and exponent of v: FP64 min and
// max have no instruction on this GPU, a pair of them is a 51-cycle sequence on the stencils'
// dependent chain and the comparisons take FP64 issue slots; this is integer work of about 12 cycles.
// (A NaN with the sign set counts as one from 0xfff80000 up, the quiet ones arithmetic makes.)
CFD2LCS_HD inline double clamp01_select(double v) {
  const int32_t h = high_word(v);
  const double top = h >= 0x3ff00000 ? 1.0 : v;                             // v >= 1, +Inf, NaN
  return h < 0 ? ((uint32_t)h >= 0xfff80000u ? 1.0 : 0.0) : top;  // negative, -0, -Inf; NaN
}

// Node search (track_lp2node, src/lp_tracking_m.f90:16-183) at an interior node: the candidate the
// 27-neighbour scan ends on, from the squared axis distances q[a][o + 1] to the lines at offsets o =
// -1, 0, 1 (their centre only along a singleton axis sa, else sa = -1).  The scan visits the offsets
// in NBR_OFFSET order (src/data_m.f90:124-152) and moves to one whose squared distance, (qx + qy) +
// qz, is below 0.99 of the best so far.  Rounded sums grow with their terms, so a candidate none of
// whose offsets brings an axis nearer is never below the centre, nor one with such an offset on a
// single axis below that axis' face: with no nearer offset the scan stays, with one it compares the
// face alone, with two it meets the two faces (offsets -1 before +1, then x, y, z) and then both
// offsets together with -1, 0, 1 on the third axis.  Three nearer offsets (rare: the sum of the three
// moves of a subcycle is at most half a cell) leave it to the full scan: returns false.
// 27 dependent compare-and-multiply steps were 540 cycles and 108 FP64 operations per pass.
template <typename T>
CFD2LCS_HD inline bool nbr_scan_short(const T q[3][3], int sa, int off[3]) {
  T g[3];  // the nearer offset's square, or the centre's
  int s[3], n = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int a = 0; a < 3; a++) {
    s[a] = a == sa ? 0 : (q[a][0] < q[a][1] ? -1 : (q[a][2] < q[a][1] ? 1 : 0));
    g[a] = s[a] < 0 ? q[a][0] : (s[a] > 0 ? q[a][2] : q[a][1]);
    n += s[a] != 0 ? 1 : 0;
    off[a] = 0;
  }
  if (n == 0) return true;
  if (n == 3) return false;
  T best = (q[0][1] + q[1][1]) + q[2][1];
  if (n == 1) {
    const T r = (g[0] + g[1]) + g[2];
    if (r < T(0.99) * best)
      for (int a = 0; a < 3; a++) off[a] = s[a];
    return true;
  }
  // the third axis c, and the nearer axes a < b
  const int c = s[0] == 0 ? 0 : (s[1] == 0 ? 1 : 2), a = c == 0 ? 1 : 0, b = c == 2 ? 1 : 2;
  const int sA = c == 0 ? s[1] : s[0], sB = c == 2 ? s[1] : s[2];
  const T fA = ((a == 0 ? g[0] : q[0][1]) + (a == 1 ? g[1] : q[1][1])) + q[2][1];
  const T fB = (q[0][1] + (b == 1 ? g[1] : q[1][1])) + (b == 2 ? g[2] : q[2][1]);
  const bool swap = sA > 0 && sB < 0;  // B's face comes first
  const T f1 = swap ? fB : fA, f2 = swap ? fA : fB;
  int pick = 0;  // 1: first face, 2: second, 3 + (o + 1): both offsets with o on the third axis
  if (f1 < T(0.99) * best) {
    best = f1;
    pick = 1;
  }
  if (f2 < T(0.99) * best) {
    best = f2;
    pick = 2;
  }
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int o = -1; o <= 1; o++) {
    if (o != 0 && c == sa) continue;
    const T x = c == 0 ? q[0][o + 1] : g[0], y = c == 1 ? q[1][o + 1] : g[1], z = c == 2 ? q[2][o + 1] : g[2];
    const T r = (x + y) + z;
    if (r < T(0.99) * best) {
      best = r;
      pick = 4 + o;
    }
  }
  const bool useA = pick >= 3 || pick == (swap ? 2 : 1), useB = pick >= 3 || pick == (swap ? 1 : 2);
  const int o = pick >= 3 ? pick - 4 : 0;
  off[0] = c == 0 ? o : (useA ? s[0] : 0);
  off[1] = c == 1 ? o : ((c == 0 ? useA : useB) ? s[1] : 0);
  off[2] = c == 2 ? o : (useB ? s[2] : 0);
  return true;
}

}  // namespace cfd2lcs
