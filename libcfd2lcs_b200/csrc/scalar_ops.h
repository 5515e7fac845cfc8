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
// in NBR_OFFSET order (src/data_m.f90:124-152), the centre first, and moves to one whose squared
// distance, (qx + qy) + qz, is below 0.99 of the best so far.  Rounded sums grow with their terms, so
// a candidate that leaves every axis as near or further is never below the centre, and one that brings
// a single axis nearer never below that axis' face: with one nearer offset the scan ends on its
// face or stays.  With two or three it ends on all of them together, r, if r is below 0.99 of every
// other candidate, that is of the smallest of those that differ from it along one axis only, by that
// axis' second nearest line.  Otherwise candidates are within a hundredth of each other (the particle
// is near the middle between two nodes, or many cells away along one axis) and the order decides:
// nbr_scan_close visits those that bring two axes or more nearer.
// The full scan is 27 dependent compare-and-multiply steps, 540 cycles and 108 FP64 operations.

// One visit of the scan: to offsets (x, y, z) at squared distance r.
template <typename T>
CFD2LCS_HD inline void nbr_visit(T r, int x, int y, int z, T &best, int off[3]) {
  if (r < T(0.99) * best) {
    best = r;
    off[0] = x;
    off[1] = y;
    off[2] = z;
  }
}

// the scan with the nearer offsets s (two or three of them; 0: none along that axis), whose squares are g
template <typename T>
CFD2LCS_HD inline void nbr_scan_close(const T q[3][3], const T g[3], const int s[3], int sa, int off[3]) {
  const T c[3] = {q[0][1], q[1][1], q[2][1]};
  T best = (c[0] + c[1]) + c[2];
  off[0] = off[1] = off[2] = 0;
  // the faces: offsets -1 along x, y, z, then +1
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int sign = -1; sign <= 1; sign += 2) {
    if (s[0] == sign) nbr_visit((g[0] + c[1]) + c[2], sign, 0, 0, best, off);
    if (s[1] == sign) nbr_visit((c[0] + g[1]) + c[2], 0, sign, 0, best, off);
    if (s[2] == sign) nbr_visit((c[0] + c[1]) + g[2], 0, 0, sign, best, off);
  }
  if (s[0] == 0 || s[1] == 0 || s[2] == 0) {
    // two: both together, with -1, 0, 1 along the third axis
    const int t = s[0] == 0 ? 0 : (s[1] == 0 ? 1 : 2);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int o = -1; o <= 1; o++) {
      if (o != 0 && t == sa) continue;
      const T x = t == 0 ? q[0][o + 1] : g[0], y = t == 1 ? q[1][o + 1] : g[1], z = t == 2 ? q[2][o + 1] : g[2];
      nbr_visit((x + y) + z, t == 0 ? o : s[0], t == 1 ? o : s[1], t == 2 ? o : s[2], best, off);
    }
    return;
  }
  // three: layer by layer along z; in the layer that is nearer the rows and columns through s[0], s[1],
  // in the others that corner alone
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int z = -1; z <= 1; z++) {
    if (z != s[2]) {
      nbr_visit((g[0] + g[1]) + q[2][z + 1], s[0], s[1], z, best, off);
      continue;
    }
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int y = -1; y <= 1; y++)
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
      for (int x = -1; x <= 1; x++)
        if ((x != 0 || y != 0) && (x == s[0] || y == s[1])) nbr_visit((q[0][x + 1] + q[1][y + 1]) + q[2][z + 1], x, y, z, best, off);
  }
}

template <typename T>
CFD2LCS_HD inline void nbr_scan_short(const T q[3][3], int sa, int off[3]) {
  T g[3], h[3];  // the nearest line's square and the second nearest's
  int n = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int a = 0; a < 3; a++) {
    const bool lo = a != sa && q[a][0] < q[a][1], hi = a != sa && !lo && q[a][2] < q[a][1];
    off[a] = lo ? -1 : (hi ? 1 : 0);
    n += lo || hi ? 1 : 0;
    g[a] = lo ? q[a][0] : (hi ? q[a][2] : q[a][1]);
    h[a] = lo || hi ? q[a][1] : (q[a][0] < q[a][2] ? q[a][0] : q[a][2]);
  }
  if (n == 0) return;
  const T r = (g[0] + g[1]) + g[2];
  if (n == 1) {
    if (!(r < T(0.99) * ((q[0][1] + q[1][1]) + q[2][1]))) off[0] = off[1] = off[2] = 0;
    return;
  }
  const T rx = (h[0] + g[1]) + g[2], ry = (g[0] + h[1]) + g[2], rz = (g[0] + g[1]) + h[2];
  if ((sa == 0 || r < T(0.99) * rx) && (sa == 1 || r < T(0.99) * ry) && (sa == 2 || r < T(0.99) * rz)) return;
  const int s[3] = {off[0], off[1], off[2]};
  nbr_scan_close(q, g, s, sa, off);
}

}  // namespace cfd2lcs
