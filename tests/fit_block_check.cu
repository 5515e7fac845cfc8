// The chunked sweeps of k_fit_block against the whole-line sweeps (k_fit_lines, k_fit_xlines), bit for
// bit: one line per combination, "<bad values> <name>".  A NaN counts as equal to a NaN.
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <random>
#include <vector>

#include "kernels.cuh"
#include "spline_host.h"

using namespace cfd2lcs;

namespace {

constexpr int FIELDS = 7;
const char *const FIELD[FIELDS] = {"random", "constant", "zero tail", "zero middle", "wide range", "nan", "zero ends"};

// value of element e of n on line l
double value(int field, std::mt19937_64 &g, long l, int e, int n) {
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  const double r = U(g);
  switch (field) {
    case 1: return 1.7 * std::sin(0.37 * (double)l);  // the same along the line
    case 2: return e < n / 4 ? r : 0.0;
    case 3: return e < n / 3 || e > 2 * n / 3 ? r : 0.0;
    case 4: return r * std::exp2(40.0 * std::sin(0.7 * e));
    case 5: return l % 5 == 2 && e == (int)((l * 13) % n) ? NAN : r;
    case 6: return e < n / 3 || e > 2 * n / 3 ? 0.0 : r;
    default: return r;
  }
}

template <typename T>
struct Case {
  int nx, ny, nz, axis;  // padded points; the axis of the solve
  std::vector<T> pull, pullT;
  SplineAxis<T> A{}, AT{};
  T *src[3], *a[3], *b[3], *dp, *dpT;
  size_t nt;

  Case(int nx_, int ny_, int nz_, int axis_, int k, bool stretched) : nx(nx_), ny(ny_), nz(nz_), axis(axis_) {
    const int n = axis == 0 ? nx : (axis == 1 ? ny : nz);
    std::vector<T> x(n);
    for (int i = 0; i < n; i++) x[i] = T(stretched ? 0.1 * i + 0.04 * std::sin(0.9 * i) : 0.1 * i);
    SplineAxisHost<T> H;
    if (!H.build(x, k)) std::printf("1 axis\n");
    pull = spline_pull_table(H);
    pullT = spline_pull_table_transposed(pull, n);
    A.n = AT.n = n;
    A.k = AT.k = k;
    spline_fit_shape<T>(pull, n, k, false, FITB_MAX_WARM, A);
    spline_fit_shape<T>(pullT, n, k, true, FITB_MAX_WARM, AT);
    cudaMalloc(&dp, pull.size() * sizeof(T));
    cudaMalloc(&dpT, pull.size() * sizeof(T));
    cudaMemcpy(dp, pull.data(), pull.size() * sizeof(T), cudaMemcpyHostToDevice);
    cudaMemcpy(dpT, pullT.data(), pull.size() * sizeof(T), cudaMemcpyHostToDevice);
    A.pull = dp;
    AT.pull = dpT;
    nt = (size_t)nx * ny * nz;
    for (int c = 0; c < 3; c++) {
      cudaMalloc(&src[c], nt * sizeof(T));
      cudaMalloc(&a[c], nt * sizeof(T));
      cudaMalloc(&b[c], nt * sizeof(T));
    }
  }
  ~Case() {
    cudaFree(dp);
    cudaFree(dpT);
    for (int c = 0; c < 3; c++) cudaFree(src[c]), cudaFree(a[c]), cudaFree(b[c]);
  }
  void fill(int field) {
    std::mt19937_64 g(17 + field);
    std::vector<T> h(nt);
    for (int c = 0; c < 3; c++) {
      for (size_t q = 0; q < nt; q++) {
        const int i = (int)(q % nx), j = (int)(q / nx % ny), k = (int)(q / ((size_t)nx * ny));
        const int e = axis == 0 ? i : (axis == 1 ? j : k);
        const long l = axis == 0 ? j + (long)ny * k : (axis == 1 ? i + (long)nx * k : i + (long)nx * j);
        h[q] = (T)value(field, g, l + c, e, A.n);
      }
      cudaMemcpy(src[c], h.data(), nt * sizeof(T), cudaMemcpyHostToDevice);
    }
  }
  FieldPtrs<T> in(T *const f[3]) const { return {{f[0], f[1], f[2]}}; }
  FieldPtrsW<T> out(T *const f[3]) const { return {{f[0], f[1], f[2]}}; }

  template <int K>
  void whole(T *const dst[3]) {
    const long sx = nx, sxy = (long)nx * ny;
    if (axis == 0) {
      const long warps = (long)((ny + 31) / 32) * nz;
      const size_t smem = sizeof(T) * 4 * 2 * 32 * (XFIT_W + 1);
      k_fit_xlines<T, K><<<dim3((unsigned)((warps + 3) / 4), 3), 128, smem>>>(A, in(src), out(dst), ny, nz, sx, sxy);
    } else {
      const long nfast = axis == 1 ? sx : sxy, nlines = axis == 1 ? sx * nz : sxy;
      k_fit_lines<T, K><<<dim3((unsigned)((nlines + 255) / 256), 3), 256>>>(A, in(src), out(dst), (int)nfast, nlines, nfast, sxy);
    }
  }
  template <int K, bool ADJ, int LINES>
  void chunked(T *const dst[3], int warm) {
    SplineAxis<T> S = ADJ ? AT : A;
    S.warm = warm;
    fit_block_launch<T, K, ADJ, LINES>(S, in(src), out(dst), axis, (long)nx, (long)nx * ny, (long)ny, (long)nz, 0);
  }
  long differ(T *const p[3], T *const q[3]) {
    std::vector<T> x(nt), y(nt);
    long bad = 0;
    for (int c = 0; c < 3; c++) {
      cudaMemcpy(x.data(), p[c], nt * sizeof(T), cudaMemcpyDeviceToHost);
      cudaMemcpy(y.data(), q[c], nt * sizeof(T), cudaMemcpyDeviceToHost);
      for (size_t r = 0; r < nt; r++) bad += !(x[r] == y[r] || (x[r] != x[r] && y[r] != y[r]));
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      std::printf("1 %s\n", cudaGetErrorString(e));
      bad++;
    }
    return bad;
  }
};

const char *type_name(double) { return "fp64"; }
const char *type_name(float) { return "fp32"; }

template <typename T, int K, int LINES>
void compare(int nx, int ny, int nz, int axis, bool stretched) {
  Case<T> c(nx, ny, nz, axis, K, stretched);
  const int n = c.A.n;
  if ((size_t)n * (LINES + 1 + (LINES < 32 ? 3 : 0)) * sizeof(T) > (size_t)(LINES > 8 ? 112 : 168) * 1024) return;
  for (int field = 0; field < FIELDS; field++) {
    c.fill(field);
    c.template whole<K>(c.a);
    // warm: the measured warm-up; 1: too short, so that nearly every chunk is swept again
    for (int too_short = 0; too_short < 2; too_short++) {
      const int warm = too_short ? 1 : c.A.warm;
      if (warm <= 0) continue;
      c.template chunked<K, false, LINES>(c.b, warm);
      std::printf("%ld %s order %d lines %d %dx%dx%d axis %d %s%s warm %d\n", c.differ(c.a, c.b), type_name(T()), K, LINES, nx, ny, nz, axis,
                  FIELD[field], stretched ? " stretched" : "", warm);
    }
    // the transposed solve against itself swept from the lines' ends (a warm-up of the whole line)
    c.template chunked<K, true, LINES>(c.a, n);
    for (int too_short = 0; too_short < 2; too_short++) {
      const int warm = too_short ? 1 : c.AT.warm;
      if (warm <= 0) continue;
      c.template chunked<K, true, LINES>(c.b, warm);
      std::printf("%ld %s order %d transposed lines %d %dx%dx%d axis %d %s%s warm %d\n", c.differ(c.a, c.b), type_name(T()), K, LINES, nx, ny, nz,
                  axis, FIELD[field], stretched ? " stretched" : "", warm);
    }
  }
}

}  // namespace

// built once per type (-DREAL=double, -DREAL=float), side by side
int main() {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) return 2;
  // the rule: many lines in y and z above 128 MB and not `whole`, x lines up to what a block holds
  auto rule = [](int n, int warm, int axis, long nlines, bool whole, int lines) {
    std::printf("%d rule %s n %d warm %d axis %d whole %d: %d lines\n", fit_block_lines<REAL>(n, warm, axis, nlines, whole) != lines,
                type_name(REAL()), n, warm, axis, whole, lines);
  };
  const bool dp = sizeof(REAL) == 8;
  for (int axis = 1; axis < 3; axis++) {
    rule(130, 41, axis, 130 * 130, false, 0);
    rule(202, 41, axis, 202 * 202, false, dp ? 32 : 0);
    rule(258, 41, axis, 258 * 258, false, 32);
    rule(258, 41, axis, 258 * 258, true, 0);
    rule(23, 41, axis, 100, false, 0);
    rule(24, 41, axis, 100, true, 32);
  }
  rule(302, 41, 0, 302 * 302, true, 32);
  rule(302, FITB_MAX_WARM + 1, 0, 100, false, 0);
  rule(1792, 41, 0, 100, false, 8);
  if (dp) rule(1793, 41, 0, 100, false, 0);
  else rule(3584, 41, 0, 100, false, 8), rule(3585, 41, 0, 100, false, 0);
  // the count of chunks swept again: below one per block on random lines (and, in FP64, constant ones), above
  // on lines at rest but for their middle, so that the whole-line sweeps take over there
  for (const int field : std::initializer_list<int>{0, 1, 6}) {
    if (field == 1 && !dp) continue;
    Case<REAL> c(150, 150, 5, 1, 4, false);
    unsigned *redo, n = 0;
    cudaMalloc(&redo, sizeof(unsigned));
    cudaMemset(redo, 0, sizeof(unsigned));
    c.fill(field);
    fit_block_launch<REAL, 4, false, 32>(c.A, c.in(c.src), c.out(c.b), 1, 150, 150 * 150, 150, 5, 0, redo);
    cudaMemcpy(&n, redo, sizeof(unsigned), cudaMemcpyDeviceToHost);
    cudaFree(redo);
    const unsigned blocks = 3 * ((150 * 5 + 31) / 32);
    std::printf("%d count %s %s: %u chunks, %u blocks\n", field == 6 ? n <= blocks : n > blocks, type_name(REAL()), FIELD[field], n, blocks);
  }
  compare<REAL, 4, 32>(5, 3, 3, 0, false);     // fewer points than chunks
  compare<REAL, 4, 32>(203, 35, 5, 0, false);  // a partial block of lines
  compare<REAL, 4, 32>(203, 35, 5, 0, true);
  compare<REAL, 4, 8>(1003, 9, 3, 0, true);
  compare<REAL, 4, 8>(1790, 3, 3, 0, false);   // the longest FP64 line of the rule
  compare<REAL, 4, 32>(37, 150, 3, 1, false);
  compare<REAL, 4, 8>(11, 1200, 3, 1, false);
  compare<REAL, 4, 32>(37, 5, 97, 2, false);
  if constexpr (sizeof(REAL) == 8) {
    compare<REAL, 4, 16>(700, 9, 3, 0, false);
    compare<REAL, 4, 16>(20, 490, 3, 1, true);
    compare<REAL, 3, 32>(203, 35, 5, 0, true);  // two off-diagonal factors on every row
    compare<REAL, 3, 32>(37, 150, 3, 1, false);
  }
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 3;
}
