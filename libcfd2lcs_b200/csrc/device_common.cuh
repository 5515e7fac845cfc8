// Device-side building blocks shared by the libcfd2lcs_b200 kernels: grid access,
// ghost rules, trilinear stencil, boundary conditions and node tracking.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "grid.h"
#include "scalar_ops.h"

namespace cfd2lcs {

// Device error word bits (folded into the library's error latch after each update).
enum : int {
  ERR_NONFINITE_VELOCITY = 1,
  ERR_TRACKING = 2,
  ERR_UNKNOWN_FLAG = 4,
  ERR_SPLINE_RANGE = 8,
  ERR_ASYNC_COPY = 16,  // a shared-memory staging copy did not complete within its wait limit
  ERR_GRID_BARRIER = 32,  // the blocks of one launch did not all reach a barrier within its wait limit
};

enum { EULER_ = 0, TRAPEZOIDAL_ = 1, RK2_ = 2, RK3_ = 3, RK4_ = 4 };
// INTERP_SPLINE: B-spline of any order per axis; INTERP_SPLINE4: cubic on every axis (3-D grid);
// INTERP_SPLINE442: cubic in x and y, order 2 in z (two-dimensional grid, z singleton);
// INTERP_TSE / INTERP_TSE_LIMIT: Taylor series about the tracked node, without / with limiter;
// INTERP_CTSE / INTERP_CTSE_LIMIT: the same on a non-rectilinear grid (least-squares gradients,
// full coordinate arrays), the only interpolators the reference runs there
enum {
  INTERP_NEAREST = 0,
  INTERP_LINEAR = 1,
  INTERP_SPLINE = 2,
  INTERP_SPLINE4 = 3,
  INTERP_TSE = 4,
  INTERP_TSE_LIMIT = 5,
  INTERP_CTSE = 6,
  INTERP_CTSE_LIMIT = 7,
  INTERP_SPLINE442 = 8
};

__host__ __device__ constexpr bool interp_is_spline(int interp) {
  return interp == INTERP_SPLINE || interp == INTERP_SPLINE4 || interp == INTERP_SPLINE442;
}
// the spline orders a B-spline variant fixes at compile time (spline.cuh): 4 on every axis, 4, 4 and
// 2, or 0 (read from the axes)
__host__ __device__ constexpr int spline_orders(int interp) { return interp == INTERP_SPLINE4 ? 4 : (interp == INTERP_SPLINE442 ? 442 : 0); }
__host__ __device__ constexpr bool interp_is_curv(int interp) { return interp == INTERP_CTSE || interp == INTERP_CTSE_LIMIT; }

// Orders `stream` after everything the caller has queued so far on the default stream (and, as the
// legacy default stream waits for them, on the streams that synchronise with it).  The library's
// streams are non-blocking: without this its kernels may read arrays that are still being written
// and write buffers that queued work still uses.  ev: any event of the device, free for reuse at once.
// About 1 us of host time; asking first whether anything is queued (cudaStreamQuery) takes longer.
inline cudaError_t wait_for_caller(cudaStream_t stream, cudaEvent_t ev) {
  const cudaError_t e = cudaEventRecord(ev, cudaStreamLegacy);
  return e != cudaSuccess ? e : cudaStreamWaitEvent(stream, ev, 0);
}

// Whether half of the device's memory stays free beside `bytes` more: the condition for buffers that
// only save time, so that the library's later ones and the caller's own still fit.
inline bool ample_memory(size_t bytes) {
  size_t free = 0, total = 0;
  return cudaMemGetInfo(&free, &total) == cudaSuccess && free >= bytes + total / 2;
}

template <typename T>
struct DevGrid {
  GridParams<T> P;
  const T *lt[3];        // node coordinate lines, index 0..n+1
  const T *li[3];        // interpolation lines, index 0..n+1
  // RN(1 / (li[a][i+1] - li[a][i])), index 0..n: the LINEAR stencils' fractions (lin_quotient)
  const T *ri[3] = {nullptr, nullptr, nullptr};
  // RN(1 / (bb[a + 3] - bb[a])) of the bounding box, for the composition's node guess (lin_quotient)
  T bbr[3] = {T(0), T(0), T(0)};
  const T *invd[3];      // inverse half spans, see HostGrid::invd
  const int8_t *flag;    // padded bcflag or nullptr
  const T *nrm[3];       // boundary normals (padded) or nullptr
  // non-rectilinear grids (P.curv), else nullptr:
  const T *X[3] = {nullptr, nullptr, nullptr};      // padded node coordinates
  const T *lsw = nullptr;                           // least-squares weights: plane nb*3 + c holds face
                                                    // neighbour nb's weight in d/dx_c
  const T *pnrm[3] = {nullptr, nullptr, nullptr};   // 2-D grids: unit normal of the data plane per interior node
  const T *invdp[3] = {nullptr, nullptr, nullptr};  // padded inverse half spans
};

template <typename T>
struct FieldPtrs {
  const T *f[3];
};

template <typename T>
struct FieldPtrsW {
  T *f[3];
};

// Forward particles (one per lcs node): position, unwrapped displacement and tracked node
// (the reference's lp%xp, lp%dx, lp%no_scfd).  Storage slot s holds the particle that started
// at interior node id[s]; slot[q] is the inverse map.  The engine re-sorts the slots by grid
// cell during an update, so that a block's particles gather neighbouring spline taps.
template <typename T>
struct Particles {
  T *x[3];
  T *dx[3];
  int *no[3];
  int *id;
  int *slot;
};

__device__ __forceinline__ int pidx(const int sx, const int sxy, int i, int j, int k) { return i + sx * j + sxy * k; }

// max(min(v,1),0) of the reference; a NaN argument yields the bound as gfortran does
__device__ __forceinline__ double clamp01(double v) { return clamp01_select(v); }
__device__ __forceinline__ float clamp01(float v) { return fmaxf(fminf(v, 1.0f), 0.0f); }

// ---------------------------------------------------------------------------------------
// Ghost fill of a padded field, written by the interior node that is the source of each
// ghost cell.  The rules restate exchange_sdata (one rank: periodic SELF copies,
// src/comms_m.f90:679-869) followed by
//   VEL: set_velocity_bc, src/sgrid_m.f90:810-866
//   FM : set_flowmap_bc,  src/flowmap_m.f90:325-392
// vpre: value the periodic copy sees (before interior boundary zeroing); vfin: final
// interior value (what a zero-gradient ghost copies).
// ---------------------------------------------------------------------------------------
enum { GHOST_VEL = 0, GHOST_FM = 1 };

__device__ __forceinline__ int ghost_rule(int kind, int f) {
  // 0: periodic image, 1: zero, 2: copy of the nearest interior node, 3: unknown flag
  if (f == LCS_INTERNAL) return 0;
  if (kind == GHOST_VEL) {
    if (f == LCS_MASK || f == LCS_WALL) return 1;
    if (f == LCS_SLIP || f == LCS_INFLOW || f == LCS_OUTFLOW || f == LCS_2D) return 2;
  } else {
    if (f == LCS_WALL || f == LCS_MASK || f == LCS_INFLOW || f == LCS_OUTFLOW) return 1;
    if (f == LCS_SLIP || f == LCS_2D) return 2;
  }
  return 3;
}

// Every ghost cell has exactly one source node: its periodic image (rule 0) or its
// nearest interior node (rules 1, 2).  The node (i,j,k) enumerates both candidate sets
// and writes the cells whose rule points back at it, so no two threads write one cell.
template <typename T, bool HAS_FLAGS, int KIND, typename TF = T>
__device__ void write_ghosts(const DevGrid<T> &g, TF *const f[3], int i, int j, int k, const TF vpre[3], const TF vfin[3],
                             int *err) {
  // a node writes ghosts at its own index and, along every axis on whose end it sits, one index
  // further out (rules 1 and 2: the near side) or at the other end of the axis (rule 0: the image).
  // The 26 cells are unrolled over compile-time offsets: index lists built at run time lived in local
  // memory and took 4700 cycles per node of a plane, whose every node is an end along z (a third of
  // a LINEAR subcycle there).
  const int n[3] = {g.P.n[0], g.P.n[1], g.P.n[2]}, v[3] = {i, j, k}, str[3] = {1, g.P.sx, g.P.sxy};
  bool lo[3], hi[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    lo[a] = v[a] == 1;
    hi[a] = v[a] == n[a];
  }
  if (!(lo[0] || lo[1] || lo[2] || hi[0] || hi[1] || hi[2])) return;
  const int p0 = pidx(g.P.sx, g.P.sxy, i, j, k);
  // near side: index 0 next to node 1, n+1 next to node n
  if (HAS_FLAGS) {
#pragma unroll
    for (int o2 = -1; o2 <= 1; o2++) {
      if ((o2 < 0 && !lo[2]) || (o2 > 0 && !hi[2])) continue;
#pragma unroll
      for (int o1 = -1; o1 <= 1; o1++) {
        if ((o1 < 0 && !lo[1]) || (o1 > 0 && !hi[1])) continue;
#pragma unroll
        for (int o0 = -1; o0 <= 1; o0++) {
          if ((o0 < 0 && !lo[0]) || (o0 > 0 && !hi[0])) continue;
          if (o0 == 0 && o1 == 0 && o2 == 0) continue;
          const int p = p0 + o0 * str[0] + o1 * str[1] + o2 * str[2];
          const int rule = ghost_rule(KIND, (int)__ldg(g.flag + p));
          if (rule == 0) continue;
          if (rule == 3) {
            atomicOr(err, ERR_UNKNOWN_FLAG);
            continue;
          }
#pragma unroll
          for (int c = 0; c < 3; c++) f[c][p] = rule == 1 ? TF(0) : vfin[c];
        }
      }
    }
  }
  // images: index n+1 is the image of node 1 and index 0 of node n, along periodic axes (a
  // singleton axis has the image of node 1 only, as an axis whose both ends it is)
  int far[3];  // padded offset of the image along each axis, 0: none
  bool any = false;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    far[a] = !g.P.per[a] ? 0 : (lo[a] ? n[a] * str[a] : (hi[a] ? -n[a] * str[a] : 0));
    any = any || far[a] != 0;
  }
  if (!any) return;
#pragma unroll
  for (int m = 1; m < 8; m++) {
    if (((m & 1) && !far[0]) || ((m & 2) && !far[1]) || ((m & 4) && !far[2])) continue;
    const int p = p0 + ((m & 1) ? far[0] : 0) + ((m & 2) ? far[1] : 0) + ((m & 4) ? far[2] : 0);
    if (HAS_FLAGS && ghost_rule(KIND, (int)__ldg(g.flag + p)) != 0) continue;
#pragma unroll
    for (int c = 0; c < 3; c++) f[c][p] = vpre[c];
  }
}

}  // namespace cfd2lcs
