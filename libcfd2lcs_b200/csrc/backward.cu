// Backward semi-Lagrangian subcycle, gathering form: every variant of k_sl_subcycle, and the LINEAR
// ones that run several subcycles per launch (k_sl_run).
#include "engine.h"
#include "launch.h"
#include "tile.cuh"

namespace cfd2lcs {

template <typename T, typename TV>
void launch_sl_gather(int iv, int integrator, bool flags, dim3 grd, dim3 blk, cudaStream_t stream, const DevGrid<T> &g,
                      const SplineAxes<T> &sa, const VelFields<TV> &V, const FieldPtrs<T> &fo, const FieldPtrsW<T> &fn, const StageTimes &S,
                      T dt, int *err) {
  for_variant(iv, [&](auto VI) {
    for_flags(flags, [&](auto FL) {
      for_integrator(integrator, [&](auto IG) {
        constexpr bool F = decltype(FL)::value || decltype(VI)::value == INTERP_SPLINE442;
        k_sl_subcycle<T, TV, decltype(IG)::value, decltype(VI)::value, F><<<grd, blk, 0, stream>>>(g, sa, V, fo, fn, S, dt, err);
      });
    });
  });
}

template <typename T, typename TV>
cudaError_t launch_sl_run(int integrator, bool flags, dim3 blk, int *max_blocks, cudaStream_t stream, const DevGrid<T> &g,
                          const VelFields<TV> &V, const FieldPtrsW<T> &fa, const FieldPtrsW<T> &fb, const StageRun &S, T dt, unsigned *bar,
                          unsigned *arrivals, int *err) {
  cudaError_t rc = cudaSuccess;
  for_flags(flags, [&](auto FL) {
    for_integrator(integrator, [&](auto IG) {
      // a plane's ghosts carry flags, so PLANE comes with them
      constexpr bool F = decltype(FL)::value;
      constexpr int I = decltype(IG)::value;
      auto *kernel = F && g.P.single_axis == 2 ? k_sl_run<T, TV, I, F, F> : k_sl_run<T, TV, I, F, false>;
      if (*max_blocks == 0) {
        int dev = 0, sms = 0, per = 0;
        if ((rc = cudaGetDevice(&dev)) != cudaSuccess || (rc = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
          return;
        rc = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, (int)(blk.x * blk.y * blk.z), 0);
        *max_blocks = per * sms;
        return;
      }
      auto tiles = [](int n, unsigned b) { return (n + (int)b - 1) / (int)b; };
      int3 nt{tiles(g.P.n[0], blk.x), tiles(g.P.n[1], blk.y), tiles(g.P.n[2], blk.z)};
      const int blocks = nt.x * nt.y * nt.z < *max_blocks ? nt.x * nt.y * nt.z : *max_blocks;
      unsigned base = *arrivals;
      T step = dt;
      void *args[] = {const_cast<DevGrid<T> *>(&g), const_cast<VelFields<TV> *>(&V), const_cast<FieldPtrsW<T> *>(&fa),
                      const_cast<FieldPtrsW<T> *>(&fb), const_cast<StageRun *>(&S), &step, &nt, &bar, &base, &err};
      rc = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel), dim3(blocks), blk, args, 0, stream);
      if (rc == cudaSuccess) *arrivals += (unsigned)((S.n - 1) * blocks);
    });
  });
  return rc;
}

#define SL_GATHER(TV)                                                                                                                  \
  template void launch_sl_gather<lcsdata_t, TV>(int, int, bool, dim3, dim3, cudaStream_t, const DevGrid<lcsdata_t> &,                     \
                                                const SplineAxes<lcsdata_t> &, const VelFields<TV> &, const FieldPtrs<lcsdata_t> &,       \
                                                const FieldPtrsW<lcsdata_t> &, const StageTimes &, lcsdata_t, int *);       \
  template cudaError_t launch_sl_run<lcsdata_t, TV>(int, bool, dim3, int *, cudaStream_t, const DevGrid<lcsdata_t> &, const VelFields<TV> &, \
                                                    const FieldPtrsW<lcsdata_t> &, const FieldPtrsW<lcsdata_t> &, const StageRun &,        \
                                                    lcsdata_t, unsigned *, unsigned *, int *);
SL_GATHER(lcsdata_t)
#ifndef CFD2LCS_SP
SL_GATHER(float)
#endif

}  // namespace cfd2lcs
