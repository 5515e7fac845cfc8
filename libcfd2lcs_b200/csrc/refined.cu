// Backward subcycle on refined lcs grids: every variant of k_sl_refined.
#include "engine.h"
#include "kernels.cuh"
#include "launch.h"

namespace cfd2lcs {

template <typename T, typename TV>
void launch_sl_refined(int iv, int integrator, bool flags_s, bool flags_l, dim3 grd, dim3 blk, cudaStream_t stream, const DevGrid<T> &gl,
                       const DevGrid<T> &gs, const SplineAxes<T> &sas, const SplineAxes<T> &sal, const FieldPtrs<T> &pos, int *no0, int *no1,
                       int *no2, const VelFields<TV> &V, const FieldPtrs<T> &fo, const FieldPtrsW<T> &fn, const StageTimes &S, T dt, int *err) {
  auto go = [&](auto VI) {
    for_flags(flags_s, [&](auto FS) {
      for_flags(flags_l, [&](auto FL) {
        for_integrator(integrator, [&](auto IG) {
          k_sl_refined<T, TV, decltype(IG)::value, decltype(VI)::value, decltype(FS)::value, decltype(FL)::value>
              <<<grd, blk, 0, stream>>>(gl, gs, sas, sal, pos, no0, no1, no2, V, fo, fn, S, dt, err);
        });
      });
    });
  };
  switch (iv) {
    case INTERP_NEAREST: go(std::integral_constant<int, INTERP_NEAREST>()); break;
    case INTERP_LINEAR: go(std::integral_constant<int, INTERP_LINEAR>()); break;
    case INTERP_TSE: go(std::integral_constant<int, INTERP_TSE>()); break;
    case INTERP_TSE_LIMIT: go(std::integral_constant<int, INTERP_TSE_LIMIT>()); break;
    case INTERP_SPLINE4: go(std::integral_constant<int, INTERP_SPLINE4>()); break;
    default: go(std::integral_constant<int, INTERP_SPLINE>()); break;
  }
}

#define SL_REFINED(TV)                                                                                                                 \
  template void launch_sl_refined<lcsdata_t, TV>(int, int, bool, bool, dim3, dim3, cudaStream_t, const DevGrid<lcsdata_t> &,              \
                                                 const DevGrid<lcsdata_t> &, const SplineAxes<lcsdata_t> &, const SplineAxes<lcsdata_t> &, \
                                                 const FieldPtrs<lcsdata_t> &, int *, int *, int *, const VelFields<TV> &,                \
                                                 const FieldPtrs<lcsdata_t> &, const FieldPtrsW<lcsdata_t> &, const StageTimes &,         \
                                                 lcsdata_t, int *);
SL_REFINED(lcsdata_t)
#ifndef CFD2LCS_SP
SL_REFINED(float)
#endif

}  // namespace cfd2lcs
