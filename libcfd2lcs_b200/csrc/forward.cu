// Forward particle subcycle, gathering form: k_fwd_subcycle for the variants whose stages are blended
// fields (LINEAR on large grids, the B-splines), k_fwd_run for the others.
#include "engine.h"
#include "kernels.cuh"
#include "launch.h"

namespace cfd2lcs {

template <typename T, typename TV>
void launch_fwd_gather(int iv, int integrator, bool flags, cudaStream_t stream, const DevGrid<T> &g, const SplineAxes<T> &sa,
                       const VelFields<TV> &V, const Particles<T> &P, const StageTimes &S, T dt, int np, int *err) {
  const int blk = 256, grd = (np + blk - 1) / blk;
  auto go = [&](auto VI) {
    for_flags(flags, [&](auto FL) {
      for_integrator(integrator, [&](auto IG) {
        constexpr bool F = decltype(FL)::value || decltype(VI)::value == INTERP_SPLINE442;
        k_fwd_subcycle<T, TV, decltype(IG)::value, decltype(VI)::value, F><<<grd, blk, 0, stream>>>(g, sa, V, P, S, dt, np, err);
      });
    });
  };
  switch (iv) {
    case INTERP_LINEAR: go(std::integral_constant<int, INTERP_LINEAR>()); break;
    case INTERP_SPLINE4: go(std::integral_constant<int, INTERP_SPLINE4>()); break;
    case INTERP_SPLINE442: go(std::integral_constant<int, INTERP_SPLINE442>()); break;
    default: go(std::integral_constant<int, INTERP_SPLINE>()); break;
  }
}

template <typename T, typename TV>
void launch_fwd_run(int iv, int integrator, bool flags, cudaStream_t stream, const DevGrid<T> &g, const VelFields<TV> &V,
                    const Particles<T> &P, const StageRun &S, T dt, int np, int *err) {
  const int blk = 256, grd = (np + blk - 1) / blk;
  for_variant(iv, [&](auto VI) {
    if constexpr (!interp_is_spline(decltype(VI)::value)) {
      for_flags(flags, [&](auto FL) {
        for_integrator(integrator, [&](auto IG) {
          k_fwd_run<T, TV, decltype(IG)::value, decltype(VI)::value, decltype(FL)::value>
              <<<grd, blk, 0, stream>>>(g, SplineAxes<T>{}, V, P, S, dt, np, err);
        });
      });
    }
  });
}

#define FWD_GATHER(TV)                                                                                                                 \
  template void launch_fwd_gather<lcsdata_t, TV>(int, int, bool, cudaStream_t, const DevGrid<lcsdata_t> &, const SplineAxes<lcsdata_t> &, \
                                                 const VelFields<TV> &, const Particles<lcsdata_t> &, const StageTimes &, lcsdata_t, int, \
                                                 int *);                                                                               \
  template void launch_fwd_run<lcsdata_t, TV>(int, int, bool, cudaStream_t, const DevGrid<lcsdata_t> &, const VelFields<TV> &,              \
                                              const Particles<lcsdata_t> &, const StageRun &, lcsdata_t, int, int *);
FWD_GATHER(lcsdata_t)
#ifndef CFD2LCS_SP
FWD_GATHER(float)
#endif

}  // namespace cfd2lcs
