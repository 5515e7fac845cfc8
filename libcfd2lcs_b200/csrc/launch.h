// Launches of the subcycle kernels that gather their taps, by interpolator variant, integrator and
// boundary flags.  Each family is instantiated in a source file of its own (backward.cu, forward.cu,
// refined.cu) for velocity stored in the interface type and, in the double library, in FP32.
#pragma once

#include "advect.cuh"

namespace cfd2lcs {

template <typename T, typename TV>
void launch_sl_gather(int iv, int integrator, bool flags, dim3 grd, dim3 blk, cudaStream_t stream, const DevGrid<T> &g,
                      const SplineAxes<T> &sa, const VelFields<TV> &V, const FieldPtrs<T> &fo, const FieldPtrsW<T> &fn, const StageTimes &S,
                      T dt, int *err);

template <typename T, typename TV>
void launch_fwd_gather(int iv, int integrator, bool flags, cudaStream_t stream, const DevGrid<T> &g, const SplineAxes<T> &sa,
                       const VelFields<TV> &V, const Particles<T> &P, const StageTimes &S, T dt, int np, int *err);

// the variants other than the B-splines: S.n subcycles in one launch (k_fwd_run)
template <typename T, typename TV>
void launch_fwd_run(int iv, int integrator, bool flags, cudaStream_t stream, const DevGrid<T> &g, const VelFields<TV> &V,
                    const Particles<T> &P, const StageRun &S, T dt, int np, int *err);

// LINEAR, S.n backward subcycles in one cooperative launch (k_sl_run) of at most max_blocks blocks
// (0: asks for that number, the blocks resident on the device at once, and launches nothing).
// *arrivals: barrier arrivals on bar so far.
template <typename T, typename TV>
cudaError_t launch_sl_run(int integrator, bool flags, dim3 blk, int *max_blocks, cudaStream_t stream, const DevGrid<T> &g,
                          const VelFields<TV> &V, const FieldPtrsW<T> &fa, const FieldPtrsW<T> &fb, const StageRun &S, T dt, unsigned *bar,
                          unsigned *arrivals, int *err);

template <typename T, typename TV>
void launch_sl_refined(int iv, int integrator, bool flags_s, bool flags_l, dim3 grd, dim3 blk, cudaStream_t stream, const DevGrid<T> &gl,
                       const DevGrid<T> &gs, const SplineAxes<T> &sas, const SplineAxes<T> &sal, const FieldPtrs<T> &pos, int *no0, int *no1,
                       int *no2, const VelFields<TV> &V, const FieldPtrs<T> &fo, const FieldPtrsW<T> &fn, const StageTimes &S, T dt, int *err);

// integer template arguments from run-time choices
template <typename F>
inline void for_integrator(int integrator, F f) {
  switch (integrator) {
    case 0: f(std::integral_constant<int, EULER_>()); break;
    case 1: f(std::integral_constant<int, TRAPEZOIDAL_>()); break;
    case 2: f(std::integral_constant<int, RK2_>()); break;
    case 3: f(std::integral_constant<int, RK3_>()); break;
    default: f(std::integral_constant<int, RK4_>()); break;
  }
}

template <typename F>
inline void for_flags(bool flags, F f) {
  if (flags) f(std::true_type());
  else f(std::false_type());
}

// the variants of a solver grid (SPLINE442 always has flags: the ghosts of its singleton axis)
template <typename F>
inline void for_variant(int iv, F f) {
  switch (iv) {
    case INTERP_NEAREST: f(std::integral_constant<int, INTERP_NEAREST>()); break;
    case INTERP_LINEAR: f(std::integral_constant<int, INTERP_LINEAR>()); break;
    case INTERP_TSE: f(std::integral_constant<int, INTERP_TSE>()); break;
    case INTERP_TSE_LIMIT: f(std::integral_constant<int, INTERP_TSE_LIMIT>()); break;
    case INTERP_CTSE: f(std::integral_constant<int, INTERP_CTSE>()); break;
    case INTERP_CTSE_LIMIT: f(std::integral_constant<int, INTERP_CTSE_LIMIT>()); break;
    case INTERP_SPLINE4: f(std::integral_constant<int, INTERP_SPLINE4>()); break;
    case INTERP_SPLINE442: f(std::integral_constant<int, INTERP_SPLINE442>()); break;
    default: f(std::integral_constant<int, INTERP_SPLINE>()); break;
  }
}

}  // namespace cfd2lcs
