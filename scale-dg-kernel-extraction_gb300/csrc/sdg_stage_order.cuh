// Per-order launch entry: resolves precision and summation order to one
// instantiation of the fused stage kernels.
#pragma once

#include "sdg_stage.cuh"
#include "sdg_stage_eo.cuh"
#include "sdg_stage_fix.cuh"
#include "sdg_stage_line.cuh"
#include "sdg_stage_loop.cuh"

namespace sdg {

template <int P>
int launch_stage_order(int prec, int opt, const StageArgs& a, cudaStream_t st) {
  constexpr bool kCanSplit = (P > 7);
  const bool split = kCanSplit && (opt != SDG_OPT_GENERAL);
  // FP64 and emulated FP64 are one arithmetic: the fixed-point stage
  if (prec != SDG_PREC_FP32)
    return opt == SDG_OPT_EVENODD ? launch_stage_fix_impl<P, true>(a, st)
                                  : launch_stage_fix_impl<P, false>(a, st);
  if (opt == SDG_OPT_EVENODD) return launch_stage_line_impl<P>(a, st);
  if (split) return launch_stage_impl<P, float, float, kCanSplit>(a, st);
  return launch_stage_impl<P, float, float, false>(a, st);
}

// A whole step call of a small box in one launch (sdg_stage_loop.cuh); with q
// null only *most, the most elements such a launch takes.
template <int P>
int launch_loop_order(int opt, const StageArgs& a, double* const* q, double dt, int nstep,
                      unsigned* bar, int polls, long long* most, cudaStream_t st) {
  const bool eo = opt == SDG_OPT_EVENODD;
  if (!q) return eo ? fix_loop_most<P, true>(most) : fix_loop_most<P, false>(most);
  return eo ? launch_stage_fix_loop<P, true>(a, q, dt, nstep, bar, polls, st)
            : launch_stage_fix_loop<P, false>(a, q, dt, nstep, bar, polls, st);
}

// The entry points of one order (one translation unit per group of orders, so
// that the build compiles them in parallel).
#define SDG_DEFINE_ORDER(p)                                                                 \
  int launch_stage_p##p(int prec, int opt, const StageArgs& a, cudaStream_t st) {           \
    return launch_stage_order<p>(prec, opt, a, st);                                         \
  }                                                                                         \
  int launch_loop_p##p(int opt, const StageArgs& a, double* const* q, double dt, int nstep, \
                       unsigned* bar, int polls, long long* most, cudaStream_t st) {        \
    return launch_loop_order<p>(opt, a, q, dt, nstep, bar, polls, most, st);                \
  }

}  // namespace sdg
