// Mixed-precision instantiations of the tiled force + integrator kernel:
// FP64 positions, velocities, shape terms, integration and reductions; FP32
// pair terms on FP64-formed offsets.
#include "cr_launch.h"
#include "cr_tile_kernel.cuh"

namespace cr {

template <int POT, int INTER, int MODE>
static void launch_mixed_t(const LaunchCfg& c, const SysParams& p, const SysArrays& a, const StepArgs& s) {
  if (c.lanes == 1) launch_k(c.pdl, k_tile<POT, INTER, MODE, 128, 1, PREC_MIXED>, dim3(c.grid), dim3(128), c.stream, 0, p, a, s);
  else if (c.lanes == 4) launch_k(c.pdl, k_tile<POT, INTER, MODE, 256, 4, PREC_MIXED>, dim3(c.grid), dim3(256), c.stream, 0, p, a, s);
  else if (c.lanes == 8) launch_k(c.pdl, k_tile<POT, INTER, MODE, 256, 8, PREC_MIXED>, dim3(c.grid), dim3(256), c.stream, 0, p, a, s);
  else launch_k(c.pdl, k_tile<POT, INTER, MODE, 192, 2, PREC_MIXED>, dim3(c.grid), dim3(192), c.stream, 0, p, a, s);
}

void launch_tile_mixed(const LaunchCfg& c, int pot, int inter, int mode, const SysParams& p, const SysArrays& a,
                       const StepArgs& s) {
#define CR_MIXED_CASE(P)                                                                \
  case P:                                                                               \
    if (inter == INT_VV) {                                                              \
      if (mode == MODE_FORCE) launch_mixed_t<P, INT_VV, MODE_FORCE>(c, p, a, s);        \
      else launch_mixed_t<P, INT_VV, MODE_STEP>(c, p, a, s);                            \
    } else {                                                                            \
      if (mode == MODE_FORCE) launch_mixed_t<P, INT_SMOOTH, MODE_FORCE>(c, p, a, s);    \
      else launch_mixed_t<P, INT_SMOOTH, MODE_STEP>(c, p, a, s);                        \
    }                                                                                   \
    break;
  switch (pot) {
    CR_MIXED_CASE(POT_HARMONIC)
    CR_MIXED_CASE(POT_LJ)
    CR_MIXED_CASE(POT_ADHESIVE)
    CR_MIXED_CASE(POT_WCA)
    default: break;
  }
#undef CR_MIXED_CASE
}


// Multi-step kernel (k_tile_steps): the shapes of tile_steps_fn_fp64.
template <int POT, int INTER>
static TileStepsFn steps_fn_l(int lanes, bool staged) {
  if (lanes == 1) {
    if (staged) return k_tile_steps<POT, INTER, 128, 1, PREC_MIXED, true>;
    return k_tile_steps<POT, INTER, 128, 1, PREC_MIXED, false>;
  }
  if (lanes == 2 && staged) return k_tile_steps<POT, INTER, 192, 2, PREC_MIXED, true>;
  return nullptr;
}

template <int POT>
static TileStepsFn steps_fn_p(int inter, int lanes, bool staged) {
  return inter == INT_VV ? steps_fn_l<POT, INT_VV>(lanes, staged) : steps_fn_l<POT, INT_SMOOTH>(lanes, staged);
}

TileStepsFn tile_steps_fn_mixed(int pot, int inter, int lanes, bool staged) {
  switch (pot) {
    case POT_HARMONIC: return steps_fn_p<POT_HARMONIC>(inter, lanes, staged);
    case POT_LJ: return steps_fn_p<POT_LJ>(inter, lanes, staged);
    case POT_ADHESIVE: return steps_fn_p<POT_ADHESIVE>(inter, lanes, staged);
    case POT_WCA: return steps_fn_p<POT_WCA>(inter, lanes, staged);
    default: return nullptr;
  }
}

}  // namespace cr
