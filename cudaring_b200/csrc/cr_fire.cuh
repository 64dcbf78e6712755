// One FIRE iteration up to the position update, per vertex, for a single
// system: used by the one-op-per-launch kernel k_fire_pre (cr_misc.cu) and by
// the multi-iteration kernel k_fire_steps (cr_tile_fire.cu).
#pragma once
#include "cr_launch.h"
#include "cr_tile.cuh"

namespace cr {

struct FireScalars {
  double dt, alpha;
  long long nstep;
};

// checkFIREParams (src/FIRE.cu:338-371) from P = v.F: the next scalars, and
// whether the step is taken back.
__device__ __forceinline__ bool fire_next(const FireParams& fp, double P, FireScalars& f) {
  if (P > 0) {
    f.nstep++;
    if (f.nstep > fp.min_step) {
      f.dt = fmin(f.dt * fp.f_inc, fp.dt_max);
      f.alpha *= fp.f_a;
    }
    return false;
  }
  f.nstep = 0;
  f.dt = fmax(f.dt * fp.f_dec, fp.dt_max / 10);
  f.alpha = fp.a_start;
  return true;
}

// The half kick (src/FIRE.cu:320-335), bendVertexVelocityTowardsForce
// (:374-394) and updateVertexPosition (:302-317) of one vertex.  |v|^2 after
// the half kick is formed from the three sums of the previous force op:
// |v + h F|^2 = vv + 2h vF + h^2 FF.
__device__ __forceinline__ void fire_move(const FireScalars& f, bool rollback, double P, double vv, double ff,
                                          double2 force, double2& x, double2& vel) {
  const double h = 0.5 * f.dt;
  const double vpost2 = rollback ? (h * h) * ff : vv + f.dt * P + (h * h) * ff;
  if (rollback) {
    x = make_double2(x.x - h * vel.x, x.y - h * vel.y);
    vel = make_double2(0.0, 0.0);
  }
  vel = make_double2(vel.x + h * force.x, vel.y + h * force.y);
  if (ff > 0) {
    const double ratio = sqrt(vpost2 / ff);
    vel = make_double2((1 - f.alpha) * vel.x + f.alpha * force.x * ratio,
                       (1 - f.alpha) * vel.y + f.alpha * force.y * ratio);
  }
  x = make_double2(x.x + f.dt * vel.x, x.y + f.dt * vel.y);
}

// Multi-iteration FIRE kernel (cr_tile_fire.cu): nullptr for lane counts other
// than one and two.
using FireStepsFn = void (*)(SysParams, SysArrays, StepArgs, FireParams, double*);
FireStepsFn fire_steps_fn(int pot, int inter, int lanes);
int fire_steps_max_blocks(FireStepsFn fn, int inter, int lanes);
cudaError_t launch_fire_steps(FireStepsFn fn, int inter, const LaunchCfg& c, const SysParams& p, const SysArrays& a,
                              const StepArgs& s, const FireParams& fp, double* fire_state);

}  // namespace cr
