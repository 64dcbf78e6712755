// FIRE iterations of one system in one launch: up to s.persist_max iterations
// with grid barriers in place of kernel boundaries (FP64, one or two lanes per
// vertex, a grid the GPU holds at once; other cases run one launch per op).
//
// Each CTA owns one tile.  An iteration:
//   pre-kick of the tile's vertices (fire_next, fire_move), displacement check
//   -- grid barrier; a check that fired ends the launch with the force op
//      pending: the list build that follows runs, the next launch starts there
//   force op of the tile (the tiled kernel's FIRE op: forces, second half
//   kick, the CTA's partial sums)
//   -- grid barrier; every CTA then reduces the partial sums itself, in the
//      one order, so all of them take the same next step and see convergence
//      together
// The lists and the topology stay in shared memory for the launch (Stage,
// cr_tile_kernel.cuh).  Bound by latency: two grid barriers and the chain of
// one tile.  As four launches per iteration, in graphs that every call captured
// and destroyed again, 200 iterations of 9,750 vertices (harmonic
// vertex-vertex) took 5.3 ms; here 2.3 ms.  One CTA of the grid per SM or less
// issues in 10% of the cycles; its first stall is the wait at the barriers.
#include "cr_fire.cuh"
#include "cr_launch.h"
#include "cr_tile_kernel.cuh"

namespace cr {

template <int POT, int INTER, int BLOCK, int L>
__global__ void __launch_bounds__(BLOCK, tile_threads_per_sm<PREC_FP64, L>() / BLOCK)
    k_fire_steps(const __grid_constant__ SysParams p, const __grid_constant__ SysArrays a,
                 const __grid_constant__ StepArgs s, const __grid_constant__ FireParams fp, double* fire_state) {
  pdl_wait();
  pdl_trigger();
  DevStatus* st = s.status;
  const volatile DevStatus* vs = st;
  if (vs->abort | vs->converged) return;
  const long long left = vs->steps_left;
  if (left <= 0) return;
  const int n = (int)(left < (long long)s.persist_max ? left : (long long)s.persist_max);
  const bool pending = vs->bpending != 0;  // the last launch left with its force op due
  StepsBarrier bar(st);
  const long long it0 = vs->fire_iters;
  __shared__ double s_sums[NSUM];
  if (threadIdx.x < NSUM) s_sums[threadIdx.x] = vs->sums[threadIdx.x];
  const volatile double* cur = fire_state + ((it0 + (pending ? 1 : 0)) & 1) * 4;
  FireScalars f{cur[0], cur[1], (long long)cur[2]};
  extern __shared__ __align__(16) unsigned char s_stage[];
  Stage<BLOCK / L> g(s_stage);
  const int4 tile = a.tiles[blockIdx.x];
  stage_build<INTER, BLOCK, L>(p, p, a, tile, s.last_pos, s.disp_cutoff, pot_range_f<POT>(p), g);
  __syncthreads();
  double2* pos = s.pos_out;
  int done = 0;
  bool stalled = false, due = false, bad = false, conv = false;
  for (int j = 0; j < n; j++) {
    if (j > 0 || !pending) {
      const double P = s_sums[S_VF], vv = s_sums[S_VV], ff = s_sums[S_FF];
      const bool rollback = fire_next(fp, P, f);
      bool moved = false;
      for (int v = tile.z + threadIdx.x; v < tile.w; v += BLOCK) {
        double2 x = pos[v], vel = s.vel[v];
        fire_move(f, rollback, P, vv, ff, s.force[v], x, vel);
        pos[v] = x;
        s.vel[v] = vel;
        moved |= moved_beyond(pbc2(p, x, s.last_pos[v]), s.disp_cutoff);
      }
      if (moved) st->rebuild = 1;
      const int b = steps_barrier(bar, __syncthreads_or(moved) != 0);
      if (b != 0) {
        stalled = b < 0;
        due = b > 0;
        break;
      }
    }
    tile_body<POT, INTER, MODE_STEP, BLOCK, L, PREC_FP64, false, 3, true>(p, a, s, pos, pos, 0ull, nullptr, j > 0, &g,
                                                                          tile, 0.5 * f.dt);
    if (steps_barrier(bar) < 0) {
      stalled = true;
      break;
    }
    reduce_partials(s.partials, gridDim.x, s_sums);
    __syncthreads();
    done++;
    bad = s_sums[S_NONFINITE] != 0.0;
    conv = s.fire_tol >= 0.0 && s_sums[S_FMAX2] <= s.fire_tol * s.fire_tol;
    if (bad || conv) break;
  }
  if (stalled || blockIdx.x != 0 || threadIdx.x != 0) return;
  // the scalars of the iteration under way (pending) or of the last one
  double* nxt = fire_state + ((it0 + done + (due ? 1 : 0)) & 1) * 4;
  nxt[0] = f.dt;
  nxt[1] = f.alpha;
  nxt[2] = (double)f.nstep;
  if (done > 0)
    for (int q = 0; q < NSUM; q++) st->sums[q] = s_sums[q];
  if (bad) {
    st->nonfinite = 1;
    st->abort = 1;
  }
  if (conv) st->converged = 1;
  st->fire_iters = it0 + done;
  st->ops_done += 2 * done;
  st->steps_left = left - done;
  st->bpending = due ? 1 : 0;
  bar.leave();
}

namespace {

size_t fire_smem(int inter, int lanes) { return stage_smem(inter, lanes == 1 ? 128 : 96); }

template <int POT, int INTER>
FireStepsFn fn_lanes(int lanes) {
  if (lanes == 1) return k_fire_steps<POT, INTER, 128, 1>;
  if (lanes == 2) return k_fire_steps<POT, INTER, 192, 2>;
  return nullptr;
}

template <int INTER>
FireStepsFn fn_pot(int pot, int lanes) {
  switch (pot) {
    case POT_HARMONIC: return fn_lanes<POT_HARMONIC, INTER>(lanes);
    case POT_LJ: return fn_lanes<POT_LJ, INTER>(lanes);
    case POT_ADHESIVE: return fn_lanes<POT_ADHESIVE, INTER>(lanes);
    default: return fn_lanes<POT_WCA, INTER>(lanes);
  }
}

}  // namespace

FireStepsFn fire_steps_fn(int pot, int inter, int lanes) {
  return inter == INT_VV ? fn_pot<INT_VV>(pot, lanes) : fn_pot<INT_SMOOTH>(pot, lanes);
}

int fire_steps_max_blocks(FireStepsFn fn, int inter, int lanes) {
  return resident_ctas(fn, lanes == 1 ? 128 : 192, fire_smem(inter, lanes));
}

cudaError_t launch_fire_steps(FireStepsFn fn, int inter, const LaunchCfg& c, const SysParams& p_in, const SysArrays& a,
                              const StepArgs& s, const FireParams& fp, double* fire_state) {
  const SysParams p = with_f32_constants(p_in);
  return launch_k(c.pdl, fn, dim3(c.grid), dim3(c.lanes == 1 ? 128 : 192), c.stream, fire_smem(inter, c.lanes), p, a, s, fp,
                  fire_state);
}

}  // namespace cr
