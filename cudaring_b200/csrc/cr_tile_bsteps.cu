// Persistent batched FIRE: up to nmax FIRE iterations of every system of a
// batch in one launch, a grid barrier after each half of an iteration in
// place of a kernel boundary.  Each CTA owns one tile (the host launches the
// kernel only when occupancy x SMs holds the grid):
//   pre-kick of the tile's vertices (bfire_prekick: the system's FIRE
//   scalars from its sums, velocity mixing, first half kick, position
//   update, displacement check)
//   -- grid barrier --
//   a system's displacement check fired: leave with the force op pending;
//   the batched list build runs and the next launch starts with that op
//   force op of the tile (the tiled kernel's FIRE op: forces, second half
//   kick, per-system sums reduced by the system's last tile, convergence)
//   -- grid barrier --
// The arithmetic is that of one launch per op (k_bfire_pre, then the tiled
// kernel), so both give the same iterates.  FP64, tile shapes (1, 128) and
// (2, 192); other configurations keep one launch per op.  Every barrier wait
// is bounded (status.spin_limit): a CTA that gives up sets stalled and
// abort, and the host reruns the chunk one launch per op.
#include "cr_bfire.cuh"
#include "cr_launch.h"
#include "cr_tile_kernel.cuh"

namespace cr {

template <int POT, int INTER, int BLOCK, int L, bool STAGED>
__global__ void __launch_bounds__(BLOCK, tile_threads_per_sm<PREC_FP64, L>() / BLOCK)
    k_bfire_steps(const __grid_constant__ SysParams p, const __grid_constant__ SysArrays a,
                  const __grid_constant__ StepArgs s, const __grid_constant__ BFire f, int nmax) {
  DevStatus* st = s.status;
  const volatile DevStatus* vs = st;
  __shared__ int s_stop;
  if (vs->abort) return;
  const int pending = vs->bpending;  // the last launch left with its force op due
  const int4 tile = a.tiles[blockIdx.x];
  StepsBarrier bar(st);
  bool stalled = false;
  int rebuild = 0;
  extern __shared__ __align__(16) unsigned char s_stage[];
  Stage<BLOCK / L> g(s_stage);
  const int n = nmax > 0 ? nmax : pending;
  if (STAGED && n > 0) {
    const BatchSys& bs = s.bsys[tile.x];
    stage_build<INTER, BLOCK, L>(p, bs.box, a, tile, s.last_pos, bs.disp_cutoff, pot_range_f<POT>(p), g);
  }
  for (int j = 0; j < n; j++) {
    if (!(j == 0 && pending)) {
      for (int v = tile.z + threadIdx.x; v < tile.w; v += BLOCK) bfire_prekick(f, v);
      if (steps_barrier(bar) < 0) {
        stalled = true;
        break;
      }
      if (threadIdx.x == 0) s_stop = (vs->rebuild ? 1 : 0) | (vs->abort ? 2 : 0);
      __syncthreads();
      const int stop = s_stop;
      __syncthreads();
      if (stop) {
        rebuild = stop & 1;
        break;
      }
    }
    tile_body<POT, INTER, MODE_STEP, BLOCK, L, PREC_FP64, true, 2, STAGED>(p, a, s, a.pos, s.pos_out, 0ull, nullptr, j > 0, &g,
                                                                           tile);
    if (steps_barrier(bar) < 0) {
      stalled = true;
      break;
    }
    if (threadIdx.x == 0) s_stop = vs->abort ? 1 : 0;
    __syncthreads();
    const int stop = s_stop;
    __syncthreads();
    if (stop) break;
  }
  if (stalled) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->bpending = rebuild;
    bar.leave();
  }
}

namespace {

// Without the stage only for smooth pairs, whose staged form leaves two CTAs an
// SM (296 tiles); the vertex-vertex kernels hold as many with it (592 with one
// lane, 444 with two).  us per iteration (calls of 200, list build included),
// unstaged against one launch per op: one lane, 592 tiles 26.7 / 35.0; two
// lanes, 444 tiles 25.7 / 33.5; staged, 296 tiles: 23.0 / 32.6 and 22.5 / 32.7.
template <int POT, int INTER, bool STAGED>
BFireStepsFn fn_shape(int lanes, int block) {
  if (lanes == 1 && block == 128) return k_bfire_steps<POT, INTER, 128, 1, STAGED>;
  if (lanes == 2 && block == 192) return k_bfire_steps<POT, INTER, 192, 2, STAGED>;
  return nullptr;
}

template <int POT>
BFireStepsFn fn_pot(int inter, int lanes, int block, bool staged) {
  if (inter == INT_VV) return staged ? fn_shape<POT, INT_VV, true>(lanes, block) : nullptr;
  return staged ? fn_shape<POT, INT_SMOOTH, true>(lanes, block) : fn_shape<POT, INT_SMOOTH, false>(lanes, block);
}

}  // namespace

BFireKernel bfire_kernel(int pot, int inter, int lanes, int block, bool staged) {
  BFireKernel k;
  switch (pot) {
    case POT_HARMONIC: k.fn = fn_pot<POT_HARMONIC>(inter, lanes, block, staged); break;
    case POT_LJ: k.fn = fn_pot<POT_LJ>(inter, lanes, block, staged); break;
    case POT_ADHESIVE: k.fn = fn_pot<POT_ADHESIVE>(inter, lanes, block, staged); break;
    default: k.fn = fn_pot<POT_WCA>(inter, lanes, block, staged); break;
  }
  k.block = block;
  k.smem = staged ? stage_smem(inter, block == 128 ? 128 : 96) : 0;
  return k;
}

int bfire_max_blocks(const BFireKernel& k) { return resident_ctas(k.fn, k.block, k.smem); }

void launch_bfire_steps(const BFireKernel& k, const LaunchCfg& c, const SysParams& p, const SysArrays& a,
                        const StepArgs& s, const BFire& f, int nmax) {
  k.fn<<<c.grid, k.block, k.smem, c.stream>>>(p, a, s, f, nmax);
}

}  // namespace cr
