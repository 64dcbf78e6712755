// Rigid rings (DPM2D::calcRigidForceEnergy, RigidNVE, RigidLangevin).
//
// One CTA per tile of whole rings, as in k_tile:
//   1. centroid of each ring from offsets to its first vertex (calcParticlePos,
//      include/cudaKernel.cuh:365-388) by a per-ring tree in shared memory;
//   2. vertex-vertex pair forces, own side only (kernelCalcVertexForceTorque,
//      :1412-1450), L lanes per vertex;
//   3. per-vertex torque about the centroid and the ring sums: force, torque /
//      moment of inertia, moment of inertia, energy
//      (kernelCalcTorqueAndMomentOfInertia / kernelCalcParticleRigidForceEnergy,
//      :1452-1492);
//   4. MODE_STEP: the ring's velocity and angular velocity complete the step
//      (RigidNVE::updateVelocity, src/Simulator.cu:348-369) and, for advancing
//      ops, take the next half kick, move the centroid and the angle
//      (updatePosition, :329-346) and every vertex is translated and rotated
//      about the new centroid (kernelTranslateVertices / kernelRotateVertices,
//      include/cudaKernel.cuh:1678-1713) into the other position buffer.
// Ring mass is 1 and the torque term is the angular acceleration, as in the
// reference.  The Langevin form here is a correct one (friction and noise
// noise*xi - gamma*v on the ring velocity with noise = sqrt(2 T gamma / dt));
// the reference's RigidLangevin adds unscaled N(0,1) draws to the velocity.
#include "cr_launch.h"
#include "cr_tile.cuh"

namespace cr {

// PREC_MIXED: the vertex pair terms in FP32 on FP64-formed offsets (as the
// deformable kernel's mixed path), accumulated per vertex in FP32; torques,
// ring sums and integration stay FP64.
//
// A step is a chain of short phases, bound by latency: the ring sums take one
// warp per ring (a tree over shared memory took a CTA barrier per level, twice
// seven of them), the rings' random numbers are drawn before the pair phase,
// the rotation's sine and cosine once per ring, and no sums over the system
// are formed (nothing reads them).  100 steps with 4 or 5 rebuilds, one graph
// captured for them: 98,304 vertices, WCA, FP64, 4.10 -> 2.82 ms; 36,024
// vertices, FP32 pairs, 2.41 -> 1.97 ms (with calls as plain launches, 2.63 and
// 1.58 ms).
template <int POT, int MODE, int BLOCK, int L, int PREC>
__global__ void __launch_bounds__(BLOCK) k_rigid(const __grid_constant__ SysParams p,
                                                 const __grid_constant__ SysArrays a,
                                                 const __grid_constant__ StepArgs s,
                                                 const __grid_constant__ RigidArgs r) {
  constexpr int TV = BLOCK / L, W = BLOCK / 32;
  __shared__ double2 s_pos[TV];
  __shared__ double s_ux[TV], s_uy[TV];   // offsets from the ring's first vertex -> centroid
  __shared__ double2 s_f[TV];             // pair force
  __shared__ double s_e[TV];
  __shared__ double s_rx[TV], s_ry[TV], s_rt[TV], s_rm[TV], s_re[TV];  // ring sums (at the first vertex)
  __shared__ int s_first[TV], s_len[TV];  // per ring of the tile: first vertex, vertices
  __shared__ double2 s_c[TV], s_shift[TV], s_rot[TV], s_noise[TV];  // per ring: centroid, translation, rotation, draws
  __shared__ double s_draw[TV];

  pdl_wait();
  pdl_trigger();
  DevStatus* st = s.status;
  if (MODE == MODE_STEP && (st->abort | st->converged)) {
    if (is_last_block(st)) {
      if (threadIdx.x == 0) {
        st->done_ctr = 0;
        if (s.use_cond) cudaGraphSetConditional(s.cond, 0u);
      }
    }
    return;
  }
  const int4 tile = a.tiles[blockIdx.x];
  const int v0 = tile.z, nvt = tile.w - tile.z;
  const int ring0 = tile.x, nrings = tile.y - tile.x;
  const int t = threadIdx.x, w = t / 32;
  const int lv = t / L, lane = t % L;
  const unsigned long long step = MODE == MODE_STEP ? (unsigned long long)st->rng_step : 0ull;
  int q0 = 0, lf = 0, k = 0, nvr = 1;  // ring in the tile, its first vertex
  if (t < nvt) {
    const int2 tp = __ldg(a.vtopo + v0 + t);
    q0 = tp.x - ring0;
    k = tp.y & 0xffff;
    nvr = tp.y >> 16;
    lf = t - k;
    s_pos[t] = __ldg(a.pos + v0 + t);
    if (k == 0) {
      s_first[q0] = t;
      s_len[q0] = nvr;
    }
  }
  // list counts and first slots, in flight across the centroid phase
  int cnt = 0, j1 = 0, j2 = 0;
  double ri = 0.0;
  if (lv < nvt) {
    cnt = min(__ldg(a.nbr_cnt + v0 + lv), a.nbr_cap);
    ri = __ldg(a.rad + v0 + lv);
    if (lane < cnt) j1 = __ldg(a.nbr + (size_t)lane * p.nv + v0 + lv);
    if (lane + L < cnt) j2 = __ldg(a.nbr + (size_t)(lane + L) * p.nv + v0 + lv);
  }
  if (MODE == MODE_STEP && BLOCK - 1 - t < nrings) {
    // the rings' random numbers, by the last threads (with two or more lanes
    // these have no vertex in the phases before the pairs)
    const int q = BLOCK - 1 - t;
    const unsigned long long ring = (unsigned long long)(ring0 + q);
    if (s.kind == KIND_LANGEVIN) s_noise[q] = philox_normal2(s.seed, 2ull * step, ring);
    if (s.active) s_draw[q] = philox_normal2(s.seed, 2ull * step + 1ull, ring).x;
  }
  __syncthreads();
  if (t < nvt) {
    const double2 u = pbc2(p, s_pos[t], s_pos[lf]);
    s_ux[t] = u.x;
    s_uy[t] = u.y;
  }
  __syncthreads();
  for (int q = w; q < nrings; q += W) {
    double* const arr[2] = {s_ux, s_uy};
    const int f = s_first[q], n = s_len[q];
    ring_sums<2>(arr, f, n);
    if ((t & 31) == 0) s_c[q] = make_double2(s_pos[f].x + s_ux[f] / n, s_pos[f].y + s_uy[f] / n);
  }

  // pair forces: the next slot's neighbour is fetched before this one's term
  {
    using T = typename std::conditional<PREC == PREC_MIXED, float, double>::type;
    typename Vec2<T>::type fi{0, 0};
    double ei = 0.0;
    if (lv < nvt) {
      const double2 xi = s_pos[lv];
      double2 nx = make_double2(0.0, 0.0);
      double nr = 0.0;
      if (lane < cnt) {
        nx = __ldg(a.pos + j1);
        nr = __ldg(a.rad + j1);
      }
      for (int sl = lane; sl < cnt; sl += L) {
        const double2 xj = nx;
        const double rj = nr;
        if (sl + L < cnt) {
          nx = __ldg(a.pos + j2);
          nr = __ldg(a.rad + j2);
          if (sl + 2 * L < cnt) j2 = __ldg(a.nbr + (size_t)(sl + 2 * L) * p.nv + v0 + lv);
        }
        if constexpr (PREC == PREC_MIXED) pair_own_f<POT>(p, f2(pbc2(p, xi, xj)), (float)(ri + rj), fi, ei);
        else pair_own<POT>(p, pbc2(p, xi, xj), ri + rj, fi, ei);
      }
    }
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) {
      fi.x += __shfl_xor_sync(0xffffffffu, fi.x, o);
      fi.y += __shfl_xor_sync(0xffffffffu, fi.y, o);
      ei += __shfl_xor_sync(0xffffffffu, ei, o);
    }
    if (lane == 0 && lv < nvt) {
      s_f[lv] = make_double2(fi.x, fi.y);
      s_e[lv] = ei;
    }
  }
  __syncthreads();

  // torque about the centroid and ring sums
  double2 F = make_double2(0.0, 0.0);
  double tau = 0.0;
  if (t < nvt) {
    F = s_f[t];
    const double2 rel = pbc2(p, s_pos[t], s_c[q0]);
    tau = rel.x * F.y - rel.y * F.x;
    s_rx[t] = F.x;
    s_ry[t] = F.y;
    s_rt[t] = tau;
    s_rm[t] = rel.x * rel.x + rel.y * rel.y;
    s_re[t] = s_e[t];
  }
  __syncthreads();
  for (int q = w; q < nrings; q += W) {
    double* const arr[5] = {s_rx, s_ry, s_rt, s_rm, s_re};
    ring_sums<5>(arr, s_first[q], s_len[q]);
  }
  __syncthreads();

  if constexpr (MODE == MODE_FORCE) {
    if (t < nvt) {
      const int v = v0 + t, ring = ring0 + q0;
      s.force[v] = F;
      s.energy[v] = s_e[t];
      r.v_torque[v] = tau;
      if (k == 0) {
        s.ppos_out[ring] = s_c[q0];
        r.p_force[ring] = make_double2(s_rx[t], s_ry[t]);
        r.p_torque[ring] = s_rt[t] / s_rm[t];
        r.p_moi[ring] = s_rm[t];
        s.p_energy[ring] = s_re[t];
      }
    }
    return;
  } else {
    int nonfinite = 0;
    if (t < nrings) {
      // ring t of the tile
      const int ring = ring0 + t, f = s_first[t];
      double2 Fp = make_double2(s_rx[f], s_ry[f]);
      const double alpha = s_rt[f] / s_rm[f];
      if (s.active) {
        // self-propulsion of the ring along its own diffusing angle
        double psi = r.sp_angle[ring];
        psi += s.sp_amp * s_draw[t];
        psi = psi + kPi;
        psi = psi - 2.0 * kPi * floor(psi / (2.0 * kPi));
        psi = psi - kPi;
        r.sp_angle[ring] = psi;
        double sn, cs;
        sincos(psi, &sn, &cs);
        Fp.x += s.driving * cs;
        Fp.y += s.driving * sn;
      }
      const double2 vh = r.p_vel[ring];
      const double wh = r.p_angvel[ring];
      if (s.kind == KIND_LANGEVIN) {
        const double2 z = s_noise[t];
        Fp.x += s.noise * z.x - s.gamma * vh.x;
        Fp.y += s.noise * z.y - s.gamma * vh.y;
      }
      const double2 vn = make_double2(vh.x + s.hdt * Fp.x, vh.y + s.hdt * Fp.y);
      const double wn = wh + s.hdt * alpha;
      if (s.advance) {
        const double2 v2 = make_double2(vn.x + s.hdt * Fp.x, vn.y + s.hdt * Fp.y);
        const double w2 = wn + s.hdt * alpha;
        r.p_vel[ring] = v2;
        r.p_angvel[ring] = w2;
        r.p_angle[ring] += s.dt * w2;
        s_shift[t] = make_double2(s.dt * v2.x, s.dt * v2.y);
        double sn, cs;
        sincos(s.dt * w2, &sn, &cs);
        s_rot[t] = make_double2(cs, sn);
      } else {
        r.p_vel[ring] = vn;
        r.p_angvel[ring] = wn;
        r.p_force[ring] = Fp;
        r.p_torque[ring] = alpha;
        r.p_moi[ring] = s_rm[f];
        s.p_energy[ring] = s_re[f];
        s.ppos_out[ring] = s_c[t];
      }
      nonfinite = !(isfinite(Fp.x) && isfinite(Fp.y) && isfinite(alpha));
    }
    const bool bad = __syncthreads_or(nonfinite) != 0;
    if (t < nvt) {
      const int v = v0 + t;
      if (s.advance) {
        // kernelTranslateVertices then kernelRotateVertices about the new centroid
        const double2 sh = s_shift[q0], rot = s_rot[q0];
        const double2 cn = make_double2(s_c[q0].x + sh.x, s_c[q0].y + sh.y);
        double2 x = make_double2(s_pos[t].x + sh.x, s_pos[t].y + sh.y);
        const double2 d = pbc2(p, x, cn);
        x.x += (d.x * rot.x - d.y * rot.y) - d.x;
        x.y += (d.x * rot.y + d.y * rot.x) - d.y;
        s.pos_out[v] = x;
        if (3.0 * dist_of(pbc2(p, x, s.last_pos[v])) > s.disp_cutoff) st->rebuild = 1;
      } else {
        s.force[v] = F;
        s.energy[v] = s_e[t];
        r.v_torque[v] = tau;
      }
    }
    if (bad && t == 0) {
      st->nonfinite = 1;
      st->abort = 1;
    }
    if (is_last_block(st)) {
      if (t == 0) {
        __threadfence();
        st->ops_done += 1;
        st->rng_step += 1;
        st->done_ctr = 0;
        if (s.use_cond) cudaGraphSetConditional(s.cond, st->rebuild ? 1u : 0u);
      }
    }
  }
}

// First half kick + move that opens a rigid NVE / Langevin sequence, from the
// stored ring forces (RigidNVE::integrate up to the force call).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_rigid_drift(const __grid_constant__ SysParams p,
                                                       const __grid_constant__ SysArrays a,
                                                       const __grid_constant__ StepArgs s,
                                                       const __grid_constant__ RigidArgs r) {
  __shared__ double2 s_shift[BLOCK];
  __shared__ double2 s_cn[BLOCK];
  __shared__ double s_dang[BLOCK];
  DevStatus* st = s.status;
  if (st->abort | st->converged) {
    if (is_last_block(st)) {
      if (threadIdx.x == 0) {
        st->done_ctr = 0;
        if (s.use_cond) cudaGraphSetConditional(s.cond, 0u);
      }
    }
    return;
  }
  const int4 tile = a.tiles[blockIdx.x];
  const int v0 = tile.z, nvt = tile.w - tile.z;
  const int t = threadIdx.x;
  int ring = -1, lf = 0;
  if (t < nvt) {
    ring = a.ring_of[v0 + t];
    lf = a.ring_first[ring] - v0;
    if (t == lf) {
      const double2 Fp = r.p_force[ring];
      const double alpha = r.p_torque[ring];
      const double2 v2 = make_double2(r.p_vel[ring].x + s.hdt * Fp.x, r.p_vel[ring].y + s.hdt * Fp.y);
      const double w2 = r.p_angvel[ring] + s.hdt * alpha;
      const double2 c = s.ppos_out[ring];
      r.p_vel[ring] = v2;
      r.p_angvel[ring] = w2;
      r.p_angle[ring] += s.dt * w2;
      s_shift[t] = make_double2(s.dt * v2.x, s.dt * v2.y);
      s_cn[t] = make_double2(c.x + s.dt * v2.x, c.y + s.dt * v2.y);
      s_dang[t] = s.dt * w2;
    }
  }
  __syncthreads();
  if (t < nvt) {
    const int v = v0 + t;
    const double2 sh = s_shift[lf];
    const double2 cn = s_cn[lf];
    double2 x = a.pos[v];
    x.x += sh.x;
    x.y += sh.y;
    const double2 d = pbc2(p, x, cn);
    double sn, cs;
    sincos(s_dang[lf], &sn, &cs);
    x.x += (d.x * cs - d.y * sn) - d.x;
    x.y += (d.x * sn + d.y * cs) - d.y;
    s.pos_out[v] = x;
    if (3.0 * dist_of(pbc2(p, x, s.last_pos[v])) > s.disp_cutoff) st->rebuild = 1;
  }
  if (is_last_block(st)) {
    if (t == 0) {
      __threadfence();
      st->ops_done += 1;
      st->done_ctr = 0;
      if (s.use_cond) cudaGraphSetConditional(s.cond, st->rebuild ? 1u : 0u);
    }
  }
}

// Ring velocities N(0, sqrt(T)) with the mean removed
// (RigidLangevin::injectKineticEnergy + kernelConserveParticleMomentum,
// src/Simulator.cu:255-262, over all rings).
__global__ void k_rigid_inject(int np, double2* p_vel, double amp, unsigned long long seed, unsigned long long stream) {
  __shared__ double2 s_sum[256];
  double2 acc = make_double2(0.0, 0.0);
  for (int q = threadIdx.x; q < np; q += blockDim.x) {
    const double2 z = philox_normal2(seed, stream, (unsigned long long)q);
    acc.x += amp * z.x;
    acc.y += amp * z.y;
  }
  s_sum[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      s_sum[threadIdx.x].x += s_sum[threadIdx.x + o].x;
      s_sum[threadIdx.x].y += s_sum[threadIdx.x + o].y;
    }
    __syncthreads();
  }
  const double2 mean = make_double2(s_sum[0].x / np, s_sum[0].y / np);
  for (int q = threadIdx.x; q < np; q += blockDim.x) {
    const double2 z = philox_normal2(seed, stream, (unsigned long long)q);
    p_vel[q] = make_double2(amp * z.x - mean.x, amp * z.y - mean.y);
  }
}

template <int POT, int MODE, int PREC>
static void launch_rigid_p(const LaunchCfg& c, const SysParams& p, const SysArrays& a, const StepArgs& s,
                           const RigidArgs& r) {
  if (c.lanes == 1) launch_k(c.pdl, k_rigid<POT, MODE, 128, 1, PREC>, dim3(c.grid), dim3(128), c.stream, 0, p, a, s, r);
  else if (c.lanes == 4) launch_k(c.pdl, k_rigid<POT, MODE, 256, 4, PREC>, dim3(c.grid), dim3(256), c.stream, 0, p, a, s, r);
  else if (c.lanes == 8) launch_k(c.pdl, k_rigid<POT, MODE, 256, 8, PREC>, dim3(c.grid), dim3(256), c.stream, 0, p, a, s, r);
  else launch_k(c.pdl, k_rigid<POT, MODE, 192, 2, PREC>, dim3(c.grid), dim3(192), c.stream, 0, p, a, s, r);  // tiles of up to 96 vertices
}

template <int POT, int MODE>
static void launch_rigid_t(const LaunchCfg& c, const SysParams& p, const SysArrays& a, const StepArgs& s,
                           const RigidArgs& r) {
  if (c.precision == CR_PRECISION_MIXED) launch_rigid_p<POT, MODE, PREC_MIXED>(c, p, a, s, r);
  else launch_rigid_p<POT, MODE, PREC_FP64>(c, p, a, s, r);
}

void launch_rigid(const LaunchCfg& c, int pot, int mode, const SysParams& p_in, const SysArrays& a,
                  const StepArgs& s, const RigidArgs& r) {
  const SysParams p = with_f32_constants(p_in);  // the FP32 pair terms read them
#define CR_RIGID_CASE(P)                                              \
  case P:                                                             \
    if (mode == MODE_FORCE) launch_rigid_t<P, MODE_FORCE>(c, p, a, s, r); \
    else launch_rigid_t<P, MODE_STEP>(c, p, a, s, r);                 \
    break;
  switch (pot) {
    CR_RIGID_CASE(POT_HARMONIC)
    CR_RIGID_CASE(POT_LJ)
    CR_RIGID_CASE(POT_ADHESIVE)
    CR_RIGID_CASE(POT_WCA)
    default: break;
  }
#undef CR_RIGID_CASE
}

void launch_rigid_drift(const LaunchCfg& c, const SysParams& p, const SysArrays& a, const StepArgs& s,
                        const RigidArgs& r) {
  // every tile holds at most 128 vertices (tile_vertices)
  k_rigid_drift<128><<<c.grid, 128, 0, c.stream>>>(p, a, s, r);
}

void launch_rigid_inject(cudaStream_t st, int np, double2* p_vel, double amp, unsigned long long seed,
                         unsigned long long stream) {
  k_rigid_inject<<<1, 256, 0, st>>>(np, p_vel, amp, seed, stream);
}

}  // namespace cr
