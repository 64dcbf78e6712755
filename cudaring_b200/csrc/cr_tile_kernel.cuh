// Tiled force + integrator kernel body (see cr_tile.cuh for the phase
// structure), shared by the FP64 instantiations (cr_tile.cu) and the
// mixed-precision ones (cr_tile_mixed.cu).
//
// Latency layout.  A step of this workload is one wave of CTAs with a few
// warps per SM, so the time of a launch is the dependent-latency chain of one
// thread, not a throughput limit.  The kernel therefore keeps that chain
// short:
//   * every per-vertex input is fetched in the prologue, in parallel: the ring
//     topology from the packed vtopo word (no ring_of -> ring_first chain),
//     rest lengths / angles into shared memory (neighbours read them there),
//     and, for a step, velocity and last-build position by cp.async straight
//     into shared memory (no registers held across the pair phase);
//   * the neighbour gather reads each listed neighbour's ring predecessors
//     from the companion list (nbr_pq), so the neighbour's position and both
//     predecessor positions are loaded together, and the next slot's list
//     entries are fetched before the current slot is evaluated;
//   * per-CTA partial sums are formed only when an op needs them (FIRE); the
//     non-finite check otherwise is one __syncthreads_or.
#pragma once
#include <type_traits>

#include "cr_bar.h"
#include "cr_tile.cuh"

namespace cr {


// Occupancy target in threads per SM, smooth interaction.  One lane per vertex:
// 512 leaves 128 registers per thread.  Two lanes per vertex (192-thread CTAs,
// tiles of up to 96 vertices): 576 threads (three CTAs, 96 registers), so that
// the grid of a 39,424-vertex system (about 430 tiles) runs as one wave.  The
// FP64 body spills 44 to 148 bytes in one op per launch and 120 to 360 with the
// staged queue of the multi-step kernels.  The mixed path takes the same
// budgets: it holds an FP64 unit body for its near-contact slots beside the
// FP32 one, and at 80 registers (four CTAs) its spills cost more than the fourth
// CTA gains (27.5 against 25.5 us per step measured at 39,424 vertices).
template <int PREC, int L = 1>
constexpr int tile_threads_per_sm() {
  return L >= 2 ? 576 : 512;
}
// One op per launch with vertex-vertex pairs: 768 threads (80 registers) hold
// four CTAs of 192, three of 256 or six of 128.  Left to itself the compiler
// takes 82 to 88 and an SM holds one CTA less (four lanes, us per step: 1,500
// rings of 24 vertices 16.8 -> 13.0, 4,096 rings 34.3 -> 26.3).
template <int INTER, int BLOCK, int PREC, int L>
constexpr int tile_ctas_per_sm() {
  return (INTER == INT_VV ? 768 : tile_threads_per_sm<PREC, L>()) / BLOCK;
}

template <typename T2> __device__ __forceinline__ T2 cvt2(double2 d);
template <> __device__ __forceinline__ double2 cvt2<double2>(double2 d) { return d; }
template <> __device__ __forceinline__ float2 cvt2<float2>(double2 d) { return f2(d); }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Box of the current tile: the system's parameters, or one system of a batch.
template <bool BATCH> struct BoxSel;
template <> struct BoxSel<false> {
  __device__ static const SysParams& get(const SysParams& p, const Box&) { return p; }
};
template <> struct BoxSel<true> {
  __device__ static const Box& get(const SysParams&, const Box& b) { return b; }
};

// Every CTA ends in the last-block protocol so that the op counter sees each
// op exactly once.
__device__ __forceinline__ void tile_skip(const StepArgs& s, DevStatus* st) {
  if (is_last_block(st)) {
    if (threadIdx.x == 0) {
      st->done_ctr = 0;
      if (s.use_cond) cudaGraphSetConditional(s.cond, st->rebuild ? 1u : 0u);
    }
  }
}

// BATCH: the grid covers the tiles of many independent systems; tile.x is
// the system, whose box, displacement cutoff, FIRE scalars and flags come
// from s.bsys, and whose last tile reduces the system's partial sums.
// Positions: the read-only path for a single-step launch; plain loads in the
// multi-step kernel, where other CTAs rewrite them between steps (the grid
// barrier's acquire makes their writes visible to plain loads, not to the
// non-coherent read-only path).
template <bool PERSIST>
__device__ __forceinline__ double2 ld_pos(const double2* p) {
  if constexpr (PERSIST) return *p;
  else return __ldg(p);
}

// ---------------------------------------------------------------------------
// Marking pass: which slots can add anything.
//
// A unit (vertex t against the segment q -> o, qq before q; tq = t - q, seg =
// o - q, pseg = q - qq) contributes only through its segment term (foot of
// the perpendicular inside the segment, a = tq . seg in [0, |seg|^2), its
// distance within range), its convex-corner term (a < 0 and tq . pseg >= 0,
// |tq| within range) or its concave-corner correction (inside the segment's
// span with |tq| within range, so within the first test).  One slot in six
// does on the smooth Lennard-Jones run, and the pass runs over all of them.
//
// Coordinates are taken as 32-bit fractions of the box: a difference of two
// is then the minimum image by itself (the integers wrap as the box does),
// and one conversion makes it a float.  Forming the differences in FP64 cost
// eight roundings and ten conversions a slot, which run at a quarter of the
// FP64 rate (16 a clock and SM, measured): that was two thirds of the pair
// phase of the multi-step kernel (12,100 of 32,400 cycles a step).
//
// The test errs towards marking.  A difference carries an error of one unit
// of the fraction, d = L 2^-32, and one float rounding; with s = |tq| + |seg|
// that moves a by up to 2 d s and the squared distance by up to 8 d s, and
// 2 d s <= 5e-4 s^2 or (s < 4000 d) <= 8000 d^2, 8 d s <= 1e-4 s^2 / 2 or
// below 1e6 d^2: the margins are 1e-3 (|tq|^2 + |seg|^2) + 1e4 d^2 on a and
// on tq . pseg, and 1% of the squared range + 1e-4 (|tq|^2 + |seg|^2) + 1e6
// d^2 on the squared distance.  Marked without a test: a segment above a
// fifth of the box or a range above 0.44 of it (beyond those a difference
// may wrap to either image), and a coordinate half a million boxes out or
// not finite.
// ---------------------------------------------------------------------------
struct MarkBox {
  double fx, fy;      // 2^32 / L
  float sx, sy;       // L 2^-32
  float ea, er;       // 1e4 d^2, 1e6 d^2
  float seg2, rng2;   // (0.2 L)^2, (0.44 L)^2 of the shorter side
  template <class B>
  __device__ __forceinline__ explicit MarkBox(const B& b) {
    fx = 4294967296.0 * b.inv_lx;
    fy = 4294967296.0 * b.inv_ly;
    sx = (float)(b.lx * 0x1p-32);
    sy = (float)(b.ly * 0x1p-32);
    const float d = fmaxf(sx, sy), l = fminf(sx, sy) * 4294967296.0f;
    ea = 1e4f * d * d;
    er = 1e6f * d * d;
    seg2 = 0.04f * l * l;
    rng2 = 0.19f * l * l;
  }
};

// x as a fraction of the box, modulo 1, in units of 2^-32: the low word of
// x 2^32 / L rounded to an integer by adding 1.5 * 2^52.  far gets bits when
// that sum leaves [2^52, 2^53).
__device__ __forceinline__ unsigned box_frac(double x, double f, unsigned& far) {
  const double y = __fma_rn(x, f, 6755399441055744.0);
  far |= ((unsigned)__double2hiint(y) ^ 0x43300000u) >> 20;
  return (unsigned)__double2loint(y);
}
__device__ __forceinline__ uint2 box_frac2(const MarkBox& m, double2 x, unsigned& far) {
  return make_uint2(box_frac(x.x, m.fx, far), box_frac(x.y, m.fy, far));
}
__device__ __forceinline__ float2 frac_diff(const MarkBox& m, uint2 a, uint2 b) {
  return make_float2((float)(int)(a.x - b.x) * m.sx, (float)(int)(a.y - b.y) * m.sy);
}

// h > 0: the mark also holds while no vertex moves more than h / 2.  Every
// difference then changes by at most h, so a by h (|tq| + |seg|) + h^2, tq .
// pseg likewise, |seg|^2 by 2 h |seg| + h^2 and the distance of t from the
// segment by h.  H: whether h may be above zero.
template <bool H>
__device__ __forceinline__ bool unit_may_contribute(const MarkBox& m, float2 tq, float2 seg, float2 pseg, float Rm2,
                                                    float h) {
  const float t2 = fmaf(tq.y, tq.y, tq.x * tq.x);
  const float l2 = fmaf(seg.y, seg.y, seg.x * seg.x);
  const float pl2 = fmaf(pseg.y, pseg.y, pseg.x * pseg.x);
  const float a = fmaf(tq.y, seg.y, tq.x * seg.x);
  const float b = fmaf(tq.y, pseg.y, tq.x * pseg.x);
  float ma = fmaf(1e-3f, t2 + l2, m.ea), mb = fmaf(1e-3f, t2 + pl2, m.ea), ml = ma;
  if constexpr (H) {
    const float sl = sqrtf(2.0f * (t2 + l2)), sp = sqrtf(2.0f * (t2 + pl2));
    ma = fmaf(h, sl + h, ma);
    mb = fmaf(h, sp + h, mb);
    ml = fmaf(2.0f * h, sl + h, ma);
  }
  const float slack = fmaf(1e-4f, t2 + l2, Rm2 + m.er);
  const bool on = a >= -ma && a < l2 + ml && !(t2 * l2 - a * a >= slack * l2);
  const bool before = a < ma && t2 < slack && b >= -mb;
  return on || before || fmaxf(l2, pl2) > m.seg2;
}

// Whether either smooth unit of a slot (vertex i against neighbour j) may
// contribute; seg_i = x_i - x_q, pseg_i = x_q - x_qq of vertex i, R = range *
// radSum.
template <bool H>
__device__ __forceinline__ bool slot_may_contribute(const MarkBox& m, uint2 ui, uint2 uq, float2 seg_i, float2 pseg_i,
                                                    uint2 uj, uint2 ujq, uint2 ujqq, float R, float h = 0.0f) {
  const float Rh = H ? R + h : R;
  const float Rm2 = 1.01f * Rh * Rh;
  return unit_may_contribute<H>(m, frac_diff(m, ui, ujq), frac_diff(m, uj, ujq), frac_diff(m, ujq, ujqq), Rm2, h) ||
         unit_may_contribute<H>(m, frac_diff(m, uj, uq), seg_i, pseg_i, Rm2, h) || Rm2 > m.rng2;
}

// ---------------------------------------------------------------------------
// Staged neighbourhood of the multi-step kernels.
//
// Between two rebuilds a tile reads the same neighbours every step: a vertex
// of the 39,424-vertex smooth Lennard-Jones run lists 9.3 vertices and reads
// three positions for each (its own and two ring predecessors'), 2,700
// gathers of 16 bytes per tile and step, each behind a list entry that comes
// from L2 too (the grid barrier's acquire empties L1).  Those positions are
// only a few hundred different ones.  So at the start of a launch each CTA
// marks the vertices its lists touch (a hash set of their rings, a bit mask
// of each ring's vertices), gives them local indices behind its own vertices
// and rewrites its list to these, one word per slot; every step then copies
// the touched positions into shared memory once and the pair phase reads
// shared memory alone.  The values read are the same, so no result changes.
// A tile that touches more rings, vertices or list entries than the stage
// holds reads global memory as before, and so does every tile of a grid that
// the GPU holds at once only without the stage's 31 to 34 KB a CTA (STAGED
// false: one lane per vertex, 445 to 592 tiles with smooth pairs, 593 to 740
// with vertex-vertex pairs).
//   Measured, with the queue of marked slots and the fixed-point marking below
// (39,424 vertices, smooth Lennard-Jones, FP64, us per step): 17.3 -> 12.1
// without rebuilds, 18.6 -> 13.9 with one in 20 steps; 9,495 vertices, smooth
// adhesive: 10.3 -> 7.5.
// ---------------------------------------------------------------------------
constexpr int kStageRings = 128;    // hash slots
constexpr int kStageHalo = 512;     // touched vertices of other tiles (own and touched: below 1024)
constexpr int kStageEntries = 1536; // list entries of the tile
template <int TV, int INTER>
constexpr size_t stage_bytes() {
  return (size_t)(TV + kStageHalo) * (sizeof(double2) + sizeof(double) + sizeof(uint2)) +
         (size_t)(kStageEntries + kStageHalo + 2 * TV + 4) * sizeof(int) +
         kStageEntries * (INTER == INT_SMOOTH ? 3 : 1);  // vertex-vertex pairs have no queue
}

inline size_t stage_smem(int inter, int tile_vertices) {
  if (inter == INT_VV) return tile_vertices == 128 ? stage_bytes<128, INT_VV>() : stage_bytes<96, INT_VV>();
  return tile_vertices == 128 ? stage_bytes<128, INT_SMOOTH>() : stage_bytes<96, INT_SMOOTH>();
}

// CTAs of a kernel with grid barriers that the current device holds at once (0
// without one); also allows the kernel that much dynamic shared memory.
template <typename Fn>
inline int resident_ctas(Fn* fn, int block, size_t smem) {
  int dev = 0, sms = 0, occ = 0;
  if (!fn || cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, block, smem) != cudaSuccess) return 0;
  return occ * sms;
}

// The list entries are in the order of the threads that collect them (own
// vertex lv, lane of it: thread lv L + lane, its slots lane, lane + L, ..), so
// each thread has one run.
template <int TV>
struct Stage {
  double2* x;    // [TV + kStageHalo] positions: own vertices, then the touched ones
  double* rad;   // [TV + kStageHalo]
  uint2* u;      // [TV + kStageHalo] positions as fractions of the box (box_frac)
  unsigned* list;  // [kStageEntries] local indices of a neighbour and its two predecessors, 10 bits each
  int* vtx;      // [kStageHalo] global vertex of each touched one
  int* start;    // [TV L + 1] first list entry of each thread
  unsigned char* owner;  // [kStageEntries] thread of each list entry
  unsigned short* place; // [kStageEntries] smooth: place of each marked entry in the queue
  int n;         // touched vertices
  int entries;   // list entries
  bool on;       // the tile's neighbourhood fits
  __device__ __forceinline__ explicit Stage(unsigned char* smem) {
    x = reinterpret_cast<double2*>(smem);
    rad = reinterpret_cast<double*>(x + TV + kStageHalo);
    u = reinterpret_cast<uint2*>(rad + TV + kStageHalo);
    list = reinterpret_cast<unsigned*>(u + TV + kStageHalo);
    vtx = reinterpret_cast<int*>(list + kStageEntries);
    start = vtx + kStageHalo;
    owner = reinterpret_cast<unsigned char*>(start + 2 * TV + 4);
    place = reinterpret_cast<unsigned short*>(owner + kStageEntries);
    n = entries = 0;
    on = false;
  }
};

// Exclusive prefix of one value per thread over the CTA; *total: the sum.
// Every thread calls it; s: BLOCK / 32 words of shared memory.
template <int BLOCK>
__device__ __forceinline__ int cta_prefix(int x, int* s, int* total) {
  const int wl = threadIdx.x & 31, w = threadIdx.x / 32;
  int incl = x;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (wl >= o) incl += y;
  }
  __syncthreads();
  if (wl == 31) s[w] = incl;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int q = 0; q < BLOCK / 32; q++) {
    const int y = s[q];
    before += q < w ? y : 0;
    all += y;
  }
  *total = all;
  return before + incl - x;
}

// Fills the stage (every thread of the CTA calls it) from the tile's lists.
// The entries are dealt to the threads evenly, four at a time, so that the
// loads of a thread (list words, then the neighbours' topology) are in flight
// together.
//
// Smooth lists are then thinned: a slot is dropped when it cannot add anything
// while every vertex stays within cutoff / 3 of its last-build position, which
// holds for every force evaluation of the launch (the first position beyond
// that ends it).  last: those positions; cutoff: DPM2D::cutoff.
template <int INTER, int BLOCK, int L, class B>
__device__ __forceinline__ void stage_build(const SysParams& p, const B& bx, const SysArrays& a, const int4& tile,
                                            const double2* last, double cutoff, float range, Stage<BLOCK / L>& g) {
  constexpr int TV = BLOCK / L;
  static_assert(TV <= 128 && TV + kStageHalo <= 1024, "7-bit ring positions, 10-bit local indices");
  static_assert(L <= 2 && BLOCK <= 256, "start holds 2 TV threads, owner is a byte");
  __shared__ int s_key[kStageRings], s_first[kStageRings];
  __shared__ unsigned s_mask[kStageRings * 4];  // touched vertices of each ring, 32 per word
  __shared__ int s_base[kStageRings * 4];       // local index of each word's first
  __shared__ int s_part[BLOCK / 32], s_bad;
  // touched flags, a byte per ring position, in the space of the positions:
  // plain stores merge where a warp's entries touch the same vertex, which
  // atomic ORs on the mask words would serialise
  unsigned char* flag = reinterpret_cast<unsigned char*>(g.x);
  static_assert(kStageRings * 128 <= (TV + kStageHalo) * (int)(sizeof(double2) + sizeof(double) + sizeof(uint2)),
                "flags fit");
  const int t = threadIdx.x, lv = t / L, lane = t % L;
  const int v0 = tile.z, nvt = tile.w - tile.z;
  for (int h = t; h < kStageRings; h += BLOCK) s_key[h] = -1;
  for (int q = t; q < kStageRings * 8; q += BLOCK) reinterpret_cast<int4*>(flag)[q] = make_int4(0, 0, 0, 0);
  if (t == 0) s_bad = 0;
  // each thread's run of the list
  const int cnt = lv < nvt ? min(__ldg(a.nbr_cnt + v0 + lv), a.nbr_cap) : 0;
  const int mine = cnt > lane ? (cnt - lane + L - 1) / L : 0;
  int total;
  const int run0 = cta_prefix<BLOCK>(mine, s_part, &total);
  if (total > kStageEntries) {
    g.on = false;
    g.n = g.entries = 0;
    __syncthreads();
    return;
  }
  g.start[t] = run0;
  if (t == 0) g.start[BLOCK] = total;
  for (int e = run0; e < run0 + mine; e++) g.owner[e] = (unsigned char)t;
  __syncthreads();
  // list words for now: hash slot and the three positions in the ring (7 bits
  // each), or bit 31 and the three indices in the tile
  for (int e0 = t; e0 < total; e0 += 4 * BLOCK) {
    int j[4], pk[4];
    int2 tp[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int e = e0 + q * BLOCK;
      j[q] = v0;
      pk[q] = 0;
      if (e < total) {
        const int o = g.owner[e];
        const size_t at = (size_t)(o % L + (e - g.start[o]) * L) * p.nv + v0 + o / L;
        j[q] = __ldg(a.nbr + at);
        if constexpr (INTER == INT_SMOOTH) pk[q] = __ldg(a.nbr_pq + at);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) tp[q] = __ldg(a.vtopo + j[q]);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int e = e0 + q * BLOCK;
      if (e >= total) break;
      if (j[q] >= v0 && j[q] < tile.w) {
        const unsigned k = j[q] - v0;
        g.list[e] = 1u << 31 | (k + pq_second(pk[q])) << 14 | (k + pq_first(pk[q])) << 7 | k;
        continue;
      }
      const unsigned k = tp[q].y & 0xffff, k1 = k + pq_first(pk[q]), k2 = k + pq_second(pk[q]);
      int h = (int)(((unsigned)tp[q].x * 2654435761u) >> 25), tries = 0;
      for (; tries < kStageRings; tries++, h = (h + 1) & (kStageRings - 1)) {
        int old = *(volatile int*)&s_key[h];
        if (old == -1) old = atomicCAS(&s_key[h], -1, tp[q].x);
        if (old == -1 || old == tp[q].x) break;
      }
      if (tries == kStageRings || (tp[q].y >> 16) > 128) {
        s_bad = 1;
        continue;
      }
      s_first[h] = j[q] - (int)k;
      flag[128 * h + k] = 1;
      if constexpr (INTER == INT_SMOOTH) {
        flag[128 * h + k1] = 1;
        flag[128 * h + k2] = 1;
      }
      g.list[e] = (unsigned)h << 21 | k2 << 14 | k1 << 7 | k;
    }
  }
  __syncthreads();
  // local indices of the touched vertices, ring after ring in hash order: each
  // thread takes the mask words of a few neighbouring hash slots
  constexpr int per = (kStageRings * 4 + BLOCK - 1) / BLOCK;
  int touched = 0;
#pragma unroll
  for (int u = 0; u < per; u++) {
    const int q = t * per + u;
    unsigned m = 0;
    if (q < kStageRings * 4) {
      if (s_key[q / 4] >= 0)
        for (int b = 0; b < 8; b++) {
          const unsigned f = reinterpret_cast<const unsigned*>(flag)[8 * q + b];  // four flags
          m |= ((f & 1u) | (f >> 7 & 2u) | (f >> 14 & 4u) | (f >> 21 & 8u)) << (4 * b);
        }
      s_mask[q] = m;
    }
    touched += __popc(m);
  }
  int n;
  int at = cta_prefix<BLOCK>(touched, s_part, &n);
  const bool fits = s_bad == 0 && n <= kStageHalo;
  if (fits) {
#pragma unroll
    for (int u = 0; u < per; u++) {
      const int q = t * per + u;
      if (q < kStageRings * 4) {
        s_base[q] = TV + at;
        for (unsigned m = s_mask[q]; m; m &= m - 1u) g.vtx[at++] = s_first[q / 4] + q % 4 * 32 + __ffs((int)m) - 1;
      }
    }
  }
  g.on = fits;
  g.n = fits ? n : 0;
  g.entries = fits ? total : 0;
  __syncthreads();
  if (!fits) return;
  if (t < nvt) g.rad[t] = __ldg(a.rad + v0 + t);
  for (int q = t; q < n; q += BLOCK) g.rad[TV + q] = __ldg(a.rad + g.vtx[q]);
  const MarkBox mb(bx);
  unsigned far = 0;
  if constexpr (INTER == INT_SMOOTH) {
    if (t < nvt) {
      const int2 tp = __ldg(a.vtopo + v0 + t);
      const int k = tp.y & 0xffff, nvr = tp.y >> 16;
      s_first[t] = t - k + (k == 0 ? nvr - 1 : k - 1);  // the own vertices' predecessors, from here on
      g.u[t] = box_frac2(mb, last[v0 + t], far);
    }
    for (int q = t; q < n; q += BLOCK) g.u[TV + q] = box_frac2(mb, last[g.vtx[q]], far);
  }
  const bool all = __syncthreads_or(far) != 0;
  const auto local = [&](unsigned h4, unsigned k) {
    const unsigned w = h4 + (k >> 5);
    return (unsigned)(s_base[w] + __popc(s_mask[w] & ((1u << (k & 31)) - 1u)));
  };
  // final list words; smooth: the thread takes its own run, so that the kept
  // entries move up in order
  const float h = fmaxf(0.0f, (float)cutoff * (2.0f / 3.0f) * 1.001f + 8.0f * fmaxf(mb.sx, mb.sy));
  unsigned* scratch = reinterpret_cast<unsigned*>(g.x);
  static_assert(kStageEntries * sizeof(unsigned) <= (TV + kStageHalo) * sizeof(double2), "scratch list fits");
  float2 seg_i = make_float2(0.0f, 0.0f), pseg_i = seg_i;
  uint2 ui = make_uint2(0u, 0u), uq = ui;
  float ri = 0.0f;
  if (INTER == INT_SMOOTH && mine > 0) {
    const int lq = s_first[lv];
    ui = g.u[lv];
    uq = g.u[lq];
    seg_i = frac_diff(mb, ui, uq);
    pseg_i = frac_diff(mb, uq, g.u[s_first[lq]]);
    ri = (float)g.rad[lv];
  }
  int kept = 0;
  for (int q = 0; q < mine; q++) {
    const unsigned e = g.list[run0 + q];
    unsigned k = e & 127u, k1 = (e >> 7) & 127u, k2 = (e >> 14) & 127u;
    if (!(e >> 31)) {
      const unsigned h4 = (e >> 21) * 4;
      k = local(h4, k);
      if constexpr (INTER == INT_SMOOTH) {
        k1 = local(h4, k1);
        k2 = local(h4, k2);
      }
    }
    bool stays = true;
    if constexpr (INTER == INT_SMOOTH)
      stays = all || slot_may_contribute<true>(mb, ui, uq, seg_i, pseg_i, g.u[k], g.u[k1], g.u[k2],
                                               range * (ri + (float)g.rad[k]), h);
    if (stays) scratch[run0 + kept++] = k2 << 20 | k1 << 10 | k;
  }
  int left;
  const int run1 = cta_prefix<BLOCK>(kept, s_part, &left);
  for (int q = 0; q < kept; q++) {
    g.list[run1 + q] = scratch[run0 + q];
    g.owner[run1 + q] = (unsigned char)t;
  }
  g.start[t] = run1;
  if (t == 0) g.start[BLOCK] = left;
  g.entries = left;
  __syncthreads();
}

// A list slot: a neighbour and its two ring predecessors, as indices into the
// positions the pair phase reads.
struct Slot {
  int j, q, qq;
};

// The pair phase's view of the tile's lists and of the positions it reads:
// global memory (plain loads where other CTAs rewrite the positions between
// steps), or the stage.  Two types rather than one with generic pointers, so
// that the staged loads are shared-memory loads with 32-bit addresses.
template <bool PERSIST>
struct GlobalSrc {
  const double2* x;
  const double* rad;
  const int* nbr;       // list of the tile's first vertex, slot stride `stride`
  const int* pq;
  size_t stride;
  int own0;             // the tile's first vertex
  __device__ __forceinline__ Slot entry(int lv, int slot) const {
    const size_t at = (size_t)slot * stride + lv;
    const int j = __ldg(nbr + at), pk = pq ? __ldg(pq + at) : 0;
    return Slot{j, j + pq_first(pk), j + pq_second(pk)};
  }
  __device__ __forceinline__ double2 pos(int i) const { return ld_pos<PERSIST>(x + i); }
  __device__ __forceinline__ double radius(int i) const { return __ldg(rad + i); }
};
template <int TV>
struct StageSrc {
  const Stage<TV>& g;
  static constexpr int own0 = 0;
  __device__ __forceinline__ Slot entry(int lv, int slot) const {
    const unsigned e = g.list[slot];  // slot: the list entry
    return Slot{(int)(e & 1023u), (int)((e >> 10) & 1023u), (int)(e >> 20)};
  }
  __device__ __forceinline__ double2 pos(int i) const { return g.x[i]; }
  __device__ __forceinline__ double radius(int i) const { return g.rad[i]; }
};

// ---------------------------------------------------------------------------
// Mixed-precision smooth units.
//
// Near contact the FP32 evaluation of a steep potential cannot meet a 1e-6
// force error: one rounding of the distance or of (radSum/d)^6 moves a unit
// force by ~1e-6 of the net force, which is a small residual of pair and
// shape forces several times larger.  So each list slot (vertex i against
// neighbour j: role 1, i against the segment prev(j) -> j; role 2, j against
// i's segment prev(i) -> i) first takes a near test in FP32: whether a live
// unit's vertex lies within f_near * radSum of its segment.  Far slots are
// evaluated in FP32 (every term of such a unit is at least that far away);
// near slots exactly as the FP64 path evaluates them (same differences, same
// arithmetic, FP64 accumulators).
// ---------------------------------------------------------------------------

// Whether t lies within Rn of the segment q -> o (tq = t - q, w = t - o,
// seg = o - q, len2 = |seg|^2, squared lengths precomputed), without a
// division: an end point within Rn, or the foot of the perpendicular on the
// segment and |tq x seg|^2 < Rn^2 |seg|^2.
__device__ __forceinline__ bool seg_near(float2 tq, float tq2, float w2, float2 seg, float len2, float Rn2) {
  if (tq2 < Rn2 || w2 < Rn2) return true;
  const float dot = tq.x * seg.x + tq.y * seg.y;
  const float cr = tq.x * seg.y - tq.y * seg.x;
  return dot > 0.0f && dot < len2 && cr * cr < Rn2 * len2;
}

// FP32 body of one slot; returns true (and evaluates nothing) when the slot
// is near and belongs to the FP64 pass.  The slot's FP32 sums enter the FP64
// accumulators.  seg_i64 = x_i - x_q (q = prev(i)).
template <int POT, class B>
__device__ __forceinline__ bool mixed_slot_f32(const SysParams& p, const B& bx, double2 xi, double2 seg_i64,
                                               float2 seg_i, float2 pseg_i, float len2_i, float len_i, double ri,
                                               double rj, double2 xj, double2 xjq, double2 xjqq, double2& fi64,
                                               double2& fq64, double& ei) {
  const double rsum64 = ri + rj;
  const float rsum = (float)rsum64;
  const float R = pot_range_f<POT>(p) * rsum;
  const double2 w64 = pbc2(bx, xi, xj);    // x_i - x_j
  const double2 tq64 = pbc2(bx, xi, xjq);  // x_i - x_jq
  const float2 w1 = f2(w64), tq1 = f2(tq64);
  // x_j - x_jq as the difference of the two offsets from x_i: the same image
  // of ring j unless x_j and x_jq have their nearest images on different
  // sides (a box under about twice the interaction range); then directly
  double2 seg1_64 = make_double2(tq64.x - w64.x, tq64.y - w64.y);
  if (fabs(seg1_64.x) > 0.25 * bx.lx || fabs(seg1_64.y) > 0.25 * bx.ly) seg1_64 = pbc2(bx, xj, xjq);
  const float2 seg1 = f2(seg1_64);
  const float2 tq2 = f2(make_double2(seg_i64.x - w64.x, seg_i64.y - w64.y));  // x_j - x_q
  const float w2 = fmaf(w1.y, w1.y, w1.x * w1.x);
  const float tq1_2 = fmaf(tq1.y, tq1.y, tq1.x * tq1.x);
  const float len1 = fmaf(seg1.y, seg1.y, seg1.x * seg1.x);
  const float tq2_2 = fmaf(tq2.y, tq2.y, tq2.x * tq2.x);
  const bool in1 = !smooth_out_of_range(R, tq1_2, w2, sqrtf(len1));
  const bool in2 = !smooth_out_of_range(R, tq2_2, w2, len_i);
  if (!(in1 | in2)) return false;
  const float Rn = p.f_near * rsum, Rn2 = Rn * Rn;
  if ((in1 && seg_near(tq1, tq1_2, w2, seg1, len1, Rn2)) || (in2 && seg_near(tq2, tq2_2, w2, seg_i, len2_i, Rn2)))
    return true;
  const float inv_rsum = 1.0f / rsum;
  float2 fs{0.0f, 0.0f}, fqs{0.0f, 0.0f}, dummy{0.0f, 0.0f};
  if (in1) {
    const float2 pseg1 = f2(pbc2(bx, xjq, xjqq));  // x_jq - x_jqq
    smooth_core<POT, true, float>(p, bx, tq1, tq1_2, w1, seg1, rsq(len1), pseg1, rsum, inv_rsum, xi, xjq, fs, dummy,
                                  dummy, ei);
  }
  if (in2) {
    const float2 mw1{-w1.x, -w1.y};  // x_j - x_i
    smooth_core<POT, false, float>(p, bx, tq2, tq2_2, mw1, seg_i, rsq(len2_i), pseg_i, rsum, inv_rsum, xj, xj, dummy,
                                   fs, fqs, ei);  // (box coordinates are read by the FP64 body only)
  }
  fi64.x += (double)fs.x;
  fi64.y += (double)fs.y;
  fq64.x += (double)fqs.x;
  fq64.y += (double)fqs.y;
  return false;
}

// FP64 body of one slot, shared by the FP64 path and the mixed path's
// near-contact slots: the reference's own differences of box coordinates
// (pbcDistance of each pair of vertices); a unit out of range adds nothing.
// seg_i = x_i - x_q, pseg_i = x_q - x_qq: vertex i's segments (q = prev(i)),
// inv_len_i = 1 / |seg_i|.
template <int POT, class B>
__device__ __forceinline__ void smooth_slot_f64(const SysParams& p, const B& bx, double2 xi, double2 xq,
                                                double2 seg_i, double2 pseg_i, double inv_len_i, double ri, double rj,
                                                double2 xj, double2 xjq, double2 xjqq, double2& fi, double2& fq,
                                                double& ei) {
  const double rsum = ri + rj;
  const double inv_rsum = 1.0 / rsum;
  const double2 w1 = pbc2(bx, xi, xj);        // x_i - x_j
  const double2 tq1 = pbc2(bx, xi, xjq);      // x_i - x_jq
  const double2 seg1 = pbc2(bx, xj, xjq);     // x_j - x_jq
  const double2 pseg1 = pbc2(bx, xjq, xjqq);  // x_jq - x_jqq
  const double2 tq2 = pbc2(bx, xj, xq);       // x_j - x_q
  const double2 mw1{-w1.x, -w1.y};            // x_j - x_i
  const double tq1_2 = fma(tq1.y, tq1.y, tq1.x * tq1.x);
  const double len1 = fma(seg1.y, seg1.y, seg1.x * seg1.x);
  const double tq2_2 = fma(tq2.y, tq2.y, tq2.x * tq2.x);
  double2 dummy{0.0, 0.0};
  smooth_core<POT, true, double>(p, bx, tq1, tq1_2, w1, seg1, rsq(len1), pseg1, rsum, inv_rsum, xi, xjq, fi, dummy,
                                 dummy, ei);
  smooth_core<POT, false, double>(p, bx, tq2, tq2_2, mw1, seg_i, inv_len_i, pseg_i, rsum, inv_rsum, xj, xq, dummy, fi,
                                  fq, ei);
}

// DPM2D::checkDisplacement's test 3 |d| > cut (include/cudaKernel.cuh and
// src/DPM2D.cu:1397-1405).  The squares decide outside a relative band of
// 1e-9, far above their rounding, so that few vertices take the square root.
__device__ __forceinline__ bool moved_beyond(double2 d, double cut) {
  const double q = 9.0 * fma(d.y, d.y, d.x * d.x), c = cut * cut;
  if (cut > 0.0 && q < c * (1.0 - 1e-9)) return false;
  return 3.0 * dist_of(d) > cut;
}

// The warp's marked slots: in FP64, or (mixed precision) in FP32 unless the
// slot is near, then in FP64.  The lanes of a warp hold uneven numbers of
// slots (0.8 on average for the smooth Lennard-Jones run, 3 to 4 for the
// warp's longest lane), and a lane-by-lane loop issues the evaluation as often
// as the longest lane needs it.  So the marked slots of the whole warp (or of
// the CTA, where its lists are staged) go into one queue, every thread
// evaluates one entry per round, and every lane then adds up the results of
// its own slots (those with slot % L = its lane) in slot order: the sums do
// not depend on how the queue was filled or dealt.
// An entry is own vertex << 24 | slot (staged: | list entry); evaluating it
// sets kNear where a mixed slot was near.
constexpr int kNear = 1 << 23;
template <int QN>
struct UnitQueue {
  int* q;        // [QN] this warp's entries
  double2* fi;   // [QN] their results: force on i, force on prev(i), energy
  double2* fq;
  double* e;
};

// W: threads that share the queue, the warp's or the CTA's.
template <int POT, int QN, int PREC, bool EN, int W, class B, class SRC>
__device__ __forceinline__ void queue_eval(const SysParams& p, const B& bx, const SRC& src,
                                           const double2* s_pos, const double2* s_seg, const double* s_il,
                                           const int* s_lp, const UnitQueue<QN>& u, int n) {
  for (int e = threadIdx.x % W; e < n; e += W) {
    const int w = u.q[e], i = (unsigned)w >> 24, lq = s_lp[i];
    const Slot en = src.entry(i, w & 0xffffff);
    const double2 seg_i = s_seg[lq], pseg_i = s_seg[s_lp[lq]], xi = s_pos[i];
    const double2 xj = src.pos(en.j), xjq = src.pos(en.q), xjqq = src.pos(en.qq);
    const double ri = src.radius(src.own0 + i), rj = src.radius(en.j);
    double2 f1{0.0, 0.0}, f2_{0.0, 0.0};
    double en_ = 0.0;
    bool wide = true;
    if constexpr (PREC == PREC_MIXED) {
      const float2 sf = f2(seg_i);
      const float len2 = fmaf(sf.y, sf.y, sf.x * sf.x);
      wide = mixed_slot_f32<POT>(p, bx, xi, seg_i, sf, f2(pseg_i), len2, sqrtf(len2), ri, rj, xj, xjq, xjqq, f1, f2_,
                                 en_);
      if (wide) u.q[e] = w | kNear;
    }
    if (wide)
      smooth_slot_f64<POT>(p, bx, xi, s_pos[lq], seg_i, pseg_i, s_il[lq], ri, rj, xj, xjq, xjqq, f1, f2_, en_);
    u.fi[e] = f1;
    u.fq[e] = f2_;
    if constexpr (EN) u.e[e] = en_;
  }
}

// Mixed precision: a vertex's far slots (pass 0) are added before its near
// ones (pass 1).
template <int QN, int PREC, bool EN>
__device__ __forceinline__ void queue_add(const UnitQueue<QN>& u, int k, int pass, double2& fi, double2& fq,
                                          double& ei) {
  if (PREC == PREC_MIXED && ((u.q[k] & kNear) != 0) != (pass != 0)) return;
  const double2 f1 = u.fi[k], f2_ = u.fq[k];
  fi.x += f1.x;
  fi.y += f1.y;
  fq.x += f2_.x;
  fq.y += f2_.y;
  if constexpr (EN) ei += u.e[k];
}

// Lists in global memory: each lane has marked its own slots (bit b of need:
// slot base + b L).  The queue is filled lane after lane, in parts of QN.
// Every lane of the warp calls it.
template <int POT, int L, int QN, int PREC, bool EN, class B, class SRC>
__device__ __forceinline__ void queue_lanes(const SysParams& p, const B& bx, const SRC& src,
                                            const double2* s_pos, const double2* s_seg, const double* s_il,
                                            const int* s_lp, const UnitQueue<QN>& u, unsigned long long need, int lv, int base,
                                            double2& fi, double2& fq, double& ei) {
  constexpr unsigned kAll = 0xffffffffu;
  const int wl = threadIdx.x & 31;
  const int n = __popcll(need);
  if (!__any_sync(kAll, n != 0)) return;
  int incl = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kAll, incl, o);
    if (wl >= o) incl += y;
  }
  const int total = __shfl_sync(kAll, incl, 31);
  const int first = incl - n;
  for (int q0 = 0; q0 < total; q0 += QN) {
    const int lo = max(first, q0), hi = min(incl, q0 + QN);  // this lane's entries in this part
    unsigned long long m = need;
    for (int k = first; k < hi; k++, m &= m - 1ull)
      if (k >= lo) u.q[k - q0] = (int)((unsigned)lv << 24 | (unsigned)(base + (__ffsll((long long)m) - 1) * L));
    __syncwarp();
    queue_eval<POT, QN, PREC, EN, 32>(p, bx, src, s_pos, s_seg, s_il, s_lp, u, min(QN, total - q0));
    __syncwarp();
    for (int pass = 0; pass < (PREC == PREC_MIXED ? 2 : 1); pass++)
      for (int k = lo; k < hi; k++) queue_add<QN, PREC, EN>(u, k - q0, pass, fi, fq, ei);
    __syncwarp();
  }
}

// What the marking pass reads of an own vertex, one record in shared memory.
struct __align__(16) OwnUnit {
  uint2 ui, uq;        // x_i and x_q as fractions of the box
  float2 seg, pseg;    // x_i - x_q, x_q - x_qq
  float rad;
  float pad[3];
};

// Staged lists: the tile's entries follow one another, so marking, evaluation
// and the queue are the CTA's.  Rounds of 32 entries are handed to the warps
// as they come free (those without a vertex start while the others still form
// the angles and shape forces); a round appends its marked entries to the
// queue, in whatever order the rounds end, and leaves its marks as one ballot
// word and each marked entry's place in the queue, by which the vertices
// collect their results in slot order.
template <int POT, int L, int TV>
__device__ __forceinline__ void mark_rounds(const SysParams& p, const MarkBox& mb, const Stage<TV>& g,
                                            const OwnUnit* own, bool far, int* round, int* queued, int cap,
                                            unsigned* bal, int* q) {
  constexpr unsigned kAll = 0xffffffffu;
  const int wl = threadIdx.x & 31;
  const int total = g.entries;
  const float range = pot_range_f<POT>(p);
  for (;;) {
    int r = 0;
    if (wl == 0) r = atomicAdd(round, 2);
    r = __shfl_sync(kAll, r, 0);
    if (32 * r >= total) return;
    // two rounds at a time, so that the loads of one overlap the other's test
    bool mark[2];
    int v[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int e = 32 * (r + u) + wl;
      mark[u] = false;
      v[u] = 0;
      if (e < total) {
        const unsigned w = g.list[e];
        v[u] = g.owner[e] / L;
        const OwnUnit& o = own[v[u]];
        const int j = w & 1023u;
        const float R = range * (o.rad + (float)g.rad[j]);
        mark[u] = far || slot_may_contribute<false>(mb, o.ui, o.uq, o.seg, o.pseg, g.u[j], g.u[(w >> 10) & 1023u],
                                             g.u[w >> 20], R);
      }
    }
    const unsigned m0 = __ballot_sync(kAll, mark[0]), m1 = __ballot_sync(kAll, mark[1]);
    int k = 0;
    if (wl == 0) {
      bal[r] = m0;
      bal[r + 1] = m1;
      if (m0 | m1) k = atomicAdd(queued, __popc(m0) + __popc(m1));
    }
    k = __shfl_sync(kAll, k, 0);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      if (!mark[u]) continue;
      const int e = 32 * (r + u) + wl;
      const int at = k + __popc((u ? m1 : m0) & ((1u << wl) - 1u)) + (u ? __popc(m0) : 0);
      g.place[e] = (unsigned short)at;
      if (at < cap) q[at] = (int)((unsigned)v[u] << 24 | (unsigned)e);
    }
  }
}

// Barrier of the CTA's first `sync` threads with all BLOCK threads: the others
// only announce that they got here (with sync = BLOCK, __syncthreads).
template <int BLOCK>
__device__ __forceinline__ void join_first(int sync) {
  if ((int)threadIdx.x < sync) asm volatile("bar.sync 1, %0;" ::"n"(BLOCK) : "memory");
  else asm volatile("bar.arrive 1, %0;" ::"n"(BLOCK) : "memory");
}

// One step (or force evaluation) of one tile.  pin / pout: positions read
// and written; step: the integrator step index (Philox stream of the noise).
// PERSIST: 0 for one op per launch; 1 the multi-step kernel: positions
// read with plain loads (other CTAs rewrite them between steps), a non-finite
// force reported in *pflag instead of the status block, whether the loop is
// to end after this step (a rebuild is due, a force is not finite) returned,
// and the last-block protocol left to the caller; 2 the persistent batched
// FIRE kernel: plain position loads, everything else as for one op; 3 the FIRE
// kernel of one system: the CTA's partial sums are all it leaves (fire_hdt:
// half the time step).  reuse: not the kernel's first op.  STAGED: the
// persistent kernel has a stage (g).
template <int POT, int INTER, int MODE, int BLOCK, int L, int PREC, bool BATCH, int PERSIST, bool STAGED>
__device__ __forceinline__ bool tile_body(const SysParams& p, const SysArrays& a, const StepArgs& s,
                                          const double2* __restrict__ pin, double2* __restrict__ pout,
                                          unsigned long long step, int* pflag, bool reuse,
                                          const Stage<BLOCK / L>* g, const int4& tile, double fire_hdt = 0.0) {
  constexpr int TV = BLOCK / L;
  // the multi-step kernel stores no energies and no sums (its ops run with
  // write_out = accumulate = 0), so its energy terms are left out at compile time
  constexpr bool kOut = PERSIST != 1;
  constexpr int TS = (MODE == MODE_STEP) ? TV : 1;
  static_assert(!STAGED || PERSIST != 0, "one op per launch has no stage");
  constexpr bool kStagedSmooth = STAGED && INTER == INT_SMOOTH;
  __shared__ double2 s_own[STAGED ? 1 : TV];
  double2* s_pos = s_own;
  if constexpr (STAGED) s_pos = g->x;
  __shared__ double2 s_seg[TV];     // pbc(pos[next] - pos[v])
  __shared__ double s_theta[TV];
  __shared__ double s_l0[TV];       // rest length of segment v -> next(v)
  __shared__ double s_il0[TV];      // its reciprocal
  __shared__ double s_th0[TV];      // rest angle at v
  __shared__ double s_il[INTER == INT_SMOOTH ? TV : 1];  // 1 / length of segment v -> next(v)
  __shared__ double s_r0[TV];       // shoelace terms -> ring area
  __shared__ double s_r1[TV];       // segment lengths -> perimeter
  __shared__ double s_r2x[TV], s_r2y[TV];  // offsets from the first vertex -> centroid
  __shared__ double2 s_fpair[TV];   // pair force on v
  __shared__ double2 s_fprev[TV];   // smooth: force on prev(v) gathered by v
  __shared__ double s_epair[TV];
  __shared__ double2 s_fsh[TV];     // shape force on v, parked across the pair phase
  __shared__ double s_esh[TV];      // shape energy booked on v
  __shared__ int s_lp[TV];
  __shared__ int2 s_tp[TV];         // topology word (ring, k | nv << 16)
  __shared__ int s_rfirst[TV];      // first vertex of each ring of the tile
  // queue of FP64 smooth units, one part per warp (see queue_eval)
  constexpr int QN = INTER != INT_SMOOTH ? 1 : (TV > 128 ? 32 : 64);  // 32: the 48 KB of static shared memory
  __shared__ int s_q[BLOCK / 32][QN];
  __shared__ OwnUnit s_ou[kStagedSmooth ? TV : 1];
  __shared__ double2 s_qi[BLOCK / 32][QN], s_qq[BLOCK / 32][QN];
  __shared__ double s_qe[kOut ? BLOCK / 32 : 1][QN];
  __shared__ double s_a0[TV];       // rest area of the vertex's ring
  __shared__ __align__(16) double2 s_vel[TS];
  __shared__ __align__(16) double2 s_last[TS];
  __shared__ double s_red[BLOCK / 32][NSUM];
  __shared__ Box s_box;
  __shared__ bool s_syslast;
  __shared__ int s_far;             // a staged coordinate beyond box_frac's range
  __shared__ int s_round;           // marking rounds handed out
  constexpr int NR = kStagedSmooth ? kStageEntries / 32 : 1;
  __shared__ unsigned s_bal[NR + 2];  // marks of each round
  __shared__ int s_queued;          // marked entries

  DevStatus* st = s.status;
  const int v0 = tile.z, nvt = tile.w - tile.z;
  const int t = threadIdx.x;
  const int sysid = BATCH ? tile.x : 0;
  if constexpr (BATCH) {
    const BatchSys& bs = s.bsys[sysid];
    if (!bs.active || (MODE == MODE_STEP && bs.converged)) {
      if constexpr (MODE == MODE_STEP) tile_skip(s, st);
      return false;
    }
    if (t == 0) s_box = bs.box;
  }
  const auto& bx = BoxSel<BATCH>::get(p, s_box);

  // ---- prologue: every per-vertex input, in parallel ------------------------
  int ring = -1, k = 0, lf = 0, lp = 0, ln = 0, nvr = 1;
  double a0r = 1.0;
  if (t < nvt) {
    const int v = v0 + t;
    int2 tp;
    // a later op of a persistent kernel: the CTA holds the same tile, so its
    // topology, rest lengths and angles and last-build positions are still in
    // shared memory; in the multi-step kernel so are its own positions and
    // velocities (stored by the last step's tail), the FIRE kernels' pre-kick
    // has stored new ones
    if (PERSIST != 0 && reuse) {
      tp = s_tp[t];
      a0r = s_a0[t];
      if constexpr (PERSIST != 1) {
        cp_async16(&s_vel[t], s.vel + v);
        cp_async_commit();
        s_pos[t] = ld_pos<true>(pin + v);
      }
    } else {
      if constexpr (MODE == MODE_STEP) {
        cp_async16(&s_vel[t], s.vel + v);
        cp_async16(&s_last[t], s.last_pos + v);
        cp_async_commit();
      }
      tp = __ldg(a.vtopo + v);
      s_pos[t] = ld_pos<(PERSIST != 0)>(pin + v);
      const double l0v = __ldg(a.l0 + v);
      s_l0[t] = l0v;
      s_il0[t] = 1.0 / l0v;
      s_th0[t] = __ldg(a.theta0 + v);
      a0r = __ldg(a.a0 + tp.x);
      s_tp[t] = tp;
      if constexpr (PERSIST != 0) s_a0[t] = a0r;
    }
    ring = tp.x;
    k = tp.y & 0xffff;
    nvr = tp.y >> 16;
    lf = t - k;
    ln = lf + (k + 1 == nvr ? 0 : k + 1);
    lp = lf + (k == 0 ? nvr - 1 : k - 1);
    s_lp[t] = lp;
  }
  if constexpr (STAGED) {
    if (t == 0) {
      s_far = s_round = s_queued = 0;
    }
    // the staged neighbourhood, in flight until the pair phase
    if (g->on) {
      for (int q = t; q < g->n; q += BLOCK) cp_async16(&g->x[TV + q], pin + g->vtx[q]);
      cp_async_commit();
    }
  }
  __syncthreads();

  // ---- phase 1: geometry --------------------------------------------------
  if (t < nvt) {
    const double2 x = s_pos[t];
    const double2 xn = s_pos[ln];
    const double2 seg = pbc2(bx, xn, x);
    s_seg[t] = seg;
    // ahead of the barrier: the pair phase reads the predecessor's too, and no
    // barrier lies between phase 2 and the unstaged pair phase
    if constexpr (INTER == INT_SMOOTH) s_il[t] = rsqrt(fma(seg.y, seg.y, seg.x * seg.x));
    const double2 x0 = s_pos[lf];
    const double2 u = pbc2(bx, x, x0);
    const double2 un = pbc2(bx, xn, x0);
    s_r0[t] = u.x * un.y - un.x * u.y;
    if constexpr (MODE == MODE_FORCE) {
      s_r1[t] = dist_of(seg);
      s_r2x[t] = u.x;
      s_r2y[t] = u.y;
    }
    if (k == 0) s_rfirst[ring - s_tp[0].x] = t;
  }
  __syncthreads();
  const MarkBox mb(bx);
  if constexpr (kStagedSmooth) {
    // the staged positions have come: each thread converts what it copied
    cp_async_wait_all();
    unsigned far = 0;
    if (t < nvt) {
      const uint2 ui = box_frac2(mb, s_pos[t], far), uq = box_frac2(mb, s_pos[lp], far);
      g->u[t] = ui;
      s_ou[t] = OwnUnit{ui, uq, f2(s_seg[lp]), f2(s_seg[s_lp[lp]]), (float)(g->on ? g->rad[t] : 0.0), {}};
    }
    for (int q = t; q < g->n; q += BLOCK) g->u[TV + q] = box_frac2(mb, g->x[TV + q], far);
    if (far) s_far = 1;
  }
  if constexpr (kStagedSmooth) __syncthreads();
  if (t < nvt) {
    // calcAngle(nextSegment, previousSegment) (include/cudaKernel.cuh:423-427)
    const double2 ns = s_seg[t];
    const double2 ps = s_seg[lp];
    s_theta[t] = atan2(ns.x * ps.y - ns.y * ps.x, ns.x * ps.x + ns.y * ps.y);
  }
  // ring sums, one warp per ring, the last warps first: with two or more
  // lanes per vertex these have no vertex of their own in this phase.  (The
  // tree over shared memory they replace took a CTA barrier per level.)
  {
    const int nrings = s_tp[nvt - 1].x - s_tp[0].x + 1;
    for (int q = BLOCK / 32 - 1 - t / 32; q < nrings; q += BLOCK / 32) {
      const int f = s_rfirst[q], n = s_tp[f].y >> 16;
      // together: one chain of shuffles for all four (163,200 vertices in 1,632
      // tiles, us a force op: vertex-vertex 19.2 -> 18.1, smooth 35.7 -> 33.9)
      if constexpr (MODE == MODE_FORCE) ring_sums<4>({s_r0, s_r1, s_r2x, s_r2y}, f, n);
      else ring_sums<1>({s_r0}, f, n);
    }
  }
  // the angles and sums go to the vertices' own threads only; in the staged
  // kernels the warps without a vertex go on to the marking pass
  if constexpr (kStagedSmooth) join_first<BLOCK>((TV + 31) / 32 * 32);
  else __syncthreads();

  // ---- phase 2: shape force (kernelCalcShapeForceEnergy, include/cudaKernel.cuh:474-529)
  double2 fsh = make_double2(0.0, 0.0);
  double esh = 0.0;
  if (t < nvt) {
    // The reference's divisions are taken as products with a few
    // reciprocals (1/A0, 1/l0 and the segments' 1/l from one rsqrt each),
    // a rounding-level difference
    const double area = fabs(s_r0[lf]) * 0.5;
    const double inv_a0 = 1.0 / a0r;
    const double dA = area * inv_a0 - 1.0;
    const double gmA = p.ea * dA * inv_a0;
    const double2 ns = s_seg[t];
    const double2 ps = s_seg[lp];
    // nRel - pRel = pos[next] - pos[prev]
    const double2 npd = make_double2(ns.x + ps.x, ns.y + ps.y);
    fsh.x += 0.5 * gmA * (-npd.y);
    fsh.y += 0.5 * gmA * (npd.x);
    esh += (0.5 * p.ea * dA * dA) / nvr;
    const double ps2 = fma(ps.y, ps.y, ps.x * ps.x), ns2 = fma(ns.y, ns.y, ns.x * ns.x);
    double r_pl, r_nl;  // 1 / |segment|
    if constexpr (INTER == INT_SMOOTH) {
      r_pl = s_il[lp];
      r_nl = s_il[t];
    } else {
      r_pl = rsqrt(ps2);
      r_nl = rsqrt(ns2);
    }
    const double plen = ps2 * r_pl, nlen = ns2 * r_nl;
    const double tl0 = s_l0[t], pl0 = s_l0[lp];
    if (p.monomer == 0) {
      const double inv_tl0 = s_il0[t], inv_pl0 = s_il0[lp];
      const double pd = plen * inv_pl0 - 1.0;
      const double nd = nlen * inv_tl0 - 1.0;
      const double cn = nd * inv_tl0 * r_nl, cp = pd * inv_pl0 * r_pl;
      fsh.x += p.el * (cn * ns.x - cp * ps.x);
      fsh.y += p.el * (cn * ns.y - cp * ps.y);
      esh += 0.5 * p.el * pd * pd;
    } else {
      const double c = 2.0 * p.el * p.stiff * p.ext_sq;
      const double an = nlen / (p.ext_sq * tl0 * tl0 - nlen * nlen);
      const double ap = plen / (p.ext_sq * pl0 * pl0 - plen * plen);
      fsh.x += c * (an * ns.x / nlen - ap * ps.x / plen);
      fsh.y += c * (an * ns.y / nlen - ap * ps.y / plen);
      esh += p.el * p.stiff * p.ext_sq * log(1.0 - plen * plen / (p.ext_sq * pl0 * pl0));
    }
    const double prevAD = s_theta[lp] - s_th0[lp];
    const double thisAD = s_theta[t] - s_th0[t];
    const double nextAD = s_theta[ln] - s_th0[ln];
    const double pvar = (thisAD - prevAD) * (r_pl * r_pl);
    const double nvar = (thisAD - nextAD) * (r_nl * r_nl);
    fsh.x += p.eb * (pvar * ps.y + nvar * ns.y);
    fsh.y += p.eb * (pvar * (-ps.x) + nvar * (-ns.x));
    esh += 0.5 * p.eb * thisAD * thisAD;
    s_fsh[t] = fsh;
    if constexpr (kOut) s_esh[t] = esh;
  }

  // ---- phase 3: pair forces ------------------------------------------------
  // L lanes per vertex stride over its list slots; each slot's list entry
  // (neighbour id and packed predecessor offsets) is fetched two slots ahead
  // and the neighbour's three positions one slot ahead, all three together.
  if constexpr (STAGED && INTER == INT_VV) {
    cp_async_wait_all();
    __syncthreads();
  }
  {
    const int lv = t / L, lane = t % L;
    using T = typename std::conditional<PREC == PREC_MIXED, float, double>::type;
    typename Vec2<T>::type fi{0, 0}, fq{0, 0};
    double2 fi64{0.0, 0.0}, fq64{0.0, 0.0};  // FP64 accumulators of the smooth units
    double ei = 0.0;
    const GlobalSrc<(PERSIST != 0)> src{pin, a.rad, a.nbr + v0, INTER == INT_SMOOTH ? a.nbr_pq + v0 : nullptr,
                                        (size_t)p.nv, v0};
    bool staged = false;
    if constexpr (STAGED) staged = g->on;
    int cnt = 0;
    if (!staged && lv < nvt) cnt = min(__ldg(a.nbr_cnt + v0 + lv), a.nbr_cap);  // an overflowed build stores counts above capacity
    if constexpr (INTER == INT_VV) {
      // first, last, step: this thread's slots
      const auto pairs = [&](const auto& from, int sl, int end, int step) {
        if (lv >= nvt) return;
        const double2 xi = s_pos[lv];
        const double ri = from.radius(from.own0 + lv);
        int j2 = 0;
        double2 nxj = make_double2(0.0, 0.0);
        double nr = 0.0;
        if (sl < end) {
          const int j = from.entry(lv, sl).j;
          if (sl + step < end) j2 = from.entry(lv, sl + step).j;
          nxj = from.pos(j);
          nr = from.radius(j);
        }
        while (sl < end) {
          const double2 xj = nxj;
          const double rj = nr;
          sl += step;
          if (sl < end) {
            nxj = from.pos(j2);
            nr = from.radius(j2);
            if (sl + step < end) j2 = from.entry(lv, sl + step).j;
          }
          if constexpr (PREC == PREC_MIXED) pair_own_f<POT>(p, f2(pbc2(bx, xi, xj)), (float)(ri + rj), fi, ei);
          else pair_own<POT>(p, pbc2(bx, xi, xj), ri + rj, fi, ei);
        }
      };
      if constexpr (STAGED) {
        if (staged) pairs(StageSrc<TV>{*g}, g->start[t], g->start[t + 1], 1);
      }
      if (!staged) pairs(src, lane, cnt, L);
    } else {
      // Smooth units of vertex i: role 1 (i against the segment prev(j) -> j)
      // and role 2 (j against i's own segment prev(i) -> i).  The marking pass
      // over the lane's slots (64 at a time) notes in a bit mask those that
      // may contribute, and these run off a queue shared by the warp
      // (queue_lanes), in slot order for each vertex: an unmarked slot adds
      // nothing when evaluated.
      if constexpr (STAGED) {
        if (staged) {
          static_assert(L <= 2, "lanes of the staged shapes");
          constexpr int QC = BLOCK / 32 * QN;
          const UnitQueue<QC> uq{&s_q[0][0], &s_qi[0][0], &s_qq[0][0], &s_qe[0][0]};
          mark_rounds<POT, L, TV>(p, mb, *g, s_ou, s_far != 0, &s_round, &s_queued, QC, s_bal, s_q[0]);
          __syncthreads();
          const int n = s_queued;
          for (int q0 = 0; q0 == 0 || q0 < n; q0 += QC) {
            if (n > QC) {
              // more entries than the queue holds: in parts, by the entries'
              // order in the lists (the rounds end in any order), so that every
              // vertex's slots still come in slot order
              if (q0 == 0)
                for (int e = t; e < g->entries; e += BLOCK) {
                  int at = __popc(s_bal[e / 32] & ((1u << e % 32) - 1u));
                  for (int w = 0; w < e / 32; w++) at += __popc(s_bal[w]);
                  g->place[e] = (unsigned short)at;
                }
              __syncthreads();
              for (int e = t; e < g->entries; e += BLOCK) {
                const int k = g->place[e] - q0;
                if ((s_bal[e / 32] >> e % 32 & 1u) && k >= 0 && k < QC)
                  s_q[0][k] = (int)((unsigned)(g->owner[e] / L) << 24 | (unsigned)e);
              }
              __syncthreads();
            }
            queue_eval<POT, QC, PREC, kOut, BLOCK>(p, bx, StageSrc<TV>{*g}, s_pos, s_seg, s_il, s_lp, uq, min(QC, n - q0));
            __syncthreads();
            // this thread's marked entries, 32 of its run at a time
            const int run = g->start[t], len = g->start[t + 1] - run;
            for (int pass = 0; pass < (PREC == PREC_MIXED ? 2 : 1); pass++)
              for (int b = 0; b < len; b += 32) {
                const int e0 = run + b;
                unsigned m = __funnelshift_r(s_bal[e0 / 32], s_bal[e0 / 32 + 1], e0 % 32);
                if (len - b < 32) m &= (1u << (len - b)) - 1u;
                for (; m; m &= m - 1u) {
                  const int k = g->place[e0 + __ffs((int)m) - 1] - q0;
                  if (k >= 0 && k < QC) queue_add<QC, PREC, kOut>(uq, k, pass, fi64, fq64, ei);
                }
              }
          }
        }
      }
      if (!staged) {
        const int li = lv < nvt ? lv : 0;
        const int lq = s_lp[li];
        const float rif = (float)src.radius(v0 + li), range = pot_range_f<POT>(p);
        const float2 seg_i = f2(s_seg[lq]), pseg_i = f2(s_seg[s_lp[lq]]);  // x_i - x_q, x_q - x_qq
        unsigned far_i = 0;
        const UnitQueue<QN> uq{s_q[t / 32], s_qi[t / 32], s_qq[t / 32], s_qe[kOut ? t / 32 : 0]};
        const uint2 ui = box_frac2(mb, s_pos[li], far_i), uqv = box_frac2(mb, s_pos[lq], far_i);
        for (int b0 = 0; __any_sync(0xffffffffu, b0 + lane < cnt); b0 += 64 * L) {
          const int base = b0 + lane, end = min(cnt, b0 + 64 * L);
          unsigned long long need = 0ull, bit = 1ull;
          if (base < end) {
            // the next slot's positions are fetched before this one is tested
            Slot e = src.entry(lv, base), e1{0, 0, 0};
            if (base + L < end) e1 = src.entry(lv, base + L);
            double2 xj = src.pos(e.j), xjq = src.pos(e.q), xjqq = src.pos(e.qq);
            double rj = src.radius(e.j);
            for (int s0 = base; s0 < end; s0 += L, bit <<= 1) {
              double2 nxj = xj, nxjq = xjq, nxjqq = xjqq;
              double nr = rj;
              Slot e2{0, 0, 0};
              if (s0 + L < end) {
                if (s0 + 2 * L < end) e2 = src.entry(lv, s0 + 2 * L);
                nxj = src.pos(e1.j);
                nxjq = src.pos(e1.q);
                nxjqq = src.pos(e1.qq);
                nr = src.radius(e1.j);
              }
              unsigned fj = far_i;
              const uint2 uj = box_frac2(mb, xj, fj), ujq = box_frac2(mb, xjq, fj), ujqq = box_frac2(mb, xjqq, fj);
              const float R = range * (rif + (float)rj);
              if (slot_may_contribute<false>(mb, ui, uqv, seg_i, pseg_i, uj, ujq, ujqq, R) || fj) need |= bit;
              xj = nxj;
              xjq = nxjq;
              xjqq = nxjqq;
              rj = nr;
              e1 = e2;
            }
          }
          queue_lanes<POT, L, QN, PREC, kOut>(p, bx, src, s_pos, s_seg, s_il, s_lp, uq, need, lv, base, fi64, fq64,
                                              ei);
        }
      }
    }
    // reduce over the L lanes of this vertex (lanes are contiguous in a warp)
    if constexpr (INTER == INT_VV) fi64 = make_double2(0.0, 0.0);
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) {
      if constexpr (kOut) ei += __shfl_xor_sync(0xffffffffu, ei, o);
      if constexpr (INTER == INT_VV) {
        fi.x += __shfl_xor_sync(0xffffffffu, fi.x, o);
        fi.y += __shfl_xor_sync(0xffffffffu, fi.y, o);
      } else {
        fi64.x += __shfl_xor_sync(0xffffffffu, fi64.x, o);
        fi64.y += __shfl_xor_sync(0xffffffffu, fi64.y, o);
        fq64.x += __shfl_xor_sync(0xffffffffu, fq64.x, o);
        fq64.y += __shfl_xor_sync(0xffffffffu, fq64.y, o);
      }
    }
    if (lane == 0 && lv < nvt) {
      if constexpr (INTER == INT_SMOOTH) {
        s_fpair[lv] = fi64;
        s_fprev[lv] = fq64;
      } else {
        s_fpair[lv] = make_double2(fi.x, fi.y);
      }
      if constexpr (kOut) s_epair[lv] = ei;
    }
  }
  __syncthreads();

  // ---- phase 4: totals and outputs ----------------------------------------
  double2 F = make_double2(0.0, 0.0);
  double evtx = 0.0;  // per-vertex energy as the reference stores it
  double epair = 0.0;
  if (t < nvt) {
    // ring topology again rather than registers held across phase 3
    const int2 tp = s_tp[t];
    ring = tp.x;
    k = tp.y & 0xffff;
    nvr = tp.y >> 16;
    lf = t - k;
    ln = lf + (k + 1 == nvr ? 0 : k + 1);
    const double2 fp = s_fpair[t];
    const double2 fsh = s_fsh[t];
    const double esh = kOut ? s_esh[t] : 0.0;
    F.x = fsh.x + fp.x;
    F.y = fsh.y + fp.y;
    if constexpr (INTER == INT_SMOOTH) {
      const double2 fn = s_fprev[ln];
      F.x += fn.x;
      F.y += fn.y;
      evtx = esh;
    } else {
      evtx = kOut ? esh + s_epair[t] : 0.0;
    }
    epair = kOut ? s_epair[t] : 0.0;
  }

  if constexpr (MODE == MODE_FORCE) {
    if (t < nvt) {
      const int v = v0 + t;
      double2 Fo = F;
      if (s.active) {
        // DPM2D::addSelfPropulsion with the angle already advanced by the caller
        const double psi = s.p_angle[ring];
        double sn, cs;
        sincos(psi, &sn, &cs);
        Fo.x += s.driving * cs;
        Fo.y += s.driving * sn;
      }
      s.force[v] = Fo;
      s.energy[v] = evtx;
      s.theta_out[v] = s_theta[t];
      s.length_out[v] = dist_of(s_seg[t]);
      if (k == 0) {
        s.area_out[ring] = fabs(s_r0[t]) * 0.5;
        s.perim_out[ring] = s_r1[t];
        const double2 x0 = s_pos[t];
        s.ppos_out[ring] = make_double2(x0.x + s_r2x[t] / nvr, x0.y + s_r2y[t] / nvr);
      }
    }
    if constexpr (INTER == INT_SMOOTH) {
      // ring energy = sum of the unit energies gathered by its vertices
      __syncthreads();
      if (t < nvt) s_r1[t] = epair;
      __syncthreads();
      for (int q = t / 32; q <= s_tp[nvt - 1].x - s_tp[0].x; q += BLOCK / 32)
        ring_sums<1>({s_r1}, s_rfirst[q], s_tp[s_rfirst[q]].y >> 16);
      __syncthreads();
      if (t < nvt && k == 0) s.p_energy[ring] = s_r1[t];
    }
    return false;
  } else {
    // ---- MODE_STEP: integrator tail (src/Simulator.cu, src/FIRE.cu) ----------
    double sums[NSUM] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int nonfinite = 0, stop = 0;
    if (s.active) {
      // addSelfPropulsion (src/DPM2D.cu:1995-2035): the ring's angle takes a
      // N(0, sqrt(2 dt / taup)) increment and is wrapped to [-pi, pi); the
      // ring's first vertex updates it once and shares it through its s_theta
      // slot, which the step tail no longer reads
      if (t < nvt && k == 0) {
        double psi = s.p_angle[ring];
        const double2 z = philox_normal2(s.seed, 2ull * step + 1ull, (unsigned long long)ring);
        psi += s.sp_amp * z.x;
        psi = psi + kPi;
        psi = psi - 2.0 * kPi * floor(psi / (2.0 * kPi));
        psi = psi - kPi;
        s.p_angle[ring] = psi;
        s_theta[t] = psi;
      }
      __syncthreads();
      if (t < nvt) {
        double sn, cs;
        sincos(s_theta[lf], &sn, &cs);
        F.x += s.driving * cs;
        F.y += s.driving * sn;
      }
    }
    if (t < nvt) {
      const int v = v0 + t;
      cp_async_wait_all();  // this thread's own copies of vel and last_pos
      double2 vh = s_vel[t];
      const double2 xl = s_last[t];
      const double2 x = s_pos[t];
      double2 vn;
      double hdt = s.hdt;
      if (s.kind == KIND_FIRE) {
        if constexpr (BATCH) hdt = 0.5 * s.bfire_state[(sysid * 2 + ((s.bsys[sysid].fire_iters + 1) & 1)) * 4];
        else if constexpr (PERSIST == 3) hdt = fire_hdt;
        else hdt = 0.5 * s.fire_state[((st->fire_iters + 1) & 1) * 4];
      }
      const double dcut = BATCH ? s.bsys[sysid].disp_cutoff : s.disp_cutoff;
      if (s.kind == KIND_LANGEVIN) {
        // langevinAddThermostatForces (src/Simulator.cu:68-73)
        const double2 z = philox_normal2(s.seed, 2ull * step, (unsigned long long)ring);
        F.x += s.noise * z.x - s.gamma * vh.x;
        F.y += s.noise * z.y - s.gamma * vh.y;
      }
      if (s.kind == KIND_BROWNIAN || s.kind == KIND_DRIVEN_BROWNIAN) {
        // updateBrownianVel / updateDrivenBrownianVel (src/Simulator.cu:168-200)
        if (s.kind == KIND_BROWNIAN) {
          const double2 z = philox_normal2(s.seed, 2ull * step, (unsigned long long)ring);
          vn = make_double2((F.x + s.noise * z.x) / s.gamma, (F.y + s.noise * z.y) / s.gamma);
        } else {
          vn = make_double2(F.x / s.gamma, F.y / s.gamma);
        }
        const double2 xn = make_double2(x.x + s.dt * vn.x, x.y + s.dt * vn.y);
        pout[v] = xn;
        s.vel[v] = vn;
        s.force[v] = F;
        if (kOut && s.write_out) s.energy[v] = evtx;
        if (moved_beyond(pbc2(bx, xn, xl), dcut)) {
          st->rebuild = 1;
          stop = 1;
          if constexpr (BATCH) s.bsys[sysid].rebuild = 1;
        }
      } else {
        // second half kick (kernelUpdateVertexVel, include/cudaKernel.cuh:1989-1996)
        vn = make_double2(vh.x + hdt * F.x, vh.y + hdt * F.y);
        if (s.advance) {
          double2 vh2, xn;
          if (s.kind == KIND_BAOAB) {
            // BAOAB::integrate (src/Simulator.cu:112-144) for the next step
            vh2 = make_double2(vn.x + s.hdt * F.x, vn.y + s.hdt * F.y);
            xn = make_double2(x.x + s.hdt * vh2.x, x.y + s.hdt * vh2.y);
            const double2 z = philox_normal2(s.seed, 2ull * (step + 1ull), (unsigned long long)ring);
            vh2 = make_double2(s.gamma_factor * vh2.x + s.noise * z.x, s.gamma_factor * vh2.y + s.noise * z.y);
            xn = make_double2(xn.x + s.hdt * vh2.x, xn.y + s.hdt * vh2.y);
          } else {
            vh2 = make_double2(vn.x + s.hdt * F.x, vn.y + s.hdt * F.y);
            xn = make_double2(x.x + s.dt * vh2.x, x.y + s.dt * vh2.y);
          }
          pout[v] = xn;
          s.vel[v] = vh2;
          if constexpr (PERSIST == 1) {
            // kept for the next step of the multi-step kernel (this thread
            // alone reads its slots until the barrier between steps)
            s_pos[t] = xn;
            s_vel[t] = vh2;
          }
          if (moved_beyond(pbc2(bx, xn, xl), dcut)) {
            st->rebuild = 1;
            stop = 1;
            if constexpr (BATCH) s.bsys[sysid].rebuild = 1;
          }
        } else {
          s.vel[v] = vn;
          s.force[v] = F;
          if (kOut && s.write_out) s.energy[v] = evtx;
        }
      }
      if (kOut && s.accumulate) {
        // products and sums rounded as written, so every kernel built on
        // this body (one op per launch, multi-step, persistent FIRE) sums alike
        sums[S_PE] = evtx + ((INTER == INT_SMOOTH) ? epair : 0.0);
        sums[S_VV] = __fma_rn(vn.y, vn.y, __dmul_rn(vn.x, vn.x));
        sums[S_VF] = __fma_rn(vn.y, F.y, __dmul_rn(vn.x, F.x));
        sums[S_FF] = __fma_rn(F.y, F.y, __dmul_rn(F.x, F.x));
        sums[S_FMAX2] = fmax(__dmul_rn(F.x, F.x), __dmul_rn(F.y, F.y));
      }
      if (!(isfinite(F.x) && isfinite(F.y))) {
        sums[S_NONFINITE] = 1.0;
        nonfinite = 1;
      }
    }
    if (kOut && s.write_out && INTER == INT_SMOOTH) {
      __syncthreads();
      if (t < nvt) s_r1[t] = epair;
      __syncthreads();
      for (int q = t / 32; q <= s_tp[nvt - 1].x - s_tp[0].x; q += BLOCK / 32)
        ring_sums<1>({s_r1}, s_rfirst[q], s_tp[s_rfirst[q]].y >> 16);
      __syncthreads();
      if (t < nvt && k == 0) s.p_energy[ring] = s_r1[t];
    }
    if (kOut && s.accumulate) {
      // per-CTA partials in a fixed order, compensated
      block_partials<BLOCK>(sums, s_red, s.partials + (size_t)blockIdx.x * NSUM);
      if constexpr (PERSIST == 3) return false;  // the caller reduces them
    } else if constexpr (PERSIST == 1) {
      if (nonfinite) *(volatile int*)pflag = 1;
      return __syncthreads_or(nonfinite | stop) != 0;
    } else if (__syncthreads_or(nonfinite) && t == 0) {
      st->nonfinite = 1;
      st->abort = 1;
    }
    if constexpr (BATCH) {
      if (kOut && s.accumulate) {
        // the system's last tile reduces the system's partials
        BatchSys& bs = s.bsys[sysid];
        __syncthreads();
        if (t == 0) {
          __threadfence();
          const unsigned int prev = atomicAdd(&bs.done_ctr, 1u);
          s_syslast = (prev == (unsigned int)(bs.tile_end - bs.tile_begin - 1));
        }
        __syncthreads();
        if (s_syslast) {
          reduce_partials(s.partials + (size_t)bs.tile_begin * NSUM, bs.tile_end - bs.tile_begin, bs.sums);
          __syncthreads();
          if (t == 0) {
            __threadfence();
            if (bs.sums[S_NONFINITE] != 0.0) {
              st->nonfinite = 1;
              st->abort = 1;
            }
            if (s.kind == KIND_FIRE) {
              bs.fire_iters += 1;
              if (bs.fire_tol >= 0.0 && bs.sums[S_FMAX2] <= bs.fire_tol * bs.fire_tol) bs.converged = 1;
            }
            bs.done_ctr = 0;
          }
        }
      }
    }
    if (is_last_block(st)) {
      if (!BATCH && kOut && s.accumulate) reduce_partials(s.partials, gridDim.x, st->sums);
      __syncthreads();
      if (t == 0) {
        __threadfence();
        if (!BATCH && kOut && s.accumulate && st->sums[S_NONFINITE] != 0.0) {
          st->nonfinite = 1;
          st->abort = 1;
        }
        if (!BATCH && s.kind == KIND_FIRE) {
          st->fire_iters += 1;
          if (s.fire_tol >= 0.0 && st->sums[S_FMAX2] <= s.fire_tol * s.fire_tol) st->converged = 1;
        }
        st->ops_done += 1;
        if (s.kind != KIND_FIRE) st->rng_step += 1;
        st->done_ctr = 0;
        if (s.use_cond) cudaGraphSetConditional(s.cond, st->rebuild ? 1u : 0u);
      }
    }
  }
  return false;
}

template <int POT, int INTER, int MODE, int BLOCK, int L, int PREC, bool BATCH = false>
__global__ void __launch_bounds__(BLOCK, (tile_ctas_per_sm<INTER, BLOCK, PREC, L>())) k_tile(const __grid_constant__ SysParams p,
                                                const __grid_constant__ SysArrays a,
                                                const __grid_constant__ StepArgs s) {
  // every input may come from the kernel before this one (positions, lists,
  // status); the next kernel (the rebuild check) may be scheduled at once and
  // waits for this one's completion itself
  pdl_wait();
  pdl_trigger();
  DevStatus* st = s.status;
  if (MODE == MODE_STEP && ((st->abort | st->converged) || (s.after_steps && st->steps_left > 0))) {
    // keep the last-block protocol intact so later ops see a consistent counter
    if (is_last_block(st)) {
      if (threadIdx.x == 0) {
        st->done_ctr = 0;
        if (s.use_cond) cudaGraphSetConditional(s.cond, 0u);
      }
    }
    return;
  }
  const int4 tile = a.tiles[blockIdx.x];
  tile_body<POT, INTER, MODE, BLOCK, L, PREC, BATCH, 0, false>(p, a, s, a.pos, s.pos_out, (unsigned long long)st->rng_step,
                                                        nullptr, false, nullptr, tile);
}

// ---------------------------------------------------------------------------
// Multi-step kernel: up to s.persist_max middle steps of an NVE / Langevin /
// BAOAB sequence in one launch, with a grid barrier between steps in place
// of a kernel boundary.  Every tile is one resident CTA (the host launches it
// only when occupancy x SMs holds the grid).  Positions ping-pong between
// pos0 (read by step 0) and pos1; a launch that ends after an odd number of
// steps copies its tiles' positions back, so the result is always in pos0.
// The launch stops after the first step whose displacement check fired (the
// one-launch build that follows it rebuilds the list) or that met a
// non-finite force.
//
// Those stop decisions must be the same in every CTA, so they travel with the
// barrier's own word (cr_bar.h): the poll that sees the barrier complete brings
// the decision too (a flag word of its own cost another trip to L2 per step).
// The word is one of two that launches take in turn: CTA 0 clears the other one
// for the next launch.  A non-finite force also goes into status.pflag.  The
// step counters and the turn are read by every CTA before barrier 0 and updated
// by CTA 0 after the loop.  Every barrier wait is bounded: a CTA that gives up
// sets stalled and abort and leaves; the others see stalled and leave too.

__device__ __forceinline__ unsigned long long pst_ld_acquire(const unsigned long long* a) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(a) : "memory");
  return v;
}

__device__ __forceinline__ unsigned long long pst_atom_add_release(unsigned long long* a, unsigned long long x) {
  unsigned long long old;
  asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;" : "=l"(old) : "l"(a), "l"(x) : "memory");
  return old;
}

// The barriers of one launch.  Every thread of the CTA makes one before the
// first barrier.
struct StepsBarrier {
  DevStatus* st;
  unsigned long long* word;
  int turn, k;  // k: barriers passed
  __device__ __forceinline__ explicit StepsBarrier(DevStatus* s) : st(s), k(0) {
    turn = *(volatile int*)&s->pturn;
    word = &s->pbar[turn];
    if (blockIdx.x == 0 && threadIdx.x == 0) s->pbar[turn ^ 1] = 0ull;
  }
  // After the last barrier, by one thread of CTA 0: the next launch takes the
  // other word.
  __device__ __forceinline__ void leave() const {
    if (k > 0) st->pturn = turn ^ 1;
  }
};

// Barrier over the grid.  stop: this CTA wants the loop to end (thread 0's
// value counts).  Returns 0: go on, 1: some CTA wanted to stop, -1: the wait
// gave up.
__device__ __forceinline__ int steps_barrier(StepsBarrier& b, bool stop = false) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    DevStatus* st = b.st;
    int ok = 0;
    pst_atom_add_release(b.word, bar_arrival(b.k, stop));
    const long long lim = barrier_poll_limit(st);
    long long it = 0;
    unsigned long long now;
    while (!bar_complete(now = pst_ld_acquire(b.word), b.k, gridDim.x)) {
      if (++it > lim || *(volatile int*)&st->stalled) {
        ok = -1;
        break;
      }
      __nanosleep(64);
    }
    if (ok < 0) {
      atomicExch(&st->stalled, 1);
      atomicExch(&st->abort, 1);
    } else if (bar_stopped(now, b.k)) {
      ok = 1;
    }
    s_ok = ok;
  }
  b.k++;
  __syncthreads();
  return s_ok;
}

// CTAs an SM the registers are held to: without the stage, five of the
// vertex-vertex form (740 tiles) rather than four.
template <int INTER, int BLOCK, int L, int PREC, bool STAGED>
constexpr int steps_ctas_per_sm() {
  return INTER == INT_VV && L == 1 && !STAGED ? 5 : tile_threads_per_sm<PREC, L>() / BLOCK;
}

template <int POT, int INTER, int BLOCK, int L, int PREC, bool STAGED>
__global__ void __launch_bounds__(BLOCK, (steps_ctas_per_sm<INTER, BLOCK, L, PREC, STAGED>()))
    k_tile_steps(const __grid_constant__ SysParams p, const __grid_constant__ SysArrays a,
                 const __grid_constant__ StepArgs s) {
  pdl_wait();
  pdl_trigger();
  DevStatus* st = s.status;
  const volatile DevStatus* vs = st;
  if (vs->abort | vs->converged) return;
  const long long left = vs->steps_left;
  if (left <= 0) return;
  const int n = (int)(left < (long long)s.persist_max ? left : (long long)s.persist_max);
  const unsigned long long step0 = (unsigned long long)vs->rng_step;
  StepsBarrier bar(st);
  double2* pos0 = const_cast<double2*>(a.pos);
  double2* pos1 = s.pos_out;
  extern __shared__ __align__(16) unsigned char s_stage[];
  Stage<BLOCK / L> g(s_stage);
  const int4 tile = a.tiles[blockIdx.x];
  if constexpr (STAGED) stage_build<INTER, BLOCK, L>(p, p, a, tile, s.last_pos, s.disp_cutoff, pot_range_f<POT>(p), g);
  int done = 0;
  bool stalled = false, stopped = false;
  for (int j = 0; j < n; j++) {
    const double2* pin = (j & 1) ? pos1 : pos0;
    double2* pout = (j & 1) ? pos0 : pos1;
    const bool stop = tile_body<POT, INTER, MODE_STEP, BLOCK, L, PREC, false, 1, STAGED>(
        p, a, s, pin, pout, step0 + (unsigned long long)j, &st->pflag, j > 0, &g, tile);
    done = j + 1;
    const int b = steps_barrier(bar, stop);
    if (b < 0) {
      stalled = true;
      break;
    }
    if (b > 0) {
      stopped = true;
      break;
    }
  }
  if (stalled) return;
  if (done & 1) {
    // the last step wrote pos1: this tile's vertices back to pos0 (every read
    // of pos0 by the last step finished before the last barrier)
    for (int v = tile.z + threadIdx.x; v < tile.w; v += BLOCK) pos0[v] = pos1[v];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && done > 0) {
    if (stopped && *(volatile int*)&st->pflag) {
      st->nonfinite = 1;
      st->abort = 1;
    }
    st->rng_step += done;
    st->ops_done += done;
    st->steps_left -= done;
    bar.leave();
  }
}

}  // namespace cr
