// Forces and energies in hyper-dual arithmetic: the derivative kernel behind
// the Hessian-vector product, the virial pressure and the parameter
// derivatives (cr_hvp, cr_calc_pressure, cr_param_derivatives).
//
// One thread per vertex evaluates the same per-vertex force and energy as the
// fused kernel (shape terms of kernelCalcShapeForceEnergy,
// include/cudaKernel.cuh:474-529, with harmonic or FENE monomers, and the pair
// terms: vertex-vertex, kernelCalcVertexInteraction :690-722, or smooth
// vertex-segment, kernelCalcSmoothInteraction :922-975, in the gather form of
// the fused kernel) with every input a hyper-dual number: positions x + t1 e1 + t2 e2, box L (1 + s1 e1 + s2 e2),
// and the shape constants and rest lengths / radii along parameter tangents.
// The e1 part of the force is then D_t1 F = -H t1 (the Hessian-vector
// product), the e1 part of the energy along the affine dilation t1 = x,
// s1 = 1 is dU/dlambda = -2 A P, and the e1 e2 parts give the mixed
// derivatives that the adjoint gradients need.  The rings' areas are summed
// once per ring by a first kernel.  These kernels serve small systems and
// iterative solves, not the time-stepping hot path.
#include <algorithm>

#include "cr_hd.cuh"
#include "cr_launch.h"
#include "cr_tile.cuh"

namespace cr {
namespace {

template <class T>
struct HBox {
  T lx, ly;
};
template <class T>
__device__ __forceinline__ HBox<T> box_of(const DiffArgs& g) {
  return HBox<T>{parts<T>(g.p.lx, g.p.lx * g.s1, g.p.lx * g.s2, 0.0), parts<T>(g.p.ly, g.p.ly * g.s1, g.p.ly * g.s2, 0.0)};
}

template <class T>
__device__ __forceinline__ T pbc_hd(T d, const T& L) {
  const double k = round(d.a / L.a);
  return d - k * L;
}

template <class T>
__device__ __forceinline__ Pair<T> pbc2_hd(const Pair<T>& a, const Pair<T>& b, const HBox<T>& bx) {
  return Pair<T>{pbc_hd(a.x - b.x, bx.lx), pbc_hd(a.y - b.y, bx.ly)};
}

template <class T>
__device__ __forceinline__ Pair<T> load_x(const DiffArgs& g, int i) {
  const double2 x = g.pos[i];
  double2 u1 = make_double2(0.0, 0.0), u2 = make_double2(0.0, 0.0);
  if (g.t1) u1 = g.t1[i];
  if (g.t2) u2 = g.t2[i];
  return Pair<T>{parts<T>(x.x, u1.x, u2.x, 0.0), parts<T>(x.y, u1.y, u2.y, 0.0)};
}

// l0 and rad scale as sqrt(calA0) (the reference's conventions: l0 from the
// preferred perimeter, rad = l0 / 2); along ln(calA0) a length w takes
// w (1 + c1/2 e1 + c2/2 e2 - c1 c2 / 4 e1 e2).
template <class T>
__device__ __forceinline__ T scaled_length(const DiffArgs& g, double w) {
  return parts<T>(w, 0.5 * g.c1 * w, 0.5 * g.c2 * w, -0.25 * g.c1 * g.c2 * w);
}

template <int POT, class T>
__device__ __forceinline__ bool pair_hd(const DiffArgs& g, T d, T rsum, T& gm, T& ep) {
  const SysParams& p = g.p;
  const double ec = p.ec;
  if constexpr (POT == POT_HARMONIC) {
    const T ov = 1.0 - d / rsum;
    if (!(ov.a > 0.0)) return false;
    gm = ec * ov / rsum;
    ep = (0.25 * ec) * ov * ov;
    return true;
  } else if constexpr (POT == POT_LJ) {
    if (!(d.a <= p.lj_cutoff * rsum.a)) return false;
    const T ratio = rsum / d;
    const T r2 = ratio * ratio;
    const T r6 = r2 * r2 * r2;
    const T r12 = r6 * r6;
    const T fshift = p.lj_fshift / rsum;
    gm = (24.0 * ec) * (2.0 * r12 - r6) / d - fshift;
    ep = 0.5 * ((4.0 * ec) * (r12 - r6) - p.lj_ecut - habs(fshift) * (d - p.lj_cutoff * rsum));
    return true;
  } else if constexpr (POT == POT_ADHESIVE) {
    if (!(d.a < (1.0 + p.l2) * rsum.a)) return false;
    const T ov = 1.0 - d / rsum;
    if (d.a < (1.0 + p.l1) * rsum.a) {
      gm = ec * ov / rsum;
      ep = (0.25 * ec) * (ov * ov - p.l1 * p.l2);
    } else {
      const double k = ec * p.l1 / (p.l2 - p.l1);
      gm = -k * (ov + p.l2) / rsum;
      ep = (-0.25 * k) * (ov + p.l2) * (ov + p.l2);
    }
    return true;
  } else {
    if (!(d.a <= kWCAcut * rsum.a)) return false;
    const T ratio = rsum / d;
    const T r2 = ratio * ratio;
    const T r6 = r2 * r2 * r2;
    const T r12 = r6 * r6;
    gm = (24.0 * ec) * (2.0 * r12 - r6) / d;
    ep = (0.5 * ec) * (4.0 * (r12 - r6) + 1.0);
    return true;
  }
}

template <class T>
__device__ __forceinline__ T cross(const Pair<T>& a, const Pair<T>& b) { return a.x * b.y - b.x * a.y; }
template <class T>
__device__ __forceinline__ T dot(const Pair<T>& a, const Pair<T>& b) { return a.x * b.x + a.y * b.y; }
template <class T>
__device__ __forceinline__ T norm(const Pair<T>& a) { return hsqrt(dot(a, a)); }
// calcAngle(nextSegment, previousSegment) (include/cudaKernel.cuh:423-427)
template <class T>
__device__ __forceinline__ T angle(const Pair<T>& ns, const Pair<T>& ps) { return hatan2(cross(ns, ps), dot(ns, ps)); }

// One smooth unit (calcGradMultipleAndEnergy / calcVertexSegmentInteraction /
// calcVertexVertexInteraction, include/cudaKernel.cuh:806-912): vertex t
// against the segment q -> o, with tq = t - q, w = t - o, seg = o - q and
// pseg = q - qq.  WHO = 1 adds the force on t, 2 the force on o, 3 the force
// on q; the unit energy is booked for WHO 1 and 2 (each unit is evaluated
// once in each role, as the fused kernel gathers it).  The branches are taken
// on the real parts.
template <int POT, int WHO, class T>
__device__ void smooth_hd(const DiffArgs& g, const Pair<T>& tq, const Pair<T>& w, const Pair<T>& seg, const Pair<T>& pseg,
                          const T& rsum, Pair<T>& f, T& e) {
  const T len2 = dot(seg, seg);
  const T inv_len = 1.0 / hsqrt(len2);
  const T inv_lsq = inv_len * inv_len;
  const T proj = dot(tq, seg) * inv_lsq;
  const T pc = dot(tq, pseg);
  const T pl2 = dot(pseg, pseg);
  auto corner = [&](double sgn) {  // sgn +1: convex (added), -1: concave (removed)
    const T d2 = norm(tq);
    T g2, ep2;
    if (pair_hd<POT>(g, d2, rsum, g2, ep2) && g2.a != 0.0) {
      const T s2 = g2 / d2;
      if (WHO == 1) {
        f.x += sgn * (s2 * tq.x);
        f.y += sgn * (s2 * tq.y);
      } else if (WHO == 3) {
        f.x -= sgn * (s2 * tq.x);
        f.y -= sgn * (s2 * tq.y);
      }
      if (WHO != 3) e += sgn * ep2;
    }
  };
  if (proj.a >= 0.0 && proj.a < 1.0) {
    const Pair<T> dp{tq.x - proj * seg.x, tq.y - proj * seg.y};
    const T d = norm(dp);
    T gm, ep;
    if (pair_hd<POT>(g, d, rsum, gm, ep) && gm.a != 0.0) {
      const T cr = seg.x * w.y - w.x * seg.y;
      const double sign = cr.a > 0.0 ? 1.0 : (cr.a < 0.0 ? -1.0 : __longlong_as_double(0x7ff8000000000000LL));
      const T gg = gm * inv_len;
      if (WHO == 1) {
        f.x += gg * (sign * (-1.0) * seg.y);
        f.y += gg * (sign * seg.x);
      } else {
        const T a = habs(cr) * inv_lsq;
        if (WHO == 2) {
          f.x += gg * (sign * tq.y - a * seg.x);
          f.y += gg * ((-sign) * tq.x - a * seg.y);
        } else {
          f.x += gg * ((-sign) * w.y + a * seg.x);
          f.y += gg * (sign * w.x + a * seg.y);
        }
      }
      if (WHO != 3) e += ep;
    }
    if (pc.a >= -pl2.a && pc.a < 0.0) corner(-1.0);
  } else if (proj.a < 0.0 && pc.a >= 0.0) {
    corner(1.0);
  }
}

// ring predecessor of vertex j from its topology
__device__ __forceinline__ int prev_of(const DiffArgs& g, int j, int back) {
  const int2 tp = g.vtopo[j];
  const int k = tp.y & 0xffff, n = tp.y >> 16;
  return j - k + (k - back + 2 * n) % n;
}

// ring area by the shoelace sum of offsets from the ring's first vertex, one
// warp per ring
template <class T>
__global__ void __launch_bounds__(128) k_ring_area(const __grid_constant__ DiffArgs g, const int* ring_first,
                                                   const int* ring_nv) {
  const int q = blockIdx.x * 4 + threadIdx.x / 32, wl = threadIdx.x & 31;
  if (q >= g.p.np || (g.skip && *g.skip)) return;
  const HBox<T> bx = box_of<T>(g);
  const int f = ring_first[q], nvr = ring_nv[q];
  const Pair<T> x0 = load_x<T>(g, f);
  T sum = num<T>(0.0);
  for (int k = wl; k < nvr; k += 32) {
    const Pair<T> u = pbc2_hd(load_x<T>(g, f + k), x0, bx);
    const Pair<T> un = pbc2_hd(load_x<T>(g, f + (k + 1 == nvr ? 0 : k + 1)), x0, bx);
    sum += cross(u, un);
  }
  double* part = reinterpret_cast<double*>(&sum);
  constexpr int np = sizeof(T) / sizeof(double);
#pragma unroll
  for (int c = 0; c < np; c++)
    for (int o = 16; o > 0; o >>= 1) part[c] += __shfl_xor_sync(0xffffffffu, part[c], o);
  if (wl) return;
  const T area = 0.5 * habs(sum);
  double* o = g.ring_area + (size_t)4 * q;
  const double* a = reinterpret_cast<const double*>(&area);
#pragma unroll
  for (int c = 0; c < np; c++) o[c] = a[c];
  if (g.diag) o[1] = sum.a >= 0.0 ? 1.0 : -1.0;  // diag mode: the ring's orientation
}

// Shape terms of one vertex (kernelCalcShapeForceEnergy,
// include/cudaKernel.cuh:474-529): ns, ps its next and previous segments, pps
// and nns the ones beyond, area its ring's.
template <class T>
__device__ __forceinline__ void shape_hd(const SysParams& p, T ea, T el, T eb, const Pair<T>& ns, const Pair<T>& ps,
                                         const Pair<T>& pps, const Pair<T>& nns, T area, double a0, int nvr, T tl0,
                                         T pl0, double th0p, double th0, double th0n, Pair<T>& F, T& E) {
  const T th = angle(ns, ps), thp = angle(ps, pps), thn = angle(nns, ns);
  // area
  const T dA = area / a0 - 1.0;
  const T gmA = ea * dA / a0;
  const Pair<T> npd{ns.x + ps.x, ns.y + ps.y};
  F.x += 0.5 * gmA * (-npd.y);
  F.y += 0.5 * gmA * npd.x;
  E += (0.5 * ea * dA * dA) / (double)nvr;
  // segment lengths: harmonic or FENE monomers (include/cudaKernel.cuh:442-471)
  const T plen = norm(ps), nlen = norm(ns);
  if (p.monomer == 0) {
    const T pd = plen / pl0 - 1.0, nd = nlen / tl0 - 1.0;
    F.x += el * (nd * ns.x / (tl0 * nlen) - pd * ps.x / (pl0 * plen));
    F.y += el * (nd * ns.y / (tl0 * nlen) - pd * ps.y / (pl0 * plen));
    E += 0.5 * el * pd * pd;
  } else {
    const T c = (2.0 * p.stiff * p.ext_sq) * el;
    const T an = nlen / (p.ext_sq * tl0 * tl0 - nlen * nlen);
    const T ap = plen / (p.ext_sq * pl0 * pl0 - plen * plen);
    F.x += c * (an * ns.x / nlen - ap * ps.x / plen);
    F.y += c * (an * ns.y / nlen - ap * ps.y / plen);
    E += (p.stiff * p.ext_sq) * el * hlog(1.0 - plen * plen / (p.ext_sq * pl0 * pl0));
  }
  // bending
  const T prevAD = thp - th0p, thisAD = th - th0, nextAD = thn - th0n;
  const T pvar = (thisAD - prevAD) / dot(ps, ps);
  const T nvar = (thisAD - nextAD) / dot(ns, ns);
  F.x += eb * (pvar * ps.y + nvar * ns.y);
  F.y += eb * (pvar * (-ps.x) + nvar * (-ns.x));
  E += 0.5 * eb * thisAD * thisAD;
}

// force on vertex v along the pair (v, j)
template <int POT, class T>
__device__ __forceinline__ void pair_force_hd(const DiffArgs& g, const Pair<T>& dl, T rsum, Pair<T>& F, T& E) {
  const T d = norm(dl);
  T gm, ep;
  if (pair_hd<POT>(g, d, rsum, gm, ep)) {
    const T s2 = gm / d;
    F.x += s2 * dl.x;
    F.y += s2 * dl.y;
    E += ep;
  }
}

template <int POT, int INTER, class T>
__global__ void __launch_bounds__(64) k_diff(const __grid_constant__ DiffArgs g) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= g.p.nv || (g.skip && *g.skip)) return;
  const SysParams& p = g.p;
  const HBox<T> bx = box_of<T>(g);
  const T ea = parts<T>(p.ea, g.pe1[0], g.pe2[0], 0.0), el = parts<T>(p.el, g.pe1[1], g.pe2[1], 0.0),
          eb = parts<T>(p.eb, g.pe1[2], g.pe2[2], 0.0);
  const int2 tp = g.vtopo[v];
  const int ring = tp.x, k = tp.y & 0xffff, nvr = tp.y >> 16;
  const int f = v - k;
  auto at = [&](int kk) { return f + ((kk % nvr) + nvr) % nvr; };
  const int vp = at(k - 1), vn = at(k + 1), vpp = at(k - 2), vnn = at(k + 2);

  const double* ra = g.ring_area + (size_t)4 * ring;
  Pair<T> x = load_x<T>(g, v);
  const Pair<T> xn = load_x<T>(g, vn), xp = load_x<T>(g, vp);
  if (g.diag) x = Pair<T>{parts<T>(x.x.a, 1.0, 0.0, 0.0), parts<T>(x.y.a, 0.0, 1.0, 0.0)};
  const Pair<T> ns = pbc2_hd(xn, x, bx), ps = pbc2_hd(x, xp, bx);
  // ring area; with the own-vertex seeding its tangents are the shoelace
  // derivatives dA/dx_v = s (y_next - y_prev) / 2, dA/dy_v = s (x_prev - x_next) / 2
  // (s the ring's orientation), second derivative zero
  const T area = g.diag ? parts<T>(ra[0], 0.5 * ra[1] * (ns.y.a + ps.y.a), -0.5 * ra[1] * (ns.x.a + ps.x.a), 0.0)
                        : parts<T>(ra[0], ra[1], ra[2], ra[3]);
  const Pair<T> pps = pbc2_hd(xp, load_x<T>(g, vpp), bx), nns = pbc2_hd(load_x<T>(g, vnn), xn, bx);
  Pair<T> F{num<T>(0.0), num<T>(0.0)};
  T E = num<T>(0.0);
  shape_hd<T>(p, ea, el, eb, ns, ps, pps, nns, area, g.a0[ring], nvr, scaled_length<T>(g, g.l0[v]),
              scaled_length<T>(g, g.l0[vp]), g.theta0[vp], g.theta0[v], g.theta0[vn], F, E);

  const T ri = scaled_length<T>(g, g.rad[v]);
  const int cnt = min(g.nbr_cnt[v], g.nbr_cap);
  if constexpr (INTER == INT_VV) {
    // vertex-vertex pairs
    for (int s = 0; s < cnt; s++) {
      const int j = g.nbr[(size_t)s * p.nv + v];
      pair_force_hd<POT>(g, pbc2_hd(x, load_x<T>(g, j), bx), ri + scaled_length<T>(g, g.rad[j]), F, E);
    }
  } else {
    // smooth units gathered as the fused kernel gathers them: this vertex
    // against each neighbour's segment prev(j) -> j (force on v), each
    // neighbour against this vertex's segment prev(v) -> v (force on v as its
    // end o), and each neighbour of next(v) against the segment v -> next(v)
    // (force on v as its start q)
    for (int s = 0; s < cnt; s++) {
      const int j = g.nbr[(size_t)s * p.nv + v];
      const Pair<T> xj = load_x<T>(g, j), xjq = load_x<T>(g, prev_of(g, j, 1)), xjqq = load_x<T>(g, prev_of(g, j, 2));
      const T rsum = ri + scaled_length<T>(g, g.rad[j]);
      smooth_hd<POT, 1>(g, pbc2_hd(x, xjq, bx), pbc2_hd(x, xj, bx), pbc2_hd(xj, xjq, bx), pbc2_hd(xjq, xjqq, bx), rsum,
                        F, E);
      smooth_hd<POT, 2>(g, pbc2_hd(xj, xp, bx), pbc2_hd(xj, x, bx), ps, pps, rsum, F, E);
    }
    const T rn = scaled_length<T>(g, g.rad[vn]);
    const int cntn = min(g.nbr_cnt[vn], g.nbr_cap);
    T none = num<T>(0.0);
    for (int s = 0; s < cntn; s++) {
      const int j = g.nbr[(size_t)s * p.nv + vn];
      const Pair<T> xj = load_x<T>(g, j);
      smooth_hd<POT, 3>(g, pbc2_hd(xj, x, bx), pbc2_hd(xj, xn, bx), ns, ps, rn + scaled_length<T>(g, g.rad[j]), F,
                        none);
    }
  }
  if (g.hv_out) {
    // the product of the Hessian with t1
    g.hv_out[v] = make_double2(-F.x.b, -F.y.b);
    return;
  }
  constexpr int np = sizeof(T) / sizeof(double);
  double* fo = g.force_out + (size_t)v * 8;
  double* eo = g.energy_out + (size_t)v * 4;
  const double *fx = reinterpret_cast<const double*>(&F.x), *fy = reinterpret_cast<const double*>(&F.y),
               *e = reinterpret_cast<const double*>(&E);
#pragma unroll
  for (int c = 0; c < np; c++) {
    fo[c] = fx[c];
    fo[4 + c] = fy[c];
    eo[c] = e[c];
  }
}

}  // namespace

namespace {
// small CTAs: the systems these derivatives serve hold a few thousand
// vertices, so 32-thread CTAs spread them over every SM
template <int INTER, class T>
void launch_diff_i(cudaStream_t st, int pot, const DiffArgs& g) {
  const int nb = (g.p.nv + 31) / 32;
  switch (pot) {
    case POT_HARMONIC: k_diff<POT_HARMONIC, INTER, T><<<nb, 32, 0, st>>>(g); break;
    case POT_LJ: k_diff<POT_LJ, INTER, T><<<nb, 32, 0, st>>>(g); break;
    case POT_ADHESIVE: k_diff<POT_ADHESIVE, INTER, T><<<nb, 32, 0, st>>>(g); break;
    default: k_diff<POT_WCA, INTER, T><<<nb, 32, 0, st>>>(g); break;
  }
}
template <class T>
void launch_diff_t(cudaStream_t st, int pot, int inter, const DiffArgs& g, const int* ring_first, const int* ring_nv) {
  k_ring_area<T><<<(g.p.np + 3) / 4, 128, 0, st>>>(g, ring_first, ring_nv);
  if (inter == INT_VV) launch_diff_i<INT_VV, T>(st, pot, g);
  else launch_diff_i<INT_SMOOTH, T>(st, pot, g);
}
}  // namespace

// hyper-dual forces and energies; with hv_out set (one position tangent t1 and
// nothing else) dual numbers and the product alone
void launch_diff(cudaStream_t st, int pot, int inter, const DiffArgs& g, const int* ring_first, const int* ring_nv) {
  if (g.hv_out) launch_diff_t<D1>(st, pot, inter, g, ring_first, ring_nv);
  else launch_diff_t<HD>(st, pot, inter, g, ring_first, ring_nv);
}

// ----------------------------------------------- device-resident CG iteration
namespace {
constexpr int kCgBlock = 256;

__device__ __forceinline__ void cg_block_sums(double* v, int n, double* out) {
  // fixed-order CTA sums of n values per thread; results in out[0..n) on thread 0
  __shared__ double s[kCgBlock / 32][4];
  for (int q = 0; q < n; q++) {
    double x = v[q];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5][q] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 0; q < n; q++) {
      double t = 0.0;
      for (int w = 0; w < kCgBlock / 32; w++) t += s[w][q];
      out[q] = t;
    }
  }
}

// partials of hp = H p: sum hp.x, sum hp.y, p.hp
__global__ void __launch_bounds__(kCgBlock) k_cg_hp(const __grid_constant__ CgArgs a) {
  if (((volatile CgState*)a.st)->done) return;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int v = blockIdx.x * kCgBlock + threadIdx.x; v < a.nv; v += a.nblk * kCgBlock) {
    const double hx = a.hp[2 * v], hy = a.hp[2 * v + 1];
    acc[0] += hx;
    acc[1] += hy;
    acc[2] += a.p[2 * v] * hx + a.p[2 * v + 1] * hy;
  }
  double out[3];
  cg_block_sums(acc, 3, out);
  if (threadIdx.x == 0)
    for (int q = 0; q < 3; q++) a.partials[(size_t)8 * blockIdx.x + q] = out[q];
}

// one thread: the mean of H p and the step alpha = r.z / p.Hp (p carries no
// translation, so p.Hp is the curvature along p of the projected Hessian)
__global__ void k_cg_alpha(const __grid_constant__ CgArgs a) {
  CgState& st = *a.st;
  if (st.done) return;
  double sx = 0.0, sy = 0.0, php = 0.0;
  for (int b = 0; b < a.nblk; b++) {
    sx += a.partials[8 * b];
    sy += a.partials[8 * b + 1];
    php += a.partials[8 * b + 2];
  }
  st.mx = sx / a.nv;
  st.my = sy / a.nv;
  if (!(php > 0.0)) {
    st.bad = 1;
    st.done = 1;
    return;
  }
  st.alpha = st.rz / php;
}

// z = M^-1 r at vertex v (2 x 2 block), or z = r without a preconditioner
__device__ __forceinline__ double2 cg_precondition(const double* minv, int v, double rx, double ry) {
  if (!minv) return make_double2(rx, ry);
  const double* m = minv + (size_t)3 * v;
  return make_double2(m[0] * rx + m[1] * ry, m[1] * rx + m[2] * ry);
}

// x += alpha p; r -= alpha (H p - mean); z = M^-1 r; partials: |r|^2, r.z,
// sum z.x, sum z.y (one vertex, both components, per thread)
__global__ void __launch_bounds__(kCgBlock) k_cg_update(const __grid_constant__ CgArgs a) {
  const CgState st = *(const CgState*)a.st;
  if (st.done) return;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int v = blockIdx.x * kCgBlock + threadIdx.x; v < a.nv; v += a.nblk * kCgBlock) {
    a.x[2 * v] += st.alpha * a.p[2 * v];
    a.x[2 * v + 1] += st.alpha * a.p[2 * v + 1];
    const double rx = a.r[2 * v] - st.alpha * (a.hp[2 * v] - st.mx);
    const double ry = a.r[2 * v + 1] - st.alpha * (a.hp[2 * v + 1] - st.my);
    a.r[2 * v] = rx;
    a.r[2 * v + 1] = ry;
    const double2 z = cg_precondition(a.minv, v, rx, ry);
    a.z[2 * v] = z.x;
    a.z[2 * v + 1] = z.y;
    acc[0] += rx * rx + ry * ry;
    acc[1] += rx * z.x + ry * z.y;
    acc[2] += z.x;
    acc[3] += z.y;
  }
  double out[4];
  cg_block_sums(acc, 4, out);
  if (threadIdx.x == 0)
    for (int q = 0; q < 4; q++) a.partials[(size_t)8 * blockIdx.x + 3 + q] = out[q];
}

// one thread: the new |r|^2 and r.z, beta = r.z / previous r.z, the mean of
// z, the iteration count and the stop tests of the host loop (relative
// residual, iteration limit)
__global__ void k_cg_beta(const __grid_constant__ CgArgs a) {
  CgState& st = *a.st;
  if (st.done) return;
  double rr2 = 0.0, rz2 = 0.0, zx = 0.0, zy = 0.0;
  for (int b = 0; b < a.nblk; b++) {
    rr2 += a.partials[8 * b + 3];
    rz2 += a.partials[8 * b + 4];
    zx += a.partials[8 * b + 5];
    zy += a.partials[8 * b + 6];
  }
  st.beta = rz2 / st.rz;
  st.rz = rz2;
  st.rr = rr2;
  st.zx = zx / a.nv;
  st.zy = zy / a.nv;
  st.iters += 1;
  if (!(sqrt(st.rr / st.bb) > st.tol) || st.iters >= st.max_iters) st.done = 1;
}

// p = (z - mean z) + beta p: the preconditioned residual without its
// translation (r carries none, so r.z needs no correction)
__global__ void __launch_bounds__(kCgBlock) k_cg_direction(const __grid_constant__ CgArgs a) {
  const CgState st = *(const CgState*)a.st;
  if (st.done) return;
  for (int i = blockIdx.x * kCgBlock + threadIdx.x; i < 2 * a.nv; i += a.nblk * kCgBlock)
    a.p[i] = (a.z[i] - ((i & 1) ? st.zy : st.zx)) + st.beta * a.p[i];
}

// inverse diagonal blocks from a diag-mode launch: H_vv = -[[Fx.b, Fx.c],
// [Fy.b, Fy.c]] symmetrised; where it is not positive definite, the inverse
// of its diagonal's magnitudes (floored at 1e-3 of the larger), and the
// identity for a zero block
__global__ void k_cg_prec(int nv, const double* fhd, double* minv) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const double* f = fhd + (size_t)8 * v;
  const double h11 = -f[1], h22 = -f[6], h12 = -0.5 * (f[2] + f[5]);
  const double det = h11 * h22 - h12 * h12;
  double* m = minv + (size_t)3 * v;
  if (h11 > 0.0 && h22 > 0.0 && det > 1e-12 * h11 * h22) {
    m[0] = h22 / det;
    m[1] = -h12 / det;
    m[2] = h11 / det;
  } else {
    const double s = fmax(fabs(h11), fabs(h22));
    m[0] = s > 0.0 ? 1.0 / fmax(fabs(h11), 1e-3 * s) : 1.0;
    m[1] = 0.0;
    m[2] = s > 0.0 ? 1.0 / fmax(fabs(h22), 1e-3 * s) : 1.0;
  }
}

// Start of a solve, by one CTA: b (in r) without its mean, z = M^-1 r and p = z
// without their means (the uniform translations, the Hessian's null space in a
// periodic box), x = 0, and the state: |b|^2, r.z and whether there is nothing
// to do.
__global__ void __launch_bounds__(1024) k_cg_start(const __grid_constant__ CgArgs a, double tol, long long max_iters) {
  __shared__ double s_part[32][2], s_tot[2];
  const auto sums = [&](double x, double y) {
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    __syncthreads();
    if (threadIdx.x % 32 == 0) {
      s_part[threadIdx.x / 32][0] = x;
      s_part[threadIdx.x / 32][1] = y;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      double t = 0.0;
      for (int w = 0; w < 32; w++) t += s_part[w][threadIdx.x];
      s_tot[threadIdx.x] = t;
    }
    __syncthreads();
    return make_double2(s_tot[0], s_tot[1]);
  };
  double2* r = reinterpret_cast<double2*>(a.r);
  double2* z = reinterpret_cast<double2*>(a.z);
  double2* p = reinterpret_cast<double2*>(a.p);
  double2* x = reinterpret_cast<double2*>(a.x);
  double2 acc = make_double2(0.0, 0.0);
  for (int v = threadIdx.x; v < a.nv; v += 1024) acc = make_double2(acc.x + r[v].x, acc.y + r[v].y);
  double2 m = sums(acc.x, acc.y);
  m = make_double2(m.x / a.nv, m.y / a.nv);
  acc = make_double2(0.0, 0.0);
  for (int v = threadIdx.x; v < a.nv; v += 1024) {
    const double2 q = make_double2(r[v].x - m.x, r[v].y - m.y), w = cg_precondition(a.minv, v, q.x, q.y);
    r[v] = q;
    z[v] = w;
    x[v] = make_double2(0.0, 0.0);
    acc = make_double2(acc.x + w.x, acc.y + w.y);
  }
  m = sums(acc.x, acc.y);
  m = make_double2(m.x / a.nv, m.y / a.nv);
  acc = make_double2(0.0, 0.0);
  for (int v = threadIdx.x; v < a.nv; v += 1024) {
    const double2 q = r[v], w = make_double2(z[v].x - m.x, z[v].y - m.y);
    z[v] = w;
    p[v] = w;
    acc = make_double2(acc.x + q.x * q.x + q.y * q.y, acc.y + q.x * w.x + q.y * w.y);
  }
  m = sums(acc.x, acc.y);
  if (threadIdx.x == 0) {
    CgState st = {};
    st.rr = st.bb = m.x;
    st.rz = m.y;
    st.tol = tol;
    st.max_iters = max_iters;
    st.done = (max_iters == 0 || !(m.x > 0.0) || !(1.0 > tol)) ? 1 : 0;
    *a.st = st;
  }
}
}  // namespace

// ------------------------------------------------- many iterations per launch
//
// The Hessian does not change during a solve, so each thread forms its vertex's
// rows once, from hyper-dual evaluations seeded on one vertex at a time: the
// 2 x 2 blocks of the shape terms with respect to the five ring vertices they
// read, the ring area's rank-one part (force coefficient c_v, area gradient
// a_v) and one symmetric block per pair in range.  A product is then some
// thirty multiplications per vertex and a sum over the ring.  Solution,
// residual and direction stay in registers, the CTA's rings in shared memory;
// CTAs exchange z and the last direction, from which a reader forms
// p = (z - mean z) + beta p_old itself, so an iteration takes two grid
// barriers (p.Hp; r.r and r.z), after each of which every CTA adds up the
// partial sums in the same order.
//   8,448 vertices, harmonic, per iteration: 63 us as seven launches of a
// captured graph (hyper-dual forces anew each time), 6.6 us here.

// Arrival and wait of one thread of the CTA (k is its barrier, from 1); false
// when the wait gave up.
__device__ __forceinline__ bool cg_wait(CgState* st, unsigned long long k, long long limit) {
  unsigned long long now;
  asm volatile("red.add.release.gpu.global.u64 [%0], %1;" ::"l"(&st->bar), "l"(1ull) : "memory");
  const long long lim = limit > 0 ? limit : (limit == 0 ? (1LL << 20) : 0);
  for (long long it = 0;;) {
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(&st->bar) : "memory");
    if (now >= k * gridDim.x) return true;
    if (++it > lim || *(volatile int*)&st->stalled) {
      atomicExch(&st->stalled, 1);
      return false;
    }
    __nanosleep(32);
  }
}

template <int POT, int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_cg_steps(const __grid_constant__ DiffArgs g, const __grid_constant__ CgArgs a,
                                                    const __grid_constant__ CgSteps ks) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int W = BLOCK / 32;
  __shared__ double2 s_u[BLOCK];
  __shared__ double s_dot[BLOCK];
  __shared__ double s_part[W][4], s_tot[4];
  __shared__ int s_rfirst[BLOCK], s_rlen[BLOCK], s_ok;
  // the first kHeld pairs of each vertex; the others stay in global memory
  constexpr int kHeld = 4;
  __shared__ double2 s_kxy[kHeld][BLOCK];
  __shared__ double s_kyy[kHeld][BLOCK];
  __shared__ int s_kj[kHeld][BLOCK];
  CgState* st = a.st;
  const CgState st0 = *st;  // no CTA writes it before the others have read it (the first barrier)
  if (st0.done || st0.stalled) return;
  const SysParams& p = g.p;
  const int t = threadIdx.x, w = t / 32, wl = t % 32;
  const int2 tile = ks.tiles[blockIdx.x];
  const int v = tile.x + t;
  const bool on = v < tile.y;
  const int2 tp = g.vtopo[on ? v : tile.x];
  const int k = tp.y & 0xffff, nvr = tp.y >> 16, lf = t - k;
  const int ring0 = g.vtopo[tile.x].x, nrings = g.vtopo[tile.y - 1].x - ring0 + 1;
  const auto near = [&](int d) { return lf + ((k + d) % nvr + nvr) % nvr; };
  if (on && k == 0) {
    s_rfirst[tp.x - ring0] = t;
    s_rlen[tp.x - ring0] = nvr;
  }
  const HBox<HD> bx = box_of<HD>(g);
  const auto pbc = [&](double2 d) {
    return make_double2(d.x - round(d.x / p.lx) * p.lx, d.y - round(d.y / p.ly) * p.ly);
  };
  // ring areas: signed shoelace sums, one warp per ring
  s_u[t] = on ? g.pos[v] : make_double2(0.0, 0.0);
  s_dot[t] = 0.0;
  __syncthreads();
  double2 e[4] = {};  // segments pps, ps, ns, nns
  if (on) {
    const double2 x0 = s_u[lf], xa = s_u[t], xb = s_u[near(1)];
    const double2 u = pbc(make_double2(xa.x - x0.x, xa.y - x0.y)), un = pbc(make_double2(xb.x - x0.x, xb.y - x0.y));
    s_dot[t] = u.x * un.y - un.x * u.y;
    for (int q = 0; q < 4; q++) {
      const double2 from = s_u[near(q - 2)], to = s_u[near(q - 1)];
      e[q] = pbc(make_double2(to.x - from.x, to.y - from.y));
    }
  }
  __syncthreads();
  const auto ring_sums = [&]() {
    for (int q = w; q < nrings; q += W) {
      const int f = s_rfirst[q], n = s_rlen[q];
      double x = 0.0;
      for (int c = wl; c < n; c += 32) x += s_dot[f + c];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kAll, x, o);
      if (wl == 0) s_dot[f] = x;
      __syncwarp();
    }
    __syncthreads();
  };
  ring_sums();
  double formed[5][4] = {};
  double2 cv = make_double2(0.0, 0.0), av = cv;
  int pairs = 0;
  if (on) {
    const double sum = s_dot[lf], area = 0.5 * fabs(sum), a0 = g.a0[tp.x];
    const int vp = tile.x + near(-1), vn = tile.x + near(1);
    for (int d = 0; d < 5; d++) {
      // vertex v + d - 2 moves along x (e1) and y (e2)
      Pair<HD> sg[4];
      for (int q = 0; q < 4; q++) {
        const double sx = q + 1 == d ? 1.0 : (q == d ? -1.0 : 0.0);  // segment q runs from v + q - 2 to v + q - 1
        sg[q] = Pair<HD>{HD{e[q].x, sx, 0.0, 0.0}, HD{e[q].y, 0.0, sx, 0.0}};
      }
      Pair<HD> F{num<HD>(0.0), num<HD>(0.0)};
      HD E = num<HD>(0.0);
      shape_hd<HD>(p, num<HD>(p.ea), num<HD>(p.el), num<HD>(p.eb), sg[2], sg[1], sg[0], sg[3], num<HD>(area), a0, nvr,
                   num<HD>(g.l0[v]), num<HD>(g.l0[vp]), g.theta0[vp], g.theta0[v], g.theta0[vn], F, E);
      formed[d][0] = F.x.b;
      formed[d][1] = F.x.c;
      formed[d][2] = F.y.b;
      formed[d][3] = F.y.c;
    }
    const double2 npd = make_double2(e[2].x + e[1].x, e[2].y + e[1].y);
    const double sgn = sum >= 0.0 ? 0.5 : -0.5, co = 0.5 * p.ea / (a0 * a0);
    av = make_double2(sgn * npd.y, -sgn * npd.x);
    cv = make_double2(-co * npd.y, co * npd.x);
    const double2 x = g.pos[v];
    const double ri = g.rad[v];
    const int cnt = min(g.nbr_cnt[v], g.nbr_cap);
    for (int s = 0; s < cnt; s++) {
      const int j = g.nbr[(size_t)s * p.nv + v];
      const double2 xj = g.pos[j];
      const Pair<HD> dl = pbc2_hd(Pair<HD>{HD{x.x, 1.0, 0.0, 0.0}, HD{x.y, 0.0, 1.0, 0.0}},
                                  Pair<HD>{num<HD>(xj.x), num<HD>(xj.y)}, bx);
      Pair<HD> F{num<HD>(0.0), num<HD>(0.0)};
      HD E = num<HD>(0.0);
      pair_force_hd<POT>(g, dl, num<HD>(ri + g.rad[j]), F, E);
      if (F.x.b != 0.0 || F.x.c != 0.0 || F.y.b != 0.0 || F.y.c != 0.0) {
        const double2 kxy = make_double2(F.x.b, 0.5 * (F.x.c + F.y.b));
        if (pairs < kHeld) {
          s_kxy[pairs][t] = kxy;
          s_kyy[pairs][t] = F.y.c;
          s_kj[pairs][t] = j;
        } else {
          const size_t at = (size_t)pairs * p.nv + v;
          ks.kxy[at] = kxy;
          ks.kyy[at] = F.y.c;
          ks.kj[at] = j;
        }
        pairs++;
      }
    }
  }
  double B[5][4];  // F_v = sum over d of B[d + 2] u(v + d): xx, xy, yx, yy
#pragma unroll
  for (int d = 0; d < 5; d++)
#pragma unroll
    for (int q = 0; q < 4; q++) B[d][q] = formed[d][q];
  double2* xg = reinterpret_cast<double2*>(a.x);
  double2* rg = reinterpret_cast<double2*>(a.r);
  double2* pg = reinterpret_cast<double2*>(a.p);
  double2* zg = reinterpret_cast<double2*>(a.z);
  const double2 zero = make_double2(0.0, 0.0);
  double2 x = on ? xg[v] : zero, r = on ? rg[v] : zero, pv = on ? pg[v] : zero, z = zero;
  double m0 = 1.0, m1 = 0.0, m2 = 1.0;
  if (on && a.minv) {
    m0 = a.minv[(size_t)3 * v];
    m1 = a.minv[(size_t)3 * v + 1];
    m2 = a.minv[(size_t)3 * v + 2];
  }
  const int l0 = near(-2), l1 = near(-1), l3 = near(1), l4 = near(2);
  __syncthreads();  // every warp has read its rings' area sums; s_dot is rewritten from here on
  double rr = st0.rr, rz = st0.rz, beta = 0.0, zx = 0.0, zy = 0.0;
  long long iters = st0.iters;
  unsigned long long bar = st0.bar / gridDim.x;
  int done = 0, bad = 0;
  // the sums of up to four values over the grid, in s_tot; false: a wait gave up
  const auto all_sums = [&](double (&acc)[4], int n) {
    for (int q = 0; q < n; q++) {
      double y = acc[q];
      for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(kAll, y, o);
      if (wl == 0) s_part[w][q] = y;
    }
    __syncthreads();
    if (t == 0) {
      for (int q = 0; q < n; q++) {
        double y = 0.0;
        for (int u = 0; u < W; u++) y += s_part[u][q];
        a.partials[(size_t)8 * blockIdx.x + q + (n == 4 ? 4 : 0)] = y;
      }
      s_ok = cg_wait(st, bar + 1, ks.spin_limit) ? 1 : 0;
    }
    bar++;
    __syncthreads();
    if (!s_ok) return false;
    for (int q = w; q < n; q += W) {
      double y = 0.0;
      for (int b = wl; b < (int)gridDim.x; b += 32) y += __ldcg(a.partials + (size_t)8 * b + q + (n == 4 ? 4 : 0));
      for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(kAll, y, o);
      if (wl == 0) s_tot[q] = y;
    }
    __syncthreads();
    return true;
  };
  for (int it = 0; it < ks.max_iters && !done; it++) {
    double2* mine = ks.pold[it & 1];
    const double2* last = ks.pold[(it & 1) ^ 1];
    s_u[t] = pv;
    s_dot[t] = av.x * pv.x + av.y * pv.y;
    if (on) mine[v] = pv;
    // the neighbours' directions: those of the held pairs are on their way
    // while the ring sums are formed
    const auto direction = [&](int j, double2& zj, double2& oj) {
      if (it == 0) {
        oj = pg[j];  // written before this launch, rewritten after its last barrier
        zj = zero;
      } else {
        zj = __ldcg(zg + j);
        oj = __ldcg(last + j);
      }
    };
    const double bt = it == 0 ? 1.0 : beta;
    double2 zj[kHeld], oj[kHeld];
#pragma unroll
    for (int s = 0; s < kHeld; s++) {
      zj[s] = oj[s] = zero;
      if (s < pairs) direction(s_kj[s][t], zj[s], oj[s]);
    }
    __syncthreads();
    ring_sums();
    double2 F = zero;
    const auto add_pair = [&](double2 kxy, double kyy, double2 zp, double2 op) {
      const double dx = pv.x - ((zp.x - zx) + bt * op.x), dy = pv.y - ((zp.y - zy) + bt * op.y);
      F.x += kxy.x * dx + kxy.y * dy;
      F.y += kxy.y * dx + kyy * dy;
    };
    if (on) {
      const double area = s_dot[lf];
      const double2 u0 = s_u[l0], u1 = s_u[l1], u3 = s_u[l3], u4 = s_u[l4];
      F.x = B[0][0] * u0.x + B[0][1] * u0.y + B[1][0] * u1.x + B[1][1] * u1.y + B[2][0] * pv.x + B[2][1] * pv.y +
            B[3][0] * u3.x + B[3][1] * u3.y + B[4][0] * u4.x + B[4][1] * u4.y + cv.x * area;
      F.y = B[0][2] * u0.x + B[0][3] * u0.y + B[1][2] * u1.x + B[1][3] * u1.y + B[2][2] * pv.x + B[2][3] * pv.y +
            B[3][2] * u3.x + B[3][3] * u3.y + B[4][2] * u4.x + B[4][3] * u4.y + cv.y * area;
#pragma unroll
      for (int s = 0; s < kHeld; s++)
        if (s < pairs) add_pair(s_kxy[s][t], s_kyy[s][t], zj[s], oj[s]);
      for (int s = kHeld; s < pairs; s++) {
        const size_t at = (size_t)s * p.nv + v;
        double2 zp, op;
        direction(ks.kj[at], zp, op);
        add_pair(ks.kxy[at], ks.kyy[at], zp, op);
      }
    }
    const double hx = -F.x, hy = -F.y;
    double acc[4] = {hx, hy, pv.x * hx + pv.y * hy, 0.0};
    if (!all_sums(acc, 3)) return;
    const double mx = s_tot[0] / a.nv, my = s_tot[1] / a.nv, php = s_tot[2];
    if (!(php > 0.0)) {
      bad = done = 1;
      break;
    }
    const double alpha = rz / php;
    if (on) {
      x = make_double2(x.x + alpha * pv.x, x.y + alpha * pv.y);
      r = make_double2(r.x - alpha * (hx - mx), r.y - alpha * (hy - my));
      z = make_double2(m0 * r.x + m1 * r.y, m1 * r.x + m2 * r.y);
      zg[v] = z;
    }
    double acc2[4] = {r.x * r.x + r.y * r.y, r.x * z.x + r.y * z.y, z.x, z.y};
    if (!all_sums(acc2, 4)) return;
    rr = s_tot[0];
    beta = s_tot[1] / rz;
    rz = s_tot[1];
    zx = s_tot[2] / a.nv;
    zy = s_tot[3] / a.nv;
    iters++;
    if (!(sqrt(rr / st0.bb) > st0.tol) || iters >= st0.max_iters) done = 1;
    if (on) pv = make_double2((z.x - zx) + beta * pv.x, (z.y - zy) + beta * pv.y);
  }
  // every product of this launch is behind a barrier: the vectors go back
  if (on) {
    xg[v] = x;
    rg[v] = r;
    pg[v] = pv;
  }
  if (blockIdx.x == 0 && t == 0) {
    st->rr = rr;
    st->rz = rz;
    st->iters = iters;
    st->bad = bad;
    st->done = done;
  }
}

namespace {
using CgStepsFn = void (*)(DiffArgs, CgArgs, CgSteps);
template <int BLOCK>
CgStepsFn cg_steps_fn(int pot) {
  switch (pot) {
    case POT_HARMONIC: return k_cg_steps<POT_HARMONIC, BLOCK>;
    case POT_LJ: return k_cg_steps<POT_LJ, BLOCK>;
    case POT_ADHESIVE: return k_cg_steps<POT_ADHESIVE, BLOCK>;
    default: return k_cg_steps<POT_WCA, BLOCK>;
  }
}
CgStepsFn cg_steps_of(int pot, int block) {
  return block == 64 ? cg_steps_fn<64>(pot) : (block == 96 ? cg_steps_fn<96>(pot) : cg_steps_fn<128>(pot));
}
}  // namespace

int cg_steps_max_blocks(int pot, int block) {
  const CgStepsFn fn = cg_steps_of(pot, block);
  int dev = 0, sms = 0, occ = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, block, 0) != cudaSuccess) return 0;
  return occ * sms;
}

cudaError_t launch_cg_steps(cudaStream_t st, int pot, int block, const DiffArgs& g, const CgArgs& a, const CgSteps& k) {
  const CgStepsFn fn = cg_steps_of(pot, block);
  fn<<<k.ntiles, block, 0, st>>>(g, a, k);
  return cudaGetLastError();
}

int cg_blocks(int nv) { return std::max(1, std::min(148, (nv + kCgBlock - 1) / kCgBlock)); }

void launch_cg_prec(cudaStream_t st, int nv, const double* fhd, double* minv) {
  k_cg_prec<<<(nv + 127) / 128, 128, 0, st>>>(nv, fhd, minv);
}

void launch_cg_start(cudaStream_t st, const CgArgs& a, double tol, long long max_iters) {
  k_cg_start<<<1, 1024, 0, st>>>(a, tol, max_iters);
}

void launch_cg_iteration(cudaStream_t st, const CgArgs& a) {
  k_cg_hp<<<a.nblk, kCgBlock, 0, st>>>(a);
  k_cg_alpha<<<1, 1, 0, st>>>(a);
  k_cg_update<<<a.nblk, kCgBlock, 0, st>>>(a);
  k_cg_beta<<<1, 1, 0, st>>>(a);
  k_cg_direction<<<a.nblk, kCgBlock, 0, st>>>(a);
}

}  // namespace cr
