// adjoint.cu — discrete adjoint of the time step and the misfit gradient.
//
// J = 1/2 sum_n sum_r |d_n,r - obs_n,r|^2 over the vx and vz traces.  The
// gradient is the exact transpose of the forward step (plain in-place
// path, plain.cu), taken stage by stage in reverse:
//
//   forward step n:  V (velocity, CPML psi_sigma)  ->  receivers  ->
//                    S (SLS stress + memory variables, CPML psi_v, free
//                    surface)  ->  explosive sources  ->  stress images
//   reverse step n:  images^T -> S^T -> r^T (v += -D^T rbar) -> residual at
//                    the receivers -> V^T -> d^T (sigma += -D^T dbar)
//
// The transpose of ddxp is -ddxm (and of ddzp, -ddzm) over cells whose
// adjoint is zero outside the update region; each psi recursion
// psi' = b psi + a d, d~ = d/kappa + psi' transposes to
// dbar = dbar~/kappa + a (psibar' + dbar~), psibar = b (psibar' + dbar~).
//
// The reverse sweep runs on 16-byte groups of cells from TMA boxes; every plane
// of the workspace has rows of a multiple of 4 cells, whatever the grid's, and
// the forward sweeps step the split pair on the same slots.
//
// Memory: the state (v, sigma, M and the current psi set) is stored every
// K (default ceil(sqrt(nt))) steps; each segment is recomputed forward into
// K + 1 state slots and walked backwards.  Wavefields and the adjoint state
// are in the plan's precision; gradients and the misfit accumulate in FP64,
// each cell gathering its own terms (no atomics, deterministic).
//
// Gradients are with respect to the medium planes (rho, c11, c13, c33,
// c55, tau) — for ISO c13 = lambda and c55 = mu carry dJ/dlambda and
// dJ/dmu.  vi_gradient_velocity maps them to (vp, vs, rho, 1/Q) and, for
// VTI, vi_gradient_thomsen to the Thomsen (epsilon, delta).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "fused.cuh"
#include "nvtx.cuh"
#include "fused_tma.cuh"
#include "gradient.cuh"
#include "pdl.cuh"
#include "plan.cuh"
#include "split.cuh"
#include "tma.cuh"
#include "vec.cuh"

namespace vb {

namespace {

template <typename T>
struct AdjArgs {
  int nx, ld, fs;  // ld: row stride of every plane (nx rounded up to a multiple of 4)
  int Lx, Rx, Tz, Bz, wx;
  T dt;
  T Dx[4], Dz[4];
  T a1[VI_MAX_SLS], a2[VI_MAX_SLS];
  const T *rho, *c11, *c13, *c33, *c55, *tau;
  const T *c15, *c35;  // TTI couplings
  const T *tx, *tz;
  long long np, psix_plane, psiz_plane;
  int nz;
  int keep_bar;  // rbar and dbar fit in half the L2: kept there between their kernels
};

// one state slot: [vx vz sxx szz sxz M(3N)] planes, then one psi set
// (4 x-strip planes, 4 z-strip planes)
template <typename T>
struct Slot {
  T *base;
  long long np, px, pz;  // plane sizes
  int nsls;
  __host__ __device__ T *vx() const { return base; }
  __host__ __device__ T *vz() const { return base + np; }
  __host__ __device__ T *sxx() const { return base + 2 * np; }
  __host__ __device__ T *szz() const { return base + 3 * np; }
  __host__ __device__ T *sxz() const { return base + 4 * np; }
  __host__ __device__ T *m() const { return base + 5 * np; }
  __host__ __device__ T *psix() const { return base + (5 + 3 * nsls) * np; }
  __host__ __device__ T *psiz() const { return psix() + 4 * px; }
  // rounded up to 64 elements, so every slot (and every plane of it, rows
  // being a multiple of 4 cells) starts on a 16-byte boundary
  __host__ __device__ static long long size(long long np, long long px, long long pz, int nsls) {
    return ((5 + 3 * nsls) * np + 4 * px + 4 * pz + 63) / 64 * 64;
  }
};

// FP64 accumulator planes of the adjoint sweep, each cell its own terms; the
// planes of half-node or buoyancy terms (H, Q) are spread over the cells they
// average once, at the end (k_adj_finish).  H and TAU carry the factor dt, the
// others get it there.
enum { ACC_HX = 0, ACC_HZ = 1, ACC_TAU = 2, ACC_Q55 = 3, ACC_11 = 4, ACC_13 = 5, ACC_33 = 6,
       ACC_15 = 7, ACC_35 = 8, ACC_Q15 = 9, ACC_Q35 = 10 };
// ISO: C11 = C33 = lambda + 2 mu share plane ACC_11
inline int acc_planes(int kind) { return kind == VI_MEDIUM_TTI ? 11 : kind == VI_MEDIUM_VTI ? 7 : 6; }

// ---- V cells (16 bytes) of a row: 4 FP32 or 2 FP64 ------------------------
template <typename T>
struct VecW {
  static constexpr int V = 16 / (int)sizeof(T);
};
template <typename T>
struct Pk {
  T v[VecW<T>::V];
};
__device__ __forceinline__ Pk<float> ldv(const float *p) {
  const float4 q = *reinterpret_cast<const float4 *>(p);
  return {{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ Pk<double> ldv(const double *p) {
  const double2 q = *reinterpret_cast<const double2 *>(p);
  return {{q.x, q.y}};
}
// Operands the kernel only reads: the non-coherent path, so their loads are
// not ordered behind its stores; volatile, so none moves ahead of pdl_wait().
__device__ __forceinline__ Pk<float> ldn(const float *p) {
  Pk<float> q;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(q.v[0]), "=f"(q.v[1]), "=f"(q.v[2]), "=f"(q.v[3])
               : "l"(p));
  return q;
}
__device__ __forceinline__ Pk<double> ldn(const double *p) {
  Pk<double> q;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(q.v[0]), "=d"(q.v[1]) : "l"(p));
  return q;
}
// state of the kernel before last, ahead of the PDL wait: read at L2
__device__ __forceinline__ Pk<float> ldcgv(const float *p) {
  const float4 q = __ldcg(reinterpret_cast<const float4 *>(p));
  return {{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ Pk<double> ldcgv(const double *p) {
  const double2 q = __ldcg(reinterpret_cast<const double2 *>(p));
  return {{q.x, q.y}};
}
__device__ __forceinline__ float ldn1(const float *p) {
  float q;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(q) : "l"(p));
  return q;
}
__device__ __forceinline__ double ldn1(const double *p) {
  double q;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(q) : "l"(p));
  return q;
}
__device__ __forceinline__ void stv(float *p, const Pk<float> &q) {
  *reinterpret_cast<float4 *>(p) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
}
__device__ __forceinline__ void stv(double *p, const Pk<double> &q) {
  *reinterpret_cast<double2 *>(p) = make_double2(q.v[0], q.v[1]);
}
// the same with an L2 eviction policy
__device__ __forceinline__ Pk<float> ldnp(const float *p, uint64_t pol) {
  Pk<float> q;
  asm volatile("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(q.v[0]), "=f"(q.v[1]), "=f"(q.v[2]), "=f"(q.v[3])
               : "l"(p), "l"(pol));
  return q;
}
__device__ __forceinline__ Pk<double> ldnp(const double *p, uint64_t pol) {
  Pk<double> q;
  asm volatile("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
               : "=d"(q.v[0]), "=d"(q.v[1])
               : "l"(p), "l"(pol));
  return q;
}
__device__ __forceinline__ void stvp(float *p, const Pk<float> &q, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "f"(q.v[0]), "f"(q.v[1]),
               "f"(q.v[2]), "f"(q.v[3]), "l"(pol)
               : "memory");
}
__device__ __forceinline__ void stvp(double *p, const Pk<double> &q, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v2.f64 [%0], {%1, %2}, %3;" ::"l"(p), "d"(q.v[0]), "d"(q.v[1]), "l"(pol)
               : "memory");
}
template <typename T>
__device__ __forceinline__ Pk<T> splat(T s) {
  Pk<T> r;
#pragma unroll
  for (int k = 0; k < VecW<T>::V; ++k) r.v[k] = s;
  return r;
}
__device__ __forceinline__ Pk<float> pfma(const Pk<float> &a, const Pk<float> &b, const Pk<float> &c) {
  const float2 l = __ffma2_rn(make_float2(a.v[0], a.v[1]), make_float2(b.v[0], b.v[1]), make_float2(c.v[0], c.v[1]));
  const float2 h = __ffma2_rn(make_float2(a.v[2], a.v[3]), make_float2(b.v[2], b.v[3]), make_float2(c.v[2], c.v[3]));
  return {{l.x, l.y, h.x, h.y}};
}
__device__ __forceinline__ Pk<double> pfma(const Pk<double> &a, const Pk<double> &b, const Pk<double> &c) {
  return {{fma(a.v[0], b.v[0], c.v[0]), fma(a.v[1], b.v[1], c.v[1])}};
}
__device__ __forceinline__ Pk<float> pmul(const Pk<float> &a, const Pk<float> &b) {
  const float2 l = __fmul2_rn(make_float2(a.v[0], a.v[1]), make_float2(b.v[0], b.v[1]));
  const float2 h = __fmul2_rn(make_float2(a.v[2], a.v[3]), make_float2(b.v[2], b.v[3]));
  return {{l.x, l.y, h.x, h.y}};
}
__device__ __forceinline__ Pk<double> pmul(const Pk<double> &a, const Pk<double> &b) {
  return {{a.v[0] * b.v[0], a.v[1] * b.v[1]}};
}
__device__ __forceinline__ Pk<float> padd(const Pk<float> &a, const Pk<float> &b) {
  const float2 l = __fadd2_rn(make_float2(a.v[0], a.v[1]), make_float2(b.v[0], b.v[1]));
  const float2 h = __fadd2_rn(make_float2(a.v[2], a.v[3]), make_float2(b.v[2], b.v[3]));
  return {{l.x, l.y, h.x, h.y}};
}
__device__ __forceinline__ Pk<double> padd(const Pk<double> &a, const Pk<double> &b) {
  return {{a.v[0] + b.v[0], a.v[1] + b.v[1]}};
}
template <typename T>
__device__ __forceinline__ Pk<T> psub(const Pk<T> &a, const Pk<T> &b) {
  return pfma(b, splat<T>(T(-1)), a);
}
template <typename T>
__device__ __forceinline__ Pk<T> pscale(T s, const Pk<T> &a) {
  return pmul(splat<T>(s), a);
}
// out[k] = term(k, in[k]), FP64: an accumulator plane read from its staged
// tile and written straight back (32-byte stores for FP32's four cells)
__device__ __forceinline__ void st_acc(double *p, const double (&t)[4]) {
  asm volatile("st.global.L2::cache_hint.v4.f64 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "d"(t[0]), "d"(t[1]), "d"(t[2]), "d"(t[3]), "l"(l2_stream())
               : "memory");
}
__device__ __forceinline__ void st_acc(double *p, const double (&t)[2]) {
  *reinterpret_cast<double2 *>(p) = make_double2(t[0], t[1]);
}
template <typename T, typename F>
__device__ __forceinline__ void acc_add(const double *in, double *out, F term) {
  constexpr int V = VecW<T>::V;
  double t[V];
#pragma unroll
  for (int q = 0; q < V; q += 2) {
    const double2 u = *reinterpret_cast<const double2 *>(in + q);
    t[q] = term(q, u.x);
    t[q + 1] = term(q + 1, u.y);
  }
  st_acc(out, t);
}

// Staggered derivatives of a plane (staged in shared memory, row stride ld)
// at the group at u.
template <typename T>
struct RowWin {  // u[c - 4 .. c + V + 3]
  T w[VecW<T>::V + 8];
};
template <typename T>
__device__ __forceinline__ RowWin<T> ldwin(const T *u) {
  constexpr int V = VecW<T>::V;
  RowWin<T> r;
#pragma unroll
  for (int q = 0; q < (V + 8) / V; ++q) {
    const Pk<T> t = ldv(u - 4 + V * q);
#pragma unroll
    for (int k = 0; k < V; ++k) r.w[V * q + k] = t.v[k];
  }
  return r;
}
template <typename T>
__device__ __forceinline__ Pk<T> at(const RowWin<T> &r, int o) {
  Pk<T> t;
#pragma unroll
  for (int k = 0; k < VecW<T>::V; ++k) t.v[k] = r.w[4 + o + k];
  return t;
}
template <typename T>
__device__ __forceinline__ Pk<T> dxp(const RowWin<T> &r, const T *D) {
  Pk<T> s = pscale(D[0], psub(at(r, 1), at(r, 0)));
#pragma unroll
  for (int q = 1; q < 4; ++q) s = pfma(splat<T>(D[q]), psub(at(r, q + 1), at(r, -q)), s);
  return s;
}
template <typename T>
__device__ __forceinline__ Pk<T> dxm(const RowWin<T> &r, const T *D) {
  Pk<T> s = pscale(D[0], psub(at(r, 0), at(r, -1)));
#pragma unroll
  for (int q = 1; q < 4; ++q) s = pfma(splat<T>(D[q]), psub(at(r, q), at(r, -q - 1)), s);
  return s;
}
template <typename T>
__device__ __forceinline__ Pk<T> dzp(const T *u, int ld, const T *D) {
  Pk<T> s = pscale(D[0], psub(ldv(u + ld), ldv(u)));
#pragma unroll
  for (int q = 1; q < 4; ++q) s = pfma(splat<T>(D[q]), psub(ldv(u + (q + 1) * ld), ldv(u - q * ld)), s);
  return s;
}
template <typename T>
__device__ __forceinline__ Pk<T> dzm(const T *u, int ld, const T *D) {
  Pk<T> s = pscale(D[0], psub(ldv(u), ldv(u - ld)));
#pragma unroll
  for (int q = 1; q < 4; ++q) s = pfma(splat<T>(D[q]), psub(ldv(u + q * ld), ldv(u - (q + 1) * ld)), s);
  return s;
}

// The CPML strips a group touches.  Profiles outside a strip are 1/kappa =
// 1, a = b = 0 and psi counts as zero there, so one vector form serves groups
// that straddle a strip's edge; only groups whose psi cells do not lie on a
// vector boundary load and store them cell by cell.
template <typename T>
struct Strips {
  bool x, z, xvec;
  int xs[VecW<T>::V];
  long long xo, zo;
};
template <typename T>
__device__ __forceinline__ Strips<T> strips_of(const AdjArgs<T> &A, int gi0, int j) {
  constexpr int V = VecW<T>::V;
  Strips<T> s;
  s.x = gi0 < A.Lx || gi0 + V - 1 >= A.nx - A.Rx;
  const int zs = strip_z(j, A.nz, A.Tz, A.Bz);
  s.z = zs >= 0;
  s.zo = (long long)zs * A.ld + gi0;
  s.xo = (long long)j * A.wx;
  s.xvec = false;
  if (s.x) {
#pragma unroll
    for (int k = 0; k < V; ++k) s.xs[k] = strip_x(gi0 + k, A.nx, A.Lx, A.Rx);
    s.xvec = s.xs[0] >= 0 && s.xs[V - 1] == s.xs[0] + V - 1 &&
             (((s.xo + s.xs[0]) | A.psix_plane | A.nx) & (V - 1)) == 0;
  }
  return s;
}
template <typename T>
__device__ __forceinline__ Pk<T> ld_psix(const Strips<T> &s, const T *plane) {
  if (s.xvec) return ldv(plane + s.xo + s.xs[0]);
  Pk<T> r;
#pragma unroll
  for (int k = 0; k < VecW<T>::V; ++k) r.v[k] = s.xs[k] >= 0 ? plane[s.xo + s.xs[k]] : T(0);
  return r;
}
template <typename T>
__device__ __forceinline__ Pk<T> ld_psix0(const Strips<T> &s, const T *plane) {  // of a forward state
  if (s.xvec) return ldn(plane + s.xo + s.xs[0]);
  Pk<T> r;
#pragma unroll
  for (int k = 0; k < VecW<T>::V; ++k) r.v[k] = s.xs[k] >= 0 ? ldn1(plane + s.xo + s.xs[k]) : T(0);
  return r;
}
template <typename T>
__device__ __forceinline__ void st_psix(const Strips<T> &s, T *plane, const Pk<T> &q) {
  if (s.xvec) {
    stv(plane + s.xo + s.xs[0], q);
    return;
  }
#pragma unroll
  for (int k = 0; k < VecW<T>::V; ++k)
    if (s.xs[k] >= 0) plane[s.xo + s.xs[k]] = q.v[k];
}
template <typename T>
__device__ __forceinline__ Pk<T> ld_tabx(const AdjArgs<T> &A, const Strips<T> &s, int row, int gi0) {
  const T *p = A.tx + row * A.nx + gi0;
  if (s.xvec) return ldn(p);
  Pk<T> r;
#pragma unroll
  for (int k = 0; k < VecW<T>::V; ++k) r.v[k] = ldn1(p + k);
  return r;
}
// Asks for the strips' operands of two x and two z derivatives ahead of the
// PDL wait (psi of the forward state and of the adjoint, the profiles): a tile
// in a strip otherwise starts four more rounds of loads after its boxes.
__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
template <typename T>
__device__ __forceinline__ void prefetch_strips(const AdjArgs<T> &A, const Strips<T> &s, int gi0, int j,
                                                const Slot<T> &x0, const T *pxb, const T *pzb, int px0, int px1,
                                                int pz0, int pz1) {
  if (s.x) {
    const int xs = s.xs[0] >= 0 ? s.xs[0] : s.xs[VecW<T>::V - 1];
    const long long o0 = px0 * A.psix_plane + s.xo + xs, o1 = px1 * A.psix_plane + s.xo + xs;
    prefetch_l1(x0.psix() + o0);
    prefetch_l1(x0.psix() + o1);
    prefetch_l1(pxb + o0);
    prefetch_l1(pxb + o1);
#pragma unroll
    for (int q = 0; q < 6; ++q) prefetch_l1(A.tx + q * A.nx + gi0);
  }
  if (s.z) {
    const long long o0 = pz0 * A.psiz_plane + s.zo, o1 = pz1 * A.psiz_plane + s.zo;
    prefetch_l1(x0.psiz() + o0);
    prefetch_l1(x0.psiz() + o1);
    prefetch_l1(pzb + o0);
    prefetch_l1(pzb + o1);
#pragma unroll
    for (int q = 0; q < 6; ++q) prefetch_l1(A.tz + q * A.nz + j);
  }
}
// forward derivative d -> d/kappa + (b psi + a d), psi of the step's start
template <typename T>
__device__ __forceinline__ void cpml_fwd_x(const AdjArgs<T> &A, const Strips<T> &s, int gi0, const T *psix, int pl,
                                           int tik, int ta, int tb, Pk<T> &d) {
  const Pk<T> p = pfma(ld_tabx(A, s, tb, gi0), ld_psix0(s, psix + pl * A.psix_plane),
                       pmul(ld_tabx(A, s, ta, gi0), d));
  d = pfma(d, ld_tabx(A, s, tik, gi0), p);
}
template <typename T>
__device__ __forceinline__ void cpml_fwd_z(const AdjArgs<T> &A, const Strips<T> &s, int j, const T *psiz, int pl,
                                           int tik, int ta, int tb, Pk<T> &d) {
  const Pk<T> p = pfma(splat<T>(A.tz[tb * A.nz + j]), ldn(psiz + pl * A.psiz_plane + s.zo),
                       pscale(A.tz[ta * A.nz + j], d));
  d = pfma(d, splat<T>(A.tz[tik * A.nz + j]), p);
}
// the transpose: P = psibar + dbar; psibar = b P, dbar = dbar/kappa + a P
template <typename T>
__device__ __forceinline__ void cpml_adj_x(const AdjArgs<T> &A, const Strips<T> &s, int gi0, T *psix, int pl, int tik,
                                           int ta, int tb, Pk<T> &d) {
  T *q = psix + pl * A.psix_plane;
  const Pk<T> P = padd(ld_psix(s, (const T *)q), d);
  st_psix(s, q, pmul(ld_tabx(A, s, tb, gi0), P));
  d = pfma(d, ld_tabx(A, s, tik, gi0), pmul(ld_tabx(A, s, ta, gi0), P));
}
template <typename T>
__device__ __forceinline__ void cpml_adj_z(const AdjArgs<T> &A, const Strips<T> &s, int j, T *psiz, int pl, int tik,
                                           int ta, int tb, Pk<T> &d) {
  T *q = psiz + pl * A.psiz_plane + s.zo;
  const Pk<T> P = padd(ldv((const T *)q), d);
  stv(q, pscale(A.tz[tb * A.nz + j], P));
  d = pfma(d, splat<T>(A.tz[tik * A.nz + j]), pscale(A.tz[ta * A.nz + j], P));
}

// L2 eviction priorities: dbar and rbar, written by one kernel and read by the
// next, are kept; the forward states (read once per kernel), the memory
// variables' adjoints and the accumulators (whose next visit is a whole step
// later) go first.  Without them 163 MB per 1024 x 512 VTI step reached DRAM;
// the reverse step 48.5 -> 41 us with 8-row tiles.
template <typename T>
__device__ __forceinline__ uint64_t bar_policy(const AdjArgs<T> &A) {
  return A.keep_bar ? l2_keep() : l2_normal();
}

// ---- the reverse step ----------------------------------------------------
// One reverse step of ISO and VTI media is two kernels, of TTI three:
//
//   k_adj_stress     sigma adjoint of the step (divergence and images
//                    transposed, below), then S^T per cell
//   k_adj_vel        v += -D^T rbar, receiver residuals, V^T per cell
//
//   TTI: k_adj_sigma_tti (sigma adjoint, forward effective rates),
//        k_adj_stress_tti (S^T, a 3 x 3 neighbourhood), k_adj_vel
//
// Every stage that reads only its own cell is in the kernel that produces its
// operands; what crosses cells goes through the planes rbar (strain-rate
// adjoints) and dbar (stress-divergence adjoints).  The ghost rows above a
// free surface are never stored: their adjoint is -D^T dbar on rows that hold
// nothing else, so the rows they mirror add it directly (adj_sigma).  The
// half-node averages and the buoyancy means are linear and do not change with
// time, so their transposes are taken once, after the sweep (k_adj_finish).
//
// A thread has up to 70 16-byte operands: loaded straight into registers they
// come in a dozen dependent rounds of L2 latency (k_adj_stress ran 33 us at
// 1024 x 512, issue slots 15 % busy, 12 us from start to end of a CTA).  One
// thread therefore requests the tile's boxes by TMA at the start of the CTA,
// the planes of the kernel before last ahead of the PDL wait; only the
// per-cell operands read once into few registers (the memory-variable sums,
// the medium) stay ordinary loads.

// Adjoint tile: rows of 512 bytes, 4 rows, one group of V cells per thread
// (1024 x 512 VTI, whole reverse step: 40.3 us; 256 bytes x 8 rows 41.8, x 4
// rows with 64 threads 41.9).
template <typename T>
struct AdjGeom {
  static constexpr int V = VecW<T>::V, TX = 512 / (int)sizeof(T), TZ = 4, NT = TX / V * TZ;
  static constexpr int WX = TX + 8;      // box with the x taps
  static constexpr int HZ = TZ + 7;      // box with the z taps of one operator
  static constexpr int WC = TX + V;      // box with one group to the right
  static constexpr int E = (int)sizeof(T);
};
constexpr int up128(int b) { return (b + 127) / 128 * 128; }

// TMA maps: dbar / rbar with x taps and with z taps, the forward states (all
// slots one 4D map: column, row, plane, slot), the adjoint planes, the
// accumulators, c55.  Kernels take the ones they use, in this order.
struct AdjMaps {
  CUtensorMap px, pz, st_a, st_b, st_c, own, mem, acc, cc, c2, c3;
};

// Shared memory of a kernel: the barrier, then its boxes (128-byte aligned).
template <typename T, int NACC, int NM>
struct StressSmem {
  using G = AdjGeom<T>;
  static constexpr int D0 = 128, D1 = D0 + up128(G::WX * G::TZ * G::E), D2 = D1 + up128(G::TX * G::HZ * G::E),
                       D3 = D2 + up128(G::WX * G::TZ * G::E), VX = D3 + up128(G::TX * G::HZ * G::E),
                       VZ = VX + up128(G::WX * G::HZ * G::E), SB = VZ + up128(G::WX * G::HZ * G::E),
                       MB = SB + 3 * G::TX * G::TZ * G::E, CC = MB + NM * G::TX * G::TZ * G::E,
                       ACC = CC + up128(G::WC * (G::TZ + 1) * G::E), SIZE = ACC + NACC * G::TX * G::TZ * 8;
  static constexpr int TAPS = (2 * G::WX * G::TZ + 2 * G::TX * G::HZ) * G::E;  // dbar boxes
  static constexpr int VBOX = 2 * G::WX * G::HZ * G::E;
  static constexpr int BYTES = TAPS + VBOX + (3 + NM) * G::TX * G::TZ * G::E + G::WC * (G::TZ + 1) * G::E +
                               NACC * G::TX * G::TZ * 8;
};
template <typename T>
struct VelSmem {
  using G = AdjGeom<T>;
  static constexpr int R0 = 128, R1 = R0 + up128(G::WX * G::TZ * G::E), R2 = R1 + up128(G::TX * G::HZ * G::E),
                       R3 = R2 + up128(G::TX * G::HZ * G::E), SXX = R3 + up128(G::WX * G::TZ * G::E),
                       SXZ = SXX + up128(G::WX * G::TZ * G::E), SZZ = SXZ + up128(G::WX * G::HZ * G::E),
                       VB = SZZ + up128(G::TX * G::HZ * G::E), ACC = VB + 2 * G::TX * G::TZ * G::E,
                       SIZE = ACC + 2 * G::TX * G::TZ * 8;
  static constexpr int BYTES = (3 * G::WX * G::TZ + 3 * G::TX * G::HZ + G::WX * G::HZ + 2 * G::TX * G::TZ) * G::E +
                               2 * G::TX * G::TZ * 8;
};
template <typename T>
struct TtiSmem {  // k_adj_stress_tti: tile and a one-cell ring (x from the group before)
  using G = AdjGeom<T>;
  static constexpr int RH = G::TZ + 2, RING = up128(G::WX * RH * G::E), NACC = 9;
  // the three planes of a 3D box follow each other without padding
  static constexpr int RP = G::WX * RH * G::E;
  static constexpr int FE = 128, SB = FE + up128(3 * RP), C15 = SB + up128(3 * RP), C35 = C15 + RING, CC = C35 + RING,
                       ACC = CC + up128(G::WC * (G::TZ + 1) * G::E), SIZE = ACC + NACC * G::TX * G::TZ * 8;
  static constexpr int BYTES = 8 * RP + G::WC * (G::TZ + 1) * G::E + NACC * G::TX * G::TZ * 8;
};

struct AdjTile {
  int x0, z0, lx, r, gi0, j;
  bool act;
};
template <typename T>
__device__ __forceinline__ AdjTile adj_tile(const AdjArgs<T> &A, int ntx) {
  using G = AdjGeom<T>;
  AdjTile t;
  const int tile = blockIdx.x;
  t.r = threadIdx.x / (G::TX / G::V);
  t.lx = G::V * (threadIdx.x % (G::TX / G::V));
  t.x0 = L + (tile % ntx) * G::TX;
  t.z0 = L + (tile / ntx) * G::TZ;
  t.gi0 = t.x0 + t.lx;
  t.j = t.z0 + t.r;
  t.act = t.gi0 < A.nx - L && t.j < A.nz - L;
  return t;
}
// every thread: the boxes have landed (or the wait gave up: kErrTimeout)
__device__ __forceinline__ bool boxes_landed(uint64_t *bar, int *err) {
  const bool ok = mbar_wait_bounded(bar, 0, 1u << 22);
  if (!__syncthreads_or(!ok)) return true;
  if (threadIdx.x == 0) {
    atomicOr(err, kErrTimeout);
    mbar_wait_bounded(bar, 0, 1u << 22);
  }
  return false;
}
// lanes of a group past the update region (nx % V != 0)
template <typename T>
__device__ __forceinline__ void zero_outside(Pk<T> &q, int n) {
#pragma unroll
  for (int k = 0; k < VecW<T>::V; ++k)
    if (k >= n) q.v[k] = T(0);
}
// The medium of lanes past the update region is the caller's and may be anything
// (0 x inf is NaN): their moduli and tau count as 0, what divides as 1.
template <typename T>
__device__ __forceinline__ void set_outside(Pk<T> &q, int n, T v) {
#pragma unroll
  for (int k = 0; k < VecW<T>::V; ++k)
    if (k >= n) q.v[k] = v;
}
// u[k + 1] of the group, u[V] from `next`
template <typename T>
__device__ __forceinline__ T right_of(const Pk<T> &u, int k, T next) {
  constexpr int V = VecW<T>::V;
  return k + 1 < V ? u.v[k + 1 < V ? k + 1 : 0] : next;
}

// sigma adjoint before the stress stage of the step: sigma - D^T dbar of the
// velocity stage after it, with the images transposed: row L + k also takes
// what -D^T dbar leaves on the ghost rows L - k (szz) and L - 1 - k (sxz),
// whose only terms are those dbar rows at or below the surface (within four
// rows of row L + k, so inside its boxes).  The image terms join the derivative
// first, so the running sigma adjoint is rounded once.  sb, d0 .. d3: the group's
// place in the boxes.
template <typename T>
__device__ __forceinline__ void adj_sigma(const AdjArgs<T> &A, const AdjTile &t, const T *sb, const T *d0, const T *d1,
                                          const T *d2, const T *d3, Pk<T> &bxx, Pk<T> &bzz, Pk<T> &bxz) {
  using G = AdjGeom<T>;
  bxx = psub(ldv(sb), dxm(ldwin(d0), A.Dx));
  Pk<T> tzz = dzm(d3, G::TX, A.Dz), txz = padd(dzp(d1, G::TX, A.Dz), dxp(ldwin(d2), A.Dx));
  if (A.fs && t.j < 2 * L) {
    const int k = t.j - L;
    Pk<T> izz = splat<T>(T(0)), ixz = izz;
    for (int q = k; q < 4; ++q) {  // grid row L - k + q: 2 k - q rows up from row L + k
      const T d = A.Dz[q];
      ixz = pfma(splat<T>(d), ldv(d1 + (q - 2 * k) * G::TX), ixz);
      if (k >= 1) izz = pfma(splat<T>(d), ldv(d3 + (q - 2 * k) * G::TX), izz);
    }
    tzz = psub(tzz, izz);
    txz = psub(txz, ixz);
  }
  bzz = psub(ldv(sb + G::TX * G::TZ), tzz);
  bxz = psub(ldv(sb + 2 * G::TX * G::TZ), txz);
  if (t.gi0 + G::V > A.nx - L) {
    zero_outside(bxx, A.nx - L - t.gi0);
    zero_outside(bzz, A.nx - L - t.gi0);
    zero_outside(bxz, A.nx - L - t.gi0);
  }
}

// Effective rates of the forward step, rounded as its kernels round them: with
// 1 + tau as one FP32 number.  The transpose uses the same number (adj_memory);
// with tau applied by itself it transposed a slightly other step, and the FP32
// gradient was 10 to 17 % further from the 64-bit one in rho, 4 to 12 % in the
// other planes (256 x 160, 48 shots; with it, as far as unfused transposes).
template <typename T>
__device__ __forceinline__ Pk<T> effective_rate(const Pk<T> &tau, const Pk<T> &rt, const Pk<T> &S) {
  return pfma(padd(tau, splat<T>(T(1))), rt, pmul(tau, S));
}
// Forward strain rates of the step from the new velocities (vx, vz: the
// group's place in the boxes) and the CPML memory before it (x0): xx, zz, xz.
template <typename T>
__device__ __forceinline__ void adj_rates(const AdjArgs<T> &A, const Slot<T> &x0, const Strips<T> &s, const AdjTile &t,
                                          const T *vx, const T *vz, Pk<T> (&rt)[3]) {
  using G = AdjGeom<T>;
  rt[0] = dxm(ldwin(vx), A.Dx);
  rt[1] = dzm(vz, G::WX, A.Dz);
  Pk<T> r3 = dxp(ldwin(vz), A.Dx), r2 = dzp(vx, G::WX, A.Dz);
  if (s.x) {
    cpml_fwd_x(A, s, t.gi0, (const T *)x0.psix(), PX_VX, T_IK, T_A, T_B, rt[0]);
    cpml_fwd_x(A, s, t.gi0, (const T *)x0.psix(), PX_VZ, T_IKH, T_AH, T_BH, r3);
  }
  if (s.z) {
    cpml_fwd_z(A, s, t.j, (const T *)x0.psiz(), PZ_VZ, T_IK, T_A, T_B, rt[1]);
    cpml_fwd_z(A, s, t.j, (const T *)x0.psiz(), PZ_VX, T_IKH, T_AH, T_BH, r2);
  }
  rt[2] = padd(r2, r3);
}

// From the effective-rate adjoints eb (times dt) of a group and its memory
// variables' adjoints mb(q): memory variables (plane 0 at mp), CPML memory,
// and the strain-rate adjoints rbar.
template <typename T, int N, typename F>
__device__ __forceinline__ void adj_memory(const AdjArgs<T> &A, F mb, T *mp, T *pxb, T *pzb, const Strips<T> &s,
                                           const AdjTile &t, long long c, bool surf, const Pk<T> &tau,
                                           const Pk<T> (&eb)[3], T *rbar) {
  const long long np = A.np;
  Pk<T> rtb[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) rtb[k] = N > 0 ? pmul(padd(tau, splat<T>(T(1))), eb[k]) : eb[k];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const T e1 = A.dt * A.a1[n], e2 = T(1) + A.dt * A.a2[n];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      T *q = mp + (k * N + n) * np;
      if (surf && k == 1) {  // Mzz' = 0 on the surface
        stvp(q, splat<T>(T(0)), l2_stream());
      } else {
        const Pk<T> m = mb(k * N + n);
        rtb[k] = pfma(splat<T>(e1), m, rtb[k]);
        stvp(q, pfma(splat<T>(e2), m, pmul(tau, eb[k])), l2_stream());  // one rounding at the size of m
      }
    }
  }
  Pk<T> rb[4] = {rtb[0], rtb[1], rtb[2], rtb[2]};
  if (s.x) {
    cpml_adj_x(A, s, t.gi0, pxb, PX_VX, T_IK, T_A, T_B, rb[0]);
    cpml_adj_x(A, s, t.gi0, pxb, PX_VZ, T_IKH, T_AH, T_BH, rb[3]);
  }
  if (s.z) {
    cpml_adj_z(A, s, t.j, pzb, PZ_VZ, T_IK, T_A, T_B, rb[1]);
    cpml_adj_z(A, s, t.j, pzb, PZ_VX, T_IKH, T_AH, T_BH, rb[2]);
  }
  if (t.gi0 + VecW<T>::V > A.nx - L)
#pragma unroll
    for (int k = 0; k < 4; ++k) zero_outside(rb[k], A.nx - L - t.gi0);
#pragma unroll
  for (int k = 0; k < 4; ++k) stvp(rbar + k * np + c, rb[k], bar_policy(A));
}

// S of a group: the sums of its memory variables
template <typename T, int N>
__device__ __forceinline__ void memory_sums(const T *m, long long np, Pk<T> (&S)[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    S[k] = splat<T>(T(0));
#pragma unroll
    for (int n = 0; n < N; ++n) S[k] = padd(S[k], ldnp(m + (k * N + n) * np, l2_stream()));
  }
}

// sigma adjoint and S^T of one step, ISO and VTI.  slot: of the step's start.
template <typename T, int KIND, int N>
struct StressK {
  static constexpr int NACC = KIND == VI_MEDIUM_ISO ? 4 : 5;
  using S = StressSmem<T, NACC, 3 * N>;
};
template <typename T, int KIND, int N>
__global__ void __launch_bounds__(AdjGeom<T>::NT, N <= 3 ? 2 : 1)
    k_adj_stress(const __grid_constant__ AdjArgs<T> A, const __grid_constant__ AdjMaps maps, Slot<T> x0, int slot,
                 int ntx, T *__restrict__ sb, T *__restrict__ mb, T *__restrict__ pxb, T *__restrict__ pzb,
                 T *__restrict__ rbar, double *__restrict__ acc, int *err) {
  using G = AdjGeom<T>;
  using SM = typename StressK<T, KIND, N>::S;
  constexpr int V = G::V, PL = G::TX * G::TZ;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
  auto box = [&](int o) { return reinterpret_cast<T *>(smem + o); };
  const AdjTile t = adj_tile(A, ntx);
  const long long ld = A.ld, np = A.np, c = (long long)t.j * ld + t.gi0;
  if (threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  Pk<T> S[3], tau{}, C11{}, C13{}, C33{};
  if (t.act) {
    memory_sums<T, N>((const T *)x0.m() + c, np, S);
    if (N > 0) tau = ldn(A.tau + c);
    C13 = ldn(A.c13 + c);
    if (KIND != VI_MEDIUM_ISO) {
      C11 = ldn(A.c11 + c);
      C33 = ldn(A.c33 + c);
    }
  }
  const Strips<T> s = strips_of(A, t.gi0, t.j);
  if (t.act) prefetch_strips(A, s, t.gi0, t.j, x0, pxb, pzb, PX_VX, PX_VZ, PZ_VZ, PZ_VX);
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar, SM::BYTES);
    tma_load_4d_hint(box(SM::VX), &maps.st_a, t.x0 - 4, t.z0 - 3, 0, slot + 1, bar, l2_stream());  // new velocities
    tma_load_4d_hint(box(SM::VZ), &maps.st_a, t.x0 - 4, t.z0 - 4, 1, slot + 1, bar, l2_stream());
    tma_load_2d(box(SM::CC), &maps.cc, t.x0, t.z0, bar);
    tma_load_3d(box(SM::SB), &maps.own, t.x0, t.z0, 0, bar);
    if (N > 0) tma_load_3d_hint(box(SM::MB), &maps.mem, t.x0, t.z0, 0, bar, l2_stream());
    tma_load_3d_hint(smem + SM::ACC, &maps.acc, t.x0, t.z0, 0, bar, l2_stream());
    pdl_wait();  // dbar: the previous kernel's
    tma_load_3d_hint(box(SM::D0), &maps.px, t.x0 - 4, t.z0, 0, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::D1), &maps.pz, t.x0, t.z0 - 3, 1, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::D2), &maps.px, t.x0 - 4, t.z0, 2, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::D3), &maps.pz, t.x0, t.z0 - 4, 3, bar, bar_policy(A));
  }
  pdl_wait();  // every thread, before its first store
  pdl_release();
  if (!boxes_landed(bar, err) || !t.act) return;
  const bool surf = A.fs && t.j == L;
  const int ow = t.r * G::WX + t.lx + 4, oz = t.r * G::TX + t.lx, oc = t.r * G::WC + t.lx;
  Pk<T> bxx, bzz, bxz;
  adj_sigma(A, t, box(SM::SB) + oz, box(SM::D0) + ow, box(SM::D1) + oz + 3 * G::TX, box(SM::D2) + ow,
            box(SM::D3) + oz + 4 * G::TX, bxx, bzz, bxz);
  stv(sb + c, bxx);
  stv(sb + np + c, surf ? splat<T>(T(0)) : bzz);  // szz' = 0 on the surface
  stv(sb + 2 * np + c, bxz);
  Pk<T> rt[3], e[3];
  adj_rates(A, x0, s, t, box(SM::VX) + ow + 3 * G::WX, box(SM::VZ) + ow + 4 * G::WX, rt);
  const T *cc = box(SM::CC) + oc;
  const Pk<T> c55 = ldv(cc), c55d = ldv(cc + G::WC);
  Pk<T> C55h;
#pragma unroll
  for (int k = 0; k < V; ++k)
    C55h.v[k] = T(0.25) * (c55.v[k] + right_of(c55, k, cc[V]) + c55d.v[k] + right_of(c55d, k, cc[G::WC + V]));
  if (KIND == VI_MEDIUM_ISO) C11 = C33 = pfma(splat<T>(T(2)), c55, C13);
  if (const int n = A.nx - L - t.gi0; n < V) {
    zero_outside(tau, n);
    zero_outside(C11, n);
    zero_outside(C13, n);
    set_outside(C33, n, T(1));
    zero_outside(C55h, n);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) e[k] = N > 0 ? effective_rate(tau, rt[k], S[k]) : rt[k];
  // accumulators: plane 0 TAU, 1 Q55, 2 C11 (ISO: C11 and C33), 3 C13, 4 C33
  const double *ai = reinterpret_cast<const double *>(smem + SM::ACC) + oz;
  double *ao = acc + c;
  Pk<T> eb[3];
  if (!surf) {
    eb[0] = pscale(A.dt, pfma(C11, bxx, pmul(C13, bzz)));
    eb[1] = pscale(A.dt, pfma(C13, bxx, pmul(C33, bzz)));
    if (KIND == VI_MEDIUM_ISO) {
      acc_add<T>(ai + 2 * PL, ao + 2 * np, [&](int k, double g) {
        return fma((double)bxx.v[k], (double)e[0].v[k], fma((double)bzz.v[k], (double)e[1].v[k], g));
      });
    } else {
      acc_add<T>(ai + 2 * PL, ao + 2 * np, [&](int k, double g) { return fma((double)bxx.v[k], (double)e[0].v[k], g); });
      acc_add<T>(ai + 4 * PL, ao + 4 * np, [&](int k, double g) { return fma((double)bzz.v[k], (double)e[1].v[k], g); });
    }
    acc_add<T>(ai + 3 * PL, ao + 3 * np, [&](int k, double g) {
      return fma((double)bxx.v[k], (double)e[1].v[k], fma((double)bzz.v[k], (double)e[0].v[k], g));
    });
  } else {
    // sxx' = sxx + dt (C11 - C13^2/C33) exx
#pragma unroll
    for (int k = 0; k < V; ++k) eb[0].v[k] = A.dt * (C11.v[k] - C13.v[k] * C13.v[k] / C33.v[k]) * bxx.v[k];
    eb[1] = splat<T>(T(0));
    auto w = [&](int k) { return (double)bxx.v[k] * (double)e[0].v[k]; };
    auto f = [&](int k) { return (double)C13.v[k] / (double)C33.v[k]; };
    if (KIND == VI_MEDIUM_ISO) {
      acc_add<T>(ai + 2 * PL, ao + 2 * np, [&](int k, double g) { return g + w(k) * (1.0 + f(k) * f(k)); });
    } else {
      acc_add<T>(ai + 2 * PL, ao + 2 * np, [&](int k, double g) { return g + w(k); });
      acc_add<T>(ai + 4 * PL, ao + 4 * np, [&](int k, double g) { return g + w(k) * (f(k) * f(k)); });
    }
    acc_add<T>(ai + 3 * PL, ao + 3 * np, [&](int k, double g) { return g - 2.0 * w(k) * f(k); });
  }
  eb[2] = pscale(A.dt, pmul(C55h, bxz));
  acc_add<T>(ai + PL, ao + np, [&](int k, double g) { return fma((double)bxz.v[k], (double)e[2].v[k], g); });
  if (N > 0)
    acc_add<T>(ai, ao, [&](int k, double g) {
      double u = (double)eb[0].v[k] * ((double)rt[0].v[k] + (double)S[0].v[k]);
      u = fma((double)eb[1].v[k], (double)rt[1].v[k] + (double)S[1].v[k], u);
      return g + fma((double)eb[2].v[k], (double)rt[2].v[k] + (double)S[2].v[k], u);
    });
  const T *ms = box(SM::MB) + oz;
  adj_memory<T, N>(A, [&](int q) { return ldv(ms + q * PL); }, mb + c, pxb, pzb, s, t, c, surf, tau, eb, rbar);
}

// v += -D^T rbar, the residual at the receivers of step it, and V^T of the
// velocity stage: dbar (4 planes: sxx-x, sxz-z, sxz-x, szz-z) and the
// buoyancy terms d(vx')/d rho = dt (-bx^2 / 2) (div + f), likewise vz.
template <typename T>
__global__ void __launch_bounds__(AdjGeom<T>::NT, 5)
    k_adj_vel(const __grid_constant__ AdjArgs<T> A, const __grid_constant__ AdjMaps maps, Slot<T> x0, Slot<T> x1,
              int slot, const __grid_constant__ FusedExtras<T> x, const T *obs, T *__restrict__ vb,
              T *__restrict__ pxb, T *__restrict__ pzb, T *__restrict__ dbar, double *__restrict__ acc) {
  using G = AdjGeom<T>;
  using SM = VelSmem<T>;
  constexpr int V = G::V, PL = G::TX * G::TZ;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
  auto box = [&](int o) { return reinterpret_cast<T *>(smem + o); };
  const AdjTile t = adj_tile(A, x.ntx);
  const long long ld = A.ld, np = A.np, c = (long long)t.j * ld + t.gi0;
  if (threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  Pk<T> r0{}, r1{};
  T rr = 0;
  if (t.act) {
    r0 = ldn(A.rho + c);
    r1 = ldn(A.rho + c + ld);
    rr = ldn1(A.rho + c + V);
  }
  const Strips<T> s = strips_of(A, t.gi0, t.j);
  if (t.act) prefetch_strips(A, s, t.gi0, t.j, x0, pxb, pzb, PX_SXX, PX_SXZ, PZ_SXZ, PZ_SZZ);
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar, SM::BYTES);
    tma_load_4d_hint(box(SM::SXX), &maps.st_a, t.x0 - 4, t.z0, 2, slot, bar, l2_stream());
    tma_load_4d_hint(box(SM::SXZ), &maps.st_b, t.x0 - 4, t.z0 - 4, 4, slot, bar, l2_stream());
    tma_load_4d_hint(box(SM::SZZ), &maps.st_c, t.x0, t.z0 - 3, 3, slot, bar, l2_stream());
    tma_load_3d(box(SM::VB), &maps.own, t.x0, t.z0, 0, bar);
    tma_load_3d_hint(smem + SM::ACC, &maps.acc, t.x0, t.z0, 0, bar, l2_stream());
    pdl_wait();  // rbar: the previous kernel's
    tma_load_3d_hint(box(SM::R0), &maps.px, t.x0 - 4, t.z0, 0, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::R1), &maps.pz, t.x0, t.z0 - 3, 1, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::R2), &maps.pz, t.x0, t.z0 - 4, 2, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::R3), &maps.px, t.x0 - 4, t.z0, 3, bar, bar_policy(A));
  }
  const int e0 = x.tile_off[blockIdx.x], e1 = x.tile_off[blockIdx.x + 1];
  pdl_wait();
  pdl_release();
  if (!boxes_landed(bar, x.err)) return;
  const int ow = t.r * G::WX + t.lx + 4, oz = t.r * G::TX + t.lx;
  Pk<T> vx{}, vz{};
  if (t.act) {
    vx = psub(ldv(box(SM::VB) + oz),
              padd(dxp(ldwin(box(SM::R0) + ow), A.Dx), dzm(box(SM::R2) + oz + 4 * G::TX, G::TX, A.Dz)));
    vz = psub(ldv(box(SM::VB) + PL + oz),
              padd(dzp(box(SM::R1) + oz + 3 * G::TX, G::TX, A.Dz), dxm(ldwin(box(SM::R3) + ow), A.Dx)));
    if (t.gi0 + V > A.nx - L) {
      zero_outside(vx, A.nx - L - t.gi0);
      zero_outside(vz, A.nx - L - t.gi0);
    }
  }
  if (e0 < e1) {  // a tile with entries: its residuals added in shared memory, one thread per receiver cell
    T *sv = box(SM::VB);
    if (t.act) {
      stv(sv + oz, vx);
      stv(sv + PL + oz, vz);
    }
    __syncthreads();
    for (int e = e0 + (int)threadIdx.x; e < e1; e += G::NT) {
      int4 en = x.tile_ent[e];
      if (en.w != TL_RECEIVER) continue;
      const int i = en.x, j = en.y;
      if (e > e0) {  // receivers of a cell follow each other: its first one's thread takes them all
        const int4 b = x.tile_ent[e - 1];
        if (b.w == TL_RECEIVER && b.x == i && b.y == j) continue;
      }
      const T dx = x1.vx()[(long long)j * ld + i], dz = x1.vz()[(long long)j * ld + i];
      const int o = (j - t.z0) * G::TX + i - t.x0;
      T ax = sv[o], az = sv[PL + o];
      int f = e;
      do {
        ax += dx - obs[(long long)en.z * x.tnt + x.it];
        az += dz - obs[(long long)(x.nrec + en.z) * x.tnt + x.it];
        if (++f == e1) break;
        en = x.tile_ent[f];
      } while (en.x == i && en.y == j);
      sv[o] = ax;
      sv[PL + o] = az;
    }
    __syncthreads();
    if (t.act) {
      vx = ldv(sv + oz);
      vz = ldv(sv + PL + oz);
    }
  }
  if (!t.act) return;
  stv(vb + c, vx);
  stv(vb + np + c, vz);
  // forward stress divergence of the step
  const T *sq = box(SM::SXZ) + ow + 4 * G::WX;
  Pk<T> d0 = dxp(ldwin(box(SM::SXX) + ow), A.Dx), d2 = dxm(ldwin(sq), A.Dx);
  Pk<T> d1 = dzm(sq, G::WX, A.Dz), d3 = dzp(box(SM::SZZ) + oz + 3 * G::TX, G::TX, A.Dz);
  if (s.x) {
    cpml_fwd_x(A, s, t.gi0, (const T *)x0.psix(), PX_SXX, T_IKH, T_AH, T_BH, d0);
    cpml_fwd_x(A, s, t.gi0, (const T *)x0.psix(), PX_SXZ, T_IK, T_A, T_B, d2);
  }
  if (s.z) {
    cpml_fwd_z(A, s, t.j, (const T *)x0.psiz(), PZ_SXZ, T_IK, T_A, T_B, d1);
    cpml_fwd_z(A, s, t.j, (const T *)x0.psiz(), PZ_SZZ, T_IKH, T_AH, T_BH, d3);
  }
  Pk<T> dx = padd(d0, d1), dz = padd(d2, d3), bx, bz;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    bx.v[k] = T(2) / (r0.v[k] + right_of(r0, k, rr));
    bz.v[k] = T(2) / (r0.v[k] + r1.v[k]);
  }
  if (t.gi0 + V > A.nx - L) {
    zero_outside(bx, A.nx - L - t.gi0);
    zero_outside(bz, A.nx - L - t.gi0);
  }
  for (int e = e0; e < e1; ++e) {  // force sources: their buoyancy factor depends on rho too
    const int4 en = x.tile_ent[e];
    if (en.w > TL_FORCE_Z) break;
    if (en.y != t.j || en.x < t.gi0 || en.x >= t.gi0 + V) continue;
    const T f = x.it < x.wnt ? x.amp[en.z] * x.wavelet[(long long)en.z * x.wnt + x.it] : T(0);
#pragma unroll
    for (int k = 0; k < V; ++k)
      if (k == en.x - t.gi0) (en.w == TL_FORCE_X ? dx.v[k] : dz.v[k]) += f;
  }
  const Pk<T> hx = pmul(pmul(pscale(A.dt * T(-0.5), pmul(bx, bx)), dx), vx);
  const Pk<T> hz = pmul(pmul(pscale(A.dt * T(-0.5), pmul(bz, bz)), dz), vz);
  const double *ai = reinterpret_cast<const double *>(smem + SM::ACC) + oz;
  acc_add<T>(ai, acc + c, [&](int k, double g) { return g + (double)hx.v[k]; });
  acc_add<T>(ai + PL, acc + np + c, [&](int k, double g) { return g + (double)hz.v[k]; });
  Pk<T> db[4];
  db[0] = db[1] = pmul(pscale(A.dt, bx), vx);
  db[2] = db[3] = pmul(pscale(A.dt, bz), vz);
  if (s.x) {
    cpml_adj_x(A, s, t.gi0, pxb, PX_SXX, T_IKH, T_AH, T_BH, db[0]);
    cpml_adj_x(A, s, t.gi0, pxb, PX_SXZ, T_IK, T_A, T_B, db[2]);
  }
  if (s.z) {
    cpml_adj_z(A, s, t.j, pzb, PZ_SXZ, T_IK, T_A, T_B, db[1]);
    cpml_adj_z(A, s, t.j, pzb, PZ_SZZ, T_IKH, T_AH, T_BH, db[3]);
  }
  if (t.gi0 + V > A.nx - L)
#pragma unroll
    for (int k = 0; k < 4; ++k) zero_outside(db[k], A.nx - L - t.gi0);
#pragma unroll
  for (int k = 0; k < 4; ++k) stvp(dbar + k * np + c, db[k], bar_policy(A));
}

// ---- TTI ----------------------------------------------------------------
// The TTI stress law couples neighbouring cells (custom_solver/Model.jl:59-108
// on the staggered grid):
//   dsxx = C11 exx + C13 ezz + C15 ebxz,   dszz = C13 exx + C33 ezz + C35 ebxz,
//   dsxz = C55h exz + C15h ebxx + C35h ebzz,
// ebxz(i,j) the mean of exz over (i,j),(i-1,j),(i,j-1),(i-1,j-1), ebxx and
// ebzz the means of exx, ezz over (i,j),(i+1,j),(i,j+1),(i+1,j+1), C15h,
// C35h, C55h the means of the stiffness over the latter four cells, and on
// the free surface (row L) ezz = -(C13 exx + C35 ebxz) / C33.  Effective
// rates and stress adjoints outside the update region are zero.

// sigma adjoint of the step, and its forward effective rates: fe holds e (3
// planes, ezz on the surface row before the surface relation) and rt + S (3
// planes: the strain rates plus the memory-variable sums, de/dtau).
template <typename T>
struct SigmaTtiSmem {
  using S = StressSmem<T, 0, 0>;
  static constexpr int SIZE = S::CC;  // the boxes up to the sigma adjoint
  static constexpr int BYTES = S::TAPS + S::VBOX + 3 * AdjGeom<T>::TX * AdjGeom<T>::TZ * AdjGeom<T>::E;
};
template <typename T, int N>
__global__ void __launch_bounds__(AdjGeom<T>::NT, 4)
    k_adj_sigma_tti(const __grid_constant__ AdjArgs<T> A, const __grid_constant__ AdjMaps maps, Slot<T> x0, int slot,
                    int ntx, T *__restrict__ sb, T *__restrict__ fe, int *err) {
  using G = AdjGeom<T>;
  using SM = typename SigmaTtiSmem<T>::S;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
  auto box = [&](int o) { return reinterpret_cast<T *>(smem + o); };
  const AdjTile t = adj_tile(A, ntx);
  const long long ld = A.ld, np = A.np, c = (long long)t.j * ld + t.gi0;
  if (threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  Pk<T> S[3], tau{};
  if (t.act) {
    memory_sums<T, N>((const T *)x0.m() + c, np, S);
    if (N > 0) tau = ldn(A.tau + c);
  }
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar, SigmaTtiSmem<T>::BYTES);
    tma_load_4d_hint(box(SM::VX), &maps.st_a, t.x0 - 4, t.z0 - 3, 0, slot + 1, bar, l2_stream());
    tma_load_4d_hint(box(SM::VZ), &maps.st_a, t.x0 - 4, t.z0 - 4, 1, slot + 1, bar, l2_stream());
    tma_load_3d(box(SM::SB), &maps.own, t.x0, t.z0, 0, bar);
    pdl_wait();  // dbar: the previous kernel's
    tma_load_3d_hint(box(SM::D0), &maps.px, t.x0 - 4, t.z0, 0, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::D1), &maps.pz, t.x0, t.z0 - 3, 1, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::D2), &maps.px, t.x0 - 4, t.z0, 2, bar, bar_policy(A));
    tma_load_3d_hint(box(SM::D3), &maps.pz, t.x0, t.z0 - 4, 3, bar, bar_policy(A));
  }
  pdl_wait();
  pdl_release();
  if (!boxes_landed(bar, err) || !t.act) return;
  const int ow = t.r * G::WX + t.lx + 4, oz = t.r * G::TX + t.lx;
  Pk<T> bxx, bzz, bxz;
  adj_sigma(A, t, box(SM::SB) + oz, box(SM::D0) + ow, box(SM::D1) + oz + 3 * G::TX, box(SM::D2) + ow,
            box(SM::D3) + oz + 4 * G::TX, bxx, bzz, bxz);
  stv(sb + c, bxx);
  stv(sb + np + c, A.fs && t.j == L ? splat<T>(T(0)) : bzz);  // szz' = 0 on the surface
  stv(sb + 2 * np + c, bxz);
  const Strips<T> s = strips_of(A, t.gi0, t.j);
  Pk<T> rt[3];
  adj_rates(A, x0, s, t, box(SM::VX) + ow + 3 * G::WX, box(SM::VZ) + ow + 4 * G::WX, rt);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const Pk<T> rs = padd(rt[k], S[k]);
    Pk<T> e = N > 0 ? effective_rate(tau, rt[k], S[k]) : rt[k];
    if (t.gi0 + G::V > A.nx - L) zero_outside(e, A.nx - L - t.gi0);
    stv(fe + k * np + c, e);
    stv(fe + (3 + k) * np + c, rs);
  }
}

// u[-1 .. V] of a row
template <typename T>
struct Row3 {
  T w[VecW<T>::V + 2];
};
template <typename T>
__device__ __forceinline__ Row3<T> ldrow3(const T *u) {
  constexpr int V = VecW<T>::V;
  Row3<T> r;
  const Pk<T> t = ldv(u);
  r.w[0] = u[-1];
  r.w[V + 1] = u[V];
#pragma unroll
  for (int k = 0; k < V; ++k) r.w[1 + k] = t.v[k];
  return r;
}
// the same of a modulus, 0 before the update region (no updated cell reads
// it there; the sigma adjoint it meets is 0)
template <typename T>
__device__ __forceinline__ Row3<T> ldrow3_med(const T *u, const AdjTile &t, int j) {
  Row3<T> r{};
  if (j < L) return r;
  r = ldrow3(u);
  if (t.gi0 == L) r.w[0] = T(0);
  return r;
}
// mean of the four cells (i, j), (i+1, j), (i, j+1), (i+1, j+1), cell o - 1 of
// the group (o = 0: the cell before it)
template <typename T>
__device__ __forceinline__ T mean_of(const Row3<T> &a, const Row3<T> &b, int o) {
  return T(0.25) * (a.w[o] + a.w[o + 1] + b.w[o] + b.w[o + 1]);
}

// S^T of one TTI step: the effective-rate adjoints gathered from the stress
// adjoints of the cells whose update reads them, the stiffness terms, the
// surface relation transposed, then memory variables, tau and CPML memory.
template <typename T, int N>
__global__ void __launch_bounds__(AdjGeom<T>::NT, 3)
    k_adj_stress_tti(const __grid_constant__ AdjArgs<T> A, const __grid_constant__ AdjMaps maps, int ntx, const T *fe,
                     T *__restrict__ mbar, T *__restrict__ pxb, T *__restrict__ pzb, T *__restrict__ rbar,
                     double *__restrict__ acc, int *err) {
  using G = AdjGeom<T>;
  using SM = TtiSmem<T>;
  constexpr int V = G::V, PL = G::TX * G::TZ, W = G::WX, RP = G::WX * SM::RH, NM = N > 0 ? 3 * N : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
  auto box = [&](int o) { return reinterpret_cast<T *>(smem + o); };
  const AdjTile t = adj_tile(A, ntx);
  const long long ld = A.ld, np = A.np, c = (long long)t.j * ld + t.gi0;
  if (threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  Pk<T> C11{}, C13{}, C33{}, tau{}, mb[NM];
  if (t.act) {
    C11 = ldn(A.c11 + c);
    C13 = ldn(A.c13 + c);
    C33 = ldn(A.c33 + c);
    if (N > 0) tau = ldn(A.tau + c);
    if (const int n = A.nx - L - t.gi0; n < V) {
      zero_outside(tau, n);
      zero_outside(C11, n);
      zero_outside(C13, n);
      set_outside(C33, n, T(1));
    }
#pragma unroll
    for (int q = 0; q < 3 * N; ++q) mb[q] = ldcgv(mbar + q * np + c);
  }
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar, SM::BYTES);
    tma_load_2d(box(SM::C15), &maps.c2, t.x0 - 4, t.z0 - 1, bar);
    tma_load_2d(box(SM::C35), &maps.c3, t.x0 - 4, t.z0 - 1, bar);
    tma_load_2d(box(SM::CC), &maps.cc, t.x0, t.z0, bar);
    tma_load_3d_hint(smem + SM::ACC, &maps.acc, t.x0, t.z0, 0, bar, l2_stream());
    pdl_wait();  // sigma adjoint and effective rates: the previous kernel's
    tma_load_3d(box(SM::FE), &maps.px, t.x0 - 4, t.z0 - 1, 0, bar);
    tma_load_3d(box(SM::SB), &maps.pz, t.x0 - 4, t.z0 - 1, 0, bar);
  }
  pdl_wait();
  pdl_release();
  Pk<T> rs[3];
  if (N > 0 && t.act)
#pragma unroll
    for (int k = 0; k < 3; ++k) rs[k] = ldcgv(fe + (3 + k) * np + c);
  if (!boxes_landed(bar, err) || !t.act) return;
  const bool surf = A.fs && t.j == L;
  const int o = (t.r + 1) * W + t.lx + 4, oc = t.r * G::WC + t.lx, oz = t.r * G::TX + t.lx;
  const T *f0 = box(SM::FE) + o, *b0 = box(SM::SB) + o;
  const double *ai = reinterpret_cast<const double *>(smem + SM::ACC) + oz;
  double *ao = acc + c;
  Pk<T> eb[3], exx, ezz, exz, ebxz, bxz, c35own;  // eb without dt until the end
  const Pk<T> bxx = ldv(b0), bzz = ldv(b0 + RP);
  eb[0] = pfma(C11, bxx, pmul(C13, bzz));
  eb[1] = pfma(C13, bxx, pmul(C33, bzz));
  // the zz effective-rate adjoint of the cell after the group (surface row)
  T zr = 0, wr = 0;
  if (surf && t.gi0 + V < A.nx - L) {
    const T *q = b0 + 2 * RP + V, *a = box(SM::C35) + o + V;
    T sz = 0;
#pragma unroll
    for (int di = 0; di <= 1; ++di)  // row L - 1 lies outside the update region
      sz += T(0.25) * (a[-di] + a[1 - di] + a[W - di] + a[W + 1 - di]) * q[-di];
    zr = ldn1(A.c13 + c + V) * b0[V] + T(0.25) * sz;
    wr = a[0] / ldn1(A.c33 + c + V);
  }
  {  // exx, ezz feed sxz of the cells (i,j), (i-1,j), (i,j-1), (i-1,j-1)
    const Row3<T> q0 = ldrow3(b0 + 2 * RP), qm = ldrow3(b0 + 2 * RP - W);
    {
      const T *cc = box(SM::CC) + oc;
      const Pk<T> c55 = ldv(cc), c55d = ldv(cc + G::WC);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        bxz.v[k] = q0.w[k + 1];
        eb[2].v[k] = T(0.25) * (c55.v[k] + right_of(c55, k, cc[V]) + c55d.v[k] + right_of(c55d, k, cc[G::WC + V])) *
                     bxz.v[k];
      }
    }
    {
      const T *a = box(SM::C15) + o;
      const Row3<T> a0 = ldrow3_med(a, t, t.j), ap = ldrow3_med(a + W, t, t.j + 1), am = ldrow3_med(a - W, t, t.j - 1);
      const Row3<T> sx0 = ldrow3(b0), sxp = ldrow3(b0 + W);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const T sx = mean_of(a0, ap, k + 1) * q0.w[k + 1] + mean_of(a0, ap, k) * q0.w[k] +
                     mean_of(am, a0, k + 1) * qm.w[k + 1] + mean_of(am, a0, k) * qm.w[k];
        eb[0].v[k] += T(0.25) * sx;
        eb[2].v[k] += T(0.25) * (a0.w[k + 1] * sx0.w[k + 1] + a0.w[k + 2] * sx0.w[k + 2] +
                                 ap.w[k + 1] * sxp.w[k + 1] + ap.w[k + 2] * sxp.w[k + 2]);
      }
    }
    {
      const T *a = box(SM::C35) + o;
      const Row3<T> a0 = ldrow3_med(a, t, t.j), ap = ldrow3_med(a + W, t, t.j + 1), am = ldrow3_med(a - W, t, t.j - 1);
      const Row3<T> sz0 = ldrow3(b0 + RP), szp = ldrow3(b0 + RP + W);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const T sz = mean_of(a0, ap, k + 1) * q0.w[k + 1] + mean_of(a0, ap, k) * q0.w[k] +
                     mean_of(am, a0, k + 1) * qm.w[k + 1] + mean_of(am, a0, k) * qm.w[k];
        eb[1].v[k] += T(0.25) * sz;
        eb[2].v[k] += T(0.25) * (a0.w[k + 1] * sz0.w[k + 1] + a0.w[k + 2] * sz0.w[k + 2] +
                                 ap.w[k + 1] * szp.w[k + 1] + ap.w[k + 2] * szp.w[k + 2]);
        c35own.v[k] = a0.w[k + 1];
      }
    }
  }
  {  // forward rates at the cell and the means its update used
    const Row3<T> z0 = ldrow3(f0 + 2 * RP), zm = ldrow3(f0 + 2 * RP - W);
    T ebx1[V + 1];
#pragma unroll
    for (int k = 0; k <= V; ++k) ebx1[k] = mean_of(zm, z0, k);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      ebxz.v[k] = ebx1[k];
      exz.v[k] = z0.w[k + 1];
    }
    const Row3<T> x0 = ldrow3(f0), xp = ldrow3(f0 + W);
    Row3<T> w0 = ldrow3(f0 + RP);
    const Row3<T> wp = ldrow3(f0 + RP + W);
    if (surf) {  // the surface relation: ezz of the group and of the cell after it
      const T *a = box(SM::C35) + o;
#pragma unroll
      for (int k = 0; k <= V; ++k)
        if (t.gi0 + k < A.nx - L)
          w0.w[k + 1] = -(ldn1(A.c13 + c + k) * x0.w[k + 1] + a[k] * ebx1[k]) / ldn1(A.c33 + c + k);
    }
    // accumulators: plane 0 TAU, 1 Q55, 2 C11, 3 C13, 4 C33, 5 C15, 6 C35, 7 Q15, 8 Q35
    acc_add<T>(ai + PL, ao + np, [&](int k, double g) { return fma((double)bxz.v[k], (double)exz.v[k], g); });
    acc_add<T>(ai + 7 * PL, ao + 7 * np,
               [&](int k, double g) { return fma((double)bxz.v[k], (double)mean_of(x0, xp, k + 1), g); });
    acc_add<T>(ai + 8 * PL, ao + 8 * np,
               [&](int k, double g) { return fma((double)bxz.v[k], (double)mean_of(w0, wp, k + 1), g); });
#pragma unroll
    for (int k = 0; k < V; ++k) {
      exx.v[k] = x0.w[k + 1];
      ezz.v[k] = w0.w[k + 1];
    }
  }
  acc_add<T>(ai + 2 * PL, ao + 2 * np, [&](int k, double g) { return fma((double)bxx.v[k], (double)exx.v[k], g); });
  acc_add<T>(ai + 5 * PL, ao + 5 * np, [&](int k, double g) { return fma((double)bxx.v[k], (double)ebxz.v[k], g); });
  if (!surf) {
    acc_add<T>(ai + 3 * PL, ao + 3 * np, [&](int k, double g) {
      return fma((double)bxx.v[k], (double)ezz.v[k], fma((double)bzz.v[k], (double)exx.v[k], g));
    });
    acc_add<T>(ai + 4 * PL, ao + 4 * np, [&](int k, double g) { return fma((double)bzz.v[k], (double)ezz.v[k], g); });
    acc_add<T>(ai + 6 * PL, ao + 6 * np, [&](int k, double g) { return fma((double)bzz.v[k], (double)ebxz.v[k], g); });
  } else {
    // the adjoint of the surface ezz moves to exx of the cell and to exz of
    // the cell and its left neighbour, with its stiffness terms (bzz = 0)
    Pk<T> zb = eb[1], wz;  // wz: C35 / C33 zb
    if (t.gi0 + V > A.nx - L) zero_outside(zb, A.nx - L - t.gi0);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      wz.v[k] = c35own.v[k] / C33.v[k] * zb.v[k];
      eb[0].v[k] -= C13.v[k] / C33.v[k] * zb.v[k];
    }
    if (t.gi0 + V > A.nx - L) zero_outside(wz, A.nx - L - t.gi0);
#pragma unroll
    for (int k = 0; k < V; ++k) eb[2].v[k] -= T(0.25) * (wz.v[k] + right_of(wz, k, wr * zr));
    eb[1] = splat<T>(T(0));
    acc_add<T>(ai + 3 * PL, ao + 3 * np, [&](int k, double g) {
      return fma((double)bxx.v[k], (double)ezz.v[k], g) - (double)zb.v[k] * (double)exx.v[k] / (double)C33.v[k];
    });
    acc_add<T>(ai + 4 * PL, ao + 4 * np,
               [&](int k, double g) { return g - (double)zb.v[k] * (double)ezz.v[k] / (double)C33.v[k]; });
    acc_add<T>(ai + 6 * PL, ao + 6 * np,
               [&](int k, double g) { return g - (double)zb.v[k] * (double)ebxz.v[k] / (double)C33.v[k]; });
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    eb[k] = pscale(A.dt, eb[k]);
    if (t.gi0 + V > A.nx - L) zero_outside(eb[k], A.nx - L - t.gi0);
  }
  if (N > 0)
    acc_add<T>(ai, ao, [&](int k, double g) {
      const double u = fma((double)eb[1].v[k], (double)rs[1].v[k], (double)eb[0].v[k] * (double)rs[0].v[k]);
      return g + fma((double)eb[2].v[k], (double)rs[2].v[k], u);
    });
  adj_memory<T, N>(A, [&](int q) { return mb[q]; }, mbar + c, pxb, pzb, strips_of(A, t.gi0, t.j), t, c, surf, tau, eb,
                   rbar);
}

// The gradient planes from the accumulators: dt applied, the buoyancy terms
// spread over the two densities of each velocity node and the half-node terms
// over the four cells of each mean.  ISO: C11 = C33 = lambda + 2 mu, C13 =
// lambda, C55 = mu.
__global__ void k_adj_finish(int kind, int nx, int nz, int ld, double dt, const double *acc, int accumulate,
                             double *grad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= nz) return;
  const long long np = (long long)ld * nz, c = (long long)j * ld + i, npo = (long long)nx * nz;
  auto half = [&](int q) {  // 1/4 of the four cells whose mean reads this one
    const double *p = acc + q * np + c;
    double t = p[0];
    if (i > 0) t += p[-1];
    if (j > 0) t += p[-ld];
    if (i > 0 && j > 0) t += p[-ld - 1];
    return 0.25 * dt * t;
  };
  double g[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const double *h = acc + ACC_HX * np + c, *v = acc + ACC_HZ * np + c;
  g[0] = h[0] + v[0] + (i > 0 ? h[-1] : 0.0) + (j > 0 ? v[-ld] : 0.0);
  g[7] = acc[ACC_TAU * np + c];
  const double g11 = dt * acc[ACC_11 * np + c], g13 = dt * acc[ACC_13 * np + c];
  if (kind == VI_MEDIUM_ISO) {
    g[2] = g11 + g13;
    g[6] = 2.0 * g11 + half(ACC_Q55);
  } else {
    g[1] = g11;
    g[2] = g13;
    g[4] = dt * acc[ACC_33 * np + c];
    g[6] = half(ACC_Q55);
  }
  if (kind == VI_MEDIUM_TTI) {
    g[3] = dt * acc[ACC_15 * np + c] + half(ACC_Q15);
    g[5] = dt * acc[ACC_35 * np + c] + half(ACC_Q35);
  }
  double *o = grad + (long long)j * nx + i;
#pragma unroll
  for (int q = 0; q < 8; ++q) o[q * npo] = accumulate ? o[q * npo] + g[q] : g[q];
}

// FP64 misfit: 1/2 sum (d - obs)^2, one partial sum per block, added in block
// order by the last kernel's thread (a fixed order).  One block alone took 53
// us for 82 k samples.
constexpr int kMisfitBlocks = 64;
template <typename T>
__global__ void k_misfit(const T *tr, const T *obs, long long n, double *part) {
  __shared__ double red[256];
  double s = 0;
  for (long long k = blockIdx.x * 256LL + threadIdx.x; k < n; k += kMisfitBlocks * 256LL) {
    const double d = (double)tr[k] - (double)obs[k];
    s += d * d;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}
__global__ void k_misfit_sum(const double *part, double *out) {
  double s = 0;
  for (int k = 0; k < kMisfitBlocks; ++k) s += part[k];
  *out = 0.5 * s;
}

// The (vp, vs, rho, 1/Q) chain rule
__global__ void k_velocity_grad(int kind, long long np, const double *g, const double *vp,
                                const double *vs, const double *rho, const double *eps,
                                const double *delta, double tau_scale, double *out) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= np) return;
  const double grho = g[0 * np + c], g11 = g[1 * np + c], g13 = g[2 * np + c];
  const double g33 = g[4 * np + c], g55 = g[6 * np + c], gtau = g[7 * np + c];
  const double p = vp[c], s = vs[c], r = rho[c];
  double gC33, gC55;
  if (kind == VI_MEDIUM_ISO) {
    // g13 slot carries dJ/dlambda, g55 slot dJ/dmu (already folded)
    const double gl = g13, gm = g55;
    gC33 = gl;          // lambda = rho (vp^2 - 2 vs^2): d/dvp via vp^2
    gC55 = gm - 2 * gl; // mu = rho vs^2
  } else {
    const double e = eps ? eps[c] : 0.0, d = delta ? delta[c] : 0.0;
    const double C33 = r * p * p, C55 = r * s * s;
    const double A = C33 - C55, B = C33 * (1 + 2 * d) - C55;
    const double sq = sqrt(fmax(A * B, 1e-300));
    const double dC13_dC33 = (B + A * (1 + 2 * d)) / (2 * sq);
    const double dC13_dC55 = (-B - A) / (2 * sq) - 1.0;
    gC33 = g33 + g11 * (1 + 2 * e) + g13 * dC13_dC33;
    gC55 = g55 + g13 * dC13_dC55;
  }
  out[0 * np + c] = gC33 * 2 * r * p;                 // dJ/dvp
  out[1 * np + c] = gC55 * 2 * r * s;                 // dJ/dvs
  out[2 * np + c] = grho + gC33 * p * p + gC55 * s * s;  // dJ/drho at fixed vp, vs
  out[3 * np + c] = gtau * tau_scale;                 // dJ/d(1/Q)
}

// VTI Thomsen parameters at fixed (vp, vs, rho): C11 = C33 (1 + 2 eps)
// gives dC11/deps = 2 C33; C13 = sqrt(A B) - C55 with A = C33 - C55,
// B = C33 (1 + 2 delta) - C55 gives dC13/ddelta = A C33 / sqrt(A B)
// (media.thomsen_vti; custom_solver/Model.jl:12-16).  gamma enters only SH
// motion: no 2D P-SV stiffness depends on it.
__global__ void k_thomsen_grad(long long np, const double *g, const double *vp, const double *vs,
                               const double *rho, const double *delta, double *out) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= np) return;
  const double g11 = g[1 * np + c], g13 = g[2 * np + c];
  const double r = rho[c], C33 = r * vp[c] * vp[c], C55 = r * vs[c] * vs[c];
  const double d = delta ? delta[c] : 0.0;
  const double A = C33 - C55, B = C33 * (1 + 2 * d) - C55;
  const double sq = sqrt(fmax(A * B, 1e-300));
  out[0 * np + c] = g11 * 2 * C33;     // dJ/deps
  out[1 * np + c] = g13 * A * C33 / sq;  // dJ/ddelta
}

// Forward-mode derivative pairs (value, d/dp) for the TTI chain rule.
struct Dual {
  double v, d;
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return {a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return {a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return {a.v * b.v, a.d * b.v + a.v * b.d}; }
__device__ __forceinline__ Dual operator*(double s, Dual a) { return {s * a.v, s * a.d}; }
__device__ __forceinline__ Dual dsqrt(Dual a) {
  const double r = sqrt(fmax(a.v, 1e-300));
  return {r, a.d / (2.0 * r)};
}

// The TTI stiffness of one cell from (vp, vs, rho, epsilon, delta, theta):
// Thomsen's VTI law (Models.jl:27-52, custom_solver/Model.jl:12-16) tilted
// by the 2D Bond rotation (the map of vi_medium_from_velocity), carried on
// derivative pairs.  out = (C11, C13, C15, C33, C35, C55).
__device__ __forceinline__ void tti_stiffness(Dual p, Dual s, Dual r, Dual e, Dual d, Dual th, Dual (&out)[6]) {
  const Dual C33 = r * p * p, C55 = r * s * s;
  const Dual C11 = C33 * Dual{1.0 + 2.0 * e.v, 2.0 * e.d};
  const Dual C13 = dsqrt((C33 - C55) * (C33 * Dual{1.0 + 2.0 * d.v, 2.0 * d.d} - C55)) - C55;
  const Dual co{cos(th.v), -sin(th.v) * th.d}, si{sin(th.v), cos(th.v) * th.d};
  const Dual c2 = co * co, s2 = si * si, cs = co * si, A = C13 + 2.0 * C55, dcs = c2 - s2;
  out[0] = c2 * c2 * C11 + 2.0 * (c2 * s2 * A) + s2 * s2 * C33;
  out[1] = c2 * s2 * (C11 + C33 - 4.0 * C55) + (c2 * c2 + s2 * s2) * C13;
  out[2] = -1.0 * (cs * (c2 * C11 - s2 * C33 - dcs * A));
  out[3] = s2 * s2 * C11 + 2.0 * (c2 * s2 * A) + c2 * c2 * C33;
  out[4] = -1.0 * (cs * (s2 * C11 - c2 * C33 + dcs * A));
  out[5] = c2 * s2 * (C11 + C33 - 2.0 * C13) + dcs * dcs * C55;
}

// dJ/d(vp, vs, rho, 1/Q, epsilon, delta, theta) of a TTI medium from the
// stiffness gradient g (vi_gradient's eight planes): the chain rule through
// tti_stiffness, one derivative direction per parameter.
__global__ void k_tti_param_grad(long long np, const double *g, const double *vp, const double *vs,
                                 const double *rho, const double *eps, const double *delta,
                                 const double *theta, double tau_scale, double *out) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= np) return;
  const double gk[6] = {g[1 * np + c], g[2 * np + c], g[3 * np + c], g[4 * np + c], g[5 * np + c], g[6 * np + c]};
  const double val[6] = {vp[c], vs[c], rho[c], eps ? eps[c] : 0.0, delta ? delta[c] : 0.0, theta ? theta[c] : 0.0};
  const int slot[6] = {0, 1, 2, 4, 5, 6};  // output plane of each parameter (3 is 1/Q)
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    Dual x[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) x[k] = {val[k], k == q ? 1.0 : 0.0};
    Dual C[6];
    tti_stiffness(x[0], x[1], x[2], x[3], x[4], x[5], C);
    double s = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) s += gk[k] * C[k].d;
    if (q == 2) s += g[c];  // rho also enters the buoyancy directly
    out[slot[q] * np + c] = s;
  }
  out[3 * np + c] = g[7 * np + c] * tau_scale;  // dJ/d(1/Q)
}

}  // namespace

// Elements of the workspace: one state slot; rbar, dbar, TTI's effective rates,
// the FP64 accumulators and the medium copies.
template <typename T>
static long long slot_elems(const vi_config &c) {
  const long long ld = (c.nx + 3) / 4 * 4, Lp = c.pml_thickness;
  const long long wx = Lp * ((c.pml_left ? 1 : 0) + (c.pml_right ? 1 : 0));
  const long long hz = Lp * ((c.pml_top ? 1 : 0) + (c.pml_bottom ? 1 : 0));
  return Slot<T>::size(ld * c.nz, wx * c.nz, ld * hz, c.nsls);
}
template <typename T>
static long long scratch_elems(const vi_config &c, int copied) {
  const long long np = (long long)((c.nx + 3) / 4 * 4) * c.nz, wide = sizeof(double) / sizeof(T);
  return (8 + (c.medium == VI_MEDIUM_TTI ? 6 : 0) + acc_planes(c.medium) * wide + copied) * np;
}
template <typename T>
static size_t gradient_bytes_t(const vi_config &c, long long nslots, int nt, int nrec, int copied) {
  // (behind the traces: the misfit and its partial sums)
  return sizeof(T) * (size_t)(nslots * slot_elems<T>(c) + scratch_elems<T>(c, copied) + 2LL * nrec * nt) + 64 +
         8 * kMisfitBlocks;
}
size_t gradient_bytes(const vi_config &c, long long nslots, int nt, int nrec, int copied) {
  return c.precision == VI_F64 ? gradient_bytes_t<double>(c, nslots, nt, nrec, copied)
                               : gradient_bytes_t<float>(c, nslots, nt, nrec, copied);
}

template <typename T>
static int gradient_impl(vi_plan *p, const vi_medium *m, const vi_shot *shot, int nt, const T *obs,
                         int K, int accumulate, double *grad, double *misfit, cudaStream_t st) {
  const vi_config &c = p->cfg;
  const bool tti = c.medium == VI_MEDIUM_TTI;
  if (c.free_surface == kFsAfda)
    return set_error(VI_ERR_ARG, "gradient: the adjoint covers the stress-imaging free surface, not H-AFDA");
  int rc = check_medium(p, m);
  if (rc) return rc;
  if (!shot || shot->nrec <= 0 || !obs) return set_error(VI_ERR_ARG, "gradient: needs receivers and observed traces");
  if (!grad) return set_error(VI_ERR_ARG, "gradient: grad buffer is NULL");
  if (nt <= 0) return set_error(VI_ERR_ARG, "gradient: nt must be positive");
  if ((rc = cuda_check(cudaSetDevice(p->device), "cudaSetDevice"))) return rc;
  const int N = c.nsls, ld = (c.nx + 3) / 4 * 4;
  // every plane of the workspace has rows of ld cells, so odd grids take the
  // same vector kernels
  const long long np = (long long)ld * c.nz;
  const long long px = (long long)p->wx * c.nz, pz = (long long)ld * p->hz;
  const long long slot = slot_elems<T>(c);
  const int nrec = shot->nrec;
  const long long ntr = 2LL * nrec * nt;
  // the medium where its planes are not laid out so already
  const void *med[8] = {m->rho, m->c11, m->c13, m->c15, m->c33, m->c35, m->c55, m->tau};
  bool copy_med = ld != c.nx;
  int nmed = 0;
  for (const void *q : med) {
    copy_med |= ((uintptr_t)q & 15) != 0;
    nmed += q != nullptr;
  }
  const int copied = copy_med ? nmed : 0;
  // K = 0: every state of the forward sweep kept in HBM when the sweep fits
  // in 60 % of the device's memory and in what is free (1024 x 512 x 3000
  // VTI FP32: 88 GB), so the adjoint reads each step's states and nothing
  // is recomputed; else checkpoints every ceil(sqrt(nt)) steps
  bool keep_all = false;
  if (K <= 0) {
    const size_t all = gradient_bytes(c, nt + 2LL, nt, nrec, copied);
    if (p->device_bytes > 0 && all <= p->fwd_bytes) {
      // the workspace holds the sweep already: nothing to ask the driver
      // (cudaMemGetInfo took up to 10 ms of a 10 ms gradient)
      keep_all = all <= (size_t)(0.6 * (double)p->device_bytes);
    } else {
      size_t fr = 0, tot = 0;
      if (cudaMemGetInfo(&fr, &tot) == cudaSuccess) {
        const size_t avail = fr + p->fwd_bytes;
        keep_all = all <= (size_t)(0.6 * (double)tot) && all + (2ull << 30) <= avail;
        p->device_bytes = tot;
      }
      cudaGetLastError();
    }
    K = (int)std::ceil(std::sqrt((double)nt));
  }
  if (K > nt) K = nt;
  const int nck = keep_all ? nt + 1 : (nt + K - 1) / K;
  // workspace: checkpoints (keep_all: every state) | segment (K + 1 slots; none when keep_all) |
  // adjoint slot | rbar, dbar (4 planes each) | TTI: forward effective rates (6 planes) | FP64
  // accumulators | medium copies | traces | misfit
  const size_t need = gradient_bytes(c, nck + (keep_all ? 0 : K + 1) + 1LL, nt, nrec, copied);
  size_t have = p->fwd_bytes;
  if ((rc = ensure_buffer(p, &p->fwd, &have, need))) return rc;
  p->fwd_bytes = have;
  T *ck = (T *)p->fwd;
  T *seg = keep_all ? ck : ck + (size_t)nck * slot;
  T *adj = keep_all ? ck + (size_t)nck * slot : seg + (size_t)(K + 1) * slot;
  T *rbar = adj + slot, *dbar = rbar + 4 * np, *fe = dbar + 4 * np;
  double *acc = (double *)(fe + (tti ? 6 * np : 0));
  T *pmed = (T *)(acc + acc_planes(c.medium) * np);
  T *tr = pmed + copied * np;
  auto mk = [&](T *b) { return Slot<T>{b, np, px, pz, N}; };
  if ((rc = stage_shot<T>(p, shot, st))) return rc;
  vi_medium mw = *m;
  if (copy_med) {
    const void **slotp[8] = {&mw.rho, &mw.c11, &mw.c13, &mw.c15, &mw.c33, &mw.c35, &mw.c55, &mw.tau};
    const T *src[8];
    T *dst[8];
    int q = 0;
    for (int k = 0; k < 8; ++k)
      if (med[k]) {
        src[q] = (const T *)med[k];
        dst[q] = pmed + q * np;
        *slotp[k] = dst[q];
        ++q;
      }
    if ((rc = cuda_check(cudaMemsetAsync(pmed, 0, nmed * np * sizeof(T), st), "zero medium copies"))) return rc;
    if ((rc = copy_planes<T>(src, dst, nmed, c.nx, ld, c.nx, c.nz, st))) return rc;
  }
  // a forward step on slots (bind() points it at them)
  vi_fields fdummy{};
  fdummy.vx = fdummy.vz = fdummy.sxx = fdummy.szz = fdummy.sxz = (void *)ck;
  fdummy.m = ck;
  fdummy.m_plane_stride = np;
  StepArgs<T> a = make_args<T>(p, &mw, &fdummy);
  a.ld = a.ldz = ld;
  a.psix_plane = px;
  a.psiz_plane = pz;
  const size_t sbytes = (size_t)slot * sizeof(T);
  // The forward sweeps (traces + checkpoints, then the segment recompute)
  // run on the split pair, the same discrete step as the plain path the
  // adjoint transposes.  TTI sweeps step out of place only (the TTI stress
  // pass reads M and psi on a ring of neighbouring cells).
  using SG = SplitGeom<T>;
  using STG = SplitTtiGeom<T>;
  using SS = SplitStressGeom<T>;
  using AG = AdjGeom<T>;
  FusedExtras<T> fx{}, fxs{}, fxa{};
  SplitMaps ms{};
  int ntiles = 0, sntiles = 0, antiles = 0;
  {
    // velocity, stress and adjoint tilings, one buffer of lists
    int ntx = 0, ntz = 0, sntx = 0, sntz = 0, antx = 0, antz = 0;
    std::vector<int> off, soff, aoff;
    std::vector<int4> ent, sent, aent;
    build_tile_lists(c.nx, c.nz, SG::TX, SG::TZ, 0, shot, off, ent, ntx, ntz);
    build_tile_lists(c.nx, c.nz, tti ? STG::TX : SS::TX, tti ? STG::TZ : SS::TZ, 0, shot, soff, sent, sntx, sntz);
    build_tile_lists(c.nx, c.nz, AG::TX, AG::TZ, 0, shot, aoff, aent, antx, antz);
    // a tile's receivers by cell, in the order of the list within one (k_adj_vel)
    for (size_t k = 0; k + 1 < aoff.size(); ++k)
      std::stable_sort(aent.begin() + aoff[k], aent.begin() + aoff[k + 1], [](const int4 &u, const int4 &v) {
        if (u.w != v.w || u.w != TL_RECEIVER) return u.w < v.w;
        return u.y != v.y ? u.y < v.y : u.x < v.x;
      });
    const int nvoff = (int)off.size();
    for (int v : soff) off.push_back(v + (int)ent.size());
    ent.insert(ent.end(), sent.begin(), sent.end());
    const int naoff = (int)off.size();
    for (int v : aoff) off.push_back(v + (int)ent.size());
    ent.insert(ent.end(), aent.begin(), aent.end());
    int *d_off = nullptr;
    int4 *d_ent = nullptr;
    if ((rc = stage_tile_lists(p, off, ent, st, &d_off, &d_ent))) return rc;
    antiles = antx * antz;
    ntiles = ntx * ntz;
    sntiles = sntx * sntz;
    fx.ntx = ntx;
    fx.fs = c.free_surface;
    fx.tile_off = d_off;
    fx.tile_ent = d_ent;
    fx.amp = (const T *)p->damp;
    fx.wavelet = shot->nsrc ? (const T *)shot->wavelet_dev : nullptr;
    fx.wnt = shot->nsrc ? shot->wavelet_nt : 0;
    fx.nrec = nrec;
    fx.tnt = nt;
    fx.err = (int *)p->errflag;
    fx.l2hint = l2_hints_fit(5LL * c.nx * c.nz * (long long)sizeof(T), p->l2_bytes);
    fxs = fx;
    fxs.ntx = sntx;
    fxs.tile_off = d_off + nvoff;
    fxa = fx;
    fxa.ntx = antx;
    fxa.tile_off = d_off + naoff;
  }
  // One forward step of slot sl, in place (ISO/VTI) or (out != nullptr) from
  // slot sl into slot *out, which then holds the next state.
  auto fwd_step = [&](const Slot<T> &sl, int it, T *traces, bool pdl, const Slot<T> *out = nullptr) -> int {
    StepArgs<T> b = a;
    b.vx = sl.vx(); b.vz = sl.vz(); b.sxx = sl.sxx(); b.szz = sl.szz(); b.sxz = sl.sxz();
    b.m = sl.m();
    b.mstride = np;
    b.psix = b.psix_o = p->wx ? sl.psix() : nullptr;
    b.psiz = b.psiz_o = p->hz ? sl.psiz() : nullptr;
    if (out) {
      b.vx_o = out->vx(); b.vz_o = out->vz();
      b.sxx_o = out->sxx(); b.szz_o = out->szz(); b.sxz_o = out->sxz();
      b.m_o = out->m();
      b.mstride_o = np;
      b.psix_o = p->wx ? out->psix() : nullptr;
      b.psiz_o = p->hz ? out->psiz() : nullptr;
    }
    fx.it = fxs.it = it;
    fx.traces = fxs.traces = traces;
    // the stress pass stages the new velocities: those of the output state
    T *nvx = out ? out->vx() : b.vx, *nvz = out ? out->vz() : b.vz;
    const int bw = tti ? STG::BW : SS::BW, bh = tti ? STG::BH : SS::BH;
    int r2 = encode_map(&ms.a, nvx, (int)sizeof(T), ld, c.nz, 1, 0, bw, bh, 1);
    if (!r2) r2 = encode_map(&ms.b, nvz, (int)sizeof(T), ld, c.nz, 1, 0, bw, bh, 1);
    if (!r2) r2 = launch_split_vel<T>(b, fx, ntiles, st, pdl);
    if (!r2)
      r2 = tti ? launch_split_stress_tti<T>(b, fxs, ms, sntiles, st, true)
               : launch_split_stress<T>(c.medium, b, fxs, ms, sntiles, st, true);
    return r2;
  };
  // the caller's hook after every enqueued step (a server's slicing)
  auto yield = [&](int units) -> int {
    if (p->yield_fn && p->yield_fn(p->yield_ctx, units)) return set_error(VI_ERR_STATE, "gradient: stopped");
    return VI_OK;
  };
  // ---- forward sweep with checkpoints and traces ----
  Slot<T> cur = mk(seg);
  // every state slot starts at zero: cells the kernels never write (outside
  // the update region, off the CPML strips) stay zero in all of them.  The
  // kept states are zeroed once per layout of the plan's buffer (the key
  // is cleared by any other user of the buffer), so slot 0, never written,
  // stays the state at rest
  const unsigned long long zkey = keep_all ? ((unsigned long long)nt << 32) ^ (unsigned long long)slot ^
                                                 ((unsigned long long)sizeof(T) << 60) ^ (uintptr_t)p->fwd
                                           : 0;
  if (keep_all && p->grad_zero_key != zkey) {
    if ((rc = cuda_check(cudaMemsetAsync(ck, 0, (size_t)nck * sbytes, st), "zero kept states"))) return rc;
    p->grad_zero_key = zkey;
  } else if (!keep_all) {
    p->grad_zero_key = 0;
    if ((rc = cuda_check(cudaMemsetAsync(seg, 0, (size_t)(K + 1) * sbytes, st), "zero segment"))) return rc;
  }
  if (keep_all) {
    NvtxRange nr("vi_gradient: forward sweep, every state kept");
    for (int it = 0; it < nt; ++it) {
      const Slot<T> out = mk(ck + (size_t)(it + 1) * slot);
      if ((rc = fwd_step(mk(ck + (size_t)it * slot), it, tr, it > 0, &out))) return rc;
      if ((rc = yield(1))) return rc;
    }
  } else {
    NvtxRange nr("vi_gradient: forward sweep");
    for (int it = 0; it < nt; ++it) {
      if (it % K == 0)
        if ((rc = cuda_check(cudaMemcpyAsync(ck + (size_t)(it / K) * slot, cur.base, sbytes,
                                             cudaMemcpyDeviceToDevice, st),
                             "checkpoint")))
          return rc;
      if (tti) {  // out of place: between the segment's first two slots
        const Slot<T> nxt = mk(cur.base == seg ? seg + slot : seg);
        if ((rc = fwd_step(cur, it, tr, it % K != 0, &nxt))) return rc;
        cur = nxt;
      } else if ((rc = fwd_step(cur, it, tr, it % K != 0))) {
        return rc;
      }
      if ((rc = yield(1))) return rc;
    }
  }
  if (shot->traces_dev && shot->traces_nt >= nt) {
    for (int k = 0; k < 2 * nrec; ++k)
      cudaMemcpyAsync((T *)shot->traces_dev + (size_t)k * shot->traces_nt, tr + (size_t)k * nt,
                      nt * sizeof(T), cudaMemcpyDeviceToDevice, st);
  }
  double *dmis = (double *)(tr + ntr);
  dmis = (double *)(((uintptr_t)dmis + 15) / 16 * 16);
  k_misfit<T><<<kMisfitBlocks, 256, 0, st>>>(tr, obs, ntr, dmis + 1);
  k_misfit_sum<<<1, 1, 0, st>>>(dmis + 1, dmis);
  // ---- adjoint sweep ----
  AdjArgs<T> A;
  A.nx = c.nx; A.nz = c.nz; A.ld = ld; A.fs = c.free_surface;
  A.Lx = p->Lx; A.Rx = p->Rx; A.Tz = p->Tz; A.Bz = p->Bz; A.wx = p->wx;
  A.dt = (T)c.dt;
  for (int k = 0; k < 4; ++k) {
    A.Dx[k] = (T)(kD8[k] / c.dx);
    A.Dz[k] = (T)(kD8[k] / c.dz);
  }
  for (int n = 0; n < N; ++n) {  // the forward step's memory-variable coefficients
    A.a1[n] = a.a1[n];
    A.a2[n] = a.a2[n];
  }
  A.rho = a.rho; A.c11 = a.c11; A.c13 = a.c13; A.c33 = a.c33; A.c55 = a.c55; A.tau = a.tau;
  A.c15 = a.c15; A.c35 = a.c35;
  A.tx = (const T *)p->tabx; A.tz = (const T *)p->tabz;
  A.np = np; A.psix_plane = px; A.psiz_plane = pz;
  A.keep_bar = l2_hints_fit(8LL * np * (long long)sizeof(T), p->l2_bytes);
  Slot<T> ab = mk(adj);
  if ((rc = cuda_check(cudaMemsetAsync(adj, 0, sbytes, st), "zero adjoint"))) return rc;
  if ((rc = cuda_check(cudaMemsetAsync(rbar, 0, (char *)pmed - (char *)rbar, st), "zero scratch"))) return rc;
  // TMA maps: the planes' and accumulators' places do not change over the sweep
  const int e = (int)sizeof(T), ntx = fxa.ntx, nslots = keep_all ? nt + 1 : K + 1;
  constexpr int TX = AG::TX, TZ = AG::TZ, WX = AG::WX, HZ = AG::HZ, WC = AG::WC;
  const int acc0 = ACC_TAU, nacc = acc_planes(c.medium) - acc0;
  double *const acck = acc + acc0 * np;
  AdjMaps ms_s{}, ms_v{}, ms_t{};  // k_adj_stress / k_adj_sigma_tti, k_adj_vel, k_adj_stress_tti
  auto em = [&](CUtensorMap *map, const void *base, int es, int depth, int bx, int bz, int bd) {
    if (!rc) rc = encode_map(map, base, es, ld, c.nz, depth, np, bx, bz, bd);
  };
  auto es4 = [&](CUtensorMap *map, int bx, int bz) {
    if (!rc) rc = encode_map_slots(map, seg, e, ld, c.nz, 5, np, nslots, slot, bx, bz);
  };
  rc = VI_OK;
  em(&ms_s.px, dbar, e, 4, WX, TZ, 1);
  em(&ms_s.pz, dbar, e, 4, TX, HZ, 1);
  es4(&ms_s.st_a, WX, HZ);
  em(&ms_s.own, ab.sxx(), e, 3, TX, TZ, 3);
  em(&ms_v.px, rbar, e, 4, WX, TZ, 1);
  em(&ms_v.pz, rbar, e, 4, TX, HZ, 1);
  es4(&ms_v.st_a, WX, TZ);
  es4(&ms_v.st_b, WX, HZ);
  es4(&ms_v.st_c, TX, HZ);
  em(&ms_v.own, ab.vx(), e, 2, TX, TZ, 2);
  em(&ms_v.acc, acc, 8, 2, TX, TZ, 2);
  if (tti) {
    em(&ms_t.px, fe, e, 3, WX, TZ + 2, 3);
    em(&ms_t.pz, ab.sxx(), e, 3, WX, TZ + 2, 3);
    em(&ms_t.cc, a.c55, e, 1, WC, TZ + 1, 1);
    em(&ms_t.c2, a.c15, e, 1, WX, TZ + 2, 1);
    em(&ms_t.c3, a.c35, e, 1, WX, TZ + 2, 1);
    em(&ms_t.acc, acck, 8, nacc, TX, TZ, nacc);
  } else {
    if (N > 0) em(&ms_s.mem, ab.m(), e, 3 * N, TX, TZ, 3 * N);
    em(&ms_s.cc, a.c55, e, 1, WC, TZ + 1, 1);
    em(&ms_s.acc, acck, 8, nacc, TX, TZ, nacc);
  }
  if (rc) return rc;
  int lrc = VI_OK;  // first launch error of the adjoint sweep
  bool opt_in = true;  // the first call per kernel only opts into its dynamic shared memory
  auto lc = [&](auto kernel, int smem, auto... args) {
    if (lrc) return;
    const cudaError_t err = opt_in ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)
                                   : launch_pdl(kernel, dim3(antiles), dim3(AG::NT), (size_t)smem, st, true, args...);
    if (err != cudaSuccess) lrc = cuda_check(err, "adjoint launch");
  };
  int *const derr = (int *)p->errflag;
  auto stress_t = [&](auto n, const Slot<T> &x0, int sl) {
    constexpr int NN = decltype(n)::value;
    if (tti) {
      lc(k_adj_sigma_tti<T, NN>, SigmaTtiSmem<T>::SIZE, A, ms_s, x0, sl, ntx, ab.sxx(), fe, derr);
      lc(k_adj_stress_tti<T, NN>, TtiSmem<T>::SIZE, A, ms_t, ntx, (const T *)fe, ab.m(), ab.psix(), ab.psiz(), rbar,
         acck, derr);
    } else if (c.medium == VI_MEDIUM_ISO) {
      lc(k_adj_stress<T, VI_MEDIUM_ISO, NN>, StressK<T, VI_MEDIUM_ISO, NN>::S::SIZE, A, ms_s, x0, sl, ntx, ab.sxx(),
         ab.m(), ab.psix(), ab.psiz(), rbar, acck, derr);
    } else {
      lc(k_adj_stress<T, VI_MEDIUM_VTI, NN>, StressK<T, VI_MEDIUM_VTI, NN>::S::SIZE, A, ms_s, x0, sl, ntx, ab.sxx(),
         ab.m(), ab.psix(), ab.psiz(), rbar, acck, derr);
    }
  };
  auto reverse_step = [&](const Slot<T> &x0, const Slot<T> &x1, int sl, int it) {
    switch (N) {
      case 0: stress_t(std::integral_constant<int, 0>{}, x0, sl); break;
      case 1: stress_t(std::integral_constant<int, 1>{}, x0, sl); break;
      case 2: stress_t(std::integral_constant<int, 2>{}, x0, sl); break;
      case 3: stress_t(std::integral_constant<int, 3>{}, x0, sl); break;
      case 4: stress_t(std::integral_constant<int, 4>{}, x0, sl); break;
      default: stress_t(std::integral_constant<int, 5>{}, x0, sl); break;
    }
    fxa.it = it;
    lc(k_adj_vel<T>, VelSmem<T>::SIZE, A, ms_v, x0, x1, sl, fxa, obs, ab.vx(), ab.psix(), ab.psiz(), dbar, acc);
  };
  reverse_step(ab, ab, 0, 0);
  opt_in = false;
  if (lrc) return lrc;
  // keep_all: one segment of nt steps whose states are all kept
  for (int qseg = keep_all ? 0 : nck - 1; qseg >= 0; --qseg) {
    const int s0 = keep_all ? 0 : qseg * K, s1 = keep_all ? nt : std::min(nt, s0 + K);
    // recompute the segment: seg[k] = state before step s0 + k
    if (!keep_all &&
        (rc = cuda_check(cudaMemcpyAsync(seg, ck + (size_t)qseg * slot, sbytes, cudaMemcpyDeviceToDevice, st),
                         "restore checkpoint")))
      return rc;
    NvtxRange nr_seg("vi_gradient: segment recompute and adjoint");
    for (int k = 0; !keep_all && k < s1 - s0; ++k) {
      // straight from slot k into slot k + 1 (no copy of the state)
      const Slot<T> out = mk(seg + (size_t)(k + 1) * slot);
      if ((rc = fwd_step(mk(seg + (size_t)k * slot), s0 + k, nullptr, k > 0, &out))) return rc;
      if ((rc = yield(1))) return rc;
    }
    for (int it = s1 - 1; it >= s0; --it) {
      const Slot<T> x0 = mk(seg + (size_t)(it - s0) * slot), x1 = mk(seg + (size_t)(it - s0 + 1) * slot);
      // every kernel of the step overlaps its predecessor's tail and waits
      // for it at entry (programmatic dependent launch)
      reverse_step(x0, x1, it - s0, it);
      if (lrc) return lrc;
      if ((rc = yield(2))) return rc;
    }
  }
  if (lrc) return lrc;
  k_adj_finish<<<dim3((c.nx + 31) / 32, (c.nz + 7) / 8), dim3(32, 8), 0, st>>>(c.medium, c.nx, c.nz, ld, (double)A.dt,
                                                                              acc, accumulate, grad);
  p->last_kernel = 1;
  if ((rc = cuda_check(cudaGetLastError(), "gradient launch"))) return rc;
  if ((rc = cuda_check(cudaMemcpyAsync(misfit, dmis, sizeof(double), cudaMemcpyDeviceToHost, st), "misfit")))
    return rc;
  return cuda_check(cudaStreamSynchronize(st), "gradient");
}

}  // namespace vb

using namespace vb;

extern "C" int vi_gradient(vi_plan *p, const vi_medium *med_dev, const vi_shot *shot, int32_t nt,
                           const void *obs_dev, int32_t checkpoint_every, int32_t accumulate,
                           double *grad_dev, double *misfit_host, void *stream) {
  if (!p || !misfit_host) return set_error(VI_ERR_ARG, "gradient: NULL argument");
  cudaStream_t st = (cudaStream_t)stream;
  if (!p->no_resident) mark_call(p, true);
  const int rc = p->cfg.precision == VI_F64
                     ? gradient_impl<double>(p, med_dev, shot, nt, (const double *)obs_dev, checkpoint_every,
                                             accumulate, grad_dev, misfit_host, st)
                     : gradient_impl<float>(p, med_dev, shot, nt, (const float *)obs_dev, checkpoint_every,
                                            accumulate, grad_dev, misfit_host, st);
  if (!p->no_resident) mark_call(p, false);
  return rc;
}

extern "C" int vi_gradient_velocity(int32_t medium, int64_t np, const double *grad8, const double *vp,
                                    const double *vs, const double *rho, const double *eps,
                                    const double *delta, double tau_scale, double *out4, void *stream) {
  if (!grad8 || !vp || !vs || !rho || !out4 || np <= 0)
    return set_error(VI_ERR_ARG, "gradient_velocity: NULL argument");
  if (medium != VI_MEDIUM_ISO && medium != VI_MEDIUM_VTI)
    return set_error(VI_ERR_ARG, "gradient_velocity: ISO or VTI only");
  k_velocity_grad<<<(unsigned)((np + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      medium, np, grad8, vp, vs, rho, eps, delta, tau_scale, out4);
  return cuda_check(cudaGetLastError(), "gradient_velocity launch");
}

extern "C" int vi_gradient_tti(int64_t np, const double *grad8, const double *vp, const double *vs,
                               const double *rho, const double *eps, const double *delta, const double *theta,
                               double tau_scale, double *out7, void *stream) {
  if (!grad8 || !vp || !vs || !rho || !out7 || np <= 0)
    return set_error(VI_ERR_ARG, "gradient_tti: NULL argument");
  k_tti_param_grad<<<(unsigned)((np + 255) / 256), 256, 0, (cudaStream_t)stream>>>(np, grad8, vp, vs, rho, eps,
                                                                                   delta, theta, tau_scale, out7);
  return cuda_check(cudaGetLastError(), "gradient_tti launch");
}

extern "C" int vi_gradient_thomsen(int64_t np, const double *grad8, const double *vp, const double *vs,
                                   const double *rho, const double *delta, double *out2, void *stream) {
  if (!grad8 || !vp || !vs || !rho || !out2 || np <= 0)
    return set_error(VI_ERR_ARG, "gradient_thomsen: NULL argument");
  k_thomsen_grad<<<(unsigned)((np + 255) / 256), 256, 0, (cudaStream_t)stream>>>(np, grad8, vp, vs, rho,
                                                                                 delta, out2);
  return cuda_check(cudaGetLastError(), "gradient_thomsen launch");
}
