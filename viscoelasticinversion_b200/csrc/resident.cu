// resident.cu — the split pair's time loop in kernels of many steps, for ISO and
// VTI grids whose state fits on the chip.
//
// A small grid's step is all latency: two dependent launches of 3.6 us each
// even at 128 x 128 (tensor maps, boxes, one round of loads and the drain
// between them), and every plane through the L2 twice.  Here one CTA per SM
// owns a rectangle of the update region for the whole launch: velocities,
// stresses and coefficients in its shared memory, memory variables in
// registers.  After each pass it hands the four cells along its edges to its
// neighbours through a shadow of the planes in which every 32-bit word travels
// beside the number of the pass that wrote it, in one 64-bit element: a reader
// polls the words themselves, so an exchange is one store and one load through
// the L2, without fences, flags or a grid barrier (flags and fences took 4 us a
// pass).  One shadow per pass suffices: a CTA rewrites its velocity edges only
// after every neighbour's stress edges have arrived, which the neighbour sent
// after it had read them, and the other way round.  All CTAs run at the same
// time (cooperative launch); every wait is bounded and reports through the
// plan's error word.
//
// The arithmetic is the split kernels' (split_tiles.cuh), operation for
// operation, so results are bitwise equal whichever form a call takes.  Us per
// step on B200 against the pair: VTI FP32 128 x 128 3.4 (7.5), 256 x 256 4.1
// (7.9), 512 x 256 5.2 (8.5), 512 x 512 8.0 (10.4); FP64 256 x 256 5.2 (10.6),
// 512 x 256 7.1 (14.4).
#include <algorithm>
#include <cstdint>
#include <vector>

#include "cpml4.cuh"
#include "fused_tma.cuh"
#include "plan.cuh"
#include "split.cuh"
#include "vec.cuh"

namespace vb {

// Tiles of 4 * txg x tz cells, px x pz of them, one per CTA; `width` cells of a
// row per thread.
struct ResGeom {
  int txg, tz, px, pz, threads, width;
  size_t smem;
};
constexpr size_t kResMaxSmem = 226 * 1024;
constexpr int kResCoef = 7;  // C11, C13, C33, C55h, tau, bx, bz
constexpr int kResPsi = 8;   // 4 planes of x-strip memory, 4 of z

template <typename T>
static size_t res_smem(int txg, int tz) {
  const size_t tx = 4 * (size_t)txg, wx = tx + 8;
  return sizeof(T) * (3 * (tz + 8) * wx + tz * wx + (tz + 8) * tx + (kResCoef + kResPsi) * tz * tx + 6 * (tx + tz));
}

// ---- W cells of a row (W = 1 or 2).  Each lane rounds as the split
// kernels' 4-cell groups do.
template <typename T, int W>
struct Pw {
  T v[W];
};
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wsplat(T s) {
  Pw<T, W> r;
#pragma unroll
  for (int k = 0; k < W; ++k) r.v[k] = s;
  return r;
}
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wfma(const Pw<T, W> &a, const Pw<T, W> &b, const Pw<T, W> &c) {
  Pw<T, W> r;
  if constexpr (sizeof(T) == 4 && W >= 2) {
#pragma unroll
    for (int k = 0; k < W; k += 2) {
      const float2 t = __ffma2_rn(make_float2(a.v[k], a.v[k + 1]), make_float2(b.v[k], b.v[k + 1]),
                                  make_float2(c.v[k], c.v[k + 1]));
      r.v[k] = t.x;
      r.v[k + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = fma_rn(a.v[k], b.v[k], c.v[k]);
  }
  return r;
}
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wmul(const Pw<T, W> &a, const Pw<T, W> &b) {
  Pw<T, W> r;
  if constexpr (sizeof(T) == 4 && W >= 2) {
#pragma unroll
    for (int k = 0; k < W; k += 2) {
      const float2 t = __fmul2_rn(make_float2(a.v[k], a.v[k + 1]), make_float2(b.v[k], b.v[k + 1]));
      r.v[k] = t.x;
      r.v[k + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = mul_rn(a.v[k], b.v[k]);
  }
  return r;
}
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wadd(const Pw<T, W> &a, const Pw<T, W> &b) {
  Pw<T, W> r;
  if constexpr (sizeof(T) == 4 && W >= 2) {
#pragma unroll
    for (int k = 0; k < W; k += 2) {
      const float2 t = __fadd2_rn(make_float2(a.v[k], a.v[k + 1]), make_float2(b.v[k], b.v[k + 1]));
      r.v[k] = t.x;
      r.v[k + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = add_rn(a.v[k], b.v[k]);
  }
  return r;
}
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wsub(const Pw<T, W> &a, const Pw<T, W> &b) {  // as sub4: one rounding
  return wfma(b, wsplat<T, W>(T(-1)), a);
}
// shared memory: vectors where the address allows
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wld(const T *p) {
  Pw<T, W> r;
  if constexpr (W == 2) {
    const Q2<T> q = lds2(p);
    r.v[0] = q.v[0];
    r.v[1] = q.v[1];
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <typename T, int W>
__device__ __forceinline__ void wst(T *p, const Pw<T, W> &q) {
  if constexpr (W == 2)
    stg2(p, Q2<T>{{q.v[0], q.v[1]}});
  else
    *p = q.v[0];
}
// the values p[-4 .. W + 3] of a row
template <typename T, int W>
struct Win {
  T w[W + 8];
  __device__ __forceinline__ explicit Win(const T *p) {
#pragma unroll
    for (int q = 0; q < W + 8; q += W) {
      const Pw<T, W> t = wld<T, W>(p - 4 + q);
#pragma unroll
      for (int k = 0; k < W; ++k) w[q + k] = t.v[k];
    }
  }
  __device__ __forceinline__ Pw<T, W> at(int o) const {
    Pw<T, W> t;
#pragma unroll
    for (int k = 0; k < W; ++k) t.v[k] = w[4 + o + k];
    return t;
  }
};
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wdxp(const Win<T, W> &u, const T *D) {  // as dps4
  Pw<T, W> s = wmul(wsplat<T, W>(D[0]), wsub(u.at(1), u.at(0)));
#pragma unroll
  for (int q = 1; q < 4; ++q) s = wfma(wsplat<T, W>(D[q]), wsub(u.at(1 + q), u.at(-q)), s);
  return s;
}
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wdxm(const Win<T, W> &u, const T *D) {  // as dms4
  Pw<T, W> s = wmul(wsplat<T, W>(D[0]), wsub(u.at(0), u.at(-1)));
#pragma unroll
  for (int q = 1; q < 4; ++q) s = wfma(wsplat<T, W>(D[q]), wsub(u.at(q), u.at(-1 - q)), s);
  return s;
}
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wdzm(const T *p, int ld, const T *D) {  // rows -4 .. 3, in the pair's order
  Pw<T, W> z = wsplat<T, W>(T(0));
#pragma unroll
  for (int q = -4; q <= 3; ++q) z = wfma(wsplat<T, W>(q >= 0 ? D[q] : -D[-q - 1]), wld<T, W>(p + q * ld), z);
  return z;
}
template <typename T, int W>
__device__ __forceinline__ Pw<T, W> wdzp(const T *p, int ld, const T *D) {  // rows -3 .. 4
  Pw<T, W> z = wsplat<T, W>(T(0));
#pragma unroll
  for (int q = -3; q <= 4; ++q) z = wfma(wsplat<T, W>(q >= 1 ? D[q - 1] : -D[-q]), wld<T, W>(p + q * ld), z);
  return z;
}
// CPML memory (psi, in shared memory) and rate of the lanes of `mask`: b, a and
// 1/kappa from the profile rows t + row * stride, one value per lane (step 1)
// or per row (step 0)
template <typename T, int W>
__device__ __forceinline__ void wcpml(unsigned mask, T *psi, const T *t, int stride, int step, int rb, int ra, int rk,
                                      Pw<T, W> &d) {
#pragma unroll
  for (int k = 0; k < W; ++k)
    if (mask >> k & 1) {
      const T p = cpml_mem(t[rb * stride + k * step], psi[k], t[ra * stride + k * step], d.v[k]);
      psi[k] = p;
      d.v[k] = cpml_rate(d.v[k], t[rk * stride + k * step], p);
    }
}
template <typename T, int W>
__device__ __forceinline__ T wlane(const Pw<T, W> &q, int k) {
  T r = q.v[0];
#pragma unroll
  for (int i = 1; i < W; ++i)
    if (i == k) r = q.v[i];
  return r;
}
template <typename T, int W>
__device__ __forceinline__ void wadd_lane(Pw<T, W> &q, int k, T d) {
#pragma unroll
  for (int i = 0; i < W; ++i)
    if (i == k) q.v[i] = add_rn(q.v[i], d);
}

// Edge cells beside their pass number: (word, pass) pairs, each one 64-bit element
// of a relaxed access, written as they come and read 4 cells at a time (the
// flag-in-word scheme of NCCL's LL protocol).  PTX promises a 64-bit element
// whole, alone or in a vector, so a pair with the right number holds that pass's
// word; the order of elements does not matter.
__device__ __forceinline__ void st_pair2(uint32_t *p, uint32_t a, uint32_t b, uint32_t n) {
  asm volatile("{\n .reg .b64 u, v;\n mov.b64 u, {%1, %3};\n mov.b64 v, {%2, %3};\n"
               " st.relaxed.gpu.global.v2.b64 [%0], {u, v};\n}" ::"l"(p), "r"(a), "r"(b), "r"(n) : "memory");
}
__device__ __forceinline__ bool ld_pair2(const uint32_t *p, uint32_t &a, uint32_t &b, uint32_t n) {
  uint32_t f, g;
  asm volatile("{\n .reg .b64 u, v;\n ld.relaxed.gpu.global.v2.b64 {u, v}, [%4];\n mov.b64 {%0, %1}, u;\n"
               " mov.b64 {%2, %3}, v;\n}" : "=r"(a), "=r"(f), "=r"(b), "=r"(g) : "l"(p) : "memory");
  return f == n && g == n;
}
template <int W>
__device__ __forceinline__ void st_edge(uint32_t *p, const Pw<float, W> &q, uint32_t n) {
  if constexpr (W == 1) {
    asm volatile("{\n .reg .b64 u;\n mov.b64 u, {%1, %2};\n st.relaxed.gpu.global.b64 [%0], u;\n}" ::"l"(p),
                 "r"(__float_as_uint(q.v[0])), "r"(n) : "memory");
  } else {
#pragma unroll
    for (int k = 0; k < W; k += 2) st_pair2(p + 2 * k, __float_as_uint(q.v[k]), __float_as_uint(q.v[k + 1]), n);
  }
}
template <int W>
__device__ __forceinline__ void st_edge(uint32_t *p, const Pw<double, W> &q, uint32_t n) {
#pragma unroll
  for (int k = 0; k < W; ++k) st_pair2(p + 4 * k, __double2loint(q.v[k]), __double2hiint(q.v[k]), n);
}
__device__ __forceinline__ bool ld_edge(const uint32_t *p, Q4<float> &q, uint32_t n) {
  uint32_t w[4];
  bool ok = ld_pair2(p, w[0], w[1], n);
  ok &= ld_pair2(p + 4, w[2], w[3], n);
#pragma unroll
  for (int k = 0; k < 4; ++k) q.v[k] = __uint_as_float(w[k]);
  return ok;
}
__device__ __forceinline__ bool ld_edge(const uint32_t *p, Q4<double> &q, uint32_t n) {
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    uint32_t lo, hi;
    ok &= ld_pair2(p + 4 * k, lo, hi, n);
    q.v[k] = __hiloint2double((int)hi, (int)lo);
  }
  return ok;
}
// One 4-cell group of a neighbour's edge: its words in the shadow and its place
// in shared memory, for the velocities and for the stresses.
struct HaloItem {
  const uint32_t *gv, *gs;
  int sv, ss;
};

// 64 registers a thread in FP32, 128 in FP64, also for blocks with fewer threads:
// at 3 mechanisms (VTI) the time loop spills 180 bytes a thread with two cells in
// FP32, 36 with one, and 76 with two in FP64.
template <typename T>
constexpr int res_max_threads() {
  return sizeof(T) == 4 ? 1024 : 512;
}

template <typename T, int KIND, int NSLS, int W>
__global__ void __launch_bounds__(res_max_threads<T>(), 1)
    k_resident(const __grid_constant__ StepArgs<T> a, const __grid_constant__ FusedExtras<T> x, const ResGeom geo,
               int it0, int nsteps, uint32_t *shadow, uint32_t pass0) {
  using P = Pw<T, W>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int TX = 4 * geo.txg, TZ = geo.tz, WX = TX + 8, NT = blockDim.x, tid = threadIdx.x;
  const int cta = blockIdx.x, bi = cta % geo.px, bj = cta / geo.px;
  const int nx = a.nx, nz = a.nz, ld = a.ld, xe = nx - L, ze = nz - L;
  const int x0 = L + bi * TX, z0 = L + bj * TZ;
  const int w = min(TX, xe - x0), h = min(TZ, ze - z0), wg = w / 4;
  const bool nl = bi > 0, nr = bi + 1 < geo.px, nu = bj > 0, nd = bj + 1 < geo.pz;
  // planes, the tile's first cell at row 4 (where there is a z halo), column 4
  T *s_vx = reinterpret_cast<T *>(smem_raw), *s_vz = s_vx + (TZ + 8) * WX, *s_xz = s_vz + (TZ + 8) * WX;
  T *s_xx = s_xz + (TZ + 8) * WX, *s_zz = s_xx + TZ * WX, *s_co = s_zz + (TZ + 8) * TX;
  const int PC = TZ * TX;
  T *s_px = s_co + kResCoef * PC, *s_pz = s_px + 4 * PC, *s_tx = s_pz + 4 * PC, *s_tz = s_tx + 6 * TX;
  constexpr int EW = sizeof(T) / 2;  // shadow words per cell
  const long long plane = (long long)ld * nz * EW;  // shadow planes: vx, vz, sxx, szz, sxz
  // ---- load the tile and its surroundings
  for (int i = tid; i < (TZ + 8) * (WX / 4); i += NT) {
    const int r = i / (WX / 4), c = 4 * (i % (WX / 4)), gi = x0 - 4 + c, gj = z0 - 4 + r;
    const bool in = gi + 4 <= ld && gj < nz;
    const long long g = (long long)gj * ld + gi;
    const Q4<T> zero = splat4<T>(T(0));
    stg4(s_vx + r * WX + c, in ? ldcg4(a.vx + g) : zero);
    stg4(s_vz + r * WX + c, in ? ldcg4(a.vz + g) : zero);
    stg4(s_xz + r * WX + c, in ? ldcg4(a.sxz + g) : zero);
    if (r >= 4 && r < TZ + 4) stg4(s_xx + (r - 4) * WX + c, in ? ldcg4(a.sxx + g) : zero);
    if (c >= 4 && c < TX + 4) stg4(s_zz + r * TX + c - 4, in ? ldcg4(a.szz + g) : zero);
  }
  for (int i = tid; i < 6 * w; i += NT) s_tx[i / w * TX + i % w] = a.tx[(long long)(i / w) * nx + x0 + i % w];
  for (int i = tid; i < 6 * h; i += NT) s_tz[i / h * TZ + i % h] = a.tz[(long long)(i / h) * nz + z0 + i % h];
  // the thread's cells: row r, columns lx .. lx + W - 1 of the tile
  const int r = tid / (w / W), lx = W * (tid % (w / W));
  const bool act = r < h;
  const int gi0 = x0 + lx, gj = z0 + r, o = r * TX + lx;
  const long long c0 = (long long)gj * ld + gi0;
  unsigned xmask = 0;
  int zs = -1;
  P m[3 * (NSLS > 0 ? NSLS : 1)];
  if (act) {
#pragma unroll
    for (int k = 0; k < 3 * NSLS; ++k)
#pragma unroll
      for (int q = 0; q < W; ++q) m[k].v[q] = __ldcg(a.m + k * a.mstride + c0 + q);
    zs = strip_z(gj, nz, a.Tz, a.Bz);
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const long long c = c0 + k;
      // coefficients as the split kernels form them
      const T c13 = __ldg(a.c13 + c), c55 = __ldg(a.c55 + c), r0 = __ldg(a.rho + c);
      const T sum = add_rn(add_rn(add_rn(c55, __ldg(a.c55 + c + 1)), __ldg(a.c55 + c + ld)), __ldg(a.c55 + c + ld + 1));
      s_co[o + k] = KIND == VI_MEDIUM_ISO ? fma_rn(T(2), c55, c13) : __ldg(a.c11 + c);
      s_co[PC + o + k] = c13;
      if (KIND != VI_MEDIUM_ISO) s_co[2 * PC + o + k] = __ldg(a.c33 + c);
      s_co[3 * PC + o + k] = mul_rn(T(0.25), sum);
      if (NSLS > 0) s_co[4 * PC + o + k] = __ldg(a.tau + c);
      s_co[5 * PC + o + k] = two_over_s(add_rn(r0, __ldg(a.rho + c + 1)));
      s_co[6 * PC + o + k] = two_over_s(add_rn(r0, __ldg(a.rho + c + ld)));
      const int xs = strip_x(gi0 + k, nx, a.Lx, a.Rx);
      if (xs >= 0) {
        xmask |= 1u << k;
#pragma unroll
        for (int q = 0; q < 4; ++q) s_px[q * PC + o + k] = a.psix[q * a.psix_plane + (long long)gj * a.wx + xs];
      }
      if (zs >= 0)
#pragma unroll
        for (int q = 0; q < 4; ++q) s_pz[q * PC + o + k] = a.psiz[q * a.psiz_plane + (long long)zs * a.ldz + gi0 + k];
    }
  }
  const unsigned zmask = zs >= 0 ? (1u << W) - 1 : 0;
  // ---- the thread's share of the neighbours' edges: 2 planes x (rows to the
  // left and right, 4 rows of groups above and below)
  constexpr int kItems = 2;
  HaloItem item[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    int q = tid + k * NT;
    item[k].gv = nullptr;
    item[k].gs = nullptr;
    item[k].sv = item[k].ss = 0;
    const int nside = 2 * h, nrow = 8 * wg;
    int side = -1, p = 0, hr = 0, hc = 0;
    if (nl) {
      if (q < nside) side = 0;
      else q -= nside;
    }
    if (side < 0 && nr) {
      if (q < nside) side = 1;
      else q -= nside;
    }
    if (side < 0 && nu) {
      if (q < nrow) side = 2;
      else q -= nrow;
    }
    if (side < 0 && nd && q < nrow) side = 3;
    if (side < 0) continue;
    if (side < 2) {
      p = q / h;
      hr = q % h;
      hc = side == 0 ? -4 : w;
    } else {
      p = q / (4 * wg);
      hr = (q % (4 * wg)) / wg + (side == 2 ? -4 : h);
      hc = 4 * (q % wg);
    }
    const uint32_t *g = shadow + ((long long)(z0 + hr) * ld + x0 + hc) * EW;
    item[k].gv = g + p * plane;
    item[k].gs = g + (p ? 4 : side < 2 ? 2 : 3) * plane;
    item[k].sv = (int)((p ? s_vz : s_vx) - s_vx) + (hr + 4) * WX + hc + 4;
    item[k].ss = p ? (int)(s_xz - s_vx) + (hr + 4) * WX + hc + 4
                   : side < 2 ? (int)(s_xx - s_vx) + hr * WX + hc + 4 : (int)(s_zz - s_vx) + (hr + 4) * TX + hc;
  }
  // waits for the neighbours' edges of pass n and stores them (every thread
  // has finished the pass before any halo is overwritten); false: gave up
  auto exchange = [&](uint32_t n, bool stress) {
    __syncthreads();
    bool ok = true;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t *g = stress ? item[k].gs : item[k].gv;
      if (!g) continue;
      Q4<T> q;
      unsigned tries = 0;
      while (!ld_edge(g, q, n) && ++tries < (1u << 22)) {}
      ok &= tries < (1u << 22);
      stg4(s_vx + (stress ? item[k].ss : item[k].sv), q);
    }
    if (!ok) atomicOr(x.err, kErrTimeout);
    return !__syncthreads_or(!ok);
  };
  const int e0 = x.tile_off[cta], e1 = x.tile_off[cta + 1];
  const bool ex = act && ((nl && lx < 4) || (nr && lx >= w - 4)), ez = act && ((nu && r < 4) || (nd && r >= h - 4));
  const bool surf = x.fs && gj == L;
  const T dt = a.dt;
  const P dt4 = wsplat<T, W>(dt);
  T *const pvx = s_vx + (r + 4) * WX + lx + 4, *const pvz = s_vz + (r + 4) * WX + lx + 4;
  T *const pxx = s_xx + r * WX + lx + 4, *const pzz = s_zz + (r + 4) * TX + lx, *const pxz = s_xz + (r + 4) * WX + lx + 4;
  uint32_t *const edge = shadow + c0 * EW;
  __syncthreads();
  for (int s = 0; s < nsteps; ++s) {
    const int it = it0 + s;
    // ---- velocity pass
    if (act) {
      const Win<T, W> wxz(pxz);
      P dxx = wdxp(Win<T, W>(pxx), a.Dx), dxxz = wdxm(wxz, a.Dx);
      P zxz = wdzm<T, W>(pxz, WX, a.Dz), zzz = wdzp<T, W>(pzz, TX, a.Dz);
      if (xmask) {
        wcpml(xmask, s_px + PX_SXX * PC + o, s_tx + lx, TX, 1, T_BH, T_AH, T_IKH, dxx);
        wcpml(xmask, s_px + PX_SXZ * PC + o, s_tx + lx, TX, 1, T_B, T_A, T_IK, dxxz);
      }
      if (zmask) {
        wcpml(zmask, s_pz + PZ_SXZ * PC + o, s_tz + r, TZ, 0, T_B, T_A, T_IK, zxz);
        wcpml(zmask, s_pz + PZ_SZZ * PC + o, s_tz + r, TZ, 0, T_BH, T_AH, T_IKH, zzz);
      }
      const P bx = wld<T, W>(s_co + 5 * PC + o), bz = wld<T, W>(s_co + 6 * PC + o);
      P vxn = wfma(wmul(dt4, bx), wadd(dxx, zxz), wld<T, W>(pvx));
      P vzn = wfma(wmul(dt4, bz), wadd(dxxz, zzz), wld<T, W>(pvz));
      for (int e = e0; e < e1; ++e) {  // force sources of this tile (listed first)
        const int4 en = x.tile_ent[e];
        if (en.w > TL_FORCE_Z) break;
        if (en.y != gj || en.x < gi0 || en.x >= gi0 + W) continue;
        const int k = en.x - gi0;
        const T wv = it < x.wnt ? x.wavelet[(long long)en.z * x.wnt + it] : T(0);
        const T f = x.amp[en.z] * wv;
        if (en.w == TL_FORCE_X)
          wadd_lane(vxn, k, dt * wlane(bx, k) * f);
        else
          wadd_lane(vzn, k, dt * wlane(bz, k) * f);
      }
      if (ex || ez) {
        st_edge(edge, vxn, pass0 + 2 * s);
        st_edge(edge + plane, vzn, pass0 + 2 * s);
      }
      wst(pvx, vxn);
      wst(pvz, vzn);
    }
    if (!exchange(pass0 + 2 * s, false)) return;
    if (x.traces && it < x.tnt)
      for (int e = e0 + tid; e < e1; e += NT) {
        const int4 en = x.tile_ent[e];
        if (en.w != TL_RECEIVER) continue;
        const int q = (en.y - z0 + 4) * WX + en.x - x0 + 4;
        x.traces[(long long)en.z * x.tnt + it] = s_vx[q];
        x.traces[(long long)(x.nrec + en.z) * x.tnt + it] = s_vz[q];
      }
    // ---- stress pass
    if (act) {
      const Win<T, W> wvx(pvx), wvz(pvz);
      P rxx = wdxm(wvx, a.Dx), dxvz = wdxp(wvz, a.Dx);
      P rzz = wdzm<T, W>(pvz, WX, a.Dz), dzvx = wdzp<T, W>(pvx, WX, a.Dz);
      if (xmask) {
        wcpml(xmask, s_px + PX_VX * PC + o, s_tx + lx, TX, 1, T_B, T_A, T_IK, rxx);
        wcpml(xmask, s_px + PX_VZ * PC + o, s_tx + lx, TX, 1, T_BH, T_AH, T_IKH, dxvz);
      }
      if (zmask) {
        wcpml(zmask, s_pz + PZ_VZ * PC + o, s_tz + r, TZ, 0, T_B, T_A, T_IK, rzz);
        wcpml(zmask, s_pz + PZ_VX * PC + o, s_tz + r, TZ, 0, T_BH, T_AH, T_IKH, dzvx);
      }
      const P rxz = wadd(dzvx, dxvz);
      P exx = rxx, ezz = rzz, exz = rxz;
      if constexpr (NSLS > 0) {
        P Sxx = m[0], Szz = m[NSLS], Sxz = m[2 * NSLS];
#pragma unroll
        for (int n = 1; n < NSLS; ++n) {
          Sxx = wadd(Sxx, m[0 * NSLS + n]);
          Szz = wadd(Szz, m[1 * NSLS + n]);
          Sxz = wadd(Sxz, m[2 * NSLS + n]);
        }
        const P tau = wld<T, W>(s_co + 4 * PC + o), t1 = wadd(tau, wsplat<T, W>(T(1)));
        exx = wfma(t1, rxx, wmul(tau, Sxx));
        ezz = wfma(t1, rzz, wmul(tau, Szz));
        exz = wfma(t1, rxz, wmul(tau, Sxz));
      }
      const P C11 = wld<T, W>(s_co + o), C13 = wld<T, W>(s_co + PC + o);
      const P C33 = KIND == VI_MEDIUM_ISO ? C11 : wld<T, W>(s_co + 2 * PC + o);
      const P C55h = wld<T, W>(s_co + 3 * PC + o);
      if (surf) {
#pragma unroll
        for (int k = 0; k < W; ++k) ezz.v[k] = -(C13.v[k] * exx.v[k]) / C33.v[k];
      }
      P sxx = wfma(dt4, wfma(C11, exx, wmul(C13, ezz)), wld<T, W>(pxx));
      P szz = wfma(dt4, wfma(C13, exx, wmul(C33, ezz)), wld<T, W>(pzz));
      P sxz = wfma(dt4, wmul(C55h, exz), wld<T, W>(pxz));
      for (int e = e0; e < e1; ++e) {  // explosive sources (after the force ones, before receivers)
        const int4 en = x.tile_ent[e];
        if (en.w < TL_EXPLOSIVE) continue;
        if (en.w > TL_EXPLOSIVE) break;
        if (en.y != gj || en.x < gi0 || en.x >= gi0 + W) continue;
        const T wv = it < x.wnt ? x.wavelet[(long long)en.z * x.wnt + it] : T(0);
        wadd_lane(sxx, en.x - gi0, dt * x.amp[en.z] * wv);
        wadd_lane(szz, en.x - gi0, dt * x.amp[en.z] * wv);
      }
      if (surf) szz = wsplat<T, W>(T(0));
      if (ex) st_edge(edge + 2 * plane, sxx, pass0 + 2 * s + 1);
      if (ez) st_edge(edge + 3 * plane, szz, pass0 + 2 * s + 1);
      if (ex || ez) st_edge(edge + 4 * plane, sxz, pass0 + 2 * s + 1);
      wst(pxx, sxx);
      wst(pzz, szz);
      wst(pxz, sxz);
#pragma unroll
      for (int n = 0; n < NSLS; ++n) {
        const P a1 = wsplat<T, W>(a.a1[n]), a2 = wsplat<T, W>(a.a2[n]);
        P &m0 = m[n], &m1 = m[NSLS + n], &m2 = m[2 * NSLS + n];
        m0 = wfma(dt4, wfma(a1, rxx, wmul(a2, m0)), m0);
        m1 = surf ? wsplat<T, W>(T(0)) : wfma(dt4, wfma(a1, rzz, wmul(a2, m1)), m1);
        m2 = wfma(dt4, wfma(a1, rxz, wmul(a2, m2)), m2);
      }
      bool bad = false;
#pragma unroll
      for (int k = 0; k < W; ++k) bad |= !isfinite((sxx.v[k] + szz.v[k]) + sxz.v[k]);
      if (bad) atomicOr(x.err, kErrNonFinite);
      if (x.fs == kFsImaging) {
        // stress images, in the halo rows above a tile that starts at the surface
        const int k = gj - L;
        P im;
        if (k >= 1 && k <= L) {
#pragma unroll
          for (int q = 0; q < W; ++q) im.v[q] = -szz.v[q];
          wst(pzz - 2 * k * TX, im);
        }
        if (k >= 0 && k < L) {
#pragma unroll
          for (int q = 0; q < W; ++q) im.v[q] = -sxz.v[q];
          wst(pxz - (2 * k + 1) * WX, im);
        }
      }
    }
    if (s + 1 < nsteps && !exchange(pass0 + 2 * s + 1, true)) return;
  }
  // ---- the state back to the global planes
  if (!act) return;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const long long c = c0 + k;
    a.vx[c] = pvx[k];
    a.vz[c] = pvz[k];
    a.sxx[c] = pxx[k];
    a.szz[c] = pzz[k];
    a.sxz[c] = pxz[k];
#pragma unroll
    for (int q = 0; q < 3 * NSLS; ++q) a.m[q * a.mstride + c] = m[q].v[k];
    if (x.fs == kFsImaging) {
      const int q = gj - L;
      if (q >= 1 && q <= L) a.szz[c - 2LL * q * ld] = -pzz[k];
      if (q >= 0 && q < L) a.sxz[c - (2LL * q + 1) * ld] = -pxz[k];
    }
    if (xmask >> k & 1) {
      const int xs = strip_x(gi0 + k, nx, a.Lx, a.Rx);
#pragma unroll
      for (int q = 0; q < 4; ++q) a.psix[q * a.psix_plane + (long long)gj * a.wx + xs] = s_px[q * PC + o + k];
    }
    if (zs >= 0)
#pragma unroll
      for (int q = 0; q < 4; ++q) a.psiz[q * a.psiz_plane + (long long)zs * a.ldz + gi0 + k] = s_pz[q * PC + o + k];
  }
}

// ------------------------------------------------------------------- host
// The tiling with the fewest groups on its fullest CTA (ties: the shortest
// edges), or none: at least 4 rows in every tile (a halo comes from one
// neighbour), at least 5 in the first under a free surface (its images), the
// CTA's state within its shared memory and registers.  A thread takes as few
// cells as the CTA's threads allow: a pass is a chain of a few hundred
// dependent operations per thread, so narrow threads finish it sooner (256 x
// 256 FP32: 4.1 us a step with one cell each, 6.3 with four) until they no
// longer fit.
template <typename T>
static bool res_geometry(const vi_config &c, int nsm, ResGeom &out) {
  const int gx = (c.nx - 2 * L) / 4, rows = c.nz - 2 * L;
  const int max_cells = 2 * res_max_threads<T>();
  bool found = false;
  long long best = 0;
  for (int txg = 1; txg <= gx; ++txg) {
    const int px = (gx + txg - 1) / txg;
    if (px > nsm) continue;
    for (int pz = std::min(nsm / px, rows / 4); pz >= 1; --pz) {
      const int tz = (rows + pz - 1) / pz, used = (rows + tz - 1) / tz, last = rows - (used - 1) * tz;
      if (last < 4 || (c.free_surface && tz < L + 1)) continue;
      const int n = txg * tz, cells = 4 * n, items = 4 * tz + 16 * txg;
      const long long cost = (long long)n * 64 + items;
      if (cells > max_cells || (found && cost >= best)) break;  // fewer rows of tiles only grow the tile
      const int width = cells <= res_max_threads<T>() ? 1 : 2;
      const int threads = (cells / width + 31) / 32 * 32;
      const size_t smem = res_smem<T>(txg, tz);
      if (items > 2 * threads || smem > kResMaxSmem) continue;
      found = true;
      best = cost;
      out = ResGeom{txg, tz, px, used, threads, width, smem};
      break;
    }
  }
  return found;
}

// the plan's tiling, looked for once
template <typename T>
static bool res_plan_geometry(vi_plan *p, ResGeom &g) {
  if (p->res_fits < 0) {
    p->res_fits = res_geometry<T>(p->cfg, p->nsm, g);
    if (p->res_fits) {
      const int v[6] = {g.txg, g.tz, g.px, g.pz, g.threads, g.width};
      std::copy(v, v + 6, p->res_geom);
      p->res_smem = g.smem;
    }
  }
  const int *v = p->res_geom;
  g = ResGeom{v[0], v[1], v[2], v[3], v[4], v[5], p->res_smem};
  return p->res_fits == 1;
}

bool resident_eligible_cfg(vi_plan *p, int nsteps, cudaStream_t st) {
  const vi_config &c = p->cfg;
  if (nsteps < kResidentMinSteps || p->no_resident || c.medium == VI_MEDIUM_TTI || c.precision == VI_F32C ||
      c.free_surface == kFsAfda || c.nx % 4 != 0)
    return false;
  ResGeom g;
  if (!(c.precision == VI_F64 ? res_plan_geometry<double>(p, g) : res_plan_geometry<float>(p, g))) return false;
  // with other plans' steps in flight only grids whose CTAs leave most of an SM
  // free: 8 streams of 128 x 128 VTI steps took 0.73 us per shot and step here
  // against 1.65 for the pair, of 512 x 256 4.7 against 2.7
  return g.threads <= 128 || !others_in_flight(p, st);
}

template <typename T, int KIND, int NSLS, int W>
static int launch_resident_w(const StepArgs<T> &a, const FusedExtras<T> &x, const ResGeom &g, int it0, int nsteps,
                             uint32_t *shadow, uint32_t pass0, cudaStream_t st) {
  auto k = k_resident<T, KIND, NSLS, W>;
  // one value whatever the tiling: the limit is the kernel's, and another thread
  // may launch it for another grid between this call and the launch
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResMaxSmem);
  if (e != cudaSuccess) return cuda_check(e, "resident step smem attribute");
  StepArgs<T> av = a;
  FusedExtras<T> xv = x;
  ResGeom gv = g;
  void *args[] = {&av, &xv, &gv, &it0, &nsteps, &shadow, &pass0};
  e = cudaLaunchCooperativeKernel((const void *)k, dim3(g.px * g.pz), dim3(g.threads), args, g.smem, st);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return set_error(VI_ERR_BUDGET, "resident step: the device cannot hold the launch");
  }
  return cuda_check(e, "resident step launch");
}
// A call runs as launches of at most this many steps, about a millisecond, so that
// a kernel of another stream that does not fit beside the resident CTAs waits for
// one launch, not for the call: a 4096^3 BF16 product issued after 3000 steps of
// 512 x 512 took 21.8 ms with one launch, 0.4 with 128 steps each, 0.37 with 64,
// 1.4 with 256 (0.16 beside the pair); of 256 x 256 10.3, 0.31, 0.23 and 0.36 ms.
// Another launch costs the state's way out and in: 3000 steps of 512 x 512 22.73
// -> 22.94 ms (64: 23.30), 256 x 256 10.74 -> 10.80 with 256 steps each (128:
// 10.89, 64: 11.06).  Tilings with one cell a thread take half as long a step.
constexpr int res_launch_steps(int width) { return width == 1 ? 256 : 128; }
template <typename T, int KIND, int NSLS>
static int launch_resident(const StepArgs<T> &a, const FusedExtras<T> &x, const ResGeom &g, int it0, int nsteps,
                           uint32_t *shadow, uint32_t pass0, cudaStream_t st) {
  const int most = res_launch_steps(g.width), launches = nsteps / most + (nsteps % most != 0);
  for (int k = 0, done = 0; k < launches; ++k) {
    const int n = (nsteps - done) / (launches - k);  // even shares
    const uint32_t pass = pass0 + 2u * (uint32_t)done;
    const int rc = g.width == 1 ? launch_resident_w<T, KIND, NSLS, 1>(a, x, g, it0 + done, n, shadow, pass, st)
                                : launch_resident_w<T, KIND, NSLS, 2>(a, x, g, it0 + done, n, shadow, pass, st);
    if (rc) return k > 0 && rc == VI_ERR_BUDGET ? VI_ERR_CUDA : rc;  // "having done nothing" holds for the first alone
    done += n;
  }
  return VI_OK;
}

template <typename T>
int resident_steps(vi_plan *p, StepArgs<T> a, const vi_shot *s, int it0, int nsteps, cudaStream_t st) {
  const vi_config &c = p->cfg;
  ResGeom g;
  if (!res_plan_geometry<T>(p, g)) return set_error(VI_ERR_ARG, "resident step: the grid does not fit on the chip");
  int ntx, ntz;
  std::vector<int> off;
  std::vector<int4> ent;
  build_tile_lists(c.nx, c.nz, 4 * g.txg, g.tz, 0, s, off, ent, ntx, ntz);
  int *d_off = nullptr;
  int4 *d_ent = nullptr;
  int rc = stage_tile_lists(p, off, ent, st, &d_off, &d_ent);
  if (rc) return rc;
  // the shadow planes, zero at first; passes are numbered on from call to call
  // (1 up; they start over, on a cleared shadow, before the count wraps)
  const size_t sbytes = 5 * (size_t)a.ld * c.nz * 2 * sizeof(T);
  const bool fresh = p->shadow_bytes < sbytes;
  if ((rc = ensure_buffer(p, &p->shadow, &p->shadow_bytes, sbytes))) return rc;
  if (fresh || p->shadow_pass > 0xffffffffu - 2u * (uint32_t)nsteps - 2u) {
    if ((rc = cuda_check(cudaMemsetAsync(p->shadow, 0, sbytes, st), "zero edge shadow"))) return rc;
    p->shadow_pass = 1;
  }
  uint32_t *const shadow = (uint32_t *)p->shadow;
  const uint32_t pass0 = p->shadow_pass;
  p->shadow_pass += 2u * (uint32_t)nsteps;
  FusedExtras<T> x{};
  x.ntx = ntx;
  x.fs = c.free_surface;
  x.tile_off = d_off;
  x.tile_ent = d_ent;
  x.amp = (const T *)p->damp;
  x.wavelet = (s && s->nsrc) ? (const T *)s->wavelet_dev : nullptr;
  x.wnt = (s && s->nsrc) ? s->wavelet_nt : 0;
  x.traces = (s && s->nrec) ? (T *)s->traces_dev : nullptr;
  x.tnt = (s && s->nrec) ? s->traces_nt : 0;
  x.nrec = s ? s->nrec : 0;
  x.err = (int *)p->errflag;
  if (a.psix) a.psix = a.psix_o = (T *)p->psix + p->psi_cur * kPsiPerSet * p->psix_plane;
  if (a.psiz) a.psiz = a.psiz_o = (T *)p->psiz + p->psi_cur * kPsiPerSet * p->psiz_plane;
#define VB_CASE(K, N) \
  if (c.medium == K && c.nsls == N) return launch_resident<T, K, N>(a, x, g, it0, nsteps, shadow, pass0, st);
#define VB_KIND(K) VB_CASE(K, 0) VB_CASE(K, 1) VB_CASE(K, 2) VB_CASE(K, 3) VB_CASE(K, 4) VB_CASE(K, 5)
  VB_KIND(VI_MEDIUM_ISO)
  VB_KIND(VI_MEDIUM_VTI)
#undef VB_KIND
#undef VB_CASE
  return set_error(VI_ERR_ARG, "the resident step covers ISO and VTI media");
}
template int resident_steps<float>(vi_plan *, StepArgs<float>, const vi_shot *, int, int, cudaStream_t);
template int resident_steps<double>(vi_plan *, StepArgs<double>, const vi_shot *, int, int, cudaStream_t);

}  // namespace vb
