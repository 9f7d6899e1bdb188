// lmc_ysweep.cuh -- y kernels of one lomacte RK3 substep for grids with many
// (kx,kz) modes: one thread per mode, sweeping along y.
//
// In the spectral layout [y][kx][kz] the threads of a warp (32 consecutive
// modes) read and write every row of their pencils as one coalesced run and
// share the coefficients of the row, so these kernels issue the fewest
// instructions per point; with enough modes to fill the device they run at
// the bandwidth of the bytes they move.  (Pencils held in registers,
// lmc_ychunk.cuh, move fewer bytes, but every chunk loads its coefficients
// anew and takes part in the scans: the RK3 update of 256 x 257 x 256 with
// float2 buffers takes 1.53 ms there and 0.73 ms here.)  What is left to save
// is passes over memory:
//  * A banded solve takes two sweeps with an FP64 scratch pencil between
//    them.  In t_post the operators applied to the result of a backward
//    sweep are factorised the other way round, A = U' L', so that their
//    first half rides on that sweep and only the second half needs another.
//  * The derivatives are gathered by linearity, lap(T) = d2T/dy2 - k2 T comes
//    from the band product dt22 - k2 dt21 (no second read of T), and only
//    the wall rows of T and Z are written by their derivatives' kernel.
// Fields are streamed through small queues of registers that are refilled K
// rows ahead of use, so every thread keeps several loads in flight.
//
// Per substep of 768 x 65 x 768 (mu = T^0.7, scalar, float2 buffers), with
// the sweeps that passed N_i, the curls and the scratch through memory:
// RK3 update 2272 -> 1588 us (with T's own update), T and Z derivatives 814
// -> 816, psi (chunked) 448 -> 393, all y kernels 5.66 -> 4.74 ms; 256 x 257 x
// 256: 1204 -> 781, 684 -> 473, 297 -> 190 us, 3.54 -> 2.44 ms.
#pragma once
#include "lmc_ytpm.cuh"

namespace lmc {
namespace tpm {

template <bool B>
struct BoolC {
  static constexpr bool value = B;
};

// this thread's scratch pencil k
__device__ __forceinline__ double2 *scr(const Dev &d, int k, int slot) {
  return d.ws[k] + slot;
}

// the same for one real coefficient per row (per-mode tables)
template <int K>
struct RdS {
  const double *p;
  size_t ld;
  int my, dir, nxt;
  double q[K];
  __device__ __forceinline__ double fetch(int r) const {
    return (r >= 0 && r < my) ? __ldg(p + (size_t)r * ld) : 0.0;
  }
  __device__ __forceinline__ void start(const double *base, size_t ld_, int my_, int dir_, int first) {
    p = base;
    ld = ld_;
    my = my_;
    dir = dir_;
    nxt = first;
#pragma unroll
    for (int t = 0; t < K; t++) {
      q[t] = fetch(nxt);
      nxt += dir;
    }
  }
  __device__ __forceinline__ double pop() {
    const double v = q[0];
#pragma unroll
    for (int t = 0; t < K - 1; t++) q[t] = q[t + 1];
    q[K - 1] = fetch(nxt);
    nxt += dir;
    return v;
  }
};

// a row pushed at the low end (descending sweeps)
__device__ __forceinline__ void push_low(Win &w, double2 v) {
#pragma unroll
  for (int t = 6; t > 0; t--) w.u[t] = w.u[t - 1];
  w.u[0] = v;
}

// band product of d/dy (dt12) and of d2/dy2 - kk (dt22 - kk dt21) at row j
__device__ __forceinline__ double2 b1(const Dev &d, int j, const Win &u) {
  const double *c = d.r_dt12 + 7 * j;
  double2 r = czero();
#pragma unroll
  for (int t = 0; t < 7; t++) {
    const double k = __ldg(c + t);
    r.x = fma(k, u.u[t].x, r.x);
    r.y = fma(k, u.u[t].y, r.y);
  }
  return r;
}
__device__ __forceinline__ double2 b2(const Dev &d, int j, double kk, const Win &u) {
  const double *c = d.r_dt22 + 5 * j, *e = d.r_dt21 + 5 * j;
  double2 r = czero();
#pragma unroll
  for (int t = 0; t < 5; t++) {
    const double k = fma(-kk, __ldg(e + t), __ldg(c + t));
    r.x = fma(k, u.u[t + 1].x, r.x);
    r.y = fma(k, u.u[t + 1].y, r.y);
  }
  return r;
}
// first and second halves of a banded solve at row j: T has B multipliers
// per row, or the reciprocal pivot and B multipliers; h the last results
template <int B>
__device__ __forceinline__ double2 half1(const double *T, int j, double2 r, Hist &h) {
  const double *l = T + B * j;
  if (B > 2) r = fms(r, __ldg(l + 2), h.c);
  r = fms(fms(r, __ldg(l + 1), h.b), __ldg(l), h.a);
  h.push(r);
  return r;
}
template <int B>
__device__ __forceinline__ double2 half2(const double *T, int j, double2 r, Hist &h) {
  const double *u = T + (B + 1) * j;
  if (B > 2) r = fms(r, __ldg(u + 3), h.c);
  r = cscale(__ldg(u), fms(fms(r, __ldg(u + 2), h.b), __ldg(u + 1), h.a));
  h.push(r);
  return r;
}

__device__ __forceinline__ bool mode_at(const Dev &d, Mode &M) {
  const int i = M.m / d.mz, k = M.m - i * d.mz;
  M.kx = __ldg(d.kx + i);
  M.kz = __ldg(d.kz + k);
  M.k2 = __ldg(d.k2 + M.m);
  return true;
}

// one mode per thread, its scratch rows at the stride of a field
#define LMC_SWEEP_MODE                                                    \
  const int my = d.my, slot = blockIdx.x * YS_TB + threadIdx.x;           \
  const size_t ld = d.nmode, ls = ld;                                     \
  Mode M;                                                                 \
  M.m = slot;                                                             \
  if (M.m >= d.nmode) return;                                             \
  mode_at(d, M);
// the modes slot, slot + stride, ... of a persistent grid, the scratch rows
// at its stride
#define LMC_SWEEP_MODES                                                                \
  const int my = d.my, slot = blockIdx.x * YS_TB + threadIdx.x, G = gridDim.x * YS_TB; \
  const size_t ld = d.nmode, ls = G;                                                   \
  Mode M;                                                                              \
  for (M.m = slot; M.m < d.nmode && mode_at(d, M); M.m += G)

// ----------------------------------------------------------------------
// (1) Lapvdvhom (cross.f:329-335, 365-372): phi -> m_y, dm_y/dy
// ----------------------------------------------------------------------
template <typename CT>
__global__ void __launch_bounds__(YS_TB) t_lapv(Dev d) {
  LMC_SWEEP_MODE
  {
    double2 *s = scr(d, 0, slot);
    {  // forward half of the Poisson solve; phi with its wall values set to zero
      Rd<double2, 8> r;
      r.start(d.phi + M.m, ld, my, 1, 0);
      RdS<8> l0, l1;
      l0.start(d.PLt + M.m, 2 * ld, my, 1, 0);
      l1.start(d.PLt + ld + M.m, 2 * ld, my, 1, 0);
      Win w;
      w.clear();
      Hist h;
      h.clear();
      for (int t = 0; t < 3; t++) {
        const double2 v = r.pop();
        w.push(t == 0 ? czero() : v);
      }
      #pragma unroll 4
      for (int j = 0; j < my; j++) {
        const double2 v = r.pop();
        w.push(j + 3 == my - 1 ? czero() : v);
        double2 b = czero();
        if (j > 0 && j < my - 1) {
          const double *c = d.r_dt21 + 5 * j;
#pragma unroll
          for (int t = 0; t < 5; t++) {
            const double k = __ldg(c + t);
            b.x = fma(k, w.u[t + 1].x, b.x);
            b.y = fma(k, w.u[t + 1].y, b.y);
          }
        }
        b = fms(fms(b, l1.pop(), h.b), l0.pop(), h.a);
        h.push(b);
        s[(size_t)j * ls] = b;
      }
    }
    double2 *s2 = scr(d, 3, slot);
    {  // backward half -> m_y
      Rd<double2, 8> r;
      r.start(s, ls, my, -1, my - 1);
      RdS<8> u0, u1, u2;
      u0.start(d.PUt + M.m, 3 * ld, my, -1, my - 1);
      u1.start(d.PUt + ld + M.m, 3 * ld, my, -1, my - 1);
      u2.start(d.PUt + 2 * ld + M.m, 3 * ld, my, -1, my - 1);
      CT *MY = wsb<CT>(d, SB_MY) + M.m;
      Hist h;
      h.clear();
      #pragma unroll 4
      for (int j = my - 1; j >= 0; j--) {
        const double p = u0.pop();
        const double2 x = cscale(p, fms(fms(r.pop(), u2.pop(), h.b), u1.pop(), h.a));  // zero for k2 = 0 (zero tables)
        h.push(x);
        put(MY, ld, j, x);
        s2[(size_t)j * ls] = x;
      }
    }
    {  // forward half of d/dy of m_y
      Rd<double2, 8> r;
      r.start(s2, ls, my, 1, 0);
      Win w;
      w.clear();
      Hist h;
      h.clear();
      for (int t = 0; t < 3; t++) w.push(r.pop());
      #pragma unroll 4
      for (int j = 0; j < my; j++) {
        w.push(r.pop());
        s[(size_t)j * ls] = d1f(d, j, w, h);
      }
    }
    {  // backward half -> dm_y/dy
      Rd<double2, 8> r;
      r.start(s, ls, my, -1, my - 1);
      CT *DMY = wsb<CT>(d, SB_DMY) + M.m;
      Hist h;
      h.clear();
      #pragma unroll 4
      for (int j = my - 1; j >= 0; j--) put(DMY, ld, j, d1b(d, j, r.pop(), h));
    }
  }
}

// ----------------------------------------------------------------------
// (2)-(3) m_x, m_z, rho u_i, xi-updates of Omega_y and phi, 00 modes
// (cross.f:315-327, 395-499)
// ----------------------------------------------------------------------
template <typename CT>
__global__ void __launch_bounds__(YS_TB) t_assemble(Dev d, int rk) {
  const double dtxi = d.scal_d[0] * d.xi[rk];
  LMC_SWEEP_MODE
  {
    const double ta = (M.k2 != 0.0) ? M.kx / M.k2 : 0.0, tb = (M.k2 != 0.0) ? M.kz / M.k2 : 0.0;
    const bool m00 = M.m == 0;
    double2 *s = scr(d, 0, slot);
    {
      Rd<double2, 3> rvor, rrom, rphi, rrph;
      Rd<CT, kq<CT>(3)> rdmy;
      Rd<double2, 4> rpsi;
      rvor.start(d.vor + M.m, ld, my, 1, 0);
      rrom.start(d.Rom + M.m, ld, my, 1, 0);
      rphi.start(d.phi + M.m, ld, my, 1, 0);
      rrph.start(d.Rphi + M.m, ld, my, 1, 0);
      rdmy.start(wsb<CT>(d, SB_DMY) + M.m, ld, my, 1, 0);
      rpsi.start(d.psi + M.m, ld, my, 1, 0);
      CT *RU = wsb<CT>(d, SB_RU) + M.m, *RW = wsb<CT>(d, SB_RW) + M.m;
      const double2 vor1 = __ldcg(d.vor + ld + M.m);  // wall BC of Omega_y, cross.f:315-327
      double2 vprev = czero();
      Win w;
      w.clear();
      Hist h;
      h.clear();
      for (int t = 0; t < 3; t++) w.push(rpsi.pop());
      #pragma unroll 4
      for (int j = 0; j < my; j++) {
        w.push(rpsi.pop());
        const double2 ps = w.c();
        const double2 vr = rvor.pop();
        const double2 vo = (j == 0) ? vor1 : (j == my - 1) ? vprev : vr;
        vprev = vr;
        const double2 a = rdmy.pop();
        double2 b = cadd(csub(cik(ta, a), cik(tb, vo)), cik(M.kx, ps));   // rho u, cross.f:402,467
        double2 c = cadd(cadd(cik(tb, a), cik(ta, vo)), cik(M.kz, ps));   // rho w, cross.f:404,469
        if (m00) {  // 00 modes injected (cross.f:486-491), then u00**, w00** (cross.f:495-498)
          b = make_double2(d.u00[j], 0.0);
          c = make_double2(d.w00[j], 0.0);
          if constexpr (mixed<CT>()) {
            d.mi[j] = b.x;
            d.mi[(size_t)2 * my + j] = c.x;
          }
          if (j >= 1 && j <= my - 2) {
            d.u00[j] += dtxi * d.rf0u[j];
            d.w00[j] += dtxi * d.rf0w[j];
          }
        }
        put(RU, ld, j, b);
        put(RW, ld, j, c);
        put(d.vor + M.m, ld, j, cadd(vo, cscale(dtxi, rrom.pop())));  // cross.f:420-424
        double2 ph = rphi.pop();
        if (j == 0 || j == my - 1) ph = czero();
        put(d.phi + M.m, ld, j, cadd(ph, cscale(dtxi, rrph.pop())));  // cross.f:424-425
        s[(size_t)j * ls] = d1f(d, j, w, h);
      }
    }
    {  // rho v = m_y + d(psi)/dy (cross.f:434-437, 471)
      Rd<double2, 4> r;
      Rd<CT, kq<CT>(4)> rmy;
      r.start(s, ls, my, -1, my - 1);
      rmy.start(wsb<CT>(d, SB_MY) + M.m, ld, my, -1, my - 1);
      CT *RV = wsb<CT>(d, SB_RV) + M.m;
      Hist h;
      h.clear();
      #pragma unroll 4
      for (int j = my - 1; j >= 0; j--) {
        double2 a = cadd(d1b(d, j, r.pop(), h), rmy.pop());
        if (m00) {
          a = make_double2(d.v00[j], 0.0);
          if constexpr (mixed<CT>()) d.mi[(size_t)my + j] = a.x;
        }
        put(RV, ld, j, a);
      }
    }
  }
}

// ----------------------------------------------------------------------
// (4) T with its wall BCs, dT/dy, lap(T) (cross.f:336-349, 521-541); Z: the
// passive scalar, treated as T (its 00 mode held at scal_d[5], scal_d[6]; mi
// rows 6, 7).  lap = d2/dy2 - k2 by the band product dt22 - k2 dt21.  Runs
// on the second stream: scratch fields 1 and 2.
// ----------------------------------------------------------------------
template <typename CT, bool Z>
__global__ void __launch_bounds__(YS_TB) t_tder(Dev d) {
  LMC_SWEEP_MODES {
    const bool m00 = M.m == 0;
    double2 *s1 = scr(d, 1, slot), *s2 = scr(d, 2, slot);
    double2 *const f = (Z ? d.zsc : d.scal) + M.m;
    {
      Rd<double2, 8> r;
      r.start(f, ld, my, 1, 0);
      r.pop();
      const double2 wb = m00 ? make_double2(Z ? d.scal_d[5] : 1.0 / d.scal_d[3], 0.0) : czero();
      const double2 wt = m00 ? make_double2(Z ? d.scal_d[6] : 1.0 / d.scal_d[4], 0.0) : czero();
      f[0] = wb;  // the wall rows of the state; the sweep does not read them from memory
      f[(size_t)(my - 1) * ld] = wt;
      Win w;
      w.clear();
      Hist h1, h2;
      h1.clear();
      h2.clear();
      w.push(wb);
      for (int t = 1; t < 3; t++) w.push(r.pop());
      #pragma unroll 4
      for (int j = 0; j < my; j++) {
        const double2 v = r.pop();
        w.push(j + 3 == my - 1 ? wt : v);
        const double2 T = w.c();
        if constexpr (mixed<CT>()) {
          put(wsb<CT>(d, Z ? SB_Z32 : SB_T32) + M.m, ld, j, T);
          if (!Z && m00) d.mi[(size_t)5 * my + j] = T.x;
        }
        s1[(size_t)j * ls] = d1f(d, j, w, h1);
        s2[(size_t)j * ls] = half1<2>(d.r_p3L, j, b2(d, j, M.k2, w), h2);
      }
    }
    {
      Rd<double2, 6> r1, r2;
      r1.start(s1, ls, my, -1, my - 1);
      r2.start(s2, ls, my, -1, my - 1);
      CT *DY = wsb<CT>(d, Z ? SB_DZDY : SB_DTDY) + M.m, *LT = wsb<CT>(d, Z ? SB_LAPZ : SB_LAPT) + M.m;
      Hist h1, h2;
      h1.clear();
      h2.clear();
      #pragma unroll 4
      for (int j = my - 1; j >= 0; j--) {
        const double2 dT = d1b(d, j, r1.pop(), h1), lT = half2<2>(d.r_p3U, j, r2.pop(), h2);
        if constexpr (mixed<CT>())
          if (m00) {
            d.mi[(size_t)(Z ? 7 : 4) * my + j] = dT.x;
            d.mi[(size_t)(Z ? 6 : 3) * my + j] = lT.x;
          }
        put(DY, ld, j, dT);
        put(LT, ld, j, lT);
      }
    }
  }
}

// ----------------------------------------------------------------------
// Variable viscosity: the spectral inputs of the strain rates.  In
// physical space d(u_i)/dx_j = T d(rho u_i)/dx_j + rho u_i dT/dx_j, and the
// stress needs d(rho u_i)/dx_j only in the symmetric sums; this kernel
// writes d(rho v)/dy and the three off-diagonal sums (d(rho u)/dx is formed
// by the x stage, d(rho w)/dz by the inverse z transforms from rho w).
// The y derivatives are deryr2's (cfdiff.f:518-601), as every first y
// derivative of the substep.  Runs after t_assemble on the same stream;
// scratch fields 0, 3 and 4 hold the forward halves (1 and 2 belong to
// t_tder on the second stream).
// The mixed forms also form the 00 profiles of the results exactly, from
// the FP64 profiles of rho u_i (mi rows 0..2) into mi rows 8..10.
// ----------------------------------------------------------------------
// an FP64 profile read as a pencil (imaginary parts zero)
struct RdM {
  RdS<4> s;
  __device__ __forceinline__ void start(const double *p, int my, int dir, int first) { s.start(p, 1, my, dir, first); }
  __device__ __forceinline__ double2 pop() { return make_double2(s.pop(), 0.0); }
};

// d/dy of the three pencils (forward halves into s0, s1, s2, then the
// backward halves), sink(j, du, dv, dw, u, v, w) per row, j descending;
// start(reader, field 0..2, direction, first row) opens the readers
template <typename RT, typename Start, typename Sink>
__device__ __forceinline__ void sgrad_pass(const Dev &d, size_t ls, double2 *s0, double2 *s1, double2 *s2,
                                           Start start, Sink sink) {
  const int my = d.my;
  {
    RT ru, rv, rw;
    start(ru, 0, 1, 0);
    start(rv, 1, 1, 0);
    start(rw, 2, 1, 0);
    Win wu, wv, ww;
    wu.clear();
    wv.clear();
    ww.clear();
    Hist hu, hv, hw;
    hu.clear();
    hv.clear();
    hw.clear();
    for (int t = 0; t < 3; t++) {
      wu.push(ru.pop());
      wv.push(rv.pop());
      ww.push(rw.pop());
    }
    #pragma unroll 2
    for (int j = 0; j < my; j++) {
      wu.push(ru.pop());
      wv.push(rv.pop());
      ww.push(rw.pop());
      s0[(size_t)j * ls] = d1f(d, j, wu, hu);
      s1[(size_t)j * ls] = d1f(d, j, wv, hv);
      s2[(size_t)j * ls] = d1f(d, j, ww, hw);
    }
  }
  Rd<double2, 3> r0, r1, r2;
  r0.start(s0, ls, my, -1, my - 1);
  r1.start(s1, ls, my, -1, my - 1);
  r2.start(s2, ls, my, -1, my - 1);
  RT ru, rv, rw;
  start(ru, 0, -1, my - 1);
  start(rv, 1, -1, my - 1);
  start(rw, 2, -1, my - 1);
  Hist hu, hv, hw;
  hu.clear();
  hv.clear();
  hw.clear();
  #pragma unroll 2
  for (int j = my - 1; j >= 0; j--) {
    const double2 du = d1b(d, j, r0.pop(), hu), dv = d1b(d, j, r1.pop(), hv), dw = d1b(d, j, r2.pop(), hw);
    sink(j, du, dv, dw, ru.pop(), rv.pop(), rw.pop());
  }
}

// The mixed forms launch one block more: its first thread runs the exact 00
// profiles (mi rows 0..2 into rows 8..10) beside the pencils; the FP32
// buffers' 00 coefficients are not read (the transforms drop them).
template <typename CT>
__global__ void __launch_bounds__(YS_TB) t_sgrad(Dev d) {
  const int my = d.my, nb = gridDim.x - (mixed<CT>() ? 1 : 0);
  const int slot = blockIdx.x * YS_TB + threadIdx.x, G = nb * YS_TB;
  const size_t ld = d.nmode, ls = G;
  if constexpr (mixed<CT>()) {
    if ((int)blockIdx.x == nb) {
      if (threadIdx.x != 0) return;
      sgrad_pass<RdM>(
          d, 1, d.vscr, d.vscr + my, d.vscr + 2 * my,
          [&](auto &r, int f, int dir, int first) { r.start(d.mi + (size_t)f * my, my, dir, first); },
          [&](int j, double2 du, double2 dv, double2 dw, double2, double2, double2) {
            d.mi[(size_t)8 * my + j] = dv.x;
            d.mi[(size_t)9 * my + j] = du.x;
            d.mi[(size_t)10 * my + j] = dw.x;
          });
      return;
    }
  }
  Mode M;
  for (M.m = slot; M.m < d.nmode && mode_at(d, M); M.m += G) {
    const CT *src[3] = {wsb<CT>(d, SB_RU) + M.m, wsb<CT>(d, SB_RV) + M.m, wsb<CT>(d, SB_RW) + M.m};
    CT *GYY = wsb<CT>(d, SB_GYY) + M.m, *G12 = wsb<CT>(d, SB_G12) + M.m;
    CT *G13 = wsb<CT>(d, SB_G13) + M.m, *G23 = wsb<CT>(d, SB_G23) + M.m;
    sgrad_pass<Rd<CT, kq<CT>(3)>>(
        d, ls, scr(d, 0, slot), scr(d, 3, slot), scr(d, 4, slot),
        [&](auto &r, int f, int dir, int first) { r.start(src[f], ld, my, dir, first); },
        [&](int j, double2 du, double2 dv, double2 dw, double2 u, double2 v, double2 w) {
          put(GYY, ld, j, dv);
          put(G12, ld, j, cadd(du, cik(M.kx, v)));
          put(G13, ld, j, cadd(cik(M.kz, u), cik(M.kx, w)));
          put(G23, ld, j, cadd(cik(M.kz, v), dw));
        });
  }
}

// ----------------------------------------------------------------------
// (6b)-(9) N_i, vorticity, the two Laplacians, RHS(Omega_y), RHS(phi) and
// the RK3 update (cross.f:652-682, 748-981), with the y derivatives of the
// three N_i, of u, w and of the two curls gathered by linearity (d = d/dy,
// lap = d2/dy2 - k2, products rho u_i u_j):
//   RHS(Omega_y) = i kz N_x - i kx N_z + lap(omega_y)/Re
//                = kx kz (uu - ww) - (kx^2 - kz^2) uw - d(i kz uv - i kx vw)
//                  + lap(i kz u - i kx w)/Re
//   (curl omega)_y = d(i kx u + i kz w) + k2 v
//   RHS(phi) = -k2 N_y - d(i kx N_x + i kz N_z) - lap((curl omega)_y)/Re
//            = k2 q + d(k2 vv - kx^2 uu - 2 kx kz uw - kz^2 ww + d q)
//              - lap((curl omega)_y)/Re,   q = i kx uv + i kz vw
// Three sweeps: up, the first halves of the four inner derivatives; down,
// their second halves, Omega_y, and the first halves (U') of the two outer
// ones; up, their second halves and phi.  (N_i and the curls through memory
// took ten sweeps: 640 bytes per point in the mixed form, 376 here.)
// Scratch fields 0, 3, 4, 5.
// ----------------------------------------------------------------------
template <typename CT>
__global__ void __launch_bounds__(YS_TB) t_post(Dev d, int rk) {
  const double dtg = post_dt(d, rk) * d.gama[rk];
  LMC_SWEEP_MODE
  {
    const double kx = M.kx, kz = M.kz, k2 = M.k2;
    double2 *sq = scr(d, 0, slot), *sr = scr(d, 3, slot), *sp = scr(d, 4, slot), *so = scr(d, 5, slot);
    // forward halves for i (kx f + kz g) (d/dy) and i (kz f - kx g) (L2 = false:
    // d/dy, true: lap); the band products are formed of f and g first
    auto up = [&](const CT *f, const CT *g, double2 *sa, double2 *sb, auto lap2) {
      constexpr bool L2 = decltype(lap2)::value;
      Rd<CT, kq<CT>(4)> rf, rg;
      rf.start(f + M.m, ld, my, 1, 0);
      rg.start(g + M.m, ld, my, 1, 0);
      Win wa, wb;
      wa.clear();
      wb.clear();
      Hist ha, hb;
      ha.clear();
      hb.clear();
      auto feed = [&]() {
        const double2 a = rf.pop(), b = rg.pop();
        wa.push(cadd(cik(kx, a), cik(kz, b)));
        wb.push(csub(cik(kz, a), cik(kx, b)));
      };
      for (int t = 0; t < 3; t++) feed();
      #pragma unroll 4
      for (int j = 0; j < my; j++) {
        feed();
        sa[(size_t)j * ls] = d1f(d, j, wa, ha);
        if constexpr (L2) sb[(size_t)j * ls] = half1<2>(d.r_p3L, j, b2(d, j, k2, wb), hb);
        else sb[(size_t)j * ls] = d1f(d, j, wb, hb);
      }
    };
    up(wsb<CT>(d, ORUV), wsb<CT>(d, ORVW), sq, sr, BoolC<false>());
    up(wsb<CT>(d, OU), wsb<CT>(d, OW), sp, so, BoolC<true>());
    {
      Rd<double2, 2> rq, rr, rp, ro, rvo;
      Rd<CT, kq<CT>(2)> ruu, rww, ruw, rvv, rv;
      rq.start(sq, ls, my, -1, my - 1);
      rr.start(sr, ls, my, -1, my - 1);
      rp.start(sp, ls, my, -1, my - 1);
      ro.start(so, ls, my, -1, my - 1);
      rvo.start(d.vor + M.m, ld, my, -1, my - 1);
      ruu.start(wsb<CT>(d, ORUU) + M.m, ld, my, -1, my - 1);
      rww.start(wsb<CT>(d, ORWW) + M.m, ld, my, -1, my - 1);
      ruw.start(wsb<CT>(d, ORUW) + M.m, ld, my, -1, my - 1);
      rvv.start(wsb<CT>(d, ORVV) + M.m, ld, my, -1, my - 1);
      rv.start(wsb<CT>(d, OV) + M.m, ld, my, -1, my - 1);
      Win we, wc;
      we.clear();
      wc.clear();
      Hist hq, hr, hp, ho, he, hc;
      hq.clear();
      hr.clear();
      hp.clear();
      ho.clear();
      he.clear();
      hc.clear();
      #pragma unroll 2
      for (int j = my - 1; j >= -3; j--) {
        double2 e = czero(), c = czero();
        if (j >= 0) {
          const double2 uu = ruu.pop(), ww = rww.pop(), uw = ruw.pop();
          const double2 dr = d1b(d, j, rr.pop(), hr), lo = half2<2>(d.r_p3U, j, ro.pop(), ho);
          double2 rom = fms(cscale(kx * kz, csub(uu, ww)), kx * kx - kz * kz, uw);
          rom = cadd(csub(rom, dr), cscale(d.ire, lo));
          put(d.Rom + M.m, ld, j, rom);
          put(d.vor + M.m, ld, j, cadd(rvo.pop(), cscale(dtg, rom)));  // cross.f:969
          e = cadd(d1b(d, j, rq.pop(), hq), cscale(k2, rvv.pop()));
          e = fms(fms(fms(e, kx * kx, uu), 2.0 * kx * kz, uw), kz * kz, ww);
          c = cadd(d1b(d, j, rp.pop(), hp), cscale(k2, rv.pop()));     // (curl omega)_y
        }
        push_low(we, e);
        push_low(wc, c);
        if (j + 3 < my) {  // rows above j are read no more: sq and sp take the new halves
          sq[(size_t)(j + 3) * ls] = half1<3>(d.r_q1U, j + 3, b1(d, j + 3, we), he);
          sp[(size_t)(j + 3) * ls] = half1<2>(d.r_q3U, j + 3, b2(d, j + 3, k2, wc), hc);
        }
      }
    }
    {
      Rd<double2, 4> re, rc, rph;
      Rd<CT, kq<CT>(4)> ruv, rvw;
      re.start(sq, ls, my, 1, 0);
      rc.start(sp, ls, my, 1, 0);
      rph.start(d.phi + M.m, ld, my, 1, 0);
      ruv.start(wsb<CT>(d, ORUV) + M.m, ld, my, 1, 0);
      rvw.start(wsb<CT>(d, ORVW) + M.m, ld, my, 1, 0);
      Hist he, hc;
      he.clear();
      hc.clear();
      #pragma unroll 4
      for (int j = 0; j < my; j++) {
        const double2 de = cscale(__ldg(d.r_fmap + j), half2<3>(d.r_q1L, j, re.pop(), he));
        const double2 lc = half2<2>(d.r_q3L, j, rc.pop(), hc);
        const double2 q = cadd(cik(kx, ruv.pop()), cik(kz, rvw.pop()));
        const double2 rp = fms(cadd(de, cscale(k2, q)), d.ire, lc);
        put(d.Rphi + M.m, ld, j, rp);
        put(d.phi + M.m, ld, j, cadd(rph.pop(), cscale(dtg, rp)));  // cross.f:978
      }
    }
  }
}

}  // namespace tpm
}  // namespace lmc
