// lmc_ytpm.cuh -- y kernels with one thread per (kx,kz) mode: the physical
// fields' export and the derivatives of the statistics (lmc_stats.cuh), which
// run once per output and not in every substep, and the 2014 variant's
// one-thread kernels.
//
// In the spectral layout [y][kx][kz] the value of mode m at row j sits at
// f[j*nmode + m], so the threads of a warp (32 consecutive modes) read and
// write every row of their pencils as one coalesced 32-value run, and the
// coefficients of a row are the same for the whole warp (one broadcast
// load).  Each banded solve A x = b with A = L U (the LU of cfdiff.f /
// laps.f in row form) runs as two sweeps along y: the forward sweep forms
// the band product of the right-hand side and applies L^-1, writing the
// intermediate pencil to an FP64 scratch field; the backward sweep reads it
// in reverse and applies U^-1.  Fields are streamed through a small queue
// of registers that is refilled K rows ahead of use, so every thread keeps
// several loads in flight.
#pragma once
#include <cuda_runtime.h>

#include "lmc_kernels.cuh"

namespace lmc {
namespace tpm {

using namespace lmcd;

constexpr int TB = 128;  // modes per block

template <typename CT>
__host__ __device__ constexpr bool mixed() { return sizeof(CT) == sizeof(float2); }

// Prefetching reader of one pencil, walking rows first, first+dir, ...
// Loads go through L2 (ld.global.cg), never the non-coherent read-only
// path: a kernel reads back scratch pencils and fields it wrote itself.
template <typename PT, int K>
struct Rd {
  const PT *p;
  size_t ld;
  int my, dir, nxt;
  PT q[K];
  __device__ __forceinline__ PT fetch(int r) const {
    PT z;
    z.x = 0;
    z.y = 0;
    return (r >= 0 && r < my) ? __ldcg(p + (size_t)r * ld) : z;
  }
  __device__ __forceinline__ void start(const PT *base, size_t ld_, int my_, int dir_, int first) {
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
  __device__ __forceinline__ double2 pop() {
    const double2 v = to_d2(q[0]);
#pragma unroll
    for (int t = 0; t < K - 1; t++) q[t] = q[t + 1];
    q[K - 1] = fetch(nxt);
    nxt += dir;
    return v;
  }
};

// queue depth giving K x 16 bytes in flight for values of type PT
template <typename PT>
__host__ __device__ constexpr int kq(int K) { return K * 16 / (int)sizeof(PT); }

template <typename PT>
__device__ __forceinline__ void put(PT *base, size_t ld, int j, double2 v) {
  base[(size_t)j * ld] = from_d2<PT>(v);
}

// u_{j-3} .. u_{j+3} around the current row j
struct Win {
  double2 u[7];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int t = 0; t < 7; t++) u[t] = czero();
  }
  __device__ __forceinline__ void push(double2 v) {
#pragma unroll
    for (int t = 0; t < 6; t++) u[t] = u[t + 1];
    u[6] = v;
  }
  __device__ __forceinline__ double2 c() const { return u[3]; }
};

// the last three results of a sweep (x_{j-+1}, x_{j-+2}, x_{j-+3})
struct Hist {
  double2 a, b, c;
  __device__ __forceinline__ void clear() { a = b = c = czero(); }
  __device__ __forceinline__ void push(double2 v) {
    c = b;
    b = a;
    a = v;
  }
};

__device__ __forceinline__ double2 fms(double2 s, double k, double2 v) {  // s - k v
  return make_double2(fma(-k, v.x, s.x), fma(-k, v.y, s.y));
}

// forward half of d/dy (deryr2, cfdiff.f:518-601): w_j = (L1^-1 dt12 u)_j
__device__ __forceinline__ double2 d1f(const Dev &d, int j, const Win &u, Hist &h) {
  const double *c = d.r_dt12 + 7 * j;
  double2 r = czero();
#pragma unroll
  for (int t = 0; t < 7; t++) {
    const double k = __ldg(c + t);
    r.x = fma(k, u.u[t].x, r.x);
    r.y = fma(k, u.u[t].y, r.y);
  }
  const double *l = d.r_p1L + 3 * j;
  r = fms(fms(fms(r, __ldg(l + 2), h.c), __ldg(l + 1), h.b), __ldg(l), h.a);
  h.push(r);
  return r;
}
// backward half of d/dy: x_j = (U1^-1 w)_j times fmap_j
__device__ __forceinline__ double2 d1b(const Dev &d, int j, double2 w, Hist &h) {
  const double *u = d.r_p1U + 4 * j;
  double2 x = fms(fms(fms(w, __ldg(u + 3), h.c), __ldg(u + 2), h.b), __ldg(u + 1), h.a);
  x = cscale(__ldg(u), x);
  h.push(x);
  return cscale(__ldg(d.r_fmap + j), x);
}
struct Mode {
  int m;
  double kx, kz, k2;
};
__device__ __forceinline__ bool mode_of(const Dev &d, Mode &M) {
  M.m = blockIdx.x * TB + threadIdx.x;
  if (M.m >= d.nmode) return false;
  const int i = M.m / d.mz, k = M.m - i * d.mz;
  M.kx = __ldg(d.kx + i);
  M.kz = __ldg(d.kz + k);
  M.k2 = __ldg(d.k2 + M.m);
  return true;
}

// the exact (FP64) 00 coefficient of transform output o at row j (mixed forms)
__device__ __forceinline__ double2 mo00_row(const Dev &d, int o, int j) {
  return make_double2(d.mo_cur[(size_t)o * d.my + j] / ((double)d.mgalx * (double)d.mgalz), 0.0);
}

// ----------------------------------------------------------------------
// Physical-field export (lmc_physical_f64), FP64: the transform inputs of
// tofis_loma's escrphys quantities from the state, without writing it:
// rho u_i assembled as the substep does (the wall conditions of Omega_y and
// phi, cross.f:315-335, then cross.f:395-499 with xi = 0), T and Z as
// stored (as tofis_loma reads them), grad T, and C = curl(rho u).  Reads
// m_y, dm_y/dy from SB_MY, SB_DMY (launch_lapv before); writes the export
// slots xslot(0..10) (lmc_kernels.cuh); scratch ws[0..3].
// ----------------------------------------------------------------------
__global__ void __launch_bounds__(TB) t_xprep(Dev d) {
  Mode M;
  if (!mode_of(d, M)) return;
  const int my = d.my;
  const size_t ld = d.nmode;
  const bool m00 = M.m == 0;
  const double ta = (M.k2 != 0.0) ? M.kx / M.k2 : 0.0, tb = (M.k2 != 0.0) ? M.kz / M.k2 : 0.0;
  double2 *s0 = d.ws[0] + M.m, *s1 = d.ws[1] + M.m, *s2 = d.ws[2] + M.m, *s3 = d.ws[3] + M.m;
  double2 *F[11];
  for (int q = 0; q < 11; q++) F[q] = d.sb[xslot(q)] + M.m;
  const double2 vor1 = d.vor[ld + M.m], vorn = d.vor[(size_t)(my - 2) * ld + M.m];  // cross.f:315-327
  {
    Rd<double2, 3> rpsi, rT, rvor, rdmy;
    rpsi.start(d.psi + M.m, ld, my, 1, 0);
    rT.start(d.scal + M.m, ld, my, 1, 0);
    rvor.start(d.vor + M.m, ld, my, 1, 0);
    rdmy.start(d.sb[SB_DMY] + M.m, ld, my, 1, 0);
    Win wp, wt, wu, ww;
    wp.clear();
    wt.clear();
    wu.clear();
    ww.clear();
    Hist hp, ht, hu, hw;
    hp.clear();
    ht.clear();
    hu.clear();
    hw.clear();
    // row r of rho u, rho w (the psi value of row r is the newest in wp)
    auto ru_rw = [&](int r, double2 ps, double2 &ru, double2 &rw) {
      const double2 a = rdmy.pop(), vr = rvor.pop();
      const double2 vo = r == 0 ? vor1 : r == my - 1 ? vorn : vr;
      ru = cadd(csub(cik(ta, a), cik(tb, vo)), cik(M.kx, ps));
      rw = cadd(cadd(cik(tb, a), cik(ta, vo)), cik(M.kz, ps));
      if (m00) {
        const bool in = r >= 0 && r < my;
        ru = make_double2(in ? d.u00[r] : 0.0, 0.0);
        rw = make_double2(in ? d.w00[r] : 0.0, 0.0);
      }
      if (r >= my) ru = rw = czero();
    };
    for (int r = 0; r < 3; r++) {
      const double2 ps = rpsi.pop();
      wp.push(ps);
      wt.push(rT.pop());
      double2 ru, rw;
      ru_rw(r, ps, ru, rw);
      wu.push(ru);
      ww.push(rw);
    }
    #pragma unroll 1
    for (int j = 0; j < my; j++) {
      const int r = j + 3;
      const double2 ps = rpsi.pop();
      wp.push(ps);
      wt.push(rT.pop());
      double2 ru, rw;
      ru_rw(r, ps, ru, rw);
      wu.push(ru);
      ww.push(rw);
      const double2 T = wt.c();
      put(F[0], ld, j, wu.c());
      put(F[2], ld, j, ww.c());
      put(F[3], ld, j, T);
      put(F[4], ld, j, cik(M.kx, T));
      put(F[6], ld, j, cik(M.kz, T));
      s0[(size_t)j * ld] = d1f(d, j, wp, hp);
      s1[(size_t)j * ld] = d1f(d, j, wt, ht);
      s2[(size_t)j * ld] = d1f(d, j, wu, hu);
      s3[(size_t)j * ld] = d1f(d, j, ww, hw);
    }
  }
  Rd<double2, 3> r0, r1, r2, r3, rmy, ru, rw;
  r0.start(s0, ld, my, -1, my - 1);
  r1.start(s1, ld, my, -1, my - 1);
  r2.start(s2, ld, my, -1, my - 1);
  r3.start(s3, ld, my, -1, my - 1);
  rmy.start(d.sb[SB_MY] + M.m, ld, my, -1, my - 1);
  ru.start(F[0], ld, my, -1, my - 1);
  rw.start(F[2], ld, my, -1, my - 1);
  Hist hp, ht, hu, hw;
  hp.clear();
  ht.clear();
  hu.clear();
  hw.clear();
  #pragma unroll 1
  for (int j = my - 1; j >= 0; j--) {
    double2 rv = cadd(d1b(d, j, r0.pop(), hp), rmy.pop());  // cross.f:434-437, 471
    if (m00) rv = make_double2(d.v00[j], 0.0);
    const double2 Ty = d1b(d, j, r1.pop(), ht), dudy = d1b(d, j, r2.pop(), hu), dwdy = d1b(d, j, r3.pop(), hw);
    const double2 u = ru.pop(), w = rw.pop();
    put(F[1], ld, j, rv);
    put(F[5], ld, j, Ty);
    put(F[7], ld, j, csub(dwdy, cik(M.kz, rv)));
    put(F[8], ld, j, csub(cik(M.kz, u), cik(M.kx, w)));
    put(F[9], ld, j, csub(cik(M.kx, rv), dudy));
    if (d.scalar) put(F[10], ld, j, d.zsc[(size_t)j * ld + M.m]);
  }
}

// 2014 variant: Deltat of the first substep of a CFL step, from the
// velocity maxima of the x stage (lomacte/cross.f:1547-1574); the new
// Deltat applies from this substep on.
__global__ void k_cfl14(Dev d, int do_cfl) {
  if (!do_cfl || threadIdx.x != 0 || blockIdx.x != 0) return;
  double hmin = d.hy[0];
  for (int j = 1; j < d.my; j++) hmin = fmin(hmin, d.hy[j]);
  const double hyy = 2.0 * d.ire * pow(fmax(1.0 / hmin, fmax(0.5 * d.hxalp, 0.5 * d.hzbet)), 2.0);
  const double cx = __longlong_as_double((long long)d.cflmax[0]) * d.hxalp;
  const double cy = __longlong_as_double((long long)d.cflmax[1]);
  const double cz = __longlong_as_double((long long)d.cflmax[2]) * d.hzbet;
  const double reig = fmax(fmax(cx, fmax(cy, cz)), hyy);
  d.scal_d[0] = (double)(float)(d.cfl / reig);  // Deltat is real*4
}

// 2014 variant, 00 modes after the substep (lomacte/cross.f:931-1002):
// rho u00 / rho w00 RK3 update, masses, rho v00 = -(cumulative trapezoid of
// d(rho)00 / (Deltat (gamma + xi)) - rho_bot trapz / (rho_top + rho_bot)),
// end-of-step time.  One thread: the sums run in the reference's order.
__global__ void k_psi00_14(Dev d, int rk) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int my = d.my;
  const double dt = d.scal_d[0], dtg = dt * d.gama[rk], den = dt * (d.gama[rk] + d.xi[rk]);
  double mu = 0.0, mv = 0.0, mw = 0.0;
  #pragma unroll 4
  for (int j = 0; j < my; j++) {
    if (j >= 1 && j <= my - 2) {
      d.u00[j] += dtg * d.rf0u[j];
      d.w00[j] += dtg * d.rf0w[j];
    }
    mu += d.u00[j] * d.hy[j];
    mv += d.v00[j] * d.hy[j];
    mw += d.w00[j] * d.hy[j];
  }
  const double2 *dr = d.sb[ODRHO];
  const size_t ld = d.nmode;
  double f = 0.0, prev = dr[0].x / den;
  d.rf0v[0] = 0.0;
  for (int j = 0; j < my - 1; j++) {
    const double nxt = dr[(size_t)(j + 1) * ld].x / den;
    f += 0.5 * (d.y[j + 1] - d.y[j]) * (nxt + prev);
    d.rf0v[j + 1] = f;
    prev = nxt;
  }
  const double trapz = f;
  const double sh = d.scal_d[3] * trapz / (d.scal_d[4] + d.scal_d[3]);
  #pragma unroll 4
  for (int j = 0; j < my; j++) {
    d.rf0v[j] -= sh;
    d.v00[j] = -d.rf0v[j];
  }
  d.diag[5] = trapz;
  d.diag[7] = mu; d.diag[8] = mv; d.diag[9] = mw;
  if (rk == 2) {
    d.diag[0] = d.scal_d[2];
    d.diag[1] = dt;
    d.scal_d[2] += dt;
    d.diag[12] = dt;
  }
}

}  // namespace tpm
}  // namespace lmc
