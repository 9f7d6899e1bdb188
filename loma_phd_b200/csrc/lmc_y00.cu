// lmc_y00.cu -- the kx = kz = 0 (00) modes of one lomacte RK3 substep, after
// the transforms and at the end of the substep.
//
// One pencil per warp: its my points are split over the lanes in chunks and
// the banded solves join the chunks by shuffles (lmc_device.cuh), so each of
// these one-block kernels is a short chain of latencies.  The six banded
// operators that the 00 modes need run on six warps at once.
#include <cuda_runtime.h>

#include "lmc_kernels.cuh"

using namespace lmcd;

namespace lmc {

namespace {

template <int C>
__device__ __forceinline__ double2 get_row(const double2 (&v)[C], const Lane &L, int row) {
  double2 r = czero();
#pragma unroll
  for (int t = 0; t < C; t++)
    if (t < L.n && L.s + t == row) r = v[t];
  return r;
}
template <int C>
__device__ __forceinline__ double2 bcast_row(const double2 (&v)[C], const Lane &L, int row) {
  double2 r = get_row(v, L, row);
  r.x = warp_sum(r.x);
  r.y = warp_sum(r.y);
  return r;
}

// compact first derivative in place (deryr2, cfdiff.f:518-601)
template <int C>
__device__ __forceinline__ void d1(const Dev &d, const Lane &L, double2 (&u)[C]) {
  matvec_ip<C, 3>(d.dt12, L, u);
  lsolve_c<C, 3>(u, d.p1L, d.k1L, L);
  usolve_c<C, 3>(u, d.p1U, d.k1U, L);
#pragma unroll
  for (int t = 0; t < C; t++)
    if (t < L.n) u[t] = cscale(tab(d.fmap, 1, t, 0, L.lane), u[t]);
}
// compact second derivative in place (deryyr2, cfdiff.f:735-797)
template <int C>
__device__ __forceinline__ void d2(const Dev &d, const Lane &L, double2 (&u)[C]) {
  matvec_ip<C, 2>(d.dt22, L, u);
  lsolve_c<C, 2>(u, d.p3L, d.k3L, L);
  usolve_c<C, 2>(u, d.p3U, d.k3U, L);
}

// 00 coefficient of transform output o at row j: the FP64 plane mean in the
// mixed forms, the spectral value otherwise
template <typename CT>
__device__ __forceinline__ double v00(const Dev &d, int o, int j) {
  if constexpr (sizeof(CT) == sizeof(float2))
    return d.mo_cur[(size_t)o * d.my + j] / ((double)d.mgalx * (double)d.mgalz);
  else return wsb<CT>(d, o)[(size_t)j * d.nmode].x;
}
template <int C, typename CT>
__device__ __forceinline__ void load00(const Dev &d, int o, const Lane &L, double2 (&v)[C]) {
#pragma unroll
  for (int t = 0; t < C; t++) v[t] = make_double2(t < L.n ? v00<CT>(d, o, L.s + t) : 0.0, 0.0);
}

// dw, dm, masst, the 00 RHS of rho u00 / rho w00, H00 and the CFL Deltat:
// cross.f:686-722, 1416-1429, 1778-1826, and the integral of d(rho)/dt00 for
// rho v00 (inty8).  Warps 0 and 1: d2/dy2 of u00 and w00; 2 and 3: d/dy of
// rho uv and rho vw; 4: the thicknesses and the mass; 5: inty8, which had its
// turn in k_psi_00 before, so that this kernel, k_psi_00 and c_psi in a row
// took longer than the RK3 update beside them (512 x 257 2-D: 0.40 ms per
// step after 0.42; 192 x 193 x 128 4.94 after 4.97).
template <int C, typename CT>
__global__ void __launch_bounds__(192, 1) k_post1_00(Dev d, int rk, int do_cfl, int do_diag) {
  extern __shared__ double R[];  // [4][my]
  const Lane L = make_lane<C>(d.lpm, d.base, d.extra);
  const int w = threadIdx.x >> 5, my = d.my;
  double2 a[C];
  if (w < 4) {
    load00<C, CT>(d, w == 0 ? OU : w == 1 ? OW : w == 2 ? ORUV : ORVW, L, a);
    if (w < 2) d2<C>(d, L, a);
    else d1<C>(d, L, a);
#pragma unroll
    for (int t = 0; t < C; t++)
      if (t < L.n) R[w * my + L.s + t] = a[t].x;
  } else if (w == 5) {
    if (!d.variant) {  // inty8 (laps.f:484-575): rf0v(y) = int d(rho)/dt00 dy with rf0v(1) = 0
      load00<C, CT>(d, ODRHO, L, a);
#pragma unroll
      for (int t = 0; t < C; t++) a[t] = make_double2((t < L.n) ? a[t].x / tab(d.fmap, 1, t, 0, L.lane) : 0.0, 0.0);
      matvec_ip<C, 3>(d.dt11, L, a);
      lsolve_c<C, 3>(a, d.i8L, d.k8L, L);
      usolve_c<C, 3>(a, d.i8U, d.k8U, L);
      const double v0 = bcast_row(a, L, 0).x, vn = bcast_row(a, L, my - 1).x;
#pragma unroll
      for (int t = 0; t < C; t++)
        if (t < L.n) d.rf0v[L.s + t] = a[t].x - v0;
      if (L.lane == 0) d.diag[5] = -(vn - v0);  // trapz, cross.f:1046
    }
  } else {
    if (rk == 2 && do_diag) {  // vorticity thickness, cross.f:692-699
      load00<C, CT>(d, OU, L, a);
      d1<C>(d, L, a);
      double mx = 0.0;
#pragma unroll
      for (int t = 0; t < C; t++)
        if (t < L.n) mx = fmax(mx, fabs(a[t].x));
      mx = warp_max(mx);
      if (L.lane == 0) {
        d.diag[3] = 1.0 / mx;
        d.diag[4] = d.diag[3] / d.ire;
      }
    }
    if (rk == 0 && do_diag) {  // momentum thickness, cross.f:1416-1429; masst, escru.f:372-376
      double s = 0.0, ms = 0.0;
      for (int j = L.lane; j < my; j += 32) {
        const double a1 = v00<CT>(d, OU, min(j + 1, my - 1)), a2 = v00<CT>(d, OU, max(j - 1, 0));
        s += d.trp[j] * (a1 * a1 + a2 * a2);
        ms += d.rhom[j] * d.hy[j];
      }
      s = warp_sum(s);
      ms = warp_sum(ms);
      if (L.lane == 0) {
        const double du0 = v00<CT>(d, OU, my - 1) - v00<CT>(d, OU, 0);
        d.diag[2] = 0.25 * (d.y[my - 1] - d.y[0]) - s / (du0 * du0);
        d.diag[6] = ms / ((double)d.mgalx * (double)d.mgalz);
      }
      if (L.lane == 0 && do_cfl) {  // cross.f:1781-1817, one compute rank
        const double cx = __longlong_as_double((long long)d.cflmax[0]) * d.hxalp * 0.5;
        const double cy = __longlong_as_double((long long)d.cflmax[1]);
        const double cz = __longlong_as_double((long long)d.cflmax[2]) * d.hzbet * 0.5;
        const double ct = __longlong_as_double((long long)d.cflmax[3]);
        d.scal_d[1] = (double)(float)(d.cfl / (cx + cy + cz + ct));  // dtr is real*4
      }
    }
  }
  __syncthreads();
  if (w < 2) {  // cross.f:705-706
    double *rf = w == 0 ? d.rf0u : d.rf0w, h = 0.0;
    for (int j = L.lane; j < my; j += 32) {
      const double r = -R[(2 + w) * my + j] + d.ire * R[w * my + j];
      rf[j] = r;
      h += r * d.hy[j];
    }
    h = warp_sum(h);
    if (L.lane == 0 && rk == 2 && do_diag) d.diag[10 + w] = 0.25 * h;
  }
}

// rho u00 / rho w00 RK3 update, masses, rho v00 with the acoustic wall
// correction, end-of-step time and Deltat: cross.f:1006-1074, 1196-1204.  One
// warp, its lanes along y.
__global__ void __launch_bounds__(32, 1) k_psi_00(Dev d, int rk, int cfl_step) {
  const double dt = d.scal_d[0], dtg = dt * d.gama[rk];
  const double corr = d.diag[5] / (1.0 + sqrt(d.scal_d[4] / d.scal_d[3]));  // cross.f:1064-1065
  double mu = 0.0, mv = 0.0, mw = 0.0;
#pragma unroll 4
  for (int j = threadIdx.x; j < d.my; j += 32) {
    const bool in = j >= 1 && j <= d.my - 2;  // cross.f:1008-1011
    const double h = d.hy[j], ru = d.rf0u[j], rw = d.rf0w[j];
    const double u = in ? d.u00[j] + dtg * ru : d.u00[j], w = in ? d.w00[j] + dtg * rw : d.w00[j];
    mu += u * h;  // cross.f:1016-1020
    mv += d.v00[j] * h;
    mw += w * h;
    d.u00[j] = u;
    d.w00[j] = w;
    d.v00[j] = d.rf0v[j] + corr;
  }
  mu = warp_sum(mu); mv = warp_sum(mv); mw = warp_sum(mw);
  if (threadIdx.x == 0) {
    d.diag[7] = mu; d.diag[8] = mv; d.diag[9] = mw;
    if (rk == 1) d.scal_d[7] = dt;
    if (rk == 2) {  // end of the time step: cross.f:1196-1204
      d.diag[0] = d.scal_d[2];
      d.diag[1] = dt;
      d.scal_d[2] += dt;  // the RK3 update beside this kernel reads scal_d[7]
      if (cfl_step) d.scal_d[0] = d.scal_d[1];
      d.diag[12] = d.scal_d[0];
    }
  }
}

template <int C, typename CT>
void post1_00(const Dev &d, int rk, int do_cfl, int do_diag, cudaStream_t s) {
  k_post1_00<C, CT><<<1, 192, (size_t)4 * d.my * sizeof(double), s>>>(d, rk, do_cfl, do_diag);
}
}  // namespace

// d.C: points per lane (the chunk sizes of pick_chunks)
#define LMC_Y00_CASE(C, CALL)                  \
  case C:                                      \
    if (d.prec) CALL(C, float2);               \
    else CALL(C, double2);                     \
    break;
#define LMC_Y00(CALL)                                                                          \
  switch (d.C) {                                                                               \
    LMC_Y00_CASE(4, CALL) LMC_Y00_CASE(5, CALL) LMC_Y00_CASE(7, CALL) LMC_Y00_CASE(9, CALL)    \
    LMC_Y00_CASE(13, CALL) default : LMC_Y00_CASE(17, CALL)                                    \
  }

void launch_post1_00(const Dev &d, int rk, int do_cfl, int do_diag, cudaStream_t s) {
  const int cfl = d.variant ? 0 : do_cfl;  // the 2014 variant sets Deltat in k_cfl14
#define CALL(C, CT) post1_00<C, CT>(d, rk, cfl, do_diag, s)
  LMC_Y00(CALL)
#undef CALL
}
void launch_psi_00(const Dev &d, int rk, int cfl_step, cudaStream_t s) { k_psi_00<<<1, 32, 0, s>>>(d, rk, cfl_step); }

}  // namespace lmc
