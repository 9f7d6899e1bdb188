// lmc_ykernels.cu -- dispatch of the y-direction kernels to the geometry of
// a case, their one-time set-up, and the layout transposes of the C ABI.
#include <cuda_runtime.h>

#include "lmc_ylaunch.h"

namespace lmc {

namespace {

// ----------------------------------------------------------------------
// layout transposes: reference [kx][kz][y] <-> device [y][kx][kz]
// ----------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_ref2dev(int my, int nkx, int mz, const double2 *__restrict__ in,
                                                 double2 *__restrict__ out) {
  __shared__ double2 t[32][33];
  const int i = blockIdx.z, y0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int k = k0 + r, y = y0 + threadIdx.x;
    if (k < mz && y < my) t[r][threadIdx.x] = in[((size_t)i * mz + k) * my + y];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int y = y0 + r, k = k0 + threadIdx.x;
    if (k < mz && y < my) out[((size_t)y * nkx + i) * mz + k] = t[threadIdx.x][r];
  }
}
__global__ void __launch_bounds__(256) k_dev2ref(int my, int nkx, int mz, const double2 *__restrict__ in,
                                                 double2 *__restrict__ out) {
  __shared__ double2 t[32][33];
  const int i = blockIdx.z, y0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int y = y0 + r, k = k0 + threadIdx.x;
    if (k < mz && y < my) t[r][threadIdx.x] = in[((size_t)y * nkx + i) * mz + k];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int k = k0 + r, y = y0 + threadIdx.x;
    if (k < mz && y < my) out[((size_t)i * mz + k) * my + y] = t[threadIdx.x][r];
  }
}

// T += Delta T, Z += Delta Z (cross.f:619-627), one value per thread; the
// mixed forms take the exact FP64 00 mode of the increment from the plane
// sums.  V: the 2014 variant advances the spectral T with this substep's
// RHS(T) (in the d(rho)/dt slot) and accumulates Delta T
// (lomacte/cross.f:563-570).
template <typename CT, bool V, bool Z>
__global__ void __launch_bounds__(256) k_tupd(Dev d, int rk) {
  const size_t n = (size_t)d.nmode * d.my;
  for (size_t p = (size_t)blockIdx.x * 256 + threadIdx.x; p < n; p += (size_t)gridDim.x * 256) {
    double2 dT = lmcd::to_d2(__ldg(wsb<CT>(d, Z ? ODZ : V ? ODRHO : ODT) + p));
    if constexpr (sizeof(CT) == sizeof(float2))
      if (p % d.nmode == 0) dT = make_double2(d.mo_cur[(size_t)(Z ? ODZ : ODT) * d.my + p / d.nmode] / ((double)d.mgalx * (double)d.mgalz), 0.0);
    if constexpr (V) {
      const double dtg = d.scal_d[0] * d.gama[rk];
      d.RT[p] = dT;
      dT = lmcd::cscale(dtg, dT);
      d.dTs[p] = lmcd::cadd(d.dTs[p], dT);
    }
    double2 *f = Z ? d.zsc : d.scal;
    f[p] = lmcd::cadd(f[p], dT);
  }
}

template <bool Z>
void tupd(const Dev &d, int rk, cudaStream_t s) {
  const size_t n = (size_t)d.nmode * d.my;
  const unsigned g = (unsigned)((n + 1023) / 1024);  // four values per thread
  if (d.prec) k_tupd<float2, false, Z><<<g, 256, 0, s>>>(d, rk);
  else if (!Z && d.variant) k_tupd<double2, true, false><<<g, 256, 0, s>>>(d, rk);
  else k_tupd<double2, false, Z><<<g, 256, 0, s>>>(d, rk);
}

}  // namespace

void launch_tupd(const Dev &d, int rk, cudaStream_t s) { tupd<false>(d, rk, s); }
void launch_zupd(const Dev &d, cudaStream_t s) { tupd<true>(d, 0, s); }

// geometry of the chunked kernels: rows per chunk and modes per block (d.yC,
// d.yMB, chosen by y_geometry in lmc_api.cu)
#define LMC_YC(CALL)                          \
  do {                                        \
    if (d.yC == 5) YC<5, 8>::CALL;            \
    else if (d.yMB == 8) YC<9, 8>::CALL;      \
    else if (d.yMB == 16) YC<9, 16>::CALL;    \
    else YC<9, 32>::CALL;                     \
  } while (0)

// d.ysb: grids with many modes sweep along y instead (lmc_ysweep.cuh)
void launch_lapv(const Dev &d, cudaStream_t s) {
  if (d.ysb) sweep_lapv(d, s);
  else LMC_YC(lapv(d, s));
}
void launch_assemble(const Dev &d, int rk, cudaStream_t s) {
  if (d.ysb) sweep_assemble(d, rk, s);
  else LMC_YC(assemble(d, rk, s));
}
void launch_tder(const Dev &d, cudaStream_t s) {
  if (d.ysb) sweep_tder(d, false, s);
  else LMC_YC(tder(d, false, s));
}
void launch_zder(const Dev &d, cudaStream_t s) {
  if (d.ysb) sweep_tder(d, true, s);
  else LMC_YC(tder(d, true, s));
}
void launch_sgrad(const Dev &d, cudaStream_t s) {
  if (d.ysb) sweep_sgrad(d, s);
  else LMC_YC(sgrad(d, s));
}
void launch_post(const Dev &d, int rk, cudaStream_t s) {
  if (d.ysb) sweep_post(d, rk, s);
  else LMC_YC(post(d, rk, !d.tpm, s));
}
void launch_psi(const Dev &d, int rk, cudaStream_t s) { LMC_YC(psi(d, rk, s)); }
void launch_op_y(const Dev &d, int op, const double2 *in, double2 *out, double2 *out2, cudaStream_t s) {
  LMC_YC(op_y(d, op, in, out, out2, s));
}
void launch_psi_tail(const Dev &d, int rk, int cfl_step, cudaStream_t s) {
  if (d.variant) tpm_psi00_14(d, rk, s);
  else launch_psi_00(d, rk, cfl_step, s);
}

// Opt the y kernels in to the device's largest dynamic shared memory.
cudaError_t ykernels_init(int limit) {
  cudaError_t e = YC<5, 8>::optin(limit);
  if (e == cudaSuccess) e = YC<9, 8>::optin(limit);
  if (e == cudaSuccess) e = YC<9, 16>::optin(limit);
  if (e == cudaSuccess) e = YC<9, 32>::optin(limit);
  return e;
}

void launch_ref2dev(const Dev &d, const double2 *in, double2 *out, cudaStream_t s) {
  dim3 g((d.my + 31) / 32, (d.mz + 31) / 32, d.nkx);
  k_ref2dev<<<g, dim3(32, 8), 0, s>>>(d.my, d.nkx, d.mz, in, out);
}
void launch_dev2ref(const Dev &d, const double2 *in, double2 *out, cudaStream_t s) {
  dim3 g((d.my + 31) / 32, (d.mz + 31) / 32, d.nkx);
  k_dev2ref<<<g, dim3(32, 8), 0, s>>>(d.my, d.nkx, d.mz, in, out);
}

}  // namespace lmc
