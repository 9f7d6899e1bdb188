// lmc_ylaunch.h -- launchers of the chunked y kernels (lmc_ychunk.cuh) for
// chunks of C rows and MB modes per block; each lmc_yc_*.cu translation unit
// instantiates one geometry so that they compile in parallel.
#pragma once
#include <cuda_runtime.h>

#include "lmc_kernels.cuh"

namespace lmc {

template <int C, int MB>
struct YC {
  static void lapv(const Dev &d, cudaStream_t s);
  static void assemble(const Dev &d, int rk, cudaStream_t s);
  static void tder(const Dev &d, bool z, cudaStream_t s);
  static void sgrad(const Dev &d, cudaStream_t s);
  static void post(const Dev &d, int rk, bool tu, cudaStream_t s);
  static void psi(const Dev &d, int rk, cudaStream_t s);
  static void op_y(const Dev &d, int op, const double2 *in, double2 *out, double2 *out2, cudaStream_t s);
  static cudaError_t optin(int limit);
};

// sweeps along y (lmc_ytpm.cu), d.ysb > 0
void sweep_lapv(const Dev &d, cudaStream_t s);
void sweep_assemble(const Dev &d, int rk, cudaStream_t s);
void sweep_tder(const Dev &d, bool z, cudaStream_t s);
void sweep_sgrad(const Dev &d, cudaStream_t s);
void sweep_post(const Dev &d, int rk, cudaStream_t s);

void launch_psi_00(const Dev &d, int rk, int cfl_step, cudaStream_t s);  // lmc_y00.cu
void tpm_psi00_14(const Dev &d, int rk, cudaStream_t s);                 // lmc_ytpm.cu

}  // namespace lmc
