// lmc_ytpm.cu -- launchers of the one-thread-per-mode y kernels
// (lmc_ytpm.cuh, lmc_ysweep.cuh) and of the statistics (lmc_stats.cuh).
#include "lmc_ylaunch.h"
#include "lmc_stats.cuh"
#include "lmc_ysweep.cuh"

namespace lmc {

namespace {
inline unsigned tgrid(const Dev &d) { return (unsigned)((d.nmode + tpm::TB - 1) / tpm::TB); }
}  // namespace

void launch_xprep(const Dev &d, cudaStream_t s) { tpm::t_xprep<<<tgrid(d), tpm::TB, 0, s>>>(d); }
void launch_cfl14(const Dev &d, int do_cfl, cudaStream_t s) { tpm::k_cfl14<<<1, 32, 0, s>>>(d, do_cfl); }
void tpm_psi00_14(const Dev &d, int rk, cudaStream_t s) { tpm::k_psi00_14<<<1, 32, 0, s>>>(d, rk); }

// the sweeps of grids with many modes (d.ysb blocks)
template <typename K, typename... A>
void sweep(K k, const Dev &d, bool persistent, int extra, cudaStream_t s, A... a) {
  const int g = persistent && d.ysb > YS_PERSIST ? YS_PERSIST : d.ysb;
  k<<<g + extra, YS_TB, 0, s>>>(a...);
}
void sweep_lapv(const Dev &d, cudaStream_t s) {
  if (d.prec) sweep(tpm::t_lapv<float2>, d, false, 0, s, d);
  else sweep(tpm::t_lapv<double2>, d, false, 0, s, d);
}
void sweep_assemble(const Dev &d, int rk, cudaStream_t s) {
  if (d.prec) sweep(tpm::t_assemble<float2>, d, false, 0, s, d, rk);
  else sweep(tpm::t_assemble<double2>, d, false, 0, s, d, rk);
}
void sweep_tder(const Dev &d, bool z, cudaStream_t s) {
  if (d.prec) z ? sweep(tpm::t_tder<float2, true>, d, true, 0, s, d) : sweep(tpm::t_tder<float2, false>, d, true, 0, s, d);
  else z ? sweep(tpm::t_tder<double2, true>, d, true, 0, s, d) : sweep(tpm::t_tder<double2, false>, d, true, 0, s, d);
}
void sweep_sgrad(const Dev &d, cudaStream_t s) {  // mixed: one more block for the exact 00 profiles
  if (d.prec) sweep(tpm::t_sgrad<float2>, d, true, 1, s, d);
  else sweep(tpm::t_sgrad<double2>, d, true, 0, s, d);
}
void sweep_post(const Dev &d, int rk, cudaStream_t s) {
  if (d.prec) sweep(tpm::t_post<float2>, d, false, 0, s, d, rk);
  else sweep(tpm::t_post<double2>, d, false, 0, s, d, rk);
}

// statistics (lmc_stats.cuh); every grid, either y family
void launch_stats1(const Dev &d, const Stats &st, cudaStream_t s) {
  if (d.prec) stats::k_srow1<float2><<<d.my, stats::SRT, 0, s>>>(d, st);
  else stats::k_srow1<double2><<<d.my, stats::SRT, 0, s>>>(d, st);
}
void launch_stats2(const Dev &d, const Stats &st, cudaStream_t s) {
  if (d.prec) {
    stats::t_sdy<float2><<<tgrid(d), tpm::TB, 0, s>>>(d, st);
    stats::k_srow2<float2><<<d.my, stats::SRT, 0, s>>>(d, st);
  } else {
    stats::t_sdy<double2><<<tgrid(d), tpm::TB, 0, s>>>(d, st);
    stats::k_srow2<double2><<<d.my, stats::SRT, 0, s>>>(d, st);
  }
  stats::k_suner<<<1, 32, 0, s>>>(d, st);
}

}  // namespace lmc
