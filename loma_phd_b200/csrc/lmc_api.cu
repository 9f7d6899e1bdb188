// lmc_api.cu -- C ABI of liblomacte_b200 (declared in include/lomacte_b200.h).
//
// One handle = one case: the tables built by lmc_host.cpp are uploaded once,
// the state lives in device memory, and lmc_step enqueues the substep
// kernels of lmc_kernels.cu on the handle's stream.  There is no CPU path:
// without a CUDA device lmc_create returns LMC_ENODEV.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "lmc_internal.h"
#include "lmc_async.cuh"
#include "lmc_kernels.cuh"

namespace lmc {
// the dense y operators on the tensor cores (lmc_yop.cu)
struct DenseY;
DenseY *dense_create(const YOps &ops, size_t ncol, cudaStream_t s, int *rc);
void dense_destroy(DenseY *z);
int dense_apply(DenseY *z, int op, int method, const double *in, double *out, cudaStream_t s);
}  // namespace lmc

struct lmc_handle {
  lmc::Grid g;
  lmc_params p;
  lmc::YOps ops;
  lmc::PoissonTables pt;
  lmc::RK3 rk;
  lmc::Dev d;
  cudaStream_t s = nullptr;
  cudaStream_t s2 = nullptr;  // side stream for the independent kernels of a substep
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  std::vector<void *> allocs;
  int steps = 0;
  int err = 0;
  // mixed form: the two FP64 plane-sum arrays alternate between substeps
  double *mo[2] = {nullptr, nullptr};
  int mo_flip = 0;
  // one CUDA graph per RK3 step variant: [CFL update step][mo_flip parity]
  bool graphs = true;
  cudaGraphExec_t gexec[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
  size_t bytes = 0;  // device bytes held
  // statistics (lmc_stats_*): device accumulators, the capacity of the
  // spectra buffers in planes, and the reference's counters
  lmc::Stats st{};
  bool st_on = false;
  int st_cap = -1;
  size_t st_spec_bytes = 0;
  int nacum = 0, nacumsp = 0;
  // slab blocks of lmc_step_split: kx planes p0 .. p0+np-1 and (z, y) lines
  // l0 .. l0+nl-1 of block r, with z-physical buffers of its planes (Z) and
  // of its lines (X), field by field
  struct Split {
    int n = 0;
    std::vector<int> p0, np, l0, nl;
    std::vector<std::vector<void *>> Z, X;
  } split;
  // dense y operators and their GEMM workspace (lmc_op_y_dense, lmc_yop_tune)
  lmc::DenseY *yop = nullptr;
  // per-kernel CUDA-event profiling (lmc_profile_start / lmc_profile_read)
  bool prof = false;
  std::vector<cudaEvent_t> ev_pool;
  std::vector<int> ev_kid;
  size_t ev_used = 0;
};

namespace {

void drop_graphs(lmc_handle *h);

#define LMC_CK(call)                                     \
  do {                                                   \
    cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) {                             \
      std::fprintf(stderr, "lomacte_b200: %s:%d %s\n", __FILE__, __LINE__, cudaGetErrorString(e_)); \
      return e_ == cudaErrorMemoryAllocation ? LMC_ENOMEM : LMC_ECUDA; \
    }                                                    \
  } while (0)

// Device buffers come from the stream-ordered allocator on the handle's
// stream and go back with cudaFreeAsync, so creating and destroying a case
// never waits for the other cases running on the device (cudaFree would
// synchronise the whole device).
template <class T>
int dalloc(lmc_handle *h, T **p, size_t n) {
  void *q = nullptr;
  cudaError_t e = cudaMallocAsync(&q, n * sizeof(T) + 16, h->s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? LMC_ENOMEM : LMC_ECUDA;
  }
  h->allocs.push_back(q);
  h->bytes += n * sizeof(T) + 16;
  *p = (T *)q;
  return LMC_OK;
}
template <class T>
int dupload(lmc_handle *h, const T **p, const std::vector<T> &v) {
  T *q = nullptr;
  int r = dalloc(h, &q, v.size());
  if (r) return r;
  // pageable source: the call returns once the data is staged
  LMC_CK(cudaMemcpyAsync(q, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, h->s));
  *p = q;
  return LMC_OK;
}

// Twiddles of the passes of a transform of length n (Fft in lmc_device.cuh):
// exp(-2 pi i m k / n) at [k M + m], k < r1, m < M = r2 r3; then
// exp(-2 pi i m k / M) at [n + k r3 + m], k < r2, m < r3; then the direct
// transform's.  C: double2 or float2
template <typename C>
std::vector<C> fft_twiddles(int n) {
  const lmc::FftRadix f = lmc::fft_radix(n, sizeof(C) == sizeof(float2));
  const int M = f.r2 * f.r3;
  std::vector<C> t;
  auto put = [&](long long e, int len) {
    const long double a = 2.0L * 3.14159265358979323846264338327950288L * (long double)(e % len) / (long double)len;
    C c;
    c.x = (decltype(c.x))cosl(a);
    c.y = (decltype(c.y))(-sinl(a));
    t.push_back(c);
  };
  for (int k = 0; k < f.r1; k++)
    for (int m = 0; m < M; m++) put((long long)k * m, n);
  for (int k = 0; k < f.r2; k++)
    for (int m = 0; m < f.r3; m++) put((long long)k * m, M);
  // of the direct transform's first twiddled pass, the tasks fastest
  const int jn = f.r3 > 1 ? f.r3 : M, fs = f.r3 > 1 ? f.r2 : f.r1, len = f.r3 > 1 ? M : n;
  for (int j = 0; j < jn; j++)
    for (int k = 0; k < fs; k++) put((long long)j * k, len);
  return t;
}

int pick_chunks(int my, int &C, int &lpm, int &base, int &extra) {
  static const int Cs[] = {4, 5, 7, 9, 13, 17};
  const int need = (my + 31) / 32;
  C = 0;
  for (int c : Cs)
    if (c >= need) { C = c; break; }
  if (!C) return LMC_EINVAL;
  lpm = (my + C - 1) / C;
  base = my / lpm;
  extra = my % lpm;
  if (lpm > 32 || base < 3) return LMC_EINVAL;
  if (!(base == C - 1 || (base == C && extra == 0))) return LMC_EINVAL;
  return LMC_OK;
}

// The x stage holds a tile's transform lines and its RHS rows in shared
// memory; with the passive scalar and the
// variable viscosity the lines of the largest lengths alone need more than
// the 227 KB a B200 block can have.
constexpr size_t SMEM_BLOCK_MAX = 227 * 1024;
bool xstage_fits(const lmc::Grid &g, int scalar, int visc) {
  lmc::Dev d;
  std::memset(&d, 0, sizeof(d));
  d.mgalx = g.mgalx;
  d.nkx = g.nkx;
  d.scalar = scalar;
  d.visc = visc;
  const size_t need = lmc::xphys_smem(d);
  return need > 0 && need + 1024 <= SMEM_BLOCK_MAX;
}

// Split of the y work by the number of modes.  LMC_YPATH=mode|warp forces the
// split of many or of few modes (tests compare them).
bool many_modes(int nmode) {
  const char *e = std::getenv("LMC_YPATH");
  if (e && std::strcmp(e, "mode") == 0) return true;
  if (e && std::strcmp(e, "warp") == 0) return false;
  return nmode >= 16384;
}

// modes up to which the chunked y kernels take short chunks (y_geometry)
constexpr int FEW_MODES = 8 * 2 * 148;

// Blocks of the sweeps along y (lmc_ysweep.cuh), which take over from the
// chunked kernels (not in the 2014 variant) for grids with many modes, where
// the sweeps fill the device (an FP64 step of 12,192 modes x 193 takes 5.3 ms
// with the chunks and 5.8 with the sweeps, one of 8,128 x 129 2.5 and
// 3.4 ms; 32,640 x 257 with mu = T^0.7, the scalar and float2 buffers 21.1
// and 17.2), and for short pencils, which a chunk or three hold (with the
// scalar and mu, 3,040 to 12,192 modes: the sweeps take 0.81 to 0.92 of the
// chunks' step at 18 rows, 0.90 to 1.03 at 24 and 1.03 to 1.24 at 33).
int sweep_blocks(const lmc::Grid &g, int variant) {
  const bool force = std::getenv("LMC_YPATH") != nullptr;
  if (variant || !(many_modes(g.nmode) || (!force && g.my <= 28 && g.nmode > FEW_MODES))) return 0;
  return (g.nmode + lmc::YS_TB - 1) / lmc::YS_TB;
}
// values of scratch field q of the sweeps: whole blocks of modes, fields 1
// and 2 those of a persistent grid
size_t sweep_scratch(int ysb, int q, const lmc::Grid &g) {
  const int nb = (q == 1 || q == 2) && ysb > lmc::YS_PERSIST ? lmc::YS_PERSIST : ysb;
  return (size_t)nb * lmc::YS_TB * g.my;
}
// Geometry of the chunked y kernels (lmc_ychunk.cuh): rows per chunk and
// modes per block.  Short chunks where the blocks of eight modes are at most
// two per SM, so that the length of one block's chain is what counts (2,016
// modes x 129, FP64: 0.93 ms per step against 1.04 with nine rows; 256 x
// 257: 0.69 against 0.79); above that nine rows, which load fewer
// coefficients per row, and as many modes per block as 512 threads allow
// (4,560 x 129, float2 buffers: 1.29 ms, 1.41 with 8 modes, 1.35 with five
// rows; 12,192 x 193, FP64: 5.29 with 16 modes, 5.65 with 8, 5.79 with five
// rows).  The scans work in whole warps, so a block has one at least: pencils of
// up to 15 points, three five-row chunks, take nine rows and 32 modes.
void y_geometry(lmc::Dev &d, const lmc::Grid &g) {
  d.ysb = sweep_blocks(g, d.variant);
  const bool few = !many_modes(g.nmode) && g.nmode <= FEW_MODES;
  const int t5 = (g.my + 4) / 5 * 8;  // threads of a block of five-row chunks
  d.yC = few && t5 >= 32 && t5 <= 512 ? 5 : 9;
  d.ync = (g.my + d.yC - 1) / d.yC;
  d.yMB = d.yC == 5 ? 8 : d.ync * 32 <= 256 ? 32 : d.ync * 16 <= 512 ? 16 : 8;
}

// Profiling: a (start, stop) pair of events around each group of launches,
// recorded on the stream that runs the group; lmc_profile_read sums the
// pairs per kernel id.  Returns the pair's index, or -1 when not profiling.
int prof_begin(lmc_handle *h, cudaStream_t st) {
  if (!h->prof) return -1;
  while (h->ev_used + 2 > h->ev_pool.size()) {
    if (h->ev_pool.size() >= 65536) return -1;
    cudaEvent_t e;
    if (cudaEventCreate(&e) != cudaSuccess) return -1;
    h->ev_pool.push_back(e);
    h->ev_kid.push_back(-1);
  }
  const int a = (int)h->ev_used;
  cudaEventRecord(h->ev_pool[a], st);
  h->ev_used += 2;
  return a;
}
void prof_end(lmc_handle *h, int kid, int a, cudaStream_t st) {
  if (a < 0) return;
  cudaEventRecord(h->ev_pool[a + 1], st);
  h->ev_kid[a] = kid;
}

int check_launch(lmc_handle *h) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    std::fprintf(stderr, "lomacte_b200: launch failed: %s\n", cudaGetErrorString(e));
    h->err = LMC_ECUDA;
    return LMC_ECUDA;
  }
  return LMC_OK;
}

int do_load(lmc_handle *h, const double *vor, const double *phi, const double *psi, const double *scal,
            const double *u00, const double *v00, const double *w00, double time) {
  const lmc::Dev &d = h->d;
  const size_t ns = (size_t)d.nmode * d.my * sizeof(double2);
  LMC_CK(cudaSetDevice(h->p.device));
  // reference layout [kx][kz][y] -> device layout [y][kx][kz]
  const double *src[4] = {vor, phi, psi, scal};
  double2 *dst[4] = {d.vor, d.phi, d.psi, d.scal};
  for (int f = 0; f < 4; f++) {  // staged through the FP64 buffers 7..9
    double2 *stage = d.sb[7 + f % 3];
    LMC_CK(cudaMemcpyAsync(stage, src[f], ns, cudaMemcpyHostToDevice, h->s));
    lmc::launch_ref2dev(d, stage, dst[f], h->s);
  }
  LMC_CK(cudaMemsetAsync(d.Rom, 0, ns, h->s));
  LMC_CK(cudaMemsetAsync(d.Rphi, 0, ns, h->s));
  if (d.variant) LMC_CK(cudaMemsetAsync(d.RT, 0, ns, h->s));
  LMC_CK(cudaMemsetAsync(d.rhst, 0, (size_t)d.my * d.mgalz * d.mgalx * sizeof(double), h->s));
  const size_t ny = (size_t)d.my * sizeof(double);
  LMC_CK(cudaMemcpyAsync(d.u00, u00, ny, cudaMemcpyHostToDevice, h->s));
  LMC_CK(cudaMemcpyAsync(d.v00, v00, ny, cudaMemcpyHostToDevice, h->s));
  LMC_CK(cudaMemcpyAsync(d.w00, w00, ny, cudaMemcpyHostToDevice, h->s));
  LMC_CK(cudaMemsetAsync(d.rf0u, 0, ny, h->s));
  LMC_CK(cudaMemsetAsync(d.rf0w, 0, ny, h->s));
  LMC_CK(cudaMemsetAsync(d.rf0v, 0, ny, h->s));
  // Densities at the walls from the 00 mode of T (cross.f:211-213).
  const double tb = scal[0], tt = scal[2 * (size_t)(d.my - 1)];
  if (!(tb > 0.0) || !(tt > 0.0)) return LMC_EINVAL;
  double sc[5] = {h->p.dt, h->p.dt, time, 1.0 / tb, 1.0 / tt};  // [5], [6]: the scalar's wall values
  LMC_CK(cudaMemcpyAsync(d.scal_d, sc, sizeof(sc), cudaMemcpyHostToDevice, h->s));
  if (d.scalar) LMC_CK(cudaMemsetAsync(d.rhsz, 0, (size_t)d.my * d.mgalz * d.mgalx * sizeof(double), h->s));
  LMC_CK(cudaMemsetAsync(d.diag, 0, 16 * sizeof(double), h->s));
  LMC_CK(cudaMemsetAsync(d.status, 0, sizeof(int), h->s));
  LMC_CK(cudaStreamSynchronize(h->s));
  h->steps = 0;
  h->err = 0;
  h->d.mean_ok = 0;  // no plane sums of a previous substep yet
  return LMC_OK;
}

}  // namespace

extern "C" {

const char *lmc_strerror(int code) {
  switch (code) {
    case LMC_OK: return "ok";
    case LMC_EINVAL: return "invalid argument or grid";
    case LMC_ENOMEM: return "device out of memory";
    case LMC_ENAN: return "non-finite value in the step's diagnostics";
    case LMC_ETIMEOUT: return "device wait timed out";
    case LMC_ECUDA: return "CUDA runtime error";
    case LMC_ENODEV: return "no CUDA device";
    default: return "unknown error";
  }
}

int lmc_create(const lmc_params *p, const double *y, lmc_handle **out) {
  if (!p || !y || !out) return LMC_EINVAL;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return LMC_ENODEV;
  }
  if (p->device < 0 || p->device >= ndev) return LMC_EINVAL;
  if (p->precision < 0 || p->precision > 2) return LMC_EINVAL;
  if (p->variant < 0 || p->variant > 1 || (p->variant == 1 && p->precision != 0)) return LMC_EINVAL;
  if (p->scalar < 0 || p->scalar > 1 || (p->scalar && p->variant)) return LMC_EINVAL;
  if (p->visc < 0 || p->visc > 1 || (p->visc && (p->variant || !(p->sigma >= 0.0 && p->sigma <= 4.0))))
    return LMC_EINVAL;
  lmc_handle *h = new (std::nothrow) lmc_handle();
  if (!h) return LMC_ENOMEM;
  h->p = *p;
  h->g.set(p->mgalx, p->mgalz, p->my);
  lmc::Dev &d = h->d;
  std::memset(&d, 0, sizeof(d));
  d.prec = p->precision;
  if (d.prec == 1) {
    const char *e = std::getenv("LMC_FFT64");
    d.fft64 = e ? (std::atoi(e) & 7) : 0;
  }
  const lmc::Grid &g = h->g;
  int rc = LMC_OK;
  // x lengths from 24 up; z also 3 (mz = 1: a 2-D run, one kz mode)
  if (g.nkx < 1 || g.mz < 1 || g.mgalx < 24 || !lmc::fft_supported(g.mgalx) || !lmc::fft_supported(g.mgalz))
    rc = LMC_EINVAL;
  if (!rc && !xstage_fits(g, p->scalar, p->visc)) rc = LMC_EINVAL;
  if (!rc) rc = pick_chunks(g.my, d.C, d.lpm, d.base, d.extra);
  if (rc) { delete h; return rc; }
  try {
    lmc::build_yops(g.my, y, h->ops);
    lmc::build_scans(h->ops, d.lpm, d.base, d.extra);
  } catch (...) {
    delete h;
    return LMC_EINVAL;
  }
  std::vector<double> kx(g.nkx), kz(g.mz);
  for (int i = 0; i < g.nkx; i++) kx[i] = p->alp * i;                         // main.f:789-792
  for (int k = 0; k < g.mz; k++) kz[k] = p->bet * ((k <= g.nz1) ? k : k - g.mz);  // main.f:769-778
  lmc::build_poisson(g, h->ops, kx.data(), kz.data(), h->pt);

  if (cudaSetDevice(p->device) != cudaSuccess ||
      cudaDeviceGetAttribute(&d.smem_limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, p->device) != cudaSuccess) {
    delete h;
    return LMC_ECUDA;
  }
  if (cudaStreamCreateWithFlags(&h->s, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithFlags(&h->s2, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming) != cudaSuccess) {
    lmc_destroy(h);
    return LMC_ECUDA;
  }
  d.my = g.my; d.mgalx = g.mgalx; d.mgalz = g.mgalz; d.nkx = g.nkx; d.mz = g.mz; d.nz1 = g.nz1; d.nmode = g.nmode;
  d.zp0 = 0; d.zkn = g.nkx; d.xt0 = 0; d.xnt = 0; d.xl0 = 0; d.msum = 1;  // the whole domain
  d.ire = 1.0 / p->Re;
  d.variant = p->variant;
  d.scalar = p->scalar;
  d.visc = p->visc;
  d.sigma = p->visc ? p->sigma : 0.0;
  // Re*Sc; Sc <= 0 takes Sc = Pr, the Schmidt number of the reference's Pe = Re*0.7f
  d.pez = p->Re * (p->schmidt > 0 ? p->schmidt : (double)0.7f);
  // Pe = Re*0.7f (main.f:569); the 2014 code uses Pe = Re (lomacte/cross.f:1301)
  d.peclet = p->peclet > 0 ? p->peclet : (d.variant ? p->Re : p->Re * (double)0.7f);
  d.cfl = (double)(float)p->cfl;
  d.hxalp = p->alp * (g.mgalx - 1) / M_PI;  // cross.f:1498
  d.hzbet = p->bet * (g.mgalz - 1) / M_PI;  // cross.f:1499
  for (int r = 0; r < 3; r++) {
    d.gama[r] = h->rk.gama[r]; d.xi[r] = h->rk.xi[r]; d.alpha[r] = h->rk.alpha[r]; d.beta[r] = h->rk.beta[r];
  }
  const lmc::YOps &o = h->ops;
  // y-operator tables go to the device chunk-major (see lmcd::tab)
  const int C = d.C, lpm = d.lpm, base = d.base, extra = d.extra, my = g.my;
  auto cm = [&](const std::vector<double> &T, int W) { return lmc::chunk_major(T, my, W, C, lpm, base, extra); };
  // the 2014 variant, the passive scalar and the variable viscosity take
  // the kernel sequence of grids that sweep along y (T's update apart)
  y_geometry(d, g);
  d.tpm = (d.variant || p->scalar || p->visc) ? 1 : d.ysb > 0 || many_modes(g.nmode);
  lmc::ChunkTables ct;
  lmc::build_chunk_tables(o, d.yC, d.ync, ct);
  // mode-fastest per-mode tables [my][band][nmode]
  const size_t nt = (size_t)g.nmode * my;
  std::vector<double> PLt(nt * 2), PUt(nt * 3), V12t(nt * 2);
  {
    const size_t n = (size_t)g.nmode;
#pragma omp parallel for schedule(static)
    for (int j = 0; j < my; j++)
      for (size_t m = 0; m < n; m++) {
        const size_t src = m * my + j;
        for (int c = 0; c < 2; c++) PLt[((size_t)j * 2 + c) * n + m] = h->pt.L[src * 2 + c];
        for (int c = 0; c < 3; c++) PUt[((size_t)j * 3 + c) * n + m] = h->pt.U[src * 3 + c];
        for (int c = 0; c < 2; c++) V12t[((size_t)j * 2 + c) * n + m] = h->pt.V12[src * 2 + c];
      }
  }
  if ((rc = dupload(h, &d.dt12, cm(o.dt12, 7))) || (rc = dupload(h, &d.dt11, cm(o.dt11, 7))) ||
      (rc = dupload(h, &d.dt22, cm(o.dt22, 5))) ||
      (rc = dupload(h, &d.p1L, cm(o.p1L, 3))) || (rc = dupload(h, &d.p1U, cm(o.p1U, 4))) ||
      (rc = dupload(h, &d.p3L, cm(o.p3L, 2))) || (rc = dupload(h, &d.p3U, cm(o.p3U, 3))) ||
      (rc = dupload(h, &d.i8L, cm(o.i8L, 3))) || (rc = dupload(h, &d.i8U, cm(o.i8U, 4))) ||
      (rc = dupload(h, &d.fmap, cm(o.fmap, 1))) || (rc = dupload(h, &d.hy, o.hy)) || (rc = dupload(h, &d.trp, o.trp)) ||
      (rc = dupload(h, &d.y, o.y)) ||
      (rc = dupload(h, &d.k1L, o.k1L)) || (rc = dupload(h, &d.k1U, o.k1U)) || (rc = dupload(h, &d.k3L, o.k3L)) ||
      (rc = dupload(h, &d.k3U, o.k3U)) || (rc = dupload(h, &d.k8L, o.k8L)) || (rc = dupload(h, &d.k8U, o.k8U)) ||
      (rc = dupload(h, &d.AAinv, h->pt.AAinv)) || (rc = dupload(h, &d.k2, h->pt.k2)) || (rc = dupload(h, &d.kx, kx)) ||
      (rc = dupload(h, &d.kz, kz))) {
    lmc_destroy(h);
    return rc;
  }
  // row form of d/dy (the statistics and the export differentiate one thread
  // per mode) and of the wall derivatives, and the per-mode tables
  if ((rc = dupload(h, &d.r_dt12, o.dt12)) || (rc = dupload(h, &d.r_p1L, o.p1L)) ||
      (rc = dupload(h, &d.r_p1U, o.p1U)) || (rc = dupload(h, &d.r_fmap, o.fmap)) ||
      (rc = dupload(h, &d.r_ebot, o.ebot)) || (rc = dupload(h, &d.r_etop, o.etop)) ||
      (rc = dupload(h, &d.PLt, PLt)) || (rc = dupload(h, &d.PUt, PUt)) || (rc = dupload(h, &d.V12t, V12t))) {
    lmc_destroy(h);
    return rc;
  }
  if (d.ysb &&
      ((rc = dupload(h, &d.r_dt22, o.dt22)) || (rc = dupload(h, &d.r_dt21, o.dt21)) ||
       (rc = dupload(h, &d.r_p3L, o.p3L)) || (rc = dupload(h, &d.r_p3U, o.p3U)) ||
       (rc = dupload(h, &d.r_q1U, o.q1U)) || (rc = dupload(h, &d.r_q1L, o.q1L)) ||
       (rc = dupload(h, &d.r_q3U, o.q3U)) || (rc = dupload(h, &d.r_q3L, o.q3L)))) {
    lmc_destroy(h);
    return rc;
  }
  {
    lmc::YChunk &q = d.ct;
    const std::pair<const double **, const std::vector<double> *> part[] = {
        {&q.fw1, &ct.fw1}, {&q.hl1, &ct.hl1}, {&q.bw1, &ct.bw1}, {&q.hu1, &ct.hu1}, {&q.m1L, &ct.m1L},
        {&q.q1L, &ct.q1L}, {&q.g1L, &ct.g1L}, {&q.m1U, &ct.m1U}, {&q.q1U, &ct.q1U}, {&q.g1U, &ct.g1U}, {&q.fw2, &ct.fw2},
        {&q.hl2, &ct.hl2}, {&q.bw2, &ct.bw2}, {&q.hu2, &ct.hu2}, {&q.m2L, &ct.m2L}, {&q.q2L, &ct.q2L}, {&q.g2L, &ct.g2L},
        {&q.m2U, &ct.m2U}, {&q.q2U, &ct.q2U}, {&q.g2U, &ct.g2U}};
    std::vector<double> all;
    std::vector<size_t> at;
    for (const auto &p : part) {
      at.push_back(all.size());
      all.insert(all.end(), p.second->begin(), p.second->end());
      all.resize((all.size() + 1) / 2 * 2, 0.0);  // 16-byte rows
    }
    const double *run = nullptr;
    if ((rc = dupload(h, &run, all)) || (rc = dupload(h, &q.fwp, ct.fwp))) {
      lmc_destroy(h);
      return rc;
    }
    for (size_t i = 0; i < at.size(); i++) *part[i].first = run + at[i];
    q.n1 = (int)at[10];
    q.n2 = (int)all.size() - q.n1;
    q.sm = 0;
  }
  // the per-mode tables are on the device now
  h->pt = lmc::PoissonTables();
  {
    const double2 *tx = nullptr, *tz = nullptr;
    if ((rc = dupload(h, &tx, fft_twiddles<double2>(g.mgalx))) || (rc = dupload(h, &tz, fft_twiddles<double2>(g.mgalz)))) {
      lmc_destroy(h);
      return rc;
    }
    d.twx = tx;
    d.twz = tz;
    if (d.prec == 1) {
      const float2 *fx = nullptr, *fz = nullptr;
      if ((rc = dupload(h, &fx, fft_twiddles<float2>(g.mgalx))) || (rc = dupload(h, &fz, fft_twiddles<float2>(g.mgalz)))) {
        lmc_destroy(h);
        return rc;
      }
      d.twxf = fx;
      d.twzf = fz;
    }
  }
  const size_t ns = (size_t)g.nmode * g.my, nzp = (size_t)g.nkx * g.my * g.mgalz;
  double2 **spec[] = {&d.vor, &d.phi, &d.psi, &d.scal, &d.Rom, &d.Rphi};
  for (auto q : spec)
    if ((rc = dalloc(h, q, ns))) { lmc_destroy(h); return rc; }
  // work buffers: FP64 in the plain form; FP32 in the mixed form, which
  // keeps three FP64 spectral buffers for the ABI transposes and lmc_op_y
  const int nsb = lmc::n_sbuf(d), nzb = lmc::n_zbuf(d);
  for (int f = 0; f < (nsb > nzb ? nsb : nzb); f++) {
    if (f < nsb && (!d.prec || (f >= 7 && f <= 9)))
      if ((rc = dalloc(h, &d.sb[f], ns))) { lmc_destroy(h); return rc; }
    if (f < nsb && d.prec)
      if ((rc = dalloc(h, &d.sbf[f], ns))) { lmc_destroy(h); return rc; }
    if (f < nzb) {
      if (!d.prec) rc = dalloc(h, &d.zb[f], nzp);
      else rc = dalloc(h, &d.zbf[f], nzp);
      if (rc) { lmc_destroy(h); return rc; }
    }
  }
  if (d.prec) {
    // partial-sum slots: one per (z tile, warp), at most mgalz tiles
    d.mpart_ld = lmc::x_block(g.mgalx, d.prec == 1 && !(d.fft64 & 2)) / 32 * g.mgalz;
    if ((d.ysb && d.visc && (rc = dalloc(h, &d.vscr, (size_t)3 * g.my))) || (rc = dalloc(h, &d.mi, (size_t)lmc::NMI * g.my)) || (rc = dalloc(h, &h->mo[0], (size_t)12 * g.my)) ||
        (rc = dalloc(h, &h->mo[1], (size_t)12 * g.my)) ||
        (rc = dalloc(h, &d.mpart, (size_t)12 * g.my * d.mpart_ld))) {
      lmc_destroy(h);
      return rc;
    }
  }
  if (d.ysb) {
    for (int q = 0; q < 6; q++)
      if ((rc = dalloc(h, &d.ws[q], sweep_scratch(d.ysb, q, g)))) { lmc_destroy(h); return rc; }
  }
  if (d.variant &&
      ((rc = dalloc(h, &d.Told, ns)) || (rc = dalloc(h, &d.dTs, ns)) || (rc = dalloc(h, &d.RT, ns)))) {
    lmc_destroy(h);
    return rc;
  }
  d.tsrc = d.variant ? d.Told : d.scal;
  if (d.scalar &&
      ((rc = dalloc(h, &d.zsc, ns)) || (rc = dalloc(h, &d.rhsz, (size_t)g.my * g.mgalz * g.mgalx)))) {
    lmc_destroy(h);
    return rc;
  }
  double **vec[] = {&d.u00, &d.v00, &d.w00, &d.rf0u, &d.rf0w, &d.rf0v, &d.rhom};
  for (auto q : vec)
    if ((rc = dalloc(h, q, (size_t)g.my))) { lmc_destroy(h); return rc; }
  if ((rc = dalloc(h, &d.rhst, (size_t)g.my * g.mgalz * g.mgalx)) || (rc = dalloc(h, &d.scal_d, (size_t)8)) ||
      (rc = dalloc(h, &d.cflmax, (size_t)4)) || (rc = dalloc(h, &d.diag, (size_t)16)) ||
      (rc = dalloc(h, &d.status, (size_t)1))) {
    lmc_destroy(h);
    return rc;
  }
  {
    const cudaError_t e = lmc::kernels_init(d);
    if (e != cudaSuccess) {
      std::fprintf(stderr, "lomacte_b200: shared-memory opt-in failed: %s\n", cudaGetErrorString(e));
      lmc_destroy(h);
      return LMC_ECUDA;
    }
  }
  if (cudaMemsetAsync(d.status, 0, sizeof(int), h->s) != cudaSuccess ||
      cudaMemsetAsync(d.diag, 0, 16 * sizeof(double), h->s) != cudaSuccess ||
      cudaStreamSynchronize(h->s) != cudaSuccess) {  // buffers and tables in place
    lmc_destroy(h);
    return LMC_ECUDA;
  }
  *out = h;
  return LMC_OK;
}

int lmc_destroy(lmc_handle *h) {
  if (!h) return LMC_EINVAL;
  cudaSetDevice(h->p.device);
  if (h->s) cudaStreamSynchronize(h->s);  // this case's own work only
  drop_graphs(h);
  lmc::dense_destroy(h->yop);
  for (void *q : h->allocs) {
    if (h->s) cudaFreeAsync(q, h->s);
    else cudaFree(q);
  }
  for (cudaEvent_t e : h->ev_pool) cudaEventDestroy(e);
  if (h->ev_fork) cudaEventDestroy(h->ev_fork);
  if (h->ev_join) cudaEventDestroy(h->ev_join);
  if (h->s2) cudaStreamSynchronize(h->s2);
  if (h->s2) cudaStreamDestroy(h->s2);
  if (h->s) cudaStreamDestroy(h->s);
  delete h;
  return LMC_OK;
}

int lmc_load_state_f64(lmc_handle *h, const double *vor, const double *phi, const double *psi, const double *scal,
                       const double *u00, const double *v00, const double *w00, double time) {
  if (!h || !vor || !phi || !psi || !scal || !u00 || !v00 || !w00) return LMC_EINVAL;
  return do_load(h, vor, phi, psi, scal, u00, v00, w00, time);
}

int lmc_load_state_f32(lmc_handle *h, const float *vor, const float *phi, const float *psi, const float *scal,
                       const double *u00, const double *v00, const double *w00, double time) {
  if (!h || !vor || !phi || !psi || !scal || !u00 || !v00 || !w00) return LMC_EINVAL;
  const size_t n = (size_t)h->d.nmode * h->d.my * 2;
  std::vector<double> a(n), b(n), c(n), e(n);
  for (size_t i = 0; i < n; i++) { a[i] = vor[i]; b[i] = phi[i]; c[i] = psi[i]; e[i] = scal[i]; }
  return do_load(h, a.data(), b.data(), c.data(), e.data(), u00, v00, w00, time);
}

int lmc_get_state_f64(lmc_handle *h, double *vor, double *phi, double *psi, double *scal, double *u00, double *v00,
                      double *w00, double *time) {
  if (!h) return LMC_EINVAL;
  const lmc::Dev &d = h->d;
  const size_t ns = (size_t)d.nmode * d.my * sizeof(double2), ny = (size_t)d.my * sizeof(double);
  LMC_CK(cudaSetDevice(h->p.device));
  // device layout -> reference layout through the spectral work buffers
  double *dsth[4] = {vor, phi, psi, scal};
  const double2 *srcd[4] = {d.vor, d.phi, d.psi, d.scal};
  for (int f = 0; f < 4; f++)
    if (dsth[f]) {
      double2 *stage = d.sb[7 + f % 3];
      lmc::launch_dev2ref(d, srcd[f], stage, h->s);
      LMC_CK(cudaMemcpyAsync(dsth[f], stage, ns, cudaMemcpyDeviceToHost, h->s));
    }
  if (u00) LMC_CK(cudaMemcpyAsync(u00, d.u00, ny, cudaMemcpyDeviceToHost, h->s));
  if (v00) LMC_CK(cudaMemcpyAsync(v00, d.v00, ny, cudaMemcpyDeviceToHost, h->s));
  if (w00) LMC_CK(cudaMemcpyAsync(w00, d.w00, ny, cudaMemcpyDeviceToHost, h->s));
  double sc[8];
  LMC_CK(cudaMemcpyAsync(sc, d.scal_d, sizeof(sc), cudaMemcpyDeviceToHost, h->s));
  LMC_CK(cudaStreamSynchronize(h->s));
  if (time) *time = sc[2];
  return h->err;
}

int lmc_physical_f64(lmc_handle *h, int nplanes, const int *jplanes, double *out) {
  if (!h || nplanes < 0 || (nplanes > 0 && (!jplanes || !out)) || h->d.variant) return LMC_EINVAL;
  if (h->err) return h->err;
  const lmc::Dev &d = h->d;
  for (int p = 0; p < nplanes; p++)
    if (jplanes[p] < 1 || jplanes[p] > d.my) return LMC_EINVAL;
  if (nplanes == 0) return LMC_OK;
  LMC_CK(cudaSetDevice(h->p.device));
  // an FP64 view of the case on buffers of its own: the state and its RK3
  // memory are read, never written
  lmc::Dev e = d;
  e.prec = 0;
  e.fft64 = 0;
  e.ysb = 0;  // Lapvdvhom with dm_y/dy written out
  const int nf = d.scalar ? 11 : 10, nq = d.scalar ? 8 : 7;
  const size_t ns = (size_t)d.nmode * d.my, nzp = (size_t)d.nkx * d.my * d.mgalz;
  const size_t nout = (size_t)nplanes * nq * d.mgalz * d.mgalx;
  std::vector<void *> tmp;
  int rc = LMC_OK;
  auto get = [&](void **q, size_t bytes) {
    if (rc) return;
    const cudaError_t err = cudaMallocAsync(q, bytes, h->s);
    if (err != cudaSuccess) {
      cudaGetLastError();
      rc = err == cudaErrorMemoryAllocation ? LMC_ENOMEM : LMC_ECUDA;
      *q = nullptr;
      return;
    }
    tmp.push_back(*q);
  };
  for (int f = 0; f < lmc::NWB; f++) {
    e.sb[f] = e.zb[f] = nullptr;
    e.sbf[f] = e.zbf[f] = nullptr;
  }
  for (int q = 0; q < nf; q++) get((void **)&e.sb[lmc::xslot(q)], ns * sizeof(double2));
  get((void **)&e.sb[lmc::SB_MY], ns * sizeof(double2));
  get((void **)&e.sb[lmc::SB_DMY], ns * sizeof(double2));
  for (int q = 0; q < nf; q++) get((void **)&e.zb[q], nzp * sizeof(double2));
  for (int k = 0; k < 4; k++) get((void **)&e.ws[k], ns * sizeof(double2));
  int *jrow = nullptr;
  double *od = nullptr;
  get((void **)&jrow, (size_t)nplanes * sizeof(int));
  get((void **)&od, nout * sizeof(double));
  std::vector<int> j0(nplanes);
  for (int p = 0; p < nplanes; p++) j0[p] = jplanes[p] - 1;
  if (!rc) {
    cudaError_t err = cudaMemcpyAsync(jrow, j0.data(), j0.size() * sizeof(int), cudaMemcpyHostToDevice, h->s);
    if (err == cudaSuccess) {
      lmc::launch_lapv(e, h->s);
      lmc::launch_xprep(e, h->s);
      lmc::launch_zinv(e, h->s, 2, 0, nf);
      lmc::launch_xexport(e, jrow, nplanes, nf, od, h->s);
      err = cudaGetLastError();
    }
    if (err == cudaSuccess) err = cudaMemcpyAsync(out, od, nout * sizeof(double), cudaMemcpyDeviceToHost, h->s);
    if (err != cudaSuccess) rc = LMC_ECUDA;
  }
  for (void *q : tmp) cudaFreeAsync(q, h->s);
  if (cudaStreamSynchronize(h->s) != cudaSuccess && !rc) rc = LMC_ECUDA;
  return rc;
}

int lmc_load_scalar_f64(lmc_handle *h, const double *z) {
  if (!h || !z || !h->d.scalar) return LMC_EINVAL;
  if (h->err) return h->err;
  const lmc::Dev &d = h->d;
  const size_t ns = (size_t)d.nmode * d.my * sizeof(double2);
  LMC_CK(cudaSetDevice(h->p.device));
  LMC_CK(cudaMemcpyAsync(d.sb[7], z, ns, cudaMemcpyHostToDevice, h->s));
  lmc::launch_ref2dev(d, d.sb[7], d.zsc, h->s);
  LMC_CK(cudaMemsetAsync(d.rhsz, 0, (size_t)d.my * d.mgalz * d.mgalx * sizeof(double), h->s));
  // wall values of the 00 mode, held by the boundary condition
  const double zw[2] = {z[0], z[2 * (size_t)(d.my - 1)]};
  LMC_CK(cudaMemcpyAsync(d.scal_d + 5, zw, sizeof(zw), cudaMemcpyHostToDevice, h->s));
  LMC_CK(cudaStreamSynchronize(h->s));
  return LMC_OK;
}

int lmc_get_scalar_f64(lmc_handle *h, double *z) {
  if (!h || !z || !h->d.scalar) return LMC_EINVAL;
  const lmc::Dev &d = h->d;
  const size_t ns = (size_t)d.nmode * d.my * sizeof(double2);
  LMC_CK(cudaSetDevice(h->p.device));
  lmc::launch_dev2ref(d, d.zsc, d.sb[7], h->s);
  LMC_CK(cudaMemcpyAsync(z, d.sb[7], ns, cudaMemcpyDeviceToHost, h->s));
  LMC_CK(cudaStreamSynchronize(h->s));
  return h->err;
}

int lmc_get_state_f32(lmc_handle *h, float *vor, float *phi, float *psi, float *scal, double *u00, double *v00,
                      double *w00, double *time) {
  if (!h) return LMC_EINVAL;
  const size_t n = (size_t)h->d.nmode * h->d.my * 2;
  std::vector<double> a(vor ? n : 0), b(phi ? n : 0), c(psi ? n : 0), e(scal ? n : 0);
  int rc = lmc_get_state_f64(h, vor ? a.data() : nullptr, phi ? b.data() : nullptr, psi ? c.data() : nullptr,
                             scal ? e.data() : nullptr, u00, v00, w00, time);
  if (rc) return rc;
  for (size_t i = 0; i < n; i++) {
    if (vor) vor[i] = (float)a[i];
    if (phi) phi[i] = (float)b[i];
    if (psi) psi[i] = (float)c[i];
    if (scal) scal[i] = (float)e[i];
  }
  return LMC_OK;
}

}  // extern "C"

namespace {

// Enqueue the kernels of one RK3 step on the handle's streams (directly, or
// into a graph being captured) and advance the host-side bookkeeping.
// Two independent pieces of each substep run on the second stream, beside
// the main chain: the T derivatives and the z transforms of the inputs made
// from T beside Lapvdvhom, the assembly of rho u_i and its z transforms
// (neither chain reads what the other writes), and the 00 RHS, the updates
// of T and Z and the psi solve beside the RK3 update of Omega_y and phi.
// The 2014 variant differentiates the T that its assembly saves, and takes
// d(rho) from a transform round trip after T's update, so it runs in one
// chain.
// The Dev of slab block r: its z transforms (kx planes, buffers Z) or its x
// stage (lines, buffers X; the mixed form's plane sums after the last block).
lmc::Dev block_dev(const lmc_handle *h, int r, bool xstage) {
  lmc::Dev e = h->d;
  const auto &sp = h->split;
  const auto &buf = xstage ? sp.X[r] : sp.Z[r];
  for (int f = 0; f < lmc::NWB; f++) {
    void *q = f < (int)buf.size() ? buf[f] : nullptr;
    if (e.prec) e.zbf[f] = (float2 *)q;
    else e.zb[f] = (double2 *)q;
  }
  if (xstage) {
    e.xt0 = e.xl0 = sp.l0[r];  // one z line per x-stage tile (mgalx >= 144)
    e.xnt = sp.nl[r];
    e.msum = r == sp.n - 1;
  } else {
    e.zp0 = sp.p0[r];
    e.zkn = sp.np[r];
  }
  return e;
}

// The plane <-> line exchanges of the slab decomposition (chpl2ln /
// chln2pl, change.f:1-143) as device copies: block r's planes of block
// r2's lines, of the z-physical fields that were transformed: the inputs
// (those that the x stage forms itself left out) or the outputs.
int exchange(lmc_handle *h, bool to_lines, cudaStream_t s) {
  const auto &sp = h->split;
  const size_t es = h->d.prec ? sizeof(float2) : sizeof(double2), nkx = (size_t)h->d.nkx;
  const int n = to_lines ? lmc::n_zin(h->d) : lmc::n_out(h->d);
  for (int i = 0; i < n; i++) {
    const int f = to_lines ? lmc::in_field(h->d, i) : i;
    for (int r = 0; r < sp.n; r++)
      for (int r2 = 0; r2 < sp.n; r2++) {
        char *z = (char *)sp.Z[r][f] + (size_t)sp.l0[r2] * sp.np[r] * es;
        char *x = (char *)sp.X[r2][f] + (size_t)sp.p0[r] * es;
        const size_t w = (size_t)sp.np[r] * es;
        if (to_lines) LMC_CK(cudaMemcpy2DAsync(x, nkx * es, z, w, w, sp.nl[r2], cudaMemcpyDeviceToDevice, s));
        else LMC_CK(cudaMemcpy2DAsync(z, w, x, nkx * es, w, sp.nl[r2], cudaMemcpyDeviceToDevice, s));
      }
  }
  return LMC_OK;
}

int enqueue_step(lmc_handle *h, int cfl_step, bool stats = false, bool split = false) {
  lmc::Dev &d = h->d;
  cudaStream_t s = h->s, s2 = h->s2;
  auto run = [&](int kid, cudaStream_t st, auto &&launch) {
    const int a = prof_begin(h, st);
    launch();
    prof_end(h, kid, a, st);
  };
  auto fork = [&]() {
    if (cudaEventRecord(h->ev_fork, s) != cudaSuccess) return false;
    return cudaStreamWaitEvent(s2, h->ev_fork, 0) == cudaSuccess;
  };
  auto join = [&]() {
    if (cudaEventRecord(h->ev_join, s2) != cudaSuccess) return false;
    return cudaStreamWaitEvent(s, h->ev_join, 0) == cudaSuccess;
  };
  const bool side = !d.variant;
  for (int rk = 0; rk < 3; rk++) {
    if (d.prec) {  // this substep's plane sums, and the previous ones
      d.mo_cur = h->mo[h->mo_flip];
      d.mo_prev = h->mo[1 - h->mo_flip];
    }
    // the T derivatives and the inverse z transforms of the four inputs
    // made from T (lap T, dT/dy, dT/dz, T) run beside Lapvdvhom, the
    // assembly of rho u_i and the z transforms of rho u_i
    if (split) {  // slab blocks: every transform after the y work, block by block
      if (!fork()) return LMC_ECUDA;
      run(2, s2, [&] { lmc::launch_tder(d, s2); });
      if (d.scalar) run(2, s2, [&] { lmc::launch_zder(d, s2); });
      if (cudaEventRecord(h->ev_join, s2) != cudaSuccess) return LMC_ECUDA;
      run(0, s, [&] { lmc::launch_lapv(d, s); });
      run(1, s, [&] { lmc::launch_assemble(d, rk, s); });
      if (d.visc) run(1, s, [&] { lmc::launch_sgrad(d, s); });
      if (cudaStreamWaitEvent(s, h->ev_join, 0) != cudaSuccess) return LMC_ECUDA;
      for (int r = 0; r < h->split.n; r++) {
        const lmc::Dev e = block_dev(h, r, false);
        run(3, s, [&] { lmc::launch_zinv(e, s); });
      }
      if (int rc = exchange(h, true, s)) return rc;
    } else {
      if (side) {
        if (!fork()) return LMC_ECUDA;
        run(2, s2, [&] { lmc::launch_tder(d, s2); });
        if (d.scalar) run(2, s2, [&] { lmc::launch_zder(d, s2); });
        run(3, s2, [&] { lmc::launch_zinv(d, s2, 0, 3, 4); });
        if (d.scalar) run(3, s2, [&] { lmc::launch_zinv(d, s2, 0, 7, 4); });
        if (cudaEventRecord(h->ev_join, s2) != cudaSuccess) return LMC_ECUDA;
      }
      run(0, s, [&] { lmc::launch_lapv(d, s); });
      run(1, s, [&] { lmc::launch_assemble(d, rk, s); });
      if (d.visc) run(1, s, [&] { lmc::launch_sgrad(d, s); });  // the strain-rate inputs
      if (side) {
        run(3, s, [&] { lmc::launch_zinv(d, s, 0, 0, 3); });
        if (d.visc) run(3, s, [&] { lmc::launch_zinv(d, s, 0, lmc::vbase(d) - 1, 5); });
        if (cudaStreamWaitEvent(s, h->ev_join, 0) != cudaSuccess) return LMC_ECUDA;
      } else {
        run(2, s, [&] { lmc::launch_tder(d, s); });
        run(3, s, [&] { lmc::launch_zinv(d, s); });
      }
    }
    // statistics of an accumulating step, first substep (cross.f:578-585,
    // 794-812, 1583-1607); id 10 in the profile
    const bool st_now = stats && rk == 0;
    if (st_now) run(10, s, [&] { lmc::launch_stats1(d, h->st, s); });
    if (st_now) run(10, s, [&] { lmc::launch_xstats(d, h->st, s); });
    if (rk == 0) {
      LMC_CK(cudaMemsetAsync(d.rhom, 0, (size_t)d.my * sizeof(double), s));
      if (cfl_step) LMC_CK(cudaMemsetAsync(d.cflmax, 0, 4 * sizeof(unsigned long long), s));
    }
    const int do_cfl = cfl_step && rk == 0;
    if (split) {
      for (int r = 0; r < h->split.n; r++) {
        const lmc::Dev e = block_dev(h, r, true);
        run(4, s, [&] { lmc::launch_xphys(e, rk, do_cfl, rk == 0, s); });
      }
      if (int rc = exchange(h, false, s)) return rc;
      for (int r = 0; r < h->split.n; r++) {
        const lmc::Dev e = block_dev(h, r, false);
        run(5, s, [&] { lmc::launch_zfwd(e, s); });
      }
    } else {
      run(4, s, [&] {
        lmc::launch_xphys(d, rk, do_cfl, rk == 0, s);
        if (d.variant && rk == 0) lmc::launch_cfl14(d, do_cfl, s);
      });
      run(5, s, [&] { lmc::launch_zfwd(d, s); });
    }
    if (st_now) run(10, s, [&] { lmc::launch_stats2(d, h->st, s); });
    if (side) {  // beside the RK3 update, which neither reads nor writes what these write
      if (!fork()) return LMC_ECUDA;
      run(6, s2, [&] { lmc::launch_post1_00(d, rk, do_cfl, 1, s2); });
      run(8, s2, [&] { lmc::launch_psi_tail(d, rk, cfl_step, s2); });
      if (d.tpm) run(6, s2, [&] { lmc::launch_tupd(d, rk, s2); });   // T += Delta T
      if (d.scalar) run(5, s2, [&] { lmc::launch_zupd(d, s2); });    // Z += Delta Z
      run(8, s2, [&] { lmc::launch_psi(d, rk, s2); });
      run(7, s, [&] { lmc::launch_post(d, rk, s); });
      if (!join()) return LMC_ECUDA;
    } else {  // the 2014 variant: d(rho) from T and Delta T (tauij2, lomacte/cross.f:877)
      run(6, s, [&] { lmc::launch_tupd(d, rk, s); });
      run(6, s, [&] { lmc::launch_post1_00(d, rk, do_cfl, 1, s); });
      run(3, s, [&] { lmc::launch_zinv(d, s, 1); });
      run(4, s, [&] { lmc::launch_xdrho(d, s); });
      run(5, s, [&] { lmc::launch_zfwd(d, s, 1); });
      run(7, s, [&] { lmc::launch_post(d, rk, s); });
      run(8, s, [&] { lmc::launch_psi(d, rk, s); });
      run(8, s, [&] { lmc::launch_psi_tail(d, rk, cfl_step, s); });
    }
    if (d.prec) {
      d.mean_ok = 1;
      h->mo_flip = 1 - h->mo_flip;
    }
  }
  return LMC_OK;
}

void drop_graphs(lmc_handle *h) {
  for (auto &row : h->gexec)
    for (auto &g : row)
      if (g) {
        cudaGraphExecDestroy(g);
        g = nullptr;
      }
}

// Capture one RK3 step into an executable graph.  The step's kernels are
// fixed by (cfl_step, mo_flip parity); everything that changes from step to
// step (Deltat, time, the state) lives in device memory.
int capture_step(lmc_handle *h, int cfl_step, cudaGraphExec_t *out) {
  cudaGraph_t g = nullptr;
  const lmc::Dev saved = h->d;
  const int flip = h->mo_flip;
  if (cudaStreamBeginCapture(h->s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return LMC_ECUDA;
  const int rc = enqueue_step(h, cfl_step);
  const cudaError_t e = cudaStreamEndCapture(h->s, &g);
  h->d = saved;  // the bookkeeping is replayed with the graph launch
  h->mo_flip = flip;
  if (rc || e != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    return LMC_ECUDA;
  }
  const cudaError_t ei = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  if (ei != cudaSuccess) {
    cudaGetLastError();
    return LMC_ECUDA;
  }
  return LMC_OK;
}

}  // namespace

extern "C" {

int lmc_step(lmc_handle *h, int nsteps) {
  if (!h || nsteps < 0) return LMC_EINVAL;
  if (h->err) return h->err;
  LMC_CK(cudaSetDevice(h->p.device));
  lmc::Dev &d = h->d;
  const int ncfl = h->p.ncfl > 0 ? h->p.ncfl : 1;
  for (int n = 0; n < nsteps; n++) {
    const int cfl_step = (h->p.dt_mode == 0) && (h->steps % ncfl == 0);  // cross.f:240
    // graphs replay steady steps; the first step after a load (whose first
    // substep has no previous plane sums) and profiled steps run directly
    const bool replay = h->graphs && !h->prof && (d.prec == 0 || d.mean_ok);
    if (replay) {
      cudaGraphExec_t &ge = h->gexec[cfl_step][h->mo_flip];
      if (!ge && capture_step(h, cfl_step, &ge) != LMC_OK) {
        std::fprintf(stderr, "lomacte_b200: step graph capture failed; running without graphs\n");
        h->graphs = false;
        drop_graphs(h);
      }
      if (ge) {
        if (cudaGraphLaunch(ge, h->s) != cudaSuccess) {
          h->err = LMC_ECUDA;
          return LMC_ECUDA;
        }
        if (d.prec) h->mo_flip ^= 1;  // three substeps: the arrays swap an odd number of times
        h->steps++;
        continue;
      }
    }
    const int rc = enqueue_step(h, cfl_step);
    if (rc) return rc;
    h->steps++;
    if (check_launch(h)) return LMC_ECUDA;
  }
  return LMC_OK;
}

int lmc_stats_reset(lmc_handle *h, int nsp, const int *jsp, double sigma) {
  if (!h || nsp < 0 || (nsp > 0 && !jsp) || h->d.variant) return LMC_EINVAL;
  if (h->err) return h->err;
  const int my = h->d.my;
  for (int i = 0; i < nsp; i++)
    if (jsp[i] < 1 || jsp[i] > my) return LMC_EINVAL;
  LMC_CK(cudaSetDevice(h->p.device));
  LMC_CK(cudaStreamSynchronize(h->s));  // no accumulating step may still read the old set-up
  lmc::Stats &st = h->st;
  lmc::Dev &d = h->d;
  int rc;
  if (!st.prof) {
    const size_t ns = (size_t)d.nmode * my;
    if ((rc = dalloc(h, &st.prof, (size_t)lmc::NSTAT * my)) || (rc = dalloc(h, &st.erow, (size_t)9 * my)) ||
        (rc = dalloc(h, &st.uner, (size_t)9)) || (rc = dalloc(h, &st.xpart, (size_t)9 * my * lmc::XGRP)))
      return rc;
    for (int q = 0; q < 3; q++)
      if ((rc = dalloc(h, &st.dy[q], ns))) return rc;
  }
  const size_t nspec = (size_t)d.nkx * 12 * nsp * (d.nz1 + 1);
  if (nsp > h->st_cap) {  // (re)size the spectra and plane buffers
    for (void *q : {(void *)st.spec, (void *)st.jsp}) {
      if (!q) continue;
      for (size_t i = 0; i < h->allocs.size(); i++)
        if (h->allocs[i] == q) {
          h->allocs.erase(h->allocs.begin() + i);
          break;
        }
      cudaFreeAsync(q, h->s);
    }
    h->bytes -= h->st_spec_bytes;
    st.spec = nullptr;
    st.jsp = nullptr;
    h->st_cap = -1;
    int *pj = nullptr;
    const size_t b0 = h->bytes;
    if ((rc = dalloc(h, &st.spec, nspec)) || (rc = dalloc(h, &pj, (size_t)(nsp > 0 ? nsp : 1)))) return rc;
    st.jsp = pj;
    h->st_spec_bytes = h->bytes - b0;
    h->st_cap = nsp;
  }
  std::vector<int> rows(nsp > 0 ? nsp : 1, 0);
  for (int i = 0; i < nsp; i++) rows[i] = jsp[i] - 1;
  LMC_CK(cudaMemcpyAsync((void *)st.jsp, rows.data(), rows.size() * sizeof(int), cudaMemcpyHostToDevice, h->s));
  LMC_CK(cudaMemsetAsync(st.prof, 0, (size_t)lmc::NSTAT * my * sizeof(double), h->s));
  LMC_CK(cudaMemsetAsync(st.spec, 0, (nspec ? nspec : 1) * sizeof(double), h->s));
  LMC_CK(cudaMemsetAsync(st.erow, 0, (size_t)9 * my * sizeof(double), h->s));
  LMC_CK(cudaMemsetAsync(st.uner, 0, 9 * sizeof(double), h->s));
  st.nsp = nsp;
  st.sigma = sigma;
  h->nacum = h->nacumsp = 0;
  h->st_on = true;
  return LMC_OK;
}

int lmc_stats_step(lmc_handle *h, int nsteps) {
  if (!h || nsteps < 0 || !h->st_on) return LMC_EINVAL;
  if (h->err) return h->err;
  LMC_CK(cudaSetDevice(h->p.device));
  const int ncfl = h->p.ncfl > 0 ? h->p.ncfl : 1;
  for (int n = 0; n < nsteps; n++) {
    const int cfl_step = (h->p.dt_mode == 0) && (h->steps % ncfl == 0);  // cross.f:240
    const int rc = enqueue_step(h, cfl_step, true);
    if (rc) return rc;
    h->steps++;
    h->nacum++;  // cross.f:800-801
    h->nacumsp++;
    if (check_launch(h)) return LMC_ECUDA;
  }
  return LMC_OK;
}

int lmc_step_split(lmc_handle *h, int nblocks, int nsteps) {
  if (!h || nsteps < 0 || nblocks < 1 || nblocks > h->d.nkx) return LMC_EINVAL;
  if (h->d.variant || h->d.mgalx < 144) return LMC_EINVAL;  // one z line per x-stage tile
  if (h->split.n && h->split.n != nblocks) return LMC_EINVAL;
  if (h->err) return h->err;
  LMC_CK(cudaSetDevice(h->p.device));
  auto &sp = h->split;
  if (!sp.n) {
    // pointers_calc (change.f:145-211): contiguous blocks, the first
    // n mod k of them one longer, of the kx planes and of the (z, y) lines
    const lmc::Dev &d = h->d;
    const int nlines = d.my * d.mgalz, nz = lmc::n_zbuf(d);
    const size_t es = d.prec ? sizeof(float2) : sizeof(double2);
    int p = 0, l = 0;
    sp.p0.clear(); sp.np.clear(); sp.l0.clear(); sp.nl.clear();  // a failed earlier attempt
    sp.Z.assign(nblocks, {});
    sp.X.assign(nblocks, {});
    for (int r = 0; r < nblocks; r++) {
      const int np = d.nkx / nblocks + (r < d.nkx % nblocks), nl = nlines / nblocks + (r < nlines % nblocks);
      sp.p0.push_back(p); sp.np.push_back(np); sp.l0.push_back(l); sp.nl.push_back(nl);
      p += np;
      l += nl;
      for (int f = 0; f < nz; f++) {
        char *z = nullptr, *x = nullptr;
        int rc = dalloc(h, &z, (size_t)nlines * np * es);
        if (!rc) rc = dalloc(h, &x, (size_t)nl * d.nkx * es);
        if (rc) return rc;
        sp.Z[r].push_back(z);
        sp.X[r].push_back(x);
      }
    }
    sp.n = nblocks;
  }
  const int ncfl = h->p.ncfl > 0 ? h->p.ncfl : 1;
  for (int n = 0; n < nsteps; n++) {
    const int cfl_step = (h->p.dt_mode == 0) && (h->steps % ncfl == 0);  // cross.f:240
    const int rc = enqueue_step(h, cfl_step, false, true);
    if (rc) return rc;
    h->steps++;
    if (check_launch(h)) return LMC_ECUDA;
  }
  return LMC_OK;
}

int lmc_stats_read(lmc_handle *h, double *prof, double *spec, double *uner, int *counts, int clear_spectra) {
  if (!h || !h->st_on) return LMC_EINVAL;
  LMC_CK(cudaSetDevice(h->p.device));
  const lmc::Stats &st = h->st;
  const size_t nspec = (size_t)h->d.nkx * 12 * st.nsp * (h->d.nz1 + 1);
  if (prof)
    LMC_CK(cudaMemcpyAsync(prof, st.prof, (size_t)lmc::NSTAT * h->d.my * sizeof(double), cudaMemcpyDeviceToHost,
                           h->s));
  if (spec && nspec) LMC_CK(cudaMemcpyAsync(spec, st.spec, nspec * sizeof(double), cudaMemcpyDeviceToHost, h->s));
  if (uner) LMC_CK(cudaMemcpyAsync(uner, st.uner, 9 * sizeof(double), cudaMemcpyDeviceToHost, h->s));
  LMC_CK(cudaStreamSynchronize(h->s));
  if (counts) {
    counts[0] = h->nacum;
    counts[1] = h->nacumsp;
  }
  if (clear_spectra) {  // escru.f:466-477
    if (nspec) LMC_CK(cudaMemsetAsync(st.spec, 0, nspec * sizeof(double), h->s));
    h->nacumsp = 0;
  }
  return h->err;
}

int lmc_use_graphs(lmc_handle *h, int on) {
  if (!h) return LMC_EINVAL;
  if (!on) drop_graphs(h);
  h->graphs = on != 0;
  return LMC_OK;
}

int lmc_query(lmc_handle *h) {
  if (!h) return LMC_EINVAL;
  if (h->err) return h->err;
  const cudaError_t e = cudaStreamQuery(h->s);
  if (e == cudaSuccess) return 1;
  if (e == cudaErrorNotReady) return 0;
  cudaGetLastError();
  return LMC_ECUDA;
}

size_t lmc_device_bytes(lmc_handle *h) { return h ? h->bytes : 0; }

int lmc_launches_per_step(lmc_handle *h) {
  if (!h) return LMC_EINVAL;
  // per substep: lapv, assemble, tder, zinv (in two launches), xphys, zfwd,
  // the 00 RHS, the RK3 update, psi and the 00 tail; grids with many modes
  // (and the extensions) update T in a kernel of its own; the mixed forms add
  // the plane-sum reduction after xphys
  // the 2014 variant: 14 kernels per substep (zinv in one launch, three for
  // the d(rho) round trip) and the Deltat kernel in the first substep
  if (h->d.variant) return 3 * 14 + 1;
  // the passive scalar adds three (its derivatives, its inverse z transforms,
  // its update); the variable viscosity two (the strain-rate inputs and
  // their inverse z transforms)
  const int per = (h->d.tpm ? 12 : 11) + (h->d.prec ? 1 : 0) + (h->d.scalar ? 3 : 0) + (h->d.visc ? 2 : 0);
  return 3 * per;
}

int lmc_y_family(lmc_handle *h) { return h ? h->d.tpm : LMC_EINVAL; }

size_t lmc_footprint(const lmc_params *p) {
  if (!p || p->precision < 0 || p->precision > 2) return 0;
  lmc::Grid g;
  g.set(p->mgalx, p->mgalz, p->my);
  int C, lpm, base, extra;
  if (g.nkx < 1 || g.mz < 1 || pick_chunks(g.my, C, lpm, base, extra) != LMC_OK) return 0;
  if (g.mgalx < 24 || !lmc::fft_supported(g.mgalx) || !lmc::fft_supported(g.mgalz)) return 0;
  if (!xstage_fits(g, p->scalar, p->visc)) return 0;
  const size_t S = (size_t)g.nmode * g.my, Z = (size_t)g.nkx * g.my * g.mgalz;
  const size_t P = (size_t)g.my * g.mgalz * g.mgalx;
  size_t b = 6 * S * 16 + P * 8;  // state, R_om, R_phi, RHS(T)
  if (p->variant) b += 3 * S * 16;  // T before the substep, Delta T, RHS(T)
  b += S * 7 * 8 + (size_t)g.nmode * 5 * 8 + (size_t)g.my * 120 * 8;  // per-mode and y tables
  for (int q = 0; q < 6; q++) b += sweep_scratch(sweep_blocks(g, p->variant), q, g) * 16;
  if (p->scalar) {  // Z, RHS(Z), one more spectral and z-physical work buffer
    b += S * 16 + P * 8 + (p->precision == 0 ? S * 16 + Z * 16 : S * 8 + Z * 8);
    b += 2 * (size_t)g.my * 8;  // mixed sums of the 12th output
  }
  if (p->visc) {  // spectral buffers up to 15, z-physical ones up to 14 (18 with the scalar)
    const size_t have = p->scalar ? 12 : 11, xs = 15 - have, xz = (p->scalar ? 18 : 14) - have;
    const size_t e = p->precision == 0 ? 16 : 8;
    b += xs * S * e + xz * Z * e + 3 * (size_t)g.my * 8;  // + mixed 00 profiles
  }
  if (p->precision == 0) b += 11 * S * 16 + 11 * Z * 16;          // FP64 work buffers
  else b += 3 * S * 16 + 11 * S * 8 + 11 * Z * 8 + 28 * (size_t)g.my * 8 +
            12 * (size_t)g.my * (lmc::x_block(g.mgalx, p->precision == 1) / 32) * g.mgalz * 8;
  b += (size_t)C * 32 * 64 * 8 + 6 * 5 * 32 * 16 * 8 + (size_t)(g.mgalx + g.mgalz) * 24;  // y tables, twiddles
  b += 64 * 16 * 64;                                              // allocation padding and scalars
  return b;
}

int lmc_sync(lmc_handle *h) {
  if (!h) return LMC_EINVAL;
  LMC_CK(cudaSetDevice(h->p.device));
  LMC_CK(cudaStreamSynchronize(h->s));
  return h->err;
}

int lmc_get_diag(lmc_handle *h, lmc_diag *out) {
  if (!h || !out) return LMC_EINVAL;
  LMC_CK(cudaSetDevice(h->p.device));
  double dg[16];
  int st = 0;
  LMC_CK(cudaMemcpyAsync(dg, h->d.diag, sizeof(dg), cudaMemcpyDeviceToHost, h->s));
  LMC_CK(cudaMemcpyAsync(&st, h->d.status, sizeof(int), cudaMemcpyDeviceToHost, h->s));
  LMC_CK(cudaStreamSynchronize(h->s));
  out->time = dg[0]; out->Deltat = dg[1]; out->dm = dg[2]; out->dw = dg[3]; out->Redw = dg[4];
  out->trapz = dg[5]; out->masst = dg[6]; out->massu = dg[7]; out->massv = dg[8]; out->massw = dg[9];
  out->H00u = dg[10]; out->H00w = dg[11]; out->Deltat_next = dg[12];
  out->step = h->steps;
  out->status = st;
  if (h->err) return h->err;
  for (int i = 0; i < 13; i++)  // a run that went non-finite
    if (!std::isfinite(dg[i])) {
      if (!st) out->status = LMC_ENAN;
      return LMC_ENAN;
    }
  return LMC_OK;
}

namespace {
// one bounded wait on an mbarrier that nothing completes: the path every
// transform kernel's wait takes when its bulk copy never lands
__global__ void k_wait_selftest(int *status, unsigned polls) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    lmcd::mbar_init(&bar, 1);
    lmcd::mbar_wait(&bar, 0, status, polls);
    lmcd::mbar_inval(&bar);
  }
}
}  // namespace

int lmc_wait_selftest(lmc_handle *h, unsigned polls) {
  if (!h || polls < 1 || polls > lmcd::LMC_WAIT_LIMIT) return LMC_EINVAL;
  LMC_CK(cudaSetDevice(h->p.device));
  k_wait_selftest<<<1, 32, 0, h->s>>>(h->d.status, polls);
  LMC_CK(cudaGetLastError());
  LMC_CK(cudaStreamSynchronize(h->s));
  return LMC_OK;
}

int lmc_status(lmc_handle *h) {
  if (!h) return LMC_EINVAL;
  lmc_diag dg;
  int rc = lmc_get_diag(h, &dg);
  return rc ? rc : dg.status;
}

void *lmc_stream(lmc_handle *h) { return h ? (void *)h->s : nullptr; }

int lmc_state_device_ptrs(lmc_handle *h, double **vor, double **phi, double **psi, double **scal) {
  if (!h) return LMC_EINVAL;
  if (vor) *vor = (double *)h->d.vor;
  if (phi) *phi = (double *)h->d.phi;
  if (psi) *psi = (double *)h->d.psi;
  if (scal) *scal = (double *)h->d.scal;
  return LMC_OK;
}

int lmc_profile_start(lmc_handle *h) {
  if (!h) return LMC_EINVAL;
  h->prof = true;
  h->ev_used = 0;
  return LMC_OK;
}

int lmc_profile_read(lmc_handle *h, int nk, double *ms, int *count) {
  if (!h || nk < 0 || (nk && (!ms || !count))) return LMC_EINVAL;
  LMC_CK(cudaSetDevice(h->p.device));
  LMC_CK(cudaStreamSynchronize(h->s));
  LMC_CK(cudaStreamSynchronize(h->s2));
  for (int k = 0; k < nk; k++) { ms[k] = 0.0; count[k] = 0; }
  for (size_t i = 0; i + 1 < h->ev_used; i += 2) {
    const int k = h->ev_kid[i];
    if (k < 0 || k >= nk) continue;
    float t = 0.f;
    if (cudaEventElapsedTime(&t, h->ev_pool[i], h->ev_pool[i + 1]) == cudaSuccess) {
      ms[k] += t;
      count[k] += 1;
    }
  }
  h->prof = false;
  h->ev_used = 0;
  return h->err;
}

int lmc_op_y(lmc_handle *h, int op, const double *in_dev, double *out_dev, double *out2_dev) {
  if (!h || op < 1 || op > 4 || !in_dev || !out_dev || (op == 3 && !out2_dev)) return LMC_EINVAL;
  LMC_CK(cudaSetDevice(h->p.device));
  // the operands use the reference layout; the operator runs on the device layout
  const lmc::Dev &d = h->d;
  lmc::launch_ref2dev(d, (const double2 *)in_dev, d.sb[7], h->s);
  lmc::launch_op_y(d, op, d.sb[7], d.sb[8], d.sb[9], h->s);
  lmc::launch_dev2ref(d, d.sb[8], (double2 *)out_dev, h->s);
  if (op == 3) lmc::launch_dev2ref(d, d.sb[9], (double2 *)out2_dev, h->s);
  if (check_launch(h)) return LMC_ECUDA;
  LMC_CK(cudaStreamSynchronize(h->s));
  return LMC_OK;
}

namespace {
// relative L2 difference of two device vectors (sums of squares by atomics:
// an error estimate, not bit-reproducible)
__global__ void k_rel_l2(const double *a, const double *b, size_t n, double *acc) {
  double d2 = 0.0, r2 = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double d = a[i] - b[i];
    d2 += d * d;
    r2 += b[i] * b[i];
  }
  d2 = lmcd::warp_sum(d2);
  r2 = lmcd::warp_sum(r2);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(acc, d2);
    atomicAdd(acc + 1, r2);
  }
}

int ensure_dense(lmc_handle *h) {
  if (h->yop) return LMC_OK;
  int rc = LMC_OK;
  h->yop = lmc::dense_create(h->ops, (size_t)2 * h->d.nmode, h->s, &rc);
  return h->yop ? LMC_OK : rc;
}
}  // namespace

int lmc_op_y_dense(lmc_handle *h, int op, int method, const double *in_dev, double *out_dev) {
  if (!h || op < 1 || op > 2 || method < 1 || method > 2 || !in_dev || !out_dev) return LMC_EINVAL;
  LMC_CK(cudaSetDevice(h->p.device));
  if (int rc = ensure_dense(h)) return rc;
  const lmc::Dev &d = h->d;
  lmc::launch_ref2dev(d, (const double2 *)in_dev, d.sb[7], h->s);
  if (int rc = lmc::dense_apply(h->yop, op, method, (const double *)d.sb[7], (double *)d.sb[8], h->s)) return rc;
  lmc::launch_dev2ref(d, d.sb[8], (double2 *)out_dev, h->s);
  if (check_launch(h)) return LMC_ECUDA;
  LMC_CK(cudaStreamSynchronize(h->s));
  return LMC_OK;
}

int lmc_yop_tune(lmc_handle *h, int op, double *out) {
  if (!h || op < 1 || op > 2 || !out) return LMC_EINVAL;
  if (h->err) return h->err;
  LMC_CK(cudaSetDevice(h->p.device));
  if (int rc = ensure_dense(h)) return rc;
  const lmc::Dev &d = h->d;
  const size_t n = (size_t)2 * d.nmode * d.my;
  const double2 *in = d.vor;  // the state's Omega_y, device layout
  double *ref = (double *)d.sb[8], *alt = (double *)d.sb[9];
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  double *acc = nullptr;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess ||
      cudaMallocAsync((void **)&acc, 2 * sizeof(double), h->s) != cudaSuccess) {
    if (e0) cudaEventDestroy(e0);  // nothing of a failed set-up is kept
    if (e1) cudaEventDestroy(e1);
    return LMC_ECUDA;
  }
  auto timed = [&](int method) -> double {  // best of three, ms
    float best = 1e30f;
    for (int rep = 0; rep < 3; rep++) {
      cudaEventRecord(e0, h->s);
      if (method == 0) lmc::launch_op_y(d, op, in, (double2 *)ref, nullptr, h->s);
      else if (lmc::dense_apply(h->yop, op, method, (const double *)in, alt, h->s)) return -1.0;
      cudaEventRecord(e1, h->s);
      cudaEventSynchronize(e1);
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (ms < best) best = ms;
    }
    return best;
  };
  double err[3] = {0.0, 0.0, 0.0};
  out[0] = timed(0);
  for (int m = 1; m <= 2; m++) {
    out[m] = timed(m);
    cudaMemsetAsync(acc, 0, 2 * sizeof(double), h->s);
    k_rel_l2<<<148 * 8, 256, 0, h->s>>>(alt, ref, n, acc);
    double hs[2] = {0.0, 0.0};
    cudaMemcpyAsync(hs, acc, sizeof(hs), cudaMemcpyDeviceToHost, h->s);
    cudaStreamSynchronize(h->s);
    err[m] = hs[1] > 0.0 ? std::sqrt(hs[0] / hs[1]) : std::sqrt(hs[0]);
  }
  out[3] = err[1];
  out[4] = err[2];
  // the fastest method whose difference from the banded solve is within
  // the form's budget (FP64 path 1e-12, mixed forms 1e-6)
  const double tol = d.prec ? 1e-6 : 1e-12;
  int best = 0;
  for (int m = 1; m <= 2; m++)
    if (out[m] > 0.0 && err[m] <= tol && out[m] < out[best]) best = m;
  out[5] = best;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(acc, h->s);
  if (check_launch(h)) return LMC_ECUDA;
  LMC_CK(cudaStreamSynchronize(h->s));
  return (out[1] < 0.0 || out[2] < 0.0) ? LMC_ECUDA : LMC_OK;
}

}  // extern "C"
