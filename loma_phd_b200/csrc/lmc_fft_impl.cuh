// lmc_fft_impl.cuh -- transform kernels of one lomacte RK3 substep,
// templated on the radices of the passes (FFT_RADIX, FFT_RADIX_F32), on the
// complex type CT of the butterflies (and of the lines in
// shared memory) and on the complex type ST of the work buffers in HBM:
//   <double2, double2>  FP64 plain form
//   <float2,  float2>   mixed form (FP32 transforms)
//   <double2, float2>   mixed form with FP64 transform arithmetic
// The pointwise products, the T update and the d(rho)/dt source are FP64
// in every form.  Included by the lmc_fft_*.cu translation units, each of which
// instantiates a group of lengths (they compile in parallel).
//
//   zinv : localyz2zy + fourz(+1) (fou3D.f:80-145): spectral [y][kx][kz]
//          -> zero-padded kz -> inverse c2c along z -> z-physical [y][z][kx]
//   xphys: phys2 (cross.f:1440-1828): per (y,z) line, inverse real x
//          transforms of 8 fields (two per complex transform), FP64
//          products, T update, d(rho)/dt source, CFL maxima, direct x
//          transforms of 11 fields truncated to kx < mx/2
//   zfwd : fourz(-1) + localzy2yz (fou3D.f:149-189): direct c2c along z,
//          truncation to the mz retained kz, back to [y][kx][kz]
#pragma once
#define LMC_FFT_TU
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "lmc_async.cuh"
#include "lmc_kernels.cuh"

using namespace lmcd;

namespace lmc {
namespace LMC_FFT_NS {

// The transforms of the x stage.  FP64: a line is padded in whole bank rows (128
// bytes of samples), so that consecutive samples, which the first and the last
// pass and the pointwise loop take, never share a bank, and the strided tasks of
// the other passes do not either; one slot per run left runs of twelve in
// conflict.  With the twiddles of the direct transforms in the order of the tasks
// (Fft) the x stage, which the L1 bounds, takes per step 9.14 ms after 10.23
// (256 x 257 x 256, mu, scalar), 12.56 after 13.97 (768 x 33), 1.70 after 2.00
// (192 x 193 x 128).  FP32, whose runs are even: one slot per run.
constexpr int x_pad(int r1, int r2, int r3, int un) {
  const int run = fft_run(r1, r2, r3);
  int p = run;
  if (r3 > 1)
    while (p % un) p += run;
  return p;
}
template <int R1, int R2, int R3, typename CT, int T = 1>
using XFft = Fft<R1, R2, R3, CT, T, x_pad(R1, R2, R3, 128 / (int)sizeof(CT))>;

// Geometry of the x stage: z lines per tile, threads of a block, and the
// blocks per SM that the registers are sized for.
template <int R1, int R2, int R3>
struct Geo {
  static constexpr int N = R1 * R2 * R3;
  static constexpr int RUN = fft_run(R1, R2, R3), LD = N + (RUN < N ? N / RUN : 0);
  static constexpr int ZB = N >= 144 ? 1 : N >= 36 ? 2 : 4;  // z lines per tile
};
template <int R1, int R2, int R3, bool F32>
struct XGeo {
  static constexpr int XT = x_block(R1 * R2 * R3, F32), MINB = x_minb(R1 * R2 * R3, F32);
};

// Geometry of the z transforms: kx lines per block, threads of k_zinv (ZI) and
// k_zfwd (ZF), and the stride of a line, which makes the passes with the
// lines fastest across the lanes free of bank conflicts.  The z-physical rows
// are touched in runs of KB values: 64 bytes from 576 points up (1152 points, 768
// x 33: k_zfwd 3.6 ms per step in FP64 against 6.4 with 32 bytes, 1.66 in FP32
// against 1.76), 128 at 384 and 288 (FP64, 256 x 257: 2.9 against 3.7; FP32, 256 x
// 129: k_zinv 1.87 against 2.06, k_zfwd 1.10 against 1.07), where the lines are
// short enough to fit; KiB at the three
// points of a 2-D grid, whose blocks are too small to be worth their launch
// otherwise (512 x 257: k_zfwd 10 us per launch after 50, k_zinv 6 after 20).
template <int R1, int R2, int R3, typename CT>
struct ZGeo {
  using F = Fft<R1, R2, R3, CT>;
  static constexpr int N = R1 * R2 * R3, W = sizeof(CT) == sizeof(float2) ? 2 : 1;
  static constexpr int KB = W * (N == 384 || N == 288 ? 8 : N >= 144 ? 4 : N == 3 ? 64 : 8);
  // FP32: a thread for every task of the larger radix, or for half of them
  // (256 x 129, k_zinv per step with the scalar and mu: 256 threads 1.87 ms, 384
  // 2.13; k_zfwd 1.14 and 1.10; 192 x 129, 160 threads 1.01 and 0.42, 288 1.10
  // and 0.45)
  static constexpr int ZI = W == 2 ? (N == 1152 ? 288 : N == 288 ? 160 : N == 576 ? 192 : N == 768 || N == 384 ? 256 : N > 384 ? 384 : 128)
                                   : N == 1152 ? 192 : N == 576 || N == 288 ? 96 : N >= 384 ? 128 : 64;
  static constexpr int ZF = W == 2 ? (N == 384 ? 384 : ZI) : N == 576 ? 144 : ZI;
  static constexpr int MI = (W == 2 ? 768 : 512) / ZI, MF = (W == 2 ? 768 : 512) / ZF;
  static constexpr int UN = 128 / (int)sizeof(CT), OD = F::RUN + 1, ST = KB >= UN ? 1 : UN / KB;
  static constexpr int LD = N == 3 ? 3 : F::LD + ((ST * OD) % UN + UN - F::LD % UN) % UN;
};

__host__ __device__ constexpr size_t round16(size_t b) { return (b + 15) / 16 * 16; }
template <typename TO, typename FROM>
__device__ __forceinline__ TO ccvt(FROM a) {
  return cmk<TO>((typename CReal<TO>::R)a.x, (typename CReal<TO>::R)a.y);
}

// one spectral row of input f
template <typename ST>
__device__ __forceinline__ const ST *zsrc(const Dev &d, int f, int mode) {
  if constexpr (sizeof(ST) == sizeof(double2)) {
    if (mode == 1) return f == 0 ? d.Told : d.dTs;
    if (mode == 2) return wsb<ST>(d, xslot(f));
  }
  const int vb = vbase(d);
  if (f >= vb) {  // variable viscosity: the sums, rho w (for d/dz)
    switch (f - vb) {
      case 1: return wsb<ST>(d, SB_GYY);
      case 2: return wsb<ST>(d, SB_RW);
      case 3: return wsb<ST>(d, SB_G12);
      case 4: return wsb<ST>(d, SB_G13);
      default: return wsb<ST>(d, SB_G23);
    }
  }
  switch (f) {
    case 0: return wsb<ST>(d, SB_RU);
    case 1: return wsb<ST>(d, SB_RV);
    case 2: return wsb<ST>(d, SB_RW);
    case 3: return wsb<ST>(d, SB_LAPT);
    case 5: return wsb<ST>(d, SB_DTDY);
    case 8: return wsb<ST>(d, SB_LAPZ);   // passive scalar: lap Z,
    case 10: return wsb<ST>(d, SB_DZDY);  // dZ/dy,
    case 9:
    case 11:                              // and Z for dZ/dx, dZ/dz
      if constexpr (sizeof(ST) == sizeof(double2)) return d.zsc;
      else return wsb<ST>(d, SB_Z32);
    default:
      if constexpr (sizeof(ST) == sizeof(double2)) return d.tsrc;
      else return wsb<ST>(d, SB_T32);
  }
}

// One block per tile (input, y, KB kx lines).  The first pass reads the
// spectral rows (lanes along kz), the last one writes its samples straight to
// the z-physical rows (lanes along kx); in between the lines cross shared
// memory once per pass.  The bound is HBM; what it takes to get near it is
// warps in flight: with its rows staged in shared memory the form with radices
// 36 and 32 had 12 on an SM at 1152 points (FP32, 131 registers and 63 KB a
// block), now it has 18.  768 x 33 with the scalar and mu, FP32: k_zinv 5.3 ms per
// step, k_zfwd 1.7; in three passes 5.5 and 2.1.
// mode 0: the transform inputs of the substep (in_field(i0) ..); mode 1 (2014
// variant, FP64): T before the substep and Delta T, for d(rho)
// (lomacte/cross.f:1760-1770); mode 2 (physical-field export, FP64): the
// export inputs, written in natural z order
template <int R1, int R2, int R3, typename CT, typename ST>
__global__ void __launch_bounds__(ZGeo<R1, R2, R3, CT>::ZI, ZGeo<R1, R2, R3, CT>::MI)
    k_zinv(Dev d, int mode, int i0) {
  using ZG = ZGeo<R1, R2, R3, CT>;
  constexpr int ZT = ZG::ZI;
  using F = Fft<R1, R2, R3, CT, ZT>;
  using Re = typename CReal<CT>::R;
  constexpr int KB = ZG::KB, LD = ZG::LD, N = F::N, SH = N / 3 + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  CT *W = (CT *)smraw;
  const CT *tw = wtwz<CT>(d);
  // the kx planes zp0 .. zp0+zkn-1 (a slab block; all planes by default),
  // written into z-physical rows of zkn values
  const int f = mode ? (int)blockIdx.z : in_field(d, i0 + (int)blockIdx.z), y = blockIdx.y;
  const int kx0 = d.zp0 + blockIdx.x * KB, nb = min(KB, d.zp0 + d.zkn - kx0);
  // i kx, i kz: of Z, T, and with the variable viscosity of rho w
  const int mult = mode ? 0 : f == vbase(d) + 2 && d.visc ? 2 : f == 9 && d.scalar ? 1 : f == 6 || (f == 11 && d.scalar) ? 2 : 0;
  const ST *src = zsrc<ST>(d, f, mode) + ((size_t)y * d.nkx + kx0) * d.mz;
  auto load = [&](int il, int n1) {
    const ST *p = src + il * d.mz + n1;
    const double *kz = d.kz + n1;
    const Re kx = mult == 1 ? (Re)__ldg(d.kx + kx0 + il) : (Re)0;
    const bool m00 = sizeof(ST) == sizeof(float2) && n1 == 0 && kx0 + il == 0;
    return [=](int o, bool up) -> CT {
      const int k = up ? o - SH : o;
      CT v = ccvt<CT>(__ldg(p + k));
      if (mult == 1) v = cik(kx, v);
      else if (mult == 2) v = cik((Re)__ldg(kz + k), v);
      if (o == 0 && m00) v = cz<CT>();  // 00 mode: added back in FP64 by xphys
      return v;
    };
  };
  F::template inv_p1<+1>(W, nb, LD, tw, load);
  if constexpr (R3 > 1) F::template inv_p2<+1>(W, nb, LD, tw);
  ST *dst = wzb<ST>(d, f) + (size_t)y * N * d.zkn + (kx0 - d.zp0);
  constexpr int RL = R3 > 1 ? R3 : R2;  // radix of the last pass
  for (int idx = threadIdx.x; idx < KB * (N / RL); idx += ZT) {
    const int il = idx % KB, q = idx / KB;
    if (il >= nb) continue;
    const CT *p = W + il * LD + (RL > 1 ? q * (RL + 1) : q);
    CT x[RL];
#pragma unroll
    for (int j = 0; j < RL; j++) x[j] = p[j];
    rdft<RL, +1>(x);
    // the samples stay in the transform's order, except for the export and
    // where the two z transforms may have different radices
    const bool nat = mode == 2 || d.fft64;
    ST *o = dst + (size_t)(nat ? F::nat(q * RL) : q * RL) * d.zkn + il;
    const int st = (nat ? F::NS : 1) * d.zkn;
#pragma unroll
    for (int j = 0; j < RL; j++) o[(size_t)j * st] = ccvt<ST>(x[j]);
  }
}

// The transpose of k_zinv, one block per tile (y, KB kx lines) and output:
// the first pass gathers its samples from the z-physical rows (R3 loads in
// flight per thread), the last one writes the retained kz of the spectral
// rows.  mode 0: the substep's outputs (field blockIdx.z in place); mode 1
// (2014 variant): d(rho) from z-physical buffer 0 into the d(rho) spectral
// slot
template <int R1, int R2, int R3, typename CT, typename ST>
__global__ void __launch_bounds__(ZGeo<R1, R2, R3, CT>::ZF, ZGeo<R1, R2, R3, CT>::MF) k_zfwd(Dev d, int mode) {
  using ZG = ZGeo<R1, R2, R3, CT>;
  constexpr int ZT = ZG::ZF;
  using F = Fft<R1, R2, R3, CT, ZT>;
  using Re = typename CReal<CT>::R;
  constexpr int KB = ZG::KB, LD = ZG::LD, N = F::N, M = F::M, SH = N / 3 + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  CT *W = (CT *)smraw;
  const CT *tw = wtwz<CT>(d);
  // the kx planes zp0 .. zp0+zkn-1, from z-physical rows of zkn values
  const int f = mode ? ODRHO : (int)blockIdx.z, y = blockIdx.y, kx0 = d.zp0 + blockIdx.x * KB;
  const int nb = min(KB, d.zp0 + d.zkn - kx0);
  const ST *src = wzb<ST>(d, mode ? 0 : f) + (size_t)y * N * d.zkn + (kx0 - d.zp0);
  constexpr int RL = R3 > 1 ? R3 : R2;  // radix of the inverse's last pass, the first one here
  for (int idx = threadIdx.x; idx < KB * (N / RL); idx += ZT) {
    const int il = idx % KB, q = idx / KB;
    if (il >= nb) continue;
    // rows as k_zinv wrote them
    const ST *r = src + (size_t)(d.fft64 ? F::nat(q * RL) : q * RL) * d.zkn + il;
    const int st = (d.fft64 ? F::NS : 1) * d.zkn;
    ST v[RL];
#pragma unroll
    for (int j = 0; j < RL; j++) v[j] = __ldg(r + (size_t)j * st);
    CT x[RL];
#pragma unroll
    for (int j = 0; j < RL; j++) x[j] = ccvt<CT>(v[j]);
    rdft<RL, -1>(x);
    CT *p = W + il * LD + (RL > 1 ? q * (RL + 1) : q);
    // twiddles: of the second pass after a third one, else of the first
    const int e = F::FW + q % F::FS;
#pragma unroll
    for (int j = 0; j < RL; j++) p[j] = (RL > 1 && j > 0) ? cmul(x[j], F::template twd<-1>(tw, e + j * F::FS)) : x[j];
  }
  __syncthreads();
  if constexpr (R3 > 1) F::template fwd_p2<-1>(W, nb, LD, tw);
  const Re dn = (Re)(1.0 / (double)N);
  ST *row = wsb<ST>(d, f) + ((size_t)y * d.nkx + kx0) * d.mz;
  line_tasks<M, ZT>(nb, [&](int il, int n1) {
    ST *o = row + il * d.mz + n1;
    F::template fwd_out<-1>(W + il * LD, n1,
                            [&](int k, bool up, CT v) { o[up ? k - SH : k] = ccvt<ST>(cscale(dn, v)); });
  });
}

__device__ __forceinline__ void atomic_max_pos(unsigned long long *a, double v) {
  atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

// The inverse x transform of one line of two real fields packed as A + iB:
// sample k of the packed spectrum from the rows' values a, c (the conjugate
// mirror in the high third; the imaginary parts of mode 0 are dropped,
// rftsingle.f:85-88)
template <typename CT>
__device__ __forceinline__ CT x_pack(CT a, CT c, int n, bool up) {
  if (up) return cmk<CT>(a.x + c.y, c.x - a.y);
  return n == 0 ? cmk<CT>(a.x, c.x) : cmk<CT>(a.x - c.y, a.y + c.x);
}

// Last pass of the direct x transforms of a tile: lines 0 .. nl-1 (ZB z lines
// each, nzb of them real) hold A + iB of the outputs ab(p, fa, fb) (fb < 0:
// none).  A thread takes the tasks n and M - n together, which hold the
// samples k and N - k of each other, and writes the retained kx of A and B.
// Radices above 12 (FP32), whose two tasks do not fit a thread's registers,
// pass the outputs through shared memory instead.
template <int R1, int R2, int R3, int T, typename CT, typename ST, typename AB>
__device__ __forceinline__ void x_out(const Dev &d, CT *sm, int nl, size_t gt, int nzb, AB &&ab) {
  using F = XFft<R1, R2, R3, CT>;
  using G = Geo<R1, R2, R3>;
  using Re = typename CReal<CT>::R;
  constexpr int N = F::N, M = F::M, Q = F::Q, ZB = G::ZB;
  const Re dn = (Re)(1.0 / (double)N), hdn = (Re)(0.5 / (double)N);
  // the retained coefficient k of A and B from the samples k and N - k
  auto emit = [&](ST *A, ST *B, int k, CT c, CT q) {
    A[k] = ccvt<ST>(cmk<CT>((c.x + q.x) * hdn, (c.y - q.y) * hdn));
    if (B) B[k] = ccvt<ST>(cmk<CT>((c.y + q.y) * hdn, (q.x - c.x) * hdn));
  };
  auto emit0 = [&](ST *A, ST *B, CT c) {
    A[0] = ccvt<ST>(cmk<CT>(c.x * dn, 0));
    if (B) B[0] = ccvt<ST>(cmk<CT>(c.y * dn, 0));
  };
  if constexpr (R1 > 12 || R1 % 3 != 0) {
    line_tasks<M, T>(nl * ZB, [&](int b, int n1) {
      if (ZB > 1 && b % ZB >= nzb) return;
      CT *line = sm + (size_t)b * G::LD + F::sk(n1);  // output n1 + o at the place of sample n1 + o
      F::template fwd_out<-1>(sm + (size_t)b * G::LD, n1, [&](int o, bool, CT v) { line[o / M * F::SM] = v; });
    });
    __syncthreads();
    line_tasks<N / 3, T>(nl * ZB, [&](int b, int k) {
      const int p = b / ZB, l = b - p * ZB;
      if (ZB > 1 && l >= nzb) return;
      int fa, fb;
      ab(p, fa, fb);
      const size_t g = gt + (size_t)l * d.nkx;
      ST *A = wzb<ST>(d, fa) + g, *B = fb >= 0 ? wzb<ST>(d, fb) + g : nullptr;
      const CT *line = sm + (size_t)b * G::LD;
      if (k == 0) emit0(A, B, line[0]);
      else emit(A, B, k, line[F::sk(k)], line[F::sk(N - k)]);
    });
  } else {
    line_tasks<(M > 1 ? M / 2 : 1), T>(nl * ZB, [&](int b, int na) {
      const int p = b / ZB, l = b - p * ZB;
      if (ZB > 1 && l >= nzb) return;
      int fa, fb;
      ab(p, fa, fb);
      const size_t g = gt + (size_t)l * d.nkx;
      ST *A = wzb<ST>(d, fa) + g, *B = fb >= 0 ? wzb<ST>(d, fb) + g : nullptr;
      const CT *line = sm + (size_t)b * G::LD;
      CT la[Q], ha[Q];
      F::template fwd_p1<-1>(line, na, la, ha);
      if (na > 0) {
        CT lb[Q], hb[Q];
        F::template fwd_p1<-1>(line, M - na, lb, hb);
#pragma unroll
        for (int j = 0; j < Q; j++) {
          emit(A, B, na + j * M, la[j], hb[Q - 1 - j]);
          emit(A, B, M - na + j * M, lb[j], ha[Q - 1 - j]);
        }
      } else {  // the two tasks that pair with themselves, 0 and M/2
        emit0(A, B, la[0]);
#pragma unroll
        for (int j = 1; j < Q; j++) emit(A, B, j * M, la[j], ha[Q - j]);
        F::template fwd_p1<-1>(line, M / 2, la, ha);
#pragma unroll
        for (int j = 0; j < Q; j++) emit(A, B, M / 2 + j * M, la[j], ha[Q - 1 - j]);
      }
    });
  }
}

// The x stage: per (y, z line), inverse x transforms of the inputs, packed two
// per complex transform,
//   (rho u, rho v) (rho w, lap T) (dT/dx, dT/dy) (dT/dz, T)
//   ZS, the passive scalar: (lap Z, dZ/dx) (dZ/dy, dZ/dz)
//   VS, the variable viscosity: the strain-rate inputs (vbase) in pairs
// the FP64 products and the T (and Z) update, and the direct transforms of
//   (u, v) (w, rho uu) (rho vv, rho ww) (rho uv, rho uw) (rho vw, drho) (DT, DZ)
// (the rounding of a packed FP32 line is that of the larger of its two fields:
// drho, which vanishes with the density contrast and is all that psi is solved
// from, shares its line with the smallest product and not with a velocity; at a
// density ratio of 1.05 psi is 1.1e-7 off beside rho vw and 1.4e-6 beside w),
// in place: every input row of a tile is read in the first pass, before any
// output row is written.  dT/dx and d(rho u)/dx are formed from the rows of T
// and rho u.  VS: T^sigma in the diffusion of T and Z, and the variable part
// of the stress taken off the products.
//
// Persistent: a block walks tiles (ZB z lines of a row y) with stride
// gridDim.x.  While a tile is transformed, its RHS rows of the previous
// substep arrive by TMA bulk copies, and the input rows of the next tile are
// brought into the L2.  What bounds it: with nine lines a tile fills 90 KB
// (FP32) or 180 KB (FP64) at 1152 points, so one or two blocks fit an SM and
// the warps that hide the latencies and the barriers between the passes have
// to come from the block: small radices in FP64, and a pointwise loop of one
// point at a time.
template <int R1, int R2, int R3, typename CT, typename ST, bool ZS, bool VS>
__global__ void __launch_bounds__(XGeo<R1, R2, R3, sizeof(CT) == sizeof(float2)>::XT,
                                  XGeo<R1, R2, R3, sizeof(CT) == sizeof(float2)>::MINB)
    k_xphys(Dev d, int rk, int do_cfl, int do_diag, int ntiles) {
  constexpr int XT = XGeo<R1, R2, R3, sizeof(CT) == sizeof(float2)>::XT;
  using F = XFft<R1, R2, R3, CT, XT>;
  using G = Geo<R1, R2, R3>;
  using Re = typename CReal<CT>::R;
  constexpr int N = F::N, ZB = G::ZB, LD = G::LD;
  constexpr int VB = ZS ? 12 : 8;  // first viscosity input
  constexpr int NI = VB + (VS ? 6 : 0), NL = NI / 2, NLM = NL > 6 ? NL : 6, NO = ZS ? 12 : 11;
  constexpr int NM = VS ? NMI : ZS ? 8 : 6;
  constexpr bool MX = sizeof(ST) == sizeof(float2);
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nkx = d.nkx;  // a multiple of 8 for every supported length
  CT *W = (CT *)smraw;                                                // NLM buffers x ZB lines x LD
  double *Sr = (double *)(smraw + round16(sizeof(CT) * NLM * ZB * LD));  // ZB*N RHS(T)
  double *Srz = Sr + ZB * N;                                          // ZB*N RHS(Z) (ZS)
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_ok;
  __shared__ unsigned long long s_tmax[ZB], s_vmax;
  __shared__ double s_red[2][XT / 32];
  __shared__ double s_min[NM], s_est[NO];  // mixed form, per tile
  const int nzk = (d.mgalz + ZB - 1) / ZB;
  // tile t of this launch is tile xt0 + t of the substep (the x stage of a
  // slab block of lines, or all of them); its z-physical rows are local to
  // the block, which starts at line xl0
  auto issue = [&](int t) {  // the RHS rows of tile t
    t += d.xt0;
    const int y = t / nzk, z0 = (t - y * nzk) * ZB, nzb = min(ZB, d.mgalz - z0);
    const uint32_t hb = d.variant ? 0u : (uint32_t)nzb * N * sizeof(double);
    mbar_expect_tx(&bar, (ZS ? 2 : 1) * hb);
    if (hb) bulk_g2s(Sr, d.rhst + ((size_t)y * d.mgalz + z0) * N, hb, &bar);
    if (ZS && hb) bulk_g2s(Srz, d.rhsz + ((size_t)y * d.mgalz + z0) * N, hb, &bar);
  };
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    s_vmax = 0ull;
  }
  for (int l = threadIdx.x; l < ZB; l += blockDim.x) s_tmax[l] = 0ull;
  __syncthreads();
  int t = blockIdx.x;
  if (threadIdx.x == 0 && t < ntiles) issue(t);
  uint32_t ph = 0;
  const double ipe = 1.0 / d.peclet, ipz = ZS ? 1.0 / d.pez : 0.0;
  const double dt = d.scal_d[0];
  const double dtxi = dt * d.xi[rk], dtg = dt * d.gama[rk], idtb = 1.0 / (dt * d.beta[rk]);
  const double ab = d.alpha[rk] / d.beta[rk];
  double mu = 0.0, mw = 0.0, cfy = 0.0, cft = 0.0;  // running maxima (cfy, cft: thread 0)
  for (; t < ntiles; t += gridDim.x) {
    const int tg = d.xt0 + t, y = tg / nzk, z0 = (tg - y * nzk) * ZB, nzb = min(ZB, d.mgalz - z0);
    if constexpr (MX) {  // the FP64 00 profiles of the inputs at this y, and the values subtracted from the
                         // outputs before they are rounded to FP32
      const int q = threadIdx.x;
      if (q < NM) s_min[q] = d.mi[(size_t)q * d.my + y];
      if (q < NO) {
        double e;
        if (d.mean_ok) {
          e = d.mo_prev[(size_t)q * d.my + y] / ((double)d.mgalx * (double)d.mgalz);
        } else {  // products of the input means
          const double ru = d.mi[y], rv = d.mi[(size_t)d.my + y], rw = d.mi[(size_t)2 * d.my + y];
          const double T = d.mi[(size_t)5 * d.my + y];
          const double u = ru * T, v = rv * T, w = rw * T;
          switch (q) {
            case OU: e = u; break;
            case OV: e = v; break;
            case OW: e = w; break;
            case ORUU: e = ru * u; break;
            case ORVV: e = rv * v; break;
            case ORWW: e = rw * w; break;
            case ORUV: e = ru * v; break;
            case ORUW: e = ru * w; break;
            case ORVW: e = rv * w; break;
            default: e = 0.0; break;
          }
        }
        s_est[q] = e;
      }
    }
    const size_t gt = ((size_t)y * d.mgalz + z0 - d.xl0) * nkx;  // the tile's rows in global memory
    auto load = [&](int b, int n1) {
      const int p = b / ZB, l = b - p * ZB;
      const bool dx = p == 2 || (VS && p == VB / 2);  // A is the x derivative of T or of rho u
      const size_t g = gt + (size_t)l * nkx;
      const ST *A = wzb<ST>(d, p == 2 ? 7 : VS && p == VB / 2 ? 0 : 2 * p) + g, *B = wzb<ST>(d, 2 * p + 1) + g;
      const bool ok = ZB == 1 || l < nzb;
      return [=, &d](int o, bool up) -> CT {
        if (!ok) return cz<CT>();
        const int k = up ? N - o - n1 : o + n1;
        CT a = ccvt<CT>(A[k]);
        const CT c = ccvt<CT>(B[k]);
        if (dx) a = cik((Re)__ldg(d.kx + k), a);
        return x_pack(a, c, o + n1, up);
      };
    };
    F::template inv_p1<+1>(W, NL * ZB, LD, wtwx<CT>(d), load);
    {  // the next tile's input rows into the L2
      const int f = threadIdx.x, tn = tg + gridDim.x;
      if (f < NI && f != 4 && !(VS && f == VB) && t + (int)gridDim.x < ntiles) {
        const int yn = tn / nzk, zn = (tn - yn * nzk) * ZB;
        bulk_prefetch_l2(wzb<ST>(d, f) + ((size_t)yn * d.mgalz + zn - d.xl0) * nkx,
                         (uint32_t)min(ZB, d.mgalz - zn) * nkx * (uint32_t)sizeof(ST));
      }
    }
    if (threadIdx.x == 0) s_ok = mbar_wait(&bar, ph, d.status);  // the RHS rows, read after the passes' barriers
    ph ^= 1;
    F::template inv_p2<+1>(W, NL * ZB, LD, wtwx<CT>(d));
    if (!s_ok) return;
    F::template inv_p3<+1>(W, NL * ZB, LD);

    double acc[12];
    if constexpr (MX) {
#pragma unroll
      for (int o = 0; o < 12; o++) acc[o] = 0.0;
    }
    double rs = 0.0, mv = 0.0;
#pragma unroll 1
    for (int q = threadIdx.x; q < nzb * N; q += XT) {
      const int l = q / N, pos = q - l * N;
      constexpr size_t LS = (size_t)ZB * LD;
      CT *c0 = W + (size_t)l * LD + F::sk(pos);
      double2 p0 = to_d2(c0[0]), p1 = to_d2(c0[LS]), p2 = to_d2(c0[2 * LS]), p3 = to_d2(c0[3 * LS]);
      if constexpr (MX) {
        p0.x += s_min[0]; p0.y += s_min[1]; p1.x += s_min[2]; p1.y += s_min[3]; p2.y += s_min[4];
        p3.y += s_min[5];
      }
      const double ru = p0.x, rv = p0.y, rw = p1.x, lapT = p1.y, tx = p2.x, ty = p2.y, tz = p3.x, T = p3.y;
      const double u = ru * T, v = rv * T, w = rw * T;                // cross.f:1613-1622
      double tn = T, d8 = 0.0;
      if (!d.variant) {
        d8 = dtxi * Sr[q];                                             // cross.f:1627
        tn = T + d8;                                                   // cross.f:1626
      }
      double tsg = 1.0;                                                // mu = k = rho D = T^sigma
      double rhs;
      if constexpr (VS) {  // branches/loma/src/cross.f:1591-1596
        tsg = exp(d.sigma * log(T));  // T > 0
        rhs = -u * tx - v * ty - w * tz + tsg * (T * lapT + d.sigma * (tx * tx + ty * ty + tz * tz)) * ipe;
      } else {
        rhs = -u * tx - v * ty - w * tz + T * lapT * ipe;              // cross.f:1632-1634
      }
      const size_t gp = ((size_t)y * d.mgalz + z0) * N + q;
      if (!d.variant) {  // the 2014 variant keeps RHS(T) spectral (lomacte/cross.f:1452-1456)
        d.rhst[gp] = rhs;
        tn = tn + dtg * rhs;                                           // cross.f:1641
        d8 = d8 + dtg * rhs;                                           // cross.f:1642
      }
      // an output pair leaves as soon as it is formed: the plane sums, the
      // estimate taken off, and the line that becomes its transform (whose
      // inputs at this point have been read)
      auto out = [&](int ln, int oa, double a, int ob, double b) {
        if constexpr (MX) {
          acc[oa] += a;
          a -= s_est[oa];
          if (ob < NO) {
            acc[ob < NO ? ob : 0] += b;
            b -= s_est[ob < NO ? ob : 0];
          }
        }
        c0[(size_t)ln * LS] = from_d2<CT>(make_double2(a, b));
      };
      double2 p4, p5, g0, g1, g2;
      if constexpr (ZS) {
        p4 = to_d2(c0[4 * LS]);
        p5 = to_d2(c0[5 * LS]);
        if constexpr (MX) {
          p4.x += s_min[6];
          p5.x += s_min[7];
        }
      }
      if constexpr (VS) {
        g0 = to_d2(c0[(VB / 2) * LS]);
        g1 = to_d2(c0[(VB / 2 + 1) * LS]);
        g2 = to_d2(c0[(VB / 2 + 2) * LS]);
        if constexpr (MX) {
          g0.y += s_min[8];
          g1.y += s_min[9];
          g2.y += s_min[10];
        }
      }
      double dz = 0.0;
      if constexpr (ZS) {  // the passive scalar, advanced as T is
        double rzs = -u * p4.y - v * p5.x - w * p5.y;
        if constexpr (VS) rzs += tsg * (T * p4.x + d.sigma * (tx * p4.y + ty * p5.x + tz * p5.y)) * ipz;
        else rzs += T * p4.x * ipz;
        dz = dtxi * Srz[q] + dtg * rzs;
        d.rhsz[gp] = rzs;
      }
      // cross.f:1670-1671: (d8 / (T tn)) / dtbeta - (alpha/beta) rhs / T^2
      double drho = rhs;
      if (!d.variant) {
        const double r = 1.0 / (T * T * tn);
        drho = r * (d8 * T * idtb - ab * rhs * tn);
      }
      double uu = ru * u, vv = rv * v, ww = rw * w, uv = ru * v, uw = ru * w, vw = rv * w;  // cross.f:1655-1666
      if constexpr (VS) {  // minus the variable part of the stress, 2 (T^sigma - 1) S_ij / Re
        const double c = d.ire * (tsg - 1.0);
        uu -= 2.0 * c * (T * g0.x + ru * tx);
        vv -= 2.0 * c * (T * g0.y + rv * ty);
        ww -= 2.0 * c * (T * g1.x + rw * tz);
        uv -= c * (T * g1.y + ru * ty + rv * tx);
        uw -= c * (T * g2.x + ru * tz + rw * tx);
        vw -= c * (T * g2.y + rv * tz + rw * ty);
      }
      out(0, OU, u, OV, v);
      out(1, OW, w, ORUU, uu);
      out(2, ORVV, vv, ORWW, ww);
      out(3, ORUV, uv, ORUW, uw);
      out(4, ORVW, vw, ODRHO, drho);
      out(5, ODT, d8, ODZ, dz);                                        // cross.f:1645-1647
      if (do_cfl) {
        mu = fmax(mu, fabs(u));
        mv = fmax(mv, fabs(v));
        mw = fmax(mw, fabs(w));
        if (!d.variant) atomic_max_pos(&s_tmax[l], fmax(T, 0.0));
      }
      if (do_diag) rs += 1.0 / T;
    }
    if (do_diag) {
      rs = warp_sum(rs);
      if ((threadIdx.x & 31) == 0) atomicAdd(d.rhom + y, rs);
    }
    if constexpr (MX) {  // FP64 partial plane sums, one slot per (tile, warp)
      const int slot = (z0 / ZB) * (XT / 32) + (threadIdx.x >> 5);
      double v[3];
      const int q0 = warp_sum12(acc, v);
      if ((threadIdx.x & 7) == 0)
#pragma unroll
        for (int i = 0; i < 3; i++)
          if (q0 + i < NO) d.mpart[((size_t)(q0 + i) * d.my + y) * d.mpart_ld + slot] = v[i];
    }
    if (do_cfl) {
      mv = warp_max(mv);
      if ((threadIdx.x & 31) == 0) atomic_max_pos(&s_vmax, mv);
    }
    __syncthreads();
    if (threadIdx.x == 0 && t + (int)gridDim.x < ntiles) {  // the RHS rows are consumed: the next tile's
      fence_proxy_async();
      issue(t + gridDim.x);
    }
    if (do_cfl && threadIdx.x == 0) {  // cross.f:1690-1708 for the lines of this tile
      const double hy = d.hy[y];
      cfy = fmax(cfy, __longlong_as_double((long long)s_vmax) / hy);
      for (int l = 0; l < nzb; l++) {
        // cross.f:1704; with the scalar the larger of the two diffusivities
        const double tm = __longlong_as_double((long long)s_tmax[l]);
        const double DD = (ZS ? fmax(ipe, ipz) : ipe) * (VS ? pow(tm, 1.0 + d.sigma) : tm);
        cft = fmax(cft, 2.0 * DD * ((d.hxalp / 2) * (d.hxalp / 2) + (d.hzbet / 2) * (d.hzbet / 2) + (1.0 / hy) * (1.0 / hy)));
        s_tmax[l] = 0ull;
      }
      s_vmax = 0ull;
    }
    const int nl = d.variant ? 5 : 6;
    F::template fwd_p3<-1>(W, nl * ZB, LD, wtwx<CT>(d));
    F::template fwd_p2<-1>(W, nl * ZB, LD, wtwx<CT>(d));
    x_out<R1, R2, R3, XT, CT, ST>(d, W, nl, gt, nzb, [](int p, int &fa, int &fb) {
      // OU .. ODT in order, two per line; the last line's second is Delta Z
      fa = 2 * p;
      fb = p < 5 || ZS ? 2 * p + 1 : -1;
    });
    __syncthreads();
  }
  if (do_cfl) {
    mu = warp_max(mu);
    mw = warp_max(mw);
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { s_red[0][wid] = mu; s_red[1][wid] = mw; }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0, c = 0;
      for (int q = 0; q < XT / 32; q++) { a = fmax(a, s_red[0][q]); c = fmax(c, s_red[1][q]); }
      atomic_max_pos(d.cflmax + 0, a);
      atomic_max_pos(d.cflmax + 1, cfy);
      atomic_max_pos(d.cflmax + 2, c);
      atomic_max_pos(d.cflmax + 3, cft);
    }
  }
}

__host__ __device__ constexpr int x_threads(int n) { return n >= 576 ? 256 : 128; }  // of the kernels below

// the three passes of nb inverse lines from rows(b, A, B) (B null: none; false:
// a padding line)
template <int R1, int R2, int R3, typename CT, typename ST, typename R>
__device__ __forceinline__ void x_inverse(const Dev &d, CT *W, int nb, R &&rows) {
  using F = XFft<R1, R2, R3, CT, x_threads(R1 * R2 * R3)>;
  constexpr int LD = Geo<R1, R2, R3>::LD;
  F::template inv_p1<+1>(W, nb, LD, wtwx<CT>(d), [&](int b, int n1) {
    const ST *A = nullptr, *B = nullptr;
    const bool ok = rows(b, A, B);
    return [=](int o, bool up) -> CT {
      if (!ok) return cz<CT>();
      const int k = up ? F::N - o - n1 : o + n1;
      return x_pack(ccvt<CT>(A[k]), B ? ccvt<CT>(B[k]) : cz<CT>(), o + n1, up);
    };
  });
  F::template inv_p2<+1>(W, nb, LD, wtwx<CT>(d));
  F::template inv_p3<+1>(W, nb, LD);
}

// Physical-field export (FP64): one block per (plane, z tile); the inverse
// x transforms of the export inputs (rows in natural z order, zinv mode 2),
// then per point u = T rho u, v, w, T, omega = T curl(rho u) + grad T x
// rho u (the quantities of tofis_loma's escrphys, trunk/tofis_loma/src/
// escru.f:101-314) and Z, written in natural x order to out[p][q][z][x]
template <int R1, int R2, int R3>
__global__ void __launch_bounds__(x_threads(R1 *R2 *R3)) k_xexport(Dev d, const int *jrow, int nplanes, int nf,
                                                                  double *out) {
  using F = XFft<R1, R2, R3, double2>;
  using G = Geo<R1, R2, R3>;
  constexpr int N = F::N, ZB = G::ZB, LD = G::LD;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2 *W = (double2 *)smraw;
  const int nkx = d.nkx, nzk = (d.mgalz + ZB - 1) / ZB, NL = (nf + 1) / 2, nq = d.scalar ? 8 : 7;
  const int p = blockIdx.x / nzk, z0 = (blockIdx.x - p * nzk) * ZB, nzb = min(ZB, d.mgalz - z0);
  if (p >= nplanes) return;
  const int y = jrow[p];
  x_inverse<R1, R2, R3, double2, double2>(d, W, NL * ZB, [&](int b, const double2 *&A, const double2 *&B) {
    const int pr = b / ZB, l = b - pr * ZB;
    const size_t g = ((size_t)y * d.mgalz + z0 + l) * nkx;
    if (l >= nzb) return false;
    A = d.zb[2 * pr] + g;
    if (2 * pr + 1 < nf) B = d.zb[2 * pr + 1] + g;
    return true;
  });
  for (int q = threadIdx.x; q < nzb * N; q += blockDim.x) {
    const int l = q / N, pos = q - l * N;
    const int x = F::nat(pos);  // natural x of the sample at pos
    const double2 *c = W + (size_t)l * LD + F::sk(pos);
    const double2 p0 = c[0], p1 = c[(size_t)ZB * LD], p2 = c[(size_t)2 * ZB * LD], p3 = c[(size_t)3 * ZB * LD];
    const double2 p4 = c[(size_t)4 * ZB * LD];
    const double ru = p0.x, rv = p0.y, rw = p1.x, T = p1.y, tx = p2.x, ty = p2.y, tz = p3.x;
    const double v[8] = {ru * T, rv * T, rw * T, T, T * p3.y + ty * rw - tz * rv, T * p4.x + tz * ru - tx * rw,
                         T * p4.y + tx * rv - ty * ru, nf > 10 ? c[(size_t)5 * ZB * LD].x : 0.0};
    double *o = out + (((size_t)p * nq) * d.mgalz + z0 + l) * d.mgalx + x;
    for (int k = 0; k < nq; k++) o[(size_t)k * d.mgalz * d.mgalx] = v[k];
  }
}

// 2014 variant: d(rho) = -Delta T / (T (T + Delta T)) at every physical
// point (tensor2, lomacte/cross.f:1819-1908): T and Delta T arrive as one
// complex line per (y, z), the result leaves in z-physical buffer 0.
template <int R1, int R2, int R3>
__global__ void __launch_bounds__(x_threads(R1 *R2 *R3)) k_xdrho(Dev d) {
  using F = XFft<R1, R2, R3, double2, x_threads(R1 * R2 * R3)>;
  using G = Geo<R1, R2, R3>;
  constexpr int N = F::N, ZB = G::ZB, LD = G::LD;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2 *W = (double2 *)smraw;
  const int y = blockIdx.y, z0 = blockIdx.x * ZB, nzb = min(ZB, d.mgalz - z0);
  const size_t gt = ((size_t)y * d.mgalz + z0) * d.nkx;
  x_inverse<R1, R2, R3, double2, double2>(d, W, ZB, [&](int l, const double2 *&A, const double2 *&B) {
    if (l >= nzb) return false;
    A = d.zb[0] + gt + (size_t)l * d.nkx;
    B = d.zb[1] + gt + (size_t)l * d.nkx;
    return true;
  });
  for (int q = threadIdx.x; q < nzb * N; q += blockDim.x) {
    const int l = q / N, pos = q - l * N;
    double2 *c = W + (size_t)l * LD + F::sk(pos);
    const double T = c->x, dT = c->y;
    *c = make_double2(-dT / (T * (T + dT)), 0.0);  // lomacte/cross.f:1881
  }
  __syncthreads();
  F::template fwd_p3<-1>(W, ZB, LD, d.twx);
  F::template fwd_p2<-1>(W, ZB, LD, d.twx);
  x_out<R1, R2, R3, x_threads(R1 * R2 * R3), double2, double2>(d, W, 1, gt, nzb, [](int, int &fa, int &fb) {
    fa = 0;
    fb = -1;
  });
}

// Statistics of the physical fields on an accumulating substep (phys2,
// cross.f:1583-1607): per y row the plane sums of u rho u, u rho v,
// u rho w, v rho v, v rho w, w rho w (u_i = rho u_i T), 1/T, T^sigma and
// T^(sigma+1).  Block (g, y) inverts rho u, rho v, rho w and T (three
// complex x transforms per z line, the same packing as k_xphys) on the z
// tiles g, g + ngrp, ... of row y before k_xphys overwrites its inputs and
// writes its partial sums to st.xpart; k_xsum adds the ngrp partials of a
// row in order, so the sums are reproducible.
template <int R1, int R2, int R3, typename CT, typename ST>
__global__ void __launch_bounds__(x_threads(R1 *R2 *R3)) k_xstats(Dev d, Stats st, int ngrp) {
  using F = XFft<R1, R2, R3, CT>;
  using G = Geo<R1, R2, R3>;
  constexpr int N = F::N, ZB = G::ZB, LD = G::LD, NW = x_threads(N) / 32;
  extern __shared__ __align__(16) unsigned char smraw[];
  CT *W = (CT *)smraw;  // 3 groups x ZB lines x LD
  __shared__ double sh[NW * 9];
  const int y = blockIdx.y, grp = blockIdx.x, nkx = d.nkx, my = d.my;
  double m0 = 0.0, m1 = 0.0, m2 = 0.0, m5 = 0.0;  // mixed form: FP64 00 profiles
  if constexpr (sizeof(ST) == sizeof(float2)) {
    m0 = d.mi[y];
    m1 = d.mi[(size_t)my + y];
    m2 = d.mi[(size_t)2 * my + y];
    m5 = d.mi[(size_t)5 * my + y];
  }
  const double sg = st.sigma, sg1 = st.sigma + 1.0;
  double a[9];
#pragma unroll
  for (int q = 0; q < 9; q++) a[q] = 0.0;
  for (int z0 = grp * ZB; z0 < d.mgalz; z0 += ngrp * ZB) {
    const int nzb = min(ZB, d.mgalz - z0);
    x_inverse<R1, R2, R3, CT, ST>(d, W, 3 * ZB, [&](int b, const ST *&A, const ST *&B) {
      const int gp = b / ZB, l = b - gp * ZB, p = gp < 2 ? gp : 3;  // line pairs (rho u, rho v), (rho w, -), (-, T)
      if (l >= nzb) return false;
      const size_t g0 = ((size_t)y * d.mgalz + z0 + l) * nkx;
      A = wzb<ST>(d, 2 * p) + g0;
      B = wzb<ST>(d, 2 * p + 1) + g0;
      return true;
    });
    for (int q = threadIdx.x; q < nzb * N; q += blockDim.x) {
      const int l = q / N, pos = q - l * N;
      const CT *c0 = W + (size_t)l * LD + F::sk(pos);
      const double2 p0 = to_d2(c0[0]), p1 = to_d2(c0[(size_t)ZB * LD]), p3 = to_d2(c0[(size_t)2 * ZB * LD]);
      const double ru = p0.x + m0, rv = p0.y + m1, rw = p1.x + m2, T = p3.y + m5;
      const double u = ru * T, v = rv * T, w = rw * T;
      a[0] += u * ru;
      a[1] += u * rv;
      a[2] += u * rw;
      a[3] += v * rv;
      a[4] += v * rw;
      a[5] += w * rw;
      a[6] += 1.0 / T;
      a[7] += pow(T, sg);
      a[8] += pow(T, sg1);
    }
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const double v = warp_sum(a[q]);
    if (lane == 0) sh[wid * 9 + q] = v;
  }
  __syncthreads();
  if (threadIdx.x < 9) {
    const int q = threadIdx.x;
    double s = 0.0;
    for (int w = 0; w < NW; w++) s += sh[w * 9 + q];
    st.xpart[((size_t)q * my + y) * ngrp + grp] = s;
  }
}

// the partial sums of k_xstats, group by group, into the profiles
template <int R1, int R2, int R3>
__global__ void k_xsum(Dev d, Stats st, int ngrp) {
  const int y = blockIdx.x, q = threadIdx.x;
  if (q >= 9) return;
  const double *src = st.xpart + ((size_t)q * d.my + y) * ngrp;
  double s = 0.0;
  for (int g = 0; g < ngrp; g++) s += src[g];
  const int dst = q < 7 ? ST_RUU + q : ST_MUM + (q - 7);  // ruu..rww, rhom, mum, num
  st.prof[(size_t)dst * d.my + y] += s;
}

// Plane sums of the mixed form's outputs from the partial sums of k_xphys,
// added in a fixed order so that a run is reproducible bit for bit.
template <int R1, int R2, int R3>
__global__ void __launch_bounds__(128) k_msum(Dev d, int nslot) {
  __shared__ double red[128];
  const int y = blockIdx.x, q = blockIdx.y;
  const double *src = d.mpart + ((size_t)q * d.my + y) * d.mpart_ld;
  double s = 0.0;
  for (int i = threadIdx.x; i < nslot; i += blockDim.x) s += src[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int h = 64; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) d.mo_cur[(size_t)q * d.my + y] = red[0];
}

template <int R1, int R2, int R3, typename CT, typename ST>
struct Launch {
  using G = Geo<R1, R2, R3>;
  using ZG = ZGeo<R1, R2, R3, CT>;
  static constexpr int XE = x_threads(G::N);
  static size_t zsm() { return (size_t)ZG::KB * ZG::LD * sizeof(CT); }
  static constexpr int nin(bool zs, bool vs) { return (zs ? 12 : 8) + (vs ? 6 : 0); }
  static size_t xphys_sm(bool zs, bool vs) {
    const int nl = nin(zs, vs) / 2 > 6 ? nin(zs, vs) / 2 : 6;
    return round16(sizeof(CT) * nl * G::ZB * G::LD) + (size_t)(zs ? 2 : 1) * G::ZB * G::N * sizeof(double);
  }
  // resident blocks per SM x SMs, for the persistent kernels
  static int grid_for(const void *fn, int threads, size_t smem, int ntiles) {
    int dev = 0, sms = 148, per = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem);
    if (per < 1) per = 1;
    const int g = sms * per;
    return g < ntiles ? g : ntiles;
  }
  static void zinv(const Dev &d, int mode, int i0, int n, cudaStream_t s) {
    if (n <= 0) {
      i0 = 0;
      n = mode == 1 ? 2 : n_zin(d);
    }
    const dim3 g((d.zkn + ZG::KB - 1) / ZG::KB, d.my, n);
    k_zinv<R1, R2, R3, CT, ST><<<g, ZG::ZI, zsm(), s>>>(d, mode, i0);
  }
  static void zfwd(const Dev &d, int mode, cudaStream_t s) {
    const dim3 g((d.zkn + ZG::KB - 1) / ZG::KB, d.my, mode ? 1 : (d.variant ? 10 : n_out(d)));
    k_zfwd<R1, R2, R3, CT, ST><<<g, ZG::ZF, zsm(), s>>>(d, mode);
  }
  static size_t xexport_sm() { return (size_t)6 * G::ZB * G::LD * sizeof(double2); }
  static void xexport(const Dev &d, const int *jrow, int nplanes, int nf, double *out, cudaStream_t s) {
    if constexpr (sizeof(CT) == sizeof(double2) && sizeof(ST) == sizeof(double2)) {
      const int nzk = (d.mgalz + G::ZB - 1) / G::ZB;
      k_xexport<R1, R2, R3><<<nplanes * nzk, XE, xexport_sm(), s>>>(d, jrow, nplanes, nf, out);
    }
  }
  static void xdrho(const Dev &d, cudaStream_t s) {
    if constexpr (sizeof(CT) == sizeof(double2) && sizeof(ST) == sizeof(double2)) {
      dim3 g((d.mgalz + G::ZB - 1) / G::ZB, d.my);
      k_xdrho<R1, R2, R3><<<g, XE, (size_t)G::ZB * G::LD * sizeof(double2), s>>>(d);
    }
  }
  template <bool ZS, bool VS>
  static void xphys_zs(const Dev &d, int rk, int do_cfl, int do_diag, cudaStream_t s) {
    const int ntiles = d.xnt > 0 ? d.xnt : d.my * ((d.mgalz + G::ZB - 1) / G::ZB);
    constexpr int XT = XGeo<R1, R2, R3, sizeof(CT) == sizeof(float2)>::XT;
    const void *fn = (const void *)k_xphys<R1, R2, R3, CT, ST, ZS, VS>;
    const size_t sm = xphys_sm(ZS, VS);
    const int g = grid_for(fn, XT, sm, ntiles);
    k_xphys<R1, R2, R3, CT, ST, ZS, VS><<<g, XT, sm, s>>>(d, rk, do_cfl, do_diag, ntiles);
    if (sizeof(ST) == sizeof(float2) && d.msum) {
      const int nslot = ((d.mgalz + G::ZB - 1) / G::ZB) * (XT / 32);
      k_msum<R1, R2, R3><<<dim3(d.my, n_out(d)), 128, 0, s>>>(d, nslot);
    }
  }
  static void xphys(const Dev &d, int rk, int do_cfl, int do_diag, cudaStream_t s) {
    if (d.visc) {
      if (d.scalar) xphys_zs<true, true>(d, rk, do_cfl, do_diag, s);
      else xphys_zs<false, true>(d, rk, do_cfl, do_diag, s);
    } else {
      if (d.scalar) xphys_zs<true, false>(d, rk, do_cfl, do_diag, s);
      else xphys_zs<false, false>(d, rk, do_cfl, do_diag, s);
    }
  }
  static size_t xstats_sm() { return (size_t)3 * G::ZB * G::LD * sizeof(CT); }
  static void xstats(const Dev &d, const Stats &st, cudaStream_t s) {
    const int ntile = (d.mgalz + G::ZB - 1) / G::ZB, ngrp = ntile < XGRP ? ntile : XGRP;
    k_xstats<R1, R2, R3, CT, ST><<<dim3(ngrp, d.my), XE, xstats_sm(), s>>>(d, st, ngrp);
    k_xsum<R1, R2, R3><<<d.my, 32, 0, s>>>(d, st, ngrp);
  }
  static cudaError_t optin1(const void *fn, int limit) {
    cudaError_t e;
    cudaFuncAttributes fa;
    if ((e = cudaFuncGetAttributes(&fa, fn)) != cudaSuccess) return e;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limit - (int)fa.sharedSizeBytes);
  }
  static cudaError_t optin(int limit) {
    cudaError_t e;
    if ((e = optin1((const void *)k_zinv<R1, R2, R3, CT, ST>, limit)) != cudaSuccess) return e;
    if ((e = optin1((const void *)k_zfwd<R1, R2, R3, CT, ST>, limit)) != cudaSuccess) return e;
    if constexpr (R2 > 1) {  // x lengths
      if ((e = optin1((const void *)k_xstats<R1, R2, R3, CT, ST>, limit)) != cudaSuccess) return e;
      if constexpr (sizeof(CT) == sizeof(double2) && sizeof(ST) == sizeof(double2)) {
        if ((e = optin1((const void *)k_xexport<R1, R2, R3>, limit)) != cudaSuccess) return e;
        if ((e = optin1((const void *)k_xdrho<R1, R2, R3>, limit)) != cudaSuccess) return e;
      }
      if ((e = optin1((const void *)k_xphys<R1, R2, R3, CT, ST, true, true>, limit)) != cudaSuccess) return e;
      if ((e = optin1((const void *)k_xphys<R1, R2, R3, CT, ST, false, true>, limit)) != cudaSuccess) return e;
      if ((e = optin1((const void *)k_xphys<R1, R2, R3, CT, ST, true, false>, limit)) != cudaSuccess) return e;
      return optin1((const void *)k_xphys<R1, R2, R3, CT, ST, false, false>, limit);
    }
    return cudaSuccess;
  }
};

// FP32 butterflies have radices of their own
template <int N>
using LaunchF32 = Launch<fft_radix(N, true).r1, fft_radix(N, true).r2, fft_radix(N, true).r3, float2, float2>;

// register-DFT twiddles exp(-2 pi i e / R) of every block size
inline cudaError_t upload_twiddles() {
  std::vector<double2> t;
  std::vector<float2> tf;
  for (int R : TW_SIZES)
    for (int e = 0; e < R; e++) {
      const long double a = 2.0L * 3.14159265358979323846264338327950288L * (long double)e / (long double)R;
      t.push_back(make_double2((double)cosl(a), (double)(-sinl(a))));
      tf.push_back(make_float2((float)cosl(a), (float)(-sinl(a))));
    }
  cudaError_t e = cudaMemcpyToSymbol(c_tw, t.data(), t.size() * sizeof(double2));
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_twf, tf.data(), tf.size() * sizeof(float2));
}

}  // namespace LMC_FFT_NS
}  // namespace lmc

// Each translation unit defines LMC_FFT_SIZES(X) as X(N, R1, R2, R3) entries and
// then expands LMC_FFT_TU_BODY(suffix) to get its dispatch functions.
#define LMC_FFT_FORMS(R1, R2, R3, CALL)                                   \
  switch (d.prec) {                                                   \
    case 1: LaunchF32<R1 * R2 * R3>::CALL; break;                         \
    case 2: Launch<R1, R2, R3, double2, float2>::CALL; break;             \
    default: Launch<R1, R2, R3, double2, double2>::CALL; break;           \
  }
// precision 1 with bit BIT of d.fft64 set: FP64 butterflies for this stage
#define LMC_FFT_FORMS_M(R1, R2, R3, BIT, CALL)                                \
  switch (d.prec) {                                                       \
    case 1:                                                               \
      if (d.fft64 & (BIT)) Launch<R1, R2, R3, double2, float2>::CALL;         \
      else LaunchF32<R1 * R2 * R3>::CALL;                                     \
      break;                                                              \
    case 2: Launch<R1, R2, R3, double2, float2>::CALL; break;                 \
    default: Launch<R1, R2, R3, double2, double2>::CALL; break;               \
  }
#define LMC_FFT_CASE_Z(N, R1, R2, R3, WHAT) \
  case N: LMC_FFT_FORMS_M(R1, R2, R3, 4, WHAT(d, mode, s)) return true;
#define LMC_FFT_CASE_XD(N, R1, R2, R3) \
  case N: Launch<R1, R2, R3, double2, double2>::xdrho(d, s); return true;
#define LMC_FFT_CASE_X(N, R1, R2, R3) \
  case N: LMC_FFT_FORMS_M(R1, R2, R3, 2, xphys(d, rk, do_cfl, do_diag, s)) return true;
#define LMC_FFT_CASE_XE(N, R1, R2, R3) \
  case N: Launch<R1, R2, R3, double2, double2>::xexport(d, jrow, nplanes, nf, out, s); return true;
#define LMC_FFT_CASE_XST(N, R1, R2, R3) \
  case N: LMC_FFT_FORMS(R1, R2, R3, xstats(d, st, s)) return true;
#define LMC_FFT_CASE_ZI(N, R1, R2, R3) \
  case N: LMC_FFT_FORMS_M(R1, R2, R3, 1, zinv(d, mode, i0, n, s)) return true;
#define LMC_FFT_CASE_ZF(N, R1, R2, R3) LMC_FFT_CASE_Z(N, R1, R2, R3, zfwd)
#define LMC_FFT_CASE_ZS(N, R1, R2, R3) case N: return Launch<R1, R2, R3, double2, double2>::zsm();
#define LMC_FFT_CASE_XS(N, R1, R2, R3) case N: return Launch<R1, R2, R3, double2, double2>::xphys_sm(zs, vs);
#define LMC_FFT_CASE_OPT(N, R1, R2, R3)                                                         \
  if ((e = Launch<R1, R2, R3, double2, double2>::optin(limit)) != cudaSuccess) return e;        \
  if ((e = LaunchF32<N>::optin(limit)) != cudaSuccess) return e;                                \
  if ((e = Launch<R1, R2, R3, double2, float2>::optin(limit)) != cudaSuccess) return e;
#define LMC_FFT_CASE_HAS(N, R1, R2, R3) case N: return true;

#define LMC_FFT_TU_BODY(SUF)                                                                      \
  namespace lmc {                                                                                 \
  using namespace LMC_FFT_NS;                                                                     \
  bool fft_has_##SUF(int n) {                                                                     \
    switch (n) { LMC_FFT_SIZES(LMC_FFT_CASE_HAS) default: return false; }                         \
  }                                                                                               \
  bool fft_zinv_##SUF(const Dev &d, int mode, int i0, int n, cudaStream_t s) {                   \
    switch (d.mgalz) { LMC_FFT_SIZES(LMC_FFT_CASE_ZI) default: return false; }                     \
  }                                                                                               \
  bool fft_zfwd_##SUF(const Dev &d, int mode, cudaStream_t s) {                                   \
    switch (d.mgalz) { LMC_FFT_SIZES(LMC_FFT_CASE_ZF) default: return false; }                     \
  }                                                                                               \
  bool fft_xdrho_##SUF(const Dev &d, cudaStream_t s) {                                            \
    switch (d.mgalx) { LMC_FFT_SIZES(LMC_FFT_CASE_XD) default: return false; }                     \
  }                                                                                               \
  bool fft_xphys_##SUF(const Dev &d, int rk, int do_cfl, int do_diag, cudaStream_t s) {           \
    switch (d.mgalx) { LMC_FFT_SIZES(LMC_FFT_CASE_X) default: return false; }                      \
  }                                                                                               \
  bool fft_xexport_##SUF(const Dev &d, const int *jrow, int nplanes, int nf, double *out, cudaStream_t s) { \
    switch (d.mgalx) { LMC_FFT_SIZES(LMC_FFT_CASE_XE) default: return false; }                     \
  }                                                                                               \
  bool fft_xstats_##SUF(const Dev &d, const Stats &st, cudaStream_t s) {                          \
    switch (d.mgalx) { LMC_FFT_SIZES(LMC_FFT_CASE_XST) default: return false; }                    \
  }                                                                                               \
  size_t fft_zsm_##SUF(int n) {                                                                   \
    switch (n) { LMC_FFT_SIZES(LMC_FFT_CASE_ZS) default: return 0; }                             \
  }                                                                                               \
  size_t fft_xsm_##SUF(int n, bool zs, bool vs) {                                                \
    switch (n) { LMC_FFT_SIZES(LMC_FFT_CASE_XS) default: return 0; }                              \
  }                                                                                               \
  cudaError_t fft_init_##SUF(int limit) {                                                         \
    cudaError_t e = upload_twiddles();                                                            \
    if (e != cudaSuccess) return e;                                                               \
    LMC_FFT_SIZES(LMC_FFT_CASE_OPT)                                                               \
    return cudaSuccess;                                                                           \
  }                                                                                               \
  }
