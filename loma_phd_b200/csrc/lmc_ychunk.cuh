// lmc_ychunk.cuh -- y kernels of one lomacte RK3 substep on pencils held in
// registers.
//
// A pencil of my points is split into NC chunks of C consecutive rows and a
// block holds MB consecutive modes, one thread per (mode, chunk).  In the
// spectral layout [y][kx][kz] the value of mode m at row j sits at
// f[j*nmode + m], so every load and store of a row moves runs of MB
// consecutive modes, straight between global memory and the registers of
// the thread that owns the rows: each field is read once and written once,
// and no intermediate pencil goes through memory.  (Two sweeps along y with
// one thread per mode, as before, spill the pencil between the forward and
// the backward half of every banded solve to an FP64 scratch field: 1.5 to
// 2.5 times the bytes a kernel cannot do without, and too few threads on
// small grids.)
//
// A banded solve A x = b with A = L U (the LU of cfdiff.f / laps.f in row
// form) runs per direction as: every chunk solves its rows with a zero
// incoming state (the particular response p), the chunks are joined by a
// scan of the affine chunk maps S_out = M S_in + p, and every row adds its
// precomputed response H to the incoming state.  The scan is two-level:
// four lanes per pencil walk a quarter of the chunks each, join their ends
// by shuffles, and every chunk adds Q S_group itself.  For the operators
// that do not depend on the mode the tables M, Q, H come from the host
// (build_chunk_tables) and are copied to shared memory where they fit (go);
// for the per-mode Poisson LUs they are formed by two
// real recurrences beside the particular one.
// Rows past my (the last chunk's padding) have zero coefficients.
//
// Kernels follow the statements of trunk/lomacte3/src/cross.f:307-1141.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "lmc_async.cuh"
#include "lmc_ylaunch.h"

namespace lmc {
namespace ych {

using namespace lmcd;

constexpr int YC_TMAX = 512;  // threads of a block at most (128 registers each)

template <typename CT>
__host__ __device__ constexpr bool mixed() { return sizeof(CT) == sizeof(float2); }

template <int C, int MB>
struct Th {
  int ml, c, nc, j0, n, m;  // mode lane, chunk, chunks, first row, rows, mode (clamped)
  bool act;                 // the mode exists
  double kx, kz, k2;
  size_t ld;
  __device__ __forceinline__ Th(const Dev &d, int blk) {
    ml = threadIdx.x % MB;
    c = threadIdx.x / MB;
    nc = blockDim.x / MB;
    j0 = c * C;
    n = min(C, d.my - j0);
    const int mm = blk * MB + ml;
    act = mm < d.nmode;
    m = act ? mm : d.nmode - 1;
    ld = (size_t)d.nmode;
    const int i = m / d.mz, k = m - i * d.mz;
    kx = __ldg(d.kx + i);
    kz = __ldg(d.kz + k);
    k2 = __ldg(d.k2 + m);
  }
};

// shared memory for F pencils worked at once (slots 0 .. F-1): edge rows of
// a pencil per thread, states of the scans (chunk-major, mode fastest), the
// groups' incoming states, and the Poisson solves' chunk maps
template <int MB>
struct Sm {
  double2 *E;  // [F][nc][6][MB]
  double2 *P;  // [F][nc][3][MB]
  double2 *G;  // [F][4][3][MB]
  double *Q;   // [nc][4][MB]
  const double *tb, *gb;  // the tables of d/dy and d2/dy2: where they are read, and in global memory
  bool two;               // d2/dy2's as well
  // TAB: the kernel uses those of d/dy (1), of both (2) or none
  template <int TAB>
  __device__ __forceinline__ void init(const Dev &d, int nc, int F, bool poisson, unsigned char *raw) {
    E = (double2 *)raw;
    P = E + F * nc * 6 * MB;
    G = P + F * nc * 3 * MB;
    Q = (double *)(G + F * 12 * MB);
    tb = gb = d.ct.fw1;
    two = TAB > 1;
    if (TAB > 0 && d.ct.sm) {  // on their way while the first rows are read
      double *t = (double *)(raw + bytes(nc, F, poisson));
      for (int i = 2 * threadIdx.x; i < d.ct.n1; i += 2 * blockDim.x) cp16(t + i, gb + i);
      cp_commit();
      if (TAB > 1)  // a group of its own
        for (int i = d.ct.n1 + 2 * threadIdx.x; i < d.ct.n1 + d.ct.n2; i += 2 * blockDim.x) cp16(t + i, gb + i);
      cp_commit();
      tb = t;
    }
  }
  // before the first use of the tables of d/dy, and of d2/dy2
  __device__ __forceinline__ void tables1() const {
    if (tb != gb) {
      cp_wait<1>();
      __syncthreads();
    }
  }
  __device__ __forceinline__ void tables2() const {
    if (two && tb != gb) {
      cp_wait<0>();
      __syncthreads();
    }
  }
  __device__ __forceinline__ const double *t(const double *p) const { return tb + (p - gb); }
  __device__ __forceinline__ const double *t2(const double *p) const { return two ? t(p) : p; }
  template <int B>  // of the tables of d/dy (B = 3) or of d2/dy2 (2)
  __device__ __forceinline__ double ld1(const double *p) const {
    return B == 3 || two ? *p : __ldg(p);
  }
  __device__ __forceinline__ double2 ld2(const double *p) const {
    return two ? *(const double2 *)p : __ldg((const double2 *)p);
  }
  __host__ __device__ static size_t bytes(int nc, int F, bool poisson) {
    return sizeof(double2) * ((size_t)F * nc * 9 * MB + F * 12 * MB) + (poisson ? sizeof(double) * nc * 4 * MB : 0);
  }
};

__device__ __forceinline__ double2 fms2(double2 s, double k, double2 v) {
  return make_double2(fma(-k, v.x, s.x), fma(-k, v.y, s.y));
}
__device__ __forceinline__ double2 fma2(double2 s, double k, double2 v) {
  return make_double2(fma(k, v.x, s.x), fma(k, v.y, s.y));
}
__device__ __forceinline__ double2 ld2(const double *p) { return *(const double2 *)p; }
__device__ __forceinline__ double2 ldg2(const double *p) { return __ldg((const double2 *)p); }

// the thread's rows of a field, and the same with three more rows on either
// side (zeros outside the pencil)
template <int C, int MB, typename PT>
__device__ __forceinline__ void rows(const Th<C, MB> &T, const PT *f, double2 (&u)[C]) {
  const PT *p = f + (size_t)T.j0 * T.ld + T.m;
#pragma unroll
  for (int t = 0; t < C; t++) u[t] = t < T.n ? to_d2(__ldcg(p + (size_t)t * T.ld)) : czero();
}
template <int C, int MB, typename PT>
__device__ __forceinline__ void rows_h(const Dev &d, const Th<C, MB> &T, const PT *f, double2 (&u)[C + 6]) {
#pragma unroll
  for (int t = 0; t < C + 6; t++) {
    const int j = T.j0 + t - 3;
    u[t] = (j >= 0 && j < d.my) ? to_d2(__ldcg(f + (size_t)j * T.ld + T.m)) : czero();
  }
}
template <int C, int MB, typename PT>
__device__ __forceinline__ void store(const Th<C, MB> &T, PT *f, const double2 (&u)[C]) {
  if (!T.act) return;
  PT *p = f + (size_t)T.j0 * T.ld + T.m;
#pragma unroll
  for (int t = 0; t < C; t++)
    if (t < T.n) p[(size_t)t * T.ld] = from_d2<PT>(u[t]);
}

// edge rows of a pencil held in registers, to and from the neighbouring
// chunks (a barrier between the two)
template <int C, int MB>
__device__ __forceinline__ void put_edges(const Th<C, MB> &T, const Sm<MB> &S, int slot, const double2 (&x)[C]) {
  double2 *e = S.E + ((size_t)slot * T.nc + T.c) * 6 * MB + T.ml;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    e[q * MB] = x[q];
    e[(3 + q) * MB] = x[C - 3 + q];
  }
}
template <int C, int MB>
__device__ __forceinline__ void with_halo(const Th<C, MB> &T, const Sm<MB> &S, int slot, const double2 (&x)[C],
                                          double2 (&u)[C + 6]) {
  const double2 *e = S.E + ((size_t)slot * T.nc + T.c) * 6 * MB + T.ml;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    u[q] = T.c > 0 ? e[(3 + q) * MB - 6 * MB] : czero();
    u[C + 3 + q] = T.c + 1 < T.nc ? e[q * MB + 6 * MB] : czero();
  }
#pragma unroll
  for (int t = 0; t < C; t++) u[t + 3] = x[t];
}

// ---------------------------------------------------------------------
// The scan of one warp's worth of pencils (eight modes, four lanes each).
// P holds every chunk's particular response on entry and, on return, the
// state that enters the chunk when its group starts from zero; G the states
// that enter the groups.  Chunks are visited from the last one if UP.
// ---------------------------------------------------------------------
template <int B>
__device__ __forceinline__ void shfl_state(double2 (&t)[B], const double2 (&s)[B], int src) {
#pragma unroll
  for (int q = 0; q < B; q++)
    t[q] = make_double2(__shfl_sync(LMC_FULL, s[q].x, src), __shfl_sync(LMC_FULL, s[q].y, src));
}
template <int B, int MB, bool UP>
__device__ __forceinline__ void scan_unit(int sub, int nc, const Sm<MB> &S, double2 *P, double2 *G, const double *__restrict__ M,
                                          const double *__restrict__ GM) {
  const int lane = threadIdx.x & 31, g = lane & 3, ml = sub * 8 + (lane >> 2);
  const int gl = (nc + 3) >> 2, i0 = g * gl, i1 = min(nc, i0 + gl);
  double2 s[B], e[B];
#pragma unroll
  for (int q = 0; q < B; q++) s[q] = e[q] = czero();
  for (int i = i0; i < i1; i++) {
    double2 *p = P + (size_t)(UP ? nc - 1 - i : i) * 3 * MB + ml;
    const double *mt = M + i * B * B;
    double2 n[B];
#pragma unroll
    for (int q = 0; q < B; q++) {
      n[q] = p[q * MB];
      p[q * MB] = s[q];
    }
#pragma unroll
    for (int r = 0; r < B; r++)
#pragma unroll
      for (int q = 0; q < B; q++) n[r] = fma2(n[r], S.template ld1<B>(mt + r * B + q), s[q]);
#pragma unroll
    for (int q = 0; q < B; q++) s[q] = n[q];
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double2 t[B];
    shfl_state(t, s, (lane & ~3) + k);
    if (k < g) {
#pragma unroll
      for (int r = 0; r < B; r++)
#pragma unroll
        for (int q = 0; q < B; q++) t[r] = fma2(t[r], S.template ld1<B>(GM + (k * B + r) * B + q), e[q]);
#pragma unroll
      for (int q = 0; q < B; q++) e[q] = t[q];
    }
  }
#pragma unroll
  for (int q = 0; q < B; q++) G[(g * 3 + q) * MB + ml] = e[q];
}
// the same for the Poisson solves, whose chunk maps (2 x 2, Sm::Q) depend
// on the mode; Q holds the maps from the group's start on return
template <int MB, bool UP>
__device__ __forceinline__ void scan_unit_p(int sub, int nc, const Sm<MB> &S) {
  const int lane = threadIdx.x & 31, g = lane & 3, ml = sub * 8 + (lane >> 2);
  const int gl = (nc + 3) >> 2, i0 = g * gl, i1 = min(nc, i0 + gl);
  double2 s[2] = {czero(), czero()}, e[2] = {czero(), czero()};
  double a = 1.0, b = 0.0, c = 0.0, f = 1.0;  // the map from the group's start
  for (int i = i0; i < i1; i++) {
    const int ch = UP ? nc - 1 - i : i;
    double2 *p = S.P + (size_t)ch * 3 * MB + ml;
    double *mt = S.Q + (size_t)ch * 4 * MB + ml;
    const double m0 = mt[0], m1 = mt[MB], m2 = mt[2 * MB], m3 = mt[3 * MB];
    mt[0] = a;
    mt[MB] = b;
    mt[2 * MB] = c;
    mt[3 * MB] = f;
    const double na = fma(m0, a, m1 * c), nb = fma(m0, b, m1 * f);
    c = fma(m2, a, m3 * c);
    f = fma(m2, b, m3 * f);
    a = na;
    b = nb;
    const double2 p0 = p[0], p1 = p[MB];
    p[0] = s[0];
    p[MB] = s[1];
    const double2 n0 = fma2(fma2(p0, m0, s[0]), m1, s[1]);
    s[1] = fma2(fma2(p1, m2, s[0]), m3, s[1]);
    s[0] = n0;
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int src = (lane & ~3) + k;
    double2 t[2];
    shfl_state(t, s, src);
    const double ta = __shfl_sync(LMC_FULL, a, src), tb = __shfl_sync(LMC_FULL, b, src);
    const double tc = __shfl_sync(LMC_FULL, c, src), tf = __shfl_sync(LMC_FULL, f, src);
    if (k < g) {
      const double2 n0 = fma2(fma2(t[0], ta, e[0]), tb, e[1]);
      e[1] = fma2(fma2(t[1], tc, e[0]), tf, e[1]);
      e[0] = n0;
    }
  }
  S.G[(g * 3) * MB + ml] = e[0];
  S.G[(g * 3 + 1) * MB + ml] = e[1];
}

// the scans of slots 0 .. F1-1 (d/dy) and F1 .. F1+F2-1 (d2/dy2), or of one
// Poisson solve, each on its own warps (a block has one at least, y_geometry);
// between barriers
template <int MB, int F1, int F2, bool UP>
__device__ __forceinline__ void scans(const Dev &d, int nc, const Sm<MB> &S) {
  constexpr int SUB = MB / 8;
  const YChunk &q = d.ct;
  __syncthreads();
  const int nw = blockDim.x >> 5, w = threadIdx.x >> 5;
  if (w < nw)  // whole warps only
    for (int u = w; u < (F1 + F2) * SUB; u += nw) {
      const int f = u / SUB, sub = u - f * SUB;
      double2 *P = S.P + (size_t)f * nc * 3 * MB, *G = S.G + f * 12 * MB;
      if (f < F1) scan_unit<3, MB, UP>(sub, nc, S, P, G, S.t(UP ? q.m1U : q.m1L), S.t(UP ? q.g1U : q.g1L));
      else scan_unit<2, MB, UP>(sub, nc, S, P, G, S.t2(UP ? q.m2U : q.m2L), S.t2(UP ? q.g2U : q.g2L));
    }
  __syncthreads();
}
template <int MB, bool UP>
__device__ __forceinline__ void scans_p(int nc, const Sm<MB> &S) {
  __syncthreads();
  const int nw = blockDim.x >> 5, w = threadIdx.x >> 5;
  if (w < nw)
    for (int u = w; u < MB / 8; u += nw) scan_unit_p<MB, UP>(u, nc, S);
  __syncthreads();
}

template <int B, int C, int MB>
__device__ __forceinline__ void put_state(const Th<C, MB> &T, const Sm<MB> &S, int slot, const double2 (&s)[B]) {
  double2 *p = S.P + ((size_t)slot * T.nc + T.c) * 3 * MB + T.ml;
#pragma unroll
  for (int q = 0; q < B; q++) p[q * MB] = s[q];
}
// state entering the thread's chunk
template <int B, bool UP, int C, int MB>
__device__ __forceinline__ void get_state(const Th<C, MB> &T, const Sm<MB> &S, int slot, const double *__restrict__ Q,
                                          double2 (&s)[B]) {
  const double2 *p = S.P + ((size_t)slot * T.nc + T.c) * 3 * MB + T.ml;
  const int i = UP ? T.nc - 1 - T.c : T.c, g = i / ((T.nc + 3) >> 2);
  const double2 *e = S.G + (slot * 12 + g * 3) * MB + T.ml;
#pragma unroll
  for (int r = 0; r < B; r++) {
    double2 v = p[r * MB];
#pragma unroll
    for (int q = 0; q < B; q++) v = fma2(v, S.template ld1<B>(Q + (i * B + r) * B + q), e[q * MB]);
    s[r] = v;
  }
}
template <bool UP, int C, int MB>
__device__ __forceinline__ void get_state_p(const Th<C, MB> &T, const Sm<MB> &S, double2 (&s)[2]) {
  const double2 *p = S.P + (size_t)T.c * 3 * MB + T.ml;
  const double *q = S.Q + (size_t)T.c * 4 * MB + T.ml;
  const int i = UP ? T.nc - 1 - T.c : T.c, g = i / ((T.nc + 3) >> 2);
  const double2 e0 = S.G[g * 3 * MB + T.ml], e1 = S.G[(g * 3 + 1) * MB + T.ml];
  s[0] = fma2(fma2(p[0], q[0], e0), q[MB], e1);
  s[1] = fma2(fma2(p[MB], q[2 * MB], e0), q[3 * MB], e1);
}

// ---------------------------------------------------------------------
// Compact first derivative (deryr2, cfdiff.f:518-601): x = fmap U^-1 L^-1
// dt12 u.  d1_fwd takes the pencil with its halo rows; then scans (L),
// d1_bwd, scans (U), d1_end.
// ---------------------------------------------------------------------
template <int C, int MB>
__device__ __forceinline__ void d1_fwd(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, int slot,
                                       const double2 (&u)[C + 6], double2 (&w)[C]) {
  const double *r = S.t(d.ct.fw1) + (size_t)T.j0 * 10;
#pragma unroll
  for (int t = 0; t < C; t++) {
    double k[10];
#pragma unroll
    for (int q = 0; q < 5; q++) {
      const double2 v = ld2(r + t * 10 + 2 * q);
      k[2 * q] = v.x;
      k[2 * q + 1] = v.y;
    }
    double2 a = czero();
#pragma unroll
    for (int q = 0; q < 7; q++) a = fma2(a, k[q], u[t + q]);
#pragma unroll
    for (int q = 2; q >= 0; q--)
      if (t - 1 - q >= 0) a = fms2(a, k[7 + q], w[t - 1 - q]);
    w[t] = a;
  }
  const double2 s[3] = {w[C - 1], w[C - 2], w[C - 3]};
  put_state<3>(T, S, slot, s);
}
template <int C, int MB, int F>
__device__ __forceinline__ void d1_bwd(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, double2 (&w)[F][C]) {
  double2 s[F][3];
#pragma unroll
  for (int f = 0; f < F; f++) get_state<3, false>(T, S, f, S.t(d.ct.q1L), s[f]);
  const double *hl = S.t(d.ct.hl1) + (size_t)T.j0 * 4, *bw = S.t(d.ct.bw1) + (size_t)T.j0 * 4;
#pragma unroll
  for (int t = C - 1; t >= 0; t--) {
    const double2 h0 = ld2(hl + t * 4), h1 = ld2(hl + t * 4 + 2), b0 = ld2(bw + t * 4), b1 = ld2(bw + t * 4 + 2);
#pragma unroll
    for (int f = 0; f < F; f++) {
      double2 a = fma2(fma2(fma2(w[f][t], h0.x, s[f][0]), h0.y, s[f][1]), h1.x, s[f][2]);
      a = cscale(b0.x, a);
      if (t + 3 < C) a = fms2(a, b1.y, w[f][t + 3]);
      if (t + 2 < C) a = fms2(a, b1.x, w[f][t + 2]);
      if (t + 1 < C) a = fms2(a, b0.y, w[f][t + 1]);
      w[f][t] = a;
    }
  }
#pragma unroll
  for (int f = 0; f < F; f++) {
    const double2 q[3] = {w[f][0], w[f][1], w[f][2]};
    put_state<3>(T, S, f, q);
  }
}
template <int C, int MB, int F>
__device__ __forceinline__ void d1_end(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, double2 (&w)[F][C]) {
  double2 s[F][3];
#pragma unroll
  for (int f = 0; f < F; f++) get_state<3, true>(T, S, f, S.t(d.ct.q1U), s[f]);
  const double *hu = S.t(d.ct.hu1) + (size_t)T.j0 * 4;
#pragma unroll
  for (int t = 0; t < C; t++) {
    const double2 h0 = ld2(hu + t * 4), h1 = ld2(hu + t * 4 + 2);
#pragma unroll
    for (int f = 0; f < F; f++)
      w[f][t] = cscale(h1.y, fma2(fma2(fma2(w[f][t], h0.x, s[f][0]), h0.y, s[f][1]), h1.x, s[f][2]));
  }
}
// F pencils from d1_fwd to the end
template <int C, int MB, int F>
__device__ __forceinline__ void d1_rest(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, double2 (&w)[F][C]) {
  scans<MB, F, 0, false>(d, T.nc, S);
  d1_bwd(d, T, S, w);
  scans<MB, F, 0, true>(d, T.nc, S);
  d1_end(d, T, S, w);
}

// ---------------------------------------------------------------------
// d2u/dy2 - kk u by the compact second derivative A2 x = B2 u (deryyr2,
// cfdiff.f:735-797): A2 x = (B2 - kk A2) u, so that the subtraction costs
// neither a second read of u nor registers to hold it.
// ---------------------------------------------------------------------
template <int C, int MB>
__device__ __forceinline__ void d2_fwd(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, int slot, double kk,
                                       const double2 (&u)[C + 6], double2 (&w)[C]) {
  const double *r = S.t2(d.ct.fw2) + (size_t)T.j0 * 12;
#pragma unroll
  for (int t = 0; t < C; t++) {
    double k[12];
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const double2 v = S.ld2(r + t * 12 + 2 * q);
      k[2 * q] = v.x;
      k[2 * q + 1] = v.y;
    }
    double2 a = czero();
#pragma unroll
    for (int q = 0; q < 5; q++) a = fma2(a, fma(-kk, k[5 + q], k[q]), u[t + q + 1]);
    if (t > 1) a = fms2(a, k[11], w[t - 2]);
    if (t > 0) a = fms2(a, k[10], w[t - 1]);
    w[t] = a;
  }
  const double2 s[2] = {w[C - 1], w[C - 2]};
  put_state<2>(T, S, slot, s);
}
template <int C, int MB>
__device__ __forceinline__ void d2_bwd(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, int slot, double2 (&w)[C]) {
  double2 s[2];
  get_state<2, false>(T, S, slot, S.t2(d.ct.q2L), s);
  const double *hl = S.t2(d.ct.hl2) + (size_t)T.j0 * 2, *bw = S.t2(d.ct.bw2) + (size_t)T.j0 * 4;
#pragma unroll
  for (int t = C - 1; t >= 0; t--) {
    const double2 h = S.ld2(hl + t * 2), b0 = S.ld2(bw + t * 4), b1 = S.ld2(bw + t * 4 + 2);
    double2 a = cscale(b0.x, fma2(fma2(w[t], h.x, s[0]), h.y, s[1]));
    if (t + 2 < C) a = fms2(a, b1.x, w[t + 2]);
    if (t + 1 < C) a = fms2(a, b0.y, w[t + 1]);
    w[t] = a;
  }
  const double2 q[2] = {w[0], w[1]};
  put_state<2>(T, S, slot, q);
}
template <int C, int MB>
__device__ __forceinline__ void d2_end(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, int slot, double2 (&w)[C]) {
  double2 s[2];
  get_state<2, true>(T, S, slot, S.t2(d.ct.q2U), s);
  const double *hu = S.t2(d.ct.hu2) + (size_t)T.j0 * 2;
#pragma unroll
  for (int t = 0; t < C; t++) {
    const double2 h = S.ld2(hu + t * 2);
    w[t] = fma2(fma2(w[t], h.x, s[0]), h.y, s[1]);
  }
}
// a first derivative in slot 0 and a second one in slot 1 from d1_fwd and
// d2_fwd to the end; they share their barriers
template <int C, int MB>
__device__ __forceinline__ void d12_rest(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, double2 (&a)[1][C],
                                         double2 (&b)[C]) {
  scans<MB, 1, 1, false>(d, T.nc, S);
  d1_bwd(d, T, S, a);
  d2_bwd(d, T, S, 1, b);
  scans<MB, 1, 1, true>(d, T.nc, S);
  d1_end(d, T, S, a);
  d2_end(d, T, S, 1, b);
}

// ---------------------------------------------------------------------
// Dirichlet Poisson solve of the thread's mode (laps.f:375-401): right-hand
// side dt21 u with zero wall rows, then the mode's LU (dt22 - k2 dt21 with
// identity wall rows); zero for k2 = 0, whose tables are zero.
// ---------------------------------------------------------------------
template <int C, int MB>
__device__ __forceinline__ void poisson(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, const double2 (&u)[C + 6],
                                        double2 (&w)[C]) {
  double2 s[2];
  double ha[C], hb[C];
  {
    const double *r = d.ct.fwp + (size_t)T.j0 * 6;
    const double *lt = d.PLt + (size_t)T.j0 * 2 * T.ld + T.m;
#pragma unroll
    for (int t = 0; t < C; t++) {
      const bool in = t < T.n;
      const double l0 = in ? __ldg(lt + (size_t)(2 * t) * T.ld) : 0.0;
      const double l1 = in ? __ldg(lt + (size_t)(2 * t + 1) * T.ld) : 0.0;
      const double2 c0 = ldg2(r + t * 6), c1 = ldg2(r + t * 6 + 2), c2 = ldg2(r + t * 6 + 4);
      double2 a = fma2(fma2(fma2(fma2(cscale(c0.x, u[t + 1]), c0.y, u[t + 2]), c1.x, u[t + 3]), c1.y, u[t + 4]), c2.x,
                       u[t + 5]);
      if (t > 1) a = fms2(a, l1, w[t - 2]);
      if (t > 0) a = fms2(a, l0, w[t - 1]);
      w[t] = a;
      ha[t] = t > 1 ? fma(-l1, ha[t - 2], -l0 * ha[t - 1]) : t == 1 ? fma(-l0, ha[0], -l1) : -l0;
      hb[t] = t > 1 ? fma(-l1, hb[t - 2], -l0 * hb[t - 1]) : t == 1 ? -l0 * hb[0] : -l1;
    }
  }
  auto put = [&](int a, int b) {
    const double2 p[2] = {w[a], w[b]};
    put_state<2>(T, S, 0, p);
    double *q = S.Q + (size_t)T.c * 4 * MB + T.ml;
    q[0] = ha[a];
    q[MB] = hb[a];
    q[2 * MB] = ha[b];
    q[3 * MB] = hb[b];
  };
  put(C - 1, C - 2);
  scans_p<MB, false>(T.nc, S);
  get_state_p<false>(T, S, s);
#pragma unroll
  for (int t = 0; t < C; t++) w[t] = fma2(fma2(w[t], ha[t], s[0]), hb[t], s[1]);
  {
    const double *ut = d.PUt + (size_t)T.j0 * 3 * T.ld + T.m;
#pragma unroll
    for (int t = C - 1; t >= 0; t--) {
      const bool in = t < T.n;
      const double u0 = in ? __ldg(ut + (size_t)(3 * t) * T.ld) : 0.0;
      const double u1 = u0 * (in ? __ldg(ut + (size_t)(3 * t + 1) * T.ld) : 0.0);
      const double u2 = u0 * (in ? __ldg(ut + (size_t)(3 * t + 2) * T.ld) : 0.0);
      double2 a = cscale(u0, w[t]);
      if (t + 2 < C) a = fms2(a, u2, w[t + 2]);
      if (t + 1 < C) a = fms2(a, u1, w[t + 1]);
      w[t] = a;
      ha[t] = t + 2 < C ? fma(-u2, ha[t + 2], -u1 * ha[t + 1]) : t + 1 < C ? fma(-u1, ha[t + 1], -u2) : -u1;
      hb[t] = t + 2 < C ? fma(-u2, hb[t + 2], -u1 * hb[t + 1]) : t + 1 < C ? -u1 * hb[t + 1] : -u2;
    }
  }
  put(0, 1);
  scans_p<MB, true>(T.nc, S);
  get_state_p<true>(T, S, s);
#pragma unroll
  for (int t = 0; t < C; t++) w[t] = fma2(fma2(w[t], ha[t], s[0]), hb[t], s[1]);
}

// the exact (FP64) 00 coefficient of transform output o at row j (mixed forms)
__device__ __forceinline__ double2 mo00(const Dev &d, int o, int j) {
  return make_double2(d.mo_cur[(size_t)o * d.my + j] / ((double)d.mgalx * (double)d.mgalz), 0.0);
}

// tables that the single operators use
__host__ __device__ constexpr int op_tables(int op) { return op == 2 ? 2 : op == 4 ? 0 : 1; }

#define LMC_YC_PROLOGUE(F, POISSON, TAB)               \
  extern __shared__ __align__(16) unsigned char raw[]; \
  const Th<C, MB> T(d, blockIdx.x);                    \
  Sm<MB> S;                                            \
  S.template init<TAB>(d, T.nc, F, POISSON, raw);

// ----------------------------------------------------------------------
// (1) Lapvdvhom: phi -> m_y, dm_y/dy (cross.f:329-335, 365-372)
// ----------------------------------------------------------------------
template <typename CT, int C, int MB>
__global__ void __launch_bounds__(YC_TMAX, 1) c_lapv(Dev d) {
  LMC_YC_PROLOGUE(1, true, 1)
  double2 x[1][C];
  {
    double2 u[C + 6];
    rows_h(d, T, d.phi, u);
#pragma unroll
    for (int t = 0; t < C + 6; t++) {  // wall values set to zero
      const int j = T.j0 + t - 3;
      if (j == 0 || j == d.my - 1) u[t] = czero();
    }
    poisson(d, T, S, u, x[0]);
    S.tables1();
  }
  store(T, wsb<CT>(d, SB_MY), x[0]);
  put_edges(T, S, 0, x[0]);
  __syncthreads();
  {
    double2 u[C + 6];
    with_halo(T, S, 0, x[0], u);
    d1_fwd(d, T, S, 0, u, x[0]);
  }
  d1_rest(d, T, S, x);
  store(T, wsb<CT>(d, SB_DMY), x[0]);
}

// ----------------------------------------------------------------------
// (2)-(3) m_x, m_z, rho u_i, xi-updates of Omega_y and phi, 00 modes
// (cross.f:315-327, 395-499).  V: the 2014 variant (trunk/lomacte/src/
// cross.f:293-461): d(Omega_y)/dy = 0 through two rows at each wall for
// m_x, m_z only, Omega_y** from the raw Omega_y, and T, T** and Delta T
// from the spectral RHS(T).
// ----------------------------------------------------------------------
template <typename CT, int C, int MB, bool V>
__global__ void __launch_bounds__(YC_TMAX, 1) c_assemble(Dev d, int rk) {
  LMC_YC_PROLOGUE(1, false, 1)
  const int my = d.my;
  const double dtxi = d.scal_d[0] * d.xi[rk];
  const double ta = (T.k2 != 0.0) ? T.kx / T.k2 : 0.0, tb = (T.k2 != 0.0) ? T.kz / T.k2 : 0.0;
  const bool m00 = T.act && T.m == 0;
  // wall condition of Omega_y (cross.f:315-327; lomacte/cross.f:306-311),
  // read before the barriers below and so before any row is overwritten
  constexpr int W = V ? 2 : 1;
  const double2 vb = __ldcg(d.vor + (size_t)W * T.ld + T.m), vt = __ldcg(d.vor + (size_t)(my - 1 - W) * T.ld + T.m);
  double2 x[1][C];
  {
    double2 u[C + 6];
    rows_h(d, T, d.psi, u);
    S.tables1();
    d1_fwd(d, T, S, 0, u, x[0]);
  }
  d1_rest(d, T, S, x);
  if (!T.act) return;
  // in batches of R rows: a batch's loads are in flight together before its
  // first store
  constexpr int R = 3;
  const size_t o = (size_t)T.j0 * T.ld + T.m;
#pragma unroll
  for (int t0 = 0; t0 < C; t0 += R) {
    double2 m[R], a[R], vr[R], ps[R], ro[R], ph[R], rp[R], Tv[V ? R : 1], RT[V ? R : 1];
#pragma unroll
    for (int r = 0; r < R; r++)
      if (t0 + r < C && t0 + r < T.n) {
        const size_t p = o + (size_t)(t0 + r) * T.ld;
        m[r] = to_d2(__ldg(wsb<CT>(d, SB_MY) + p));
        a[r] = to_d2(__ldg(wsb<CT>(d, SB_DMY) + p));
        ps[r] = __ldg(d.psi + p);
        ro[r] = __ldg(d.Rom + p);
        rp[r] = __ldg(d.Rphi + p);
        vr[r] = __ldcg(d.vor + p);
        ph[r] = __ldcg(d.phi + p);
        if constexpr (V) {
          Tv[r] = __ldcg(d.scal + p);
          RT[r] = __ldg(d.RT + p);
        }
      }
#pragma unroll
    for (int r = 0; r < R; r++)
      if (t0 + r < C && t0 + r < T.n) {
        const int j = T.j0 + t0 + r;
        const size_t p = o + (size_t)(t0 + r) * T.ld;
        const double2 vo = j < W ? vb : j > my - 1 - W ? vt : vr[r];
        double2 b = cadd(csub(cik(ta, a[r]), cik(tb, vo)), cik(T.kx, ps[r]));  // rho u, cross.f:402,467
        double2 c = cadd(cadd(cik(tb, a[r]), cik(ta, vo)), cik(T.kz, ps[r]));  // rho w, cross.f:404,469
        double2 e = cadd(x[0][t0 + r], m[r]);                                   // rho v, cross.f:434-437, 471
        if (m00) {  // 00 modes injected (cross.f:486-491), then u00**, w00** (cross.f:495-498)
          b = make_double2(d.u00[j], 0.0);
          c = make_double2(d.w00[j], 0.0);
          e = make_double2(d.v00[j], 0.0);
          if constexpr (mixed<CT>()) {
            d.mi[j] = b.x;
            d.mi[(size_t)my + j] = e.x;
            d.mi[(size_t)2 * my + j] = c.x;
          }
          if (j >= 1 && j <= my - 2) {
            d.u00[j] += dtxi * d.rf0u[j];
            d.w00[j] += dtxi * d.rf0w[j];
          }
        }
        wsb<CT>(d, SB_RU)[p] = from_d2<CT>(b);
        wsb<CT>(d, SB_RW)[p] = from_d2<CT>(c);
        wsb<CT>(d, SB_RV)[p] = from_d2<CT>(e);
        d.vor[p] = fma2(V ? vr[r] : vo, dtxi, ro[r]);  // cross.f:420-424
        if constexpr (V) {  // T saved, T** and Delta T: lomacte/cross.f:368-396
          const double2 inc = cscale(dtxi, RT[r]);
          d.Told[p] = Tv[r];
          d.scal[p] = cadd(Tv[r], inc);
          d.dTs[p] = inc;
        }
        d.phi[p] = fma2((j == 0 || j == my - 1) ? czero() : ph[r], dtxi, rp[r]);  // cross.f:424-425
      }
  }
}

// ----------------------------------------------------------------------
// (4) T with its wall BCs, dT/dy, lap(T) (cross.f:336-349, 521-541).  V: the
// 2014 variant differentiates the T saved before its update, with no wall
// values imposed (lomacte/cross.f:486-519).  Z: the passive scalar, treated
// as T, its 00 mode held at scal_d[5], scal_d[6] (mi rows 6, 7).
// ----------------------------------------------------------------------
template <typename CT, int C, int MB, bool V, bool Z, int TAB>
__global__ void __launch_bounds__(YC_TMAX, 1) c_tder(Dev d) {
  LMC_YC_PROLOGUE(2, false, TAB)
  const int my = d.my;
  const bool m00 = T.act && T.m == 0;
  double2 *const f = Z ? d.zsc : V ? d.Told : d.scal;
  double2 a[1][C], b[C];
  {
    double2 u[C + 6];
    rows_h(d, T, f, u);
    if constexpr (!V) {
      const double2 wb = T.m != 0 ? czero() : make_double2(Z ? d.scal_d[5] : 1.0 / d.scal_d[3], 0.0);
      const double2 wt = T.m != 0 ? czero() : make_double2(Z ? d.scal_d[6] : 1.0 / d.scal_d[4], 0.0);
#pragma unroll
      for (int t = 0; t < C + 6; t++) {
        const int j = T.j0 + t - 3;
        if (j == 0) u[t] = wb;
        if (j == my - 1) u[t] = wt;
      }
      if (T.act) {  // the wall rows of the state; nobody reads them from memory in this kernel
        if (T.c == 0) f[T.m] = wb;
        if (T.c == T.nc - 1) f[(size_t)(my - 1) * T.ld + T.m] = wt;
      }
    }
    if constexpr (mixed<CT>()) {
      double2 v[C];
#pragma unroll
      for (int t = 0; t < C; t++) {
        v[t] = u[t + 3];
        if (!Z && m00 && t < T.n) d.mi[(size_t)5 * my + T.j0 + t] = v[t].x;
      }
      store(T, wsb<CT>(d, Z ? SB_Z32 : SB_T32), v);
    }
    S.tables1();
    d1_fwd(d, T, S, 0, u, a[0]);
    S.tables2();
    d2_fwd(d, T, S, 1, T.k2, u, b);
  }
  d12_rest(d, T, S, a, b);
  if constexpr (mixed<CT>())
    if (m00) {
#pragma unroll
      for (int t = 0; t < C; t++)
        if (t < T.n) {
          d.mi[(size_t)(Z ? 7 : 4) * my + T.j0 + t] = a[0][t].x;
          d.mi[(size_t)(Z ? 6 : 3) * my + T.j0 + t] = b[t].x;
        }
    }
  store(T, wsb<CT>(d, Z ? SB_DZDY : SB_DTDY), a[0]);
  store(T, wsb<CT>(d, Z ? SB_LAPZ : SB_LAPT), b);
}

// ----------------------------------------------------------------------
// Variable viscosity: the spectral inputs of the strain rates.  In
// physical space d(u_i)/dx_j = T d(rho u_i)/dx_j + rho u_i dT/dx_j, and the
// stress needs d(rho u_i)/dx_j only in the symmetric sums; this kernel
// writes d(rho v)/dy and the three off-diagonal sums (d(rho u)/dx is formed
// by the x stage, d(rho w)/dz by the inverse z transforms from rho w).
// The y derivatives are deryr2's (cfdiff.f:518-601), as every first y
// derivative of the substep.  Runs after c_assemble on the same stream.
// The mixed forms launch one block more: its modes 0, 1, 2 are the exact
// 00 profiles of rho u, rho v, rho w (mi rows 0..2), differentiated into mi
// rows 9, 8, 10; the FP32 buffers' 00 coefficients are not read (the
// transforms drop them).  parts = 3: a block forms one of the derivatives
// (sgrad_parts).
// ----------------------------------------------------------------------
template <typename CT, int C, int MB>
__global__ void __launch_bounds__(YC_TMAX, 1) c_sgrad(Dev d, int parts) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int part = parts == 3 ? (int)blockIdx.x % 3 : -1;
  const Th<C, MB> T(d, parts == 3 ? blockIdx.x / 3 : blockIdx.x);
  Sm<MB> S;
  S.template init<1>(d, T.nc, 1, false, raw);
  double2 x[1][C];
  if constexpr (mixed<CT>()) {
    if (blockIdx.x == gridDim.x - 1) {
      const double *p = d.mi + (size_t)(T.ml < 3 ? T.ml : 0) * d.my;
      double2 u[C + 6];
#pragma unroll
      for (int t = 0; t < C + 6; t++) {
        const int j = T.j0 + t - 3;
        u[t] = make_double2((j >= 0 && j < d.my) ? p[j] : 0.0, 0.0);
      }
      S.tables1();
      d1_fwd(d, T, S, 0, u, x[0]);
      d1_rest(d, T, S, x);
      if (T.ml < 3) {
        double *q = d.mi + (size_t)(T.ml == 0 ? 9 : T.ml == 1 ? 8 : 10) * d.my + T.j0;
#pragma unroll
        for (int t = 0; t < C; t++)
          if (t < T.n) q[t] = x[0][t].x;
      }
      return;
    }
  }
  const CT *RU = wsb<CT>(d, SB_RU), *RV = wsb<CT>(d, SB_RV), *RW = wsb<CT>(d, SB_RW);
  S.tables1();
  auto deriv = [&](const CT *f) {
    double2 u[C + 6];
    rows_h(d, T, f, u);
    d1_fwd(d, T, S, 0, u, x[0]);
    d1_rest(d, T, S, x);
  };
  double2 v[C];
  if (part <= 0) {
    deriv(RV);
    store(T, wsb<CT>(d, SB_GYY), x[0]);
    rows(T, RU, v);
    rows(T, RW, x[0]);
#pragma unroll
    for (int t = 0; t < C; t++) x[0][t] = cadd(cik(T.kz, v[t]), cik(T.kx, x[0][t]));
    store(T, wsb<CT>(d, SB_G13), x[0]);
  }
  if (part == -1 || part == 1) {
    deriv(RU);
    rows(T, RV, v);
#pragma unroll
    for (int t = 0; t < C; t++) x[0][t] = cadd(x[0][t], cik(T.kx, v[t]));
    store(T, wsb<CT>(d, SB_G12), x[0]);
  }
  if (part == -1 || part == 2) {
    deriv(RW);
    rows(T, RV, v);
#pragma unroll
    for (int t = 0; t < C; t++) x[0][t] = cadd(x[0][t], cik(T.kz, v[t]));
    store(T, wsb<CT>(d, SB_G23), x[0]);
  }
}

// ----------------------------------------------------------------------
// (6b)-(9) N_i, vorticity, the two Laplacians, RHS(Omega_y), RHS(phi) and
// the RK3 update (cross.f:652-682, 748-981), with the y derivatives of the
// three N_i, of u, w and of the two curls gathered by linearity (d = d/dy,
// lap = d2/dy2 - k2):
//   RHS(Omega_y) = i kz N_x - i kx N_z + lap(omega_y)/Re
//                = kx kz (uu - ww) - (kx^2 - kz^2) uw - d(i kz uv - i kx vw)
//                  + lap(i kz u - i kx w)/Re
//   (curl omega)_y = d(i kx u + i kz w) + k2 v
//   RHS(phi) = -k2 N_y - d(i kx N_x + i kz N_z) - lap((curl omega)_y)/Re
//            = k2 q + d(k2 vv - kx^2 uu - 2 kx kz uw - kz^2 ww + d q)
//              - lap((curl omega)_y)/Re,   q = i kx uv + i kz vw
// (products rho u_i u_j): four first derivatives instead of six, and no
// N_i or curl goes through memory.  TU: T += Delta T as well (cross.f:
// 619-627); grids with many modes leave that to k_tupd on the second stream.
// halves = 2: even blocks take RHS(phi), odd ones RHS(Omega_y) (post_halves);
// neither reads what the other writes.
// ----------------------------------------------------------------------
template <typename CT, int C, int MB, bool TU, int TAB>
__global__ void __launch_bounds__(YC_TMAX, 1) c_post(Dev d, int rk, int halves) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int half = halves == 2 ? (int)blockIdx.x & 1 : -1;
  const Th<C, MB> T(d, halves == 2 ? blockIdx.x >> 1 : blockIdx.x);
  Sm<MB> S;
  S.template init<TAB>(d, T.nc, 2, false, raw);
  const double kx = T.kx, kz = T.kz, k2 = T.k2, dtg = post_dt(d, rk) * d.gama[rk];
  const CT *U = wsb<CT>(d, OU), *V = wsb<CT>(d, OV), *W = wsb<CT>(d, OW);
  const CT *UU = wsb<CT>(d, ORUU), *VV = wsb<CT>(d, ORVV), *WW = wsb<CT>(d, ORWW);
  const CT *UV = wsb<CT>(d, ORUV), *UW = wsb<CT>(d, ORUW), *VW = wsb<CT>(d, ORVW);
  // i (a f + b g) with its halo rows
  auto comb = [&](double a, const CT *f, double b, const CT *g, double2 (&u)[C + 6]) {
#pragma unroll
    for (int t = 0; t < C + 6; t++) {
      const int j = T.j0 + t - 3;
      u[t] = czero();
      if (j >= 0 && j < d.my) {
        const size_t p = (size_t)j * T.ld + T.m;
        u[t] = cadd(cik(a, to_d2(__ldg(f + p))), cik(b, to_d2(__ldg(g + p))));
      }
    }
  };
  const size_t o = (size_t)T.j0 * T.ld + T.m;
  if (half != 1) {  // RHS(phi)
    double2 x[2][C];
    {
      double2 u[C + 6];
      comb(kx, UV, kz, VW, u);
      S.tables1();
      d1_fwd(d, T, S, 0, u, x[0]);
      comb(kx, U, kz, W, u);
      d1_fwd(d, T, S, 1, u, x[1]);
    }
    d1_rest(d, T, S, x);
    S.tables2();
#pragma unroll
    for (int t = 0; t < C; t++) {
      if (t < T.n) {
        const size_t p = o + (size_t)t * T.ld;
        double2 e = fma2(x[0][t], k2, to_d2(__ldg(VV + p)));
        e = fms2(e, kx * kx, to_d2(__ldg(UU + p)));
        e = fms2(e, 2.0 * kx * kz, to_d2(__ldg(UW + p)));
        x[0][t] = fms2(e, kz * kz, to_d2(__ldg(WW + p)));
        x[1][t] = fma2(x[1][t], k2, to_d2(__ldg(V + p)));
      } else {
        x[0][t] = x[1][t] = czero();
      }
    }
    put_edges(T, S, 0, x[0]);
    put_edges(T, S, 1, x[1]);
    __syncthreads();
    double2 a[1][C];
    {
      double2 u[C + 6];
      with_halo(T, S, 0, x[0], u);
      d1_fwd(d, T, S, 0, u, a[0]);
      with_halo(T, S, 1, x[1], u);
      d2_fwd(d, T, S, 1, k2, u, x[1]);
    }
    d12_rest(d, T, S, a, x[1]);
#pragma unroll
    for (int t = 0; t < C; t++)
      if (t < T.n) {
        const size_t p = o + (size_t)t * T.ld;
        a[0][t] = fms2(a[0][t], d.ire, x[1][t]);
        a[0][t] = fma2(a[0][t], k2, cadd(cik(kx, to_d2(__ldg(UV + p))), cik(kz, to_d2(__ldg(VW + p)))));
        x[1][t] = __ldcg(d.phi + p);
      }
    store(T, d.Rphi, a[0]);
#pragma unroll
    for (int t = 0; t < C; t++) x[1][t] = fma2(x[1][t], dtg, a[0][t]);  // cross.f:978
    store(T, d.phi, x[1]);
    if (half == 0) return;
  }
  {  // RHS(Omega_y)
    double2 a[1][C], b[C];
    {
      double2 u[C + 6];
      comb(kz, UV, -kx, VW, u);
      if (half == 1) {
        S.tables1();
        S.tables2();
      }
      d1_fwd(d, T, S, 0, u, a[0]);
      comb(kz, U, -kx, W, u);
      d2_fwd(d, T, S, 1, k2, u, b);
    }
    d12_rest(d, T, S, a, b);
#pragma unroll
    for (int t = 0; t < C; t++)
      if (t < T.n) {
        const size_t p = o + (size_t)t * T.ld;
        const double2 uu = to_d2(__ldg(UU + p)), ww = to_d2(__ldg(WW + p)), uw = to_d2(__ldg(UW + p));
        a[0][t] = fma2(csub(fms2(cscale(kx * kz, csub(uu, ww)), kx * kx - kz * kz, uw), a[0][t]), d.ire, b[t]);
        b[t] = __ldcg(d.vor + p);
      }
    store(T, d.Rom, a[0]);
#pragma unroll
    for (int t = 0; t < C; t++) b[t] = fma2(b[t], dtg, a[0][t]);  // cross.f:969
    store(T, d.vor, b);
  }
  if constexpr (TU) {
    double2 a[C], b[C];
    rows(T, wsb<CT>(d, ODT), a);
    rows(T, d.scal, b);
#pragma unroll
    for (int t = 0; t < C; t++) {
      if constexpr (mixed<CT>())
        if (T.m == 0 && t < T.n) a[t] = mo00(d, ODT, T.j0 + t);
      b[t] = cadd(b[t], a[t]);
    }
    store(T, d.scal, b);
  }
}

// ----------------------------------------------------------------------
// (8) psi^{n+1} by solvepsi (cross.f:1092-1104, laps.f:580-730): the
// Dirichlet solution of the thread's mode, then Neumann walls through the
// homogeneous solutions v1, v2 and the inverse of their 2 x 2 wall matrix.
// V: the 2014 variant solves the Dirichlet problem for
// psi = -d(rho) / (Deltat (gamma + xi)) (lomacte/cross.f:970-983).
// ----------------------------------------------------------------------
template <int C, int MB>
__device__ __forceinline__ void neumann(const Dev &d, const Th<C, MB> &T, const Sm<MB> &S, double2 (&x)[C]) {
  double2 db = czero(), dt = czero();
#pragma unroll
  for (int t = 0; t < C; t++)
    if (t < T.n) {
      db = fma2(db, __ldg(d.r_ebot + T.j0 + t), x[t]);
      dt = fma2(dt, __ldg(d.r_etop + T.j0 + t), x[t]);
    }
  double2 *e = S.E + (size_t)T.c * 2 * MB + T.ml;
  e[0] = db;
  e[MB] = dt;
  __syncthreads();
  const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (w < nw)
    for (int u = w; u < MB / 8; u += nw) {
      const int ml = u * 8 + (lane >> 2);
      double2 a = czero(), b = czero();
      for (int c = lane & 3; c < T.nc; c += 4) {
        a = cadd(a, S.E[(size_t)c * 2 * MB + ml]);
        b = cadd(b, S.E[((size_t)c * 2 + 1) * MB + ml]);
      }
#pragma unroll
      for (int off = 1; off < 4; off <<= 1) {
        a.x += __shfl_xor_sync(LMC_FULL, a.x, off);
        a.y += __shfl_xor_sync(LMC_FULL, a.y, off);
        b.x += __shfl_xor_sync(LMC_FULL, b.x, off);
        b.y += __shfl_xor_sync(LMC_FULL, b.y, off);
      }
      if ((lane & 3) == 0) {
        S.G[ml] = a;
        S.G[MB + ml] = b;
      }
    }
  __syncthreads();
  db = S.G[T.ml];
  dt = S.G[MB + T.ml];
  const double *ai = d.AAinv + (size_t)T.m * 4;
  const double a0 = __ldg(ai), a1 = __ldg(ai + 1), a2 = __ldg(ai + 2), a3 = __ldg(ai + 3);
  const double2 c1 = make_double2(-(a0 * db.x + a1 * dt.x), -(a0 * db.y + a1 * dt.y));
  const double2 c2 = make_double2(-(a2 * db.x + a3 * dt.x), -(a2 * db.y + a3 * dt.y));
  const double *v = d.V12t + (size_t)T.j0 * 2 * T.ld + T.m;
#pragma unroll
  for (int t = 0; t < C; t++)
    if (t < T.n)
      x[t] = fma2(fma2(x[t], __ldg(v + (size_t)(2 * t) * T.ld), c1), __ldg(v + (size_t)(2 * t + 1) * T.ld), c2);
}
template <typename CT, int C, int MB, bool V>
__global__ void __launch_bounds__(YC_TMAX, 1) c_psi(Dev d, int rk) {
  LMC_YC_PROLOGUE(1, true, 0)
  double2 x[C];
  {
    double2 u[C + 6];
    rows_h(d, T, wsb<CT>(d, ODRHO), u);
    if constexpr (V) {
      const double sc = -1.0 / (d.scal_d[0] * (d.gama[rk] + d.xi[rk]));
#pragma unroll
      for (int t = 0; t < C + 6; t++) u[t] = cscale(sc, u[t]);
    }
    poisson(d, T, S, u, x);
  }
  if constexpr (!V) neumann(d, T, S, x);
  store(T, d.psi, x);
}

// single y operator on FP64 device-layout fields: OP 1 d/dy, 2 d2/dy2,
// 3 Lapvdvhom (out = v, out2 = dv/dy), 4 solvepsi.  A block forms nothing but
// its operator: with both derivatives formed for either one lmc_op_y took 0.24 ms
// on 512 x 33 x 512 and 0.22 on 256 x 129 x 256, now 0.15 and 0.15 (d/dy; one
// thread per mode before that 0.17 and 0.21).
template <int C, int MB, int OP>
__global__ void __launch_bounds__(YC_TMAX, 1) c_op(Dev d, const double2 *in, double2 *out, double2 *out2) {
  LMC_YC_PROLOGUE(1, OP > 2, op_tables(OP))
  double2 x[1][C];
  {
    double2 u[C + 6];
    rows_h(d, T, in, u);
    if constexpr (OP == 1) {
      S.tables1();
      d1_fwd(d, T, S, 0, u, x[0]);
    } else if constexpr (OP == 2) {
      S.tables2();
      d2_fwd(d, T, S, 0, 0.0, u, x[0]);
    } else {
      poisson(d, T, S, u, x[0]);
    }
  }
  if constexpr (OP == 1) {
    d1_rest(d, T, S, x);
  } else if constexpr (OP == 2) {
    scans<MB, 0, 1, false>(d, T.nc, S);
    d2_bwd(d, T, S, 0, x[0]);
    scans<MB, 0, 1, true>(d, T.nc, S);
    d2_end(d, T, S, 0, x[0]);
  }
  if constexpr (OP == 4) neumann(d, T, S, x[0]);
  store(T, out, x[0]);
  if constexpr (OP == 3) {
    S.tables1();
    put_edges(T, S, 0, x[0]);
    __syncthreads();
    {
      double2 u[C + 6];
      with_halo(T, S, 0, x[0], u);
      d1_fwd(d, T, S, 0, u, x[0]);
    }
    d1_rest(d, T, S, x);
    store(T, out2, x[0]);
  }
}

}  // namespace ych

namespace ych {
// Blocks from which c_tder and c_post take the tables of d2/dy2 from shared
// memory as well as those of d/dy: with several waves of blocks they are out
// of the L1 each time (12,192 modes x 193, FP64, five waves: 5.29 ms per step
// against 5.43); with one or two a block waits for more bytes than it saves
// (2,016 x 129: 0.93 against 0.98; 4,560 x 129 1.29 against 1.32).
template <int MB>
bool many_waves(const Dev &d) {
  return (d.nmode + MB - 1) / MB > 4 * 148;
}
// Blocks of nt threads that the registers of the device hold (128 each).
inline int resident(int nt) { return std::max(64 / ((nt + 31) / 32 * 4), 1) * 148; }
// c_post as two blocks per MB modes, one for each right-hand side: shorter
// chains where twice the blocks still run at once (24 x 25 x 24: 0.173 ms per
// step against 0.205; 512 x 257 2-D 0.618 against 0.627), and shorter last
// waves where they come in waves anyway (12,192 x 193: 4.97 against 5.24;
// 8,128 x 129 2.40 against 2.45; 6,096 x 129 with the scalar and mu 2.53
// against 2.65).  In between the second wave costs more (2,016 x 129 with
// both: 0.93 against 0.88).
inline int post_halves(int g, int nt) { return 2 * g <= resident(nt) || g > resident(nt) ? 2 : 1; }
// c_sgrad as three, one for each derivative, where they all run at once
// (1,128 modes x 97: 0.525 ms per step against 0.560; 4,560 x 97, where they
// do not: 1.472 against 1.461).
inline int sgrad_parts(int g, int nt) { return 3 * g <= resident(nt) ? 3 : 1; }

// `parts` blocks per MB modes (and `extra` blocks), shared memory for F pencils and for
// the tables of d/dy (tabs 1) and of d2/dy2 (tabs 2), which every block reads
// several times: from global memory they come out of the L2 with each pass,
// as the pencils' rows push them out of the L1 (c_post, 12,192 x 193: 16 of
// 25 cycles between a warp's instructions were waits for loads).  They stay
// there where shared memory has no room for them or would hold fewer blocks
// per SM than the registers do.  24 x 25 x 24: 0.230 ms per step after 0.240;
// 64 x 129 x 64 with the scalar and mu 0.93 after 1.00; 96 x 129 x 96, float2
// buffers, 1.29 after 1.33; 192 x 193 x 128 5.29 after 5.60.
template <int MB, typename K, typename... A>
void go(K k, const Dev &d, int F, bool poisson, int tabs, int parts, int extra, cudaStream_t s, A... a) {
  const int g = (d.nmode + MB - 1) / MB * parts + extra, nt = d.ync * MB;
  const size_t base = Sm<MB>::bytes(d.ync, F, poisson);
  const size_t tab = sizeof(double) * (tabs == 2 ? d.ct.n1 + d.ct.n2 : tabs == 1 ? d.ct.n1 : 0);
  const size_t sm = 228 * 1024, res = 1024;                // shared memory of an SM, and what each block reserves of it
  const size_t per = std::min<size_t>(resident(nt) / 148, std::min<size_t>(sm / (base + res), (g + 147) / 148));
  Dev e = d;
  e.ct.sm = tab > 0 && base + tab <= (size_t)d.smem_limit && per * (base + tab + res) <= sm;
  k<<<g, nt, base + (e.ct.sm ? tab : 0), s>>>(e, a...);
}
}  // namespace ych

template <int C, int MB>
void YC<C, MB>::lapv(const Dev &d, cudaStream_t s) {
  if (d.prec) ych::go<MB>(ych::c_lapv<float2, C, MB>, d, 1, true, 1, 1, 0, s);
  else ych::go<MB>(ych::c_lapv<double2, C, MB>, d, 1, true, 1, 1, 0, s);
}
template <int C, int MB>
void YC<C, MB>::assemble(const Dev &d, int rk, cudaStream_t s) {
  if (d.prec) ych::go<MB>(ych::c_assemble<float2, C, MB, false>, d, 1, false, 1, 1, 0, s, rk);
  else if (d.variant) ych::go<MB>(ych::c_assemble<double2, C, MB, true>, d, 1, false, 1, 1, 0, s, rk);
  else ych::go<MB>(ych::c_assemble<double2, C, MB, false>, d, 1, false, 1, 1, 0, s, rk);
}
template <int C, int MB>
void YC<C, MB>::tder(const Dev &d, bool z, cudaStream_t s) {
  using namespace ych;
  auto run = [&](auto t) {
    constexpr int TAB = decltype(t)::value;
    if (z) {
      if (d.prec) go<MB>(c_tder<float2, C, MB, false, true, TAB>, d, 2, false, TAB, 1, 0, s);
      else go<MB>(c_tder<double2, C, MB, false, true, TAB>, d, 2, false, TAB, 1, 0, s);
    } else if (d.prec) {
      go<MB>(c_tder<float2, C, MB, false, false, TAB>, d, 2, false, TAB, 1, 0, s);
    } else if (d.variant) {
      go<MB>(c_tder<double2, C, MB, true, false, TAB>, d, 2, false, TAB, 1, 0, s);
    } else {
      go<MB>(c_tder<double2, C, MB, false, false, TAB>, d, 2, false, TAB, 1, 0, s);
    }
  };
  if (many_waves<MB>(d)) run(std::integral_constant<int, 2>());
  else run(std::integral_constant<int, 1>());
}
template <int C, int MB>
void YC<C, MB>::sgrad(const Dev &d, cudaStream_t s) {  // mixed: one more block for the exact 00 profiles
  const int parts = ych::sgrad_parts((d.nmode + MB - 1) / MB, d.ync * MB);
  if (d.prec) ych::go<MB>(ych::c_sgrad<float2, C, MB>, d, 1, false, 1, parts, 1, s, parts);
  else ych::go<MB>(ych::c_sgrad<double2, C, MB>, d, 1, false, 1, parts, 0, s, parts);
}
template <int C, int MB>
void YC<C, MB>::post(const Dev &d, int rk, bool tu, cudaStream_t s) {
  using namespace ych;
  const int g = (d.nmode + MB - 1) / MB, halves = post_halves(g, d.ync * MB);
  auto run = [&](auto t) {
    constexpr int TAB = decltype(t)::value;
    if (d.prec) {
      if (tu) go<MB>(c_post<float2, C, MB, true, TAB>, d, 2, false, TAB, halves, 0, s, rk, halves);
      else go<MB>(c_post<float2, C, MB, false, TAB>, d, 2, false, TAB, halves, 0, s, rk, halves);
    } else {
      if (tu) go<MB>(c_post<double2, C, MB, true, TAB>, d, 2, false, TAB, halves, 0, s, rk, halves);
      else go<MB>(c_post<double2, C, MB, false, TAB>, d, 2, false, TAB, halves, 0, s, rk, halves);
    }
  };
  if (many_waves<MB>(d)) run(std::integral_constant<int, 2>());
  else run(std::integral_constant<int, 1>());
}
template <int C, int MB>
void YC<C, MB>::psi(const Dev &d, int rk, cudaStream_t s) {
  if (d.prec) ych::go<MB>(ych::c_psi<float2, C, MB, false>, d, 1, true, 0, 1, 0, s, rk);
  else if (d.variant) ych::go<MB>(ych::c_psi<double2, C, MB, true>, d, 1, true, 0, 1, 0, s, rk);
  else ych::go<MB>(ych::c_psi<double2, C, MB, false>, d, 1, true, 0, 1, 0, s, rk);
}
template <int C, int MB>
void YC<C, MB>::op_y(const Dev &d, int op, const double2 *in, double2 *out, double2 *out2, cudaStream_t s) {
  auto run = [&](auto o) {
    constexpr int OP = decltype(o)::value;
    ych::go<MB>(ych::c_op<C, MB, OP>, d, 1, OP > 2, ych::op_tables(OP), 1, 0, s, in, out, out2);
  };
  if (op == 1) run(std::integral_constant<int, 1>());
  else if (op == 2) run(std::integral_constant<int, 2>());
  else if (op == 3) run(std::integral_constant<int, 3>());
  else run(std::integral_constant<int, 4>());
}
template <int C, int MB>
cudaError_t YC<C, MB>::optin(int limit) {
  using namespace ych;
  const void *fns[] = {(const void *)c_lapv<float2, C, MB>, (const void *)c_lapv<double2, C, MB>,
                       (const void *)c_assemble<float2, C, MB, false>, (const void *)c_assemble<double2, C, MB, true>,
                       (const void *)c_assemble<double2, C, MB, false>, (const void *)c_tder<float2, C, MB, false, true, 1>,
                       (const void *)c_tder<double2, C, MB, false, true, 1>, (const void *)c_tder<float2, C, MB, false, false, 1>,
                       (const void *)c_tder<double2, C, MB, true, false, 1>, (const void *)c_tder<double2, C, MB, false, false, 1>,
                       (const void *)c_tder<float2, C, MB, false, true, 2>, (const void *)c_tder<double2, C, MB, false, true, 2>,
                       (const void *)c_tder<float2, C, MB, false, false, 2>, (const void *)c_tder<double2, C, MB, true, false, 2>,
                       (const void *)c_tder<double2, C, MB, false, false, 2>,
                       (const void *)c_sgrad<float2, C, MB>, (const void *)c_sgrad<double2, C, MB>,
                       (const void *)c_post<float2, C, MB, true, 1>, (const void *)c_post<float2, C, MB, false, 1>,
                       (const void *)c_post<double2, C, MB, true, 1>, (const void *)c_post<double2, C, MB, false, 1>,
                       (const void *)c_post<float2, C, MB, true, 2>, (const void *)c_post<float2, C, MB, false, 2>,
                       (const void *)c_post<double2, C, MB, true, 2>, (const void *)c_post<double2, C, MB, false, 2>,
                       (const void *)c_psi<float2, C, MB, false>, (const void *)c_psi<double2, C, MB, true>,
                       (const void *)c_psi<double2, C, MB, false>, (const void *)c_op<C, MB, 1>,
                       (const void *)c_op<C, MB, 2>, (const void *)c_op<C, MB, 3>, (const void *)c_op<C, MB, 4>};
  for (const void *fn : fns) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace lmc
