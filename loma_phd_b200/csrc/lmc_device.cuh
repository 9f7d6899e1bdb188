// lmc_device.cuh -- device building blocks of the lomacte substep kernels.
//
// y-direction operators of the 00 modes and of the no-allocation d/dy: one warp
// per pencil.  The my points are split into chunks of n in {C-1, C}
// consecutive points, one chunk per active lane (LPM active lanes).  Banded
// matrix-vector products exchange a halo of H points with the neighbour lanes
// by shuffles.  Banded triangular solves run each chunk's recurrence in
// registers and join the chunks with a Kogge-Stone scan of the affine chunk
// maps state_out = M state_in + p, whose matrices come from the host (the
// compact-derivative LUs), so only the particular responses p travel between
// lanes.
//
// x/z transforms: FFTs in passes of register DFTs over lines in shared memory
// (Fft below).
#pragma once
#include <cuda_runtime.h>

namespace lmcd {

#define LMC_FULL 0xffffffffu

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cscale(double s, double2 a) { return make_double2(s * a.x, s * a.y); }
// (i k) * a
__device__ __forceinline__ double2 cik(double k, double2 a) { return make_double2(-k * a.y, k * a.x); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 czero() { return make_double2(0.0, 0.0); }

// The same operations on single-precision complex values (the transform
// work buffers of the mixed-precision form).
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cscale(float s, float2 a) { return make_float2(s * a.x, s * a.y); }
__device__ __forceinline__ float2 cik(float k, float2 a) { return make_float2(-k * a.y, k * a.x); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }

// real type and constructors of a complex type
template <typename CT>
struct CReal;
template <>
struct CReal<double2> { using R = double; };
template <>
struct CReal<float2> { using R = float; };
template <typename CT>
__device__ __forceinline__ CT cmk(typename CReal<CT>::R a, typename CReal<CT>::R b) {
  CT c;
  c.x = a;
  c.y = b;
  return c;
}
template <typename CT>
__device__ __forceinline__ CT cz() { return cmk<CT>(0, 0); }
// FP64 value of a stored work-buffer element and back
__device__ __forceinline__ double2 to_d2(double2 a) { return a; }
__device__ __forceinline__ double2 to_d2(float2 a) { return make_double2(a.x, a.y); }
template <typename CT>
__device__ __forceinline__ CT from_d2(double2 a) { return cmk<CT>((typename CReal<CT>::R)a.x, (typename CReal<CT>::R)a.y); }

__device__ __forceinline__ double2 shfl_up2(double2 v, int d) {
  return make_double2(__shfl_up_sync(LMC_FULL, v.x, d), __shfl_up_sync(LMC_FULL, v.y, d));
}
__device__ __forceinline__ double2 shfl_down2(double2 v, int d) {
  return make_double2(__shfl_down_sync(LMC_FULL, v.x, d), __shfl_down_sync(LMC_FULL, v.y, d));
}

// ---------------------------------------------------------------------
// Chunk geometry of one lane
// ---------------------------------------------------------------------
struct Lane {
  int lane, s, n, lpm;
  bool full;  // n == C
};

template <int C>
__device__ __forceinline__ Lane make_lane(int lpm, int base, int extra) {
  Lane L;
  L.lane = threadIdx.x & 31;
  L.lpm = lpm;
  if (L.lane < lpm) {
    L.n = base + (L.lane < extra ? 1 : 0);
    L.s = L.lane * base + (L.lane < extra ? L.lane : extra);
  } else {
    L.n = 0;
    L.s = 0;
  }
  L.full = (L.n == C);
  return L;
}

// Row tables are stored chunk-major: entry (row s+t, coefficient c) of
// lane l is T[(t*W + c)*32 + l], so a warp reads 32 consecutive doubles.
__device__ __forceinline__ double tab(const double *__restrict__ T, int W, int t, int c, int lane) {
  return __ldg(T + ((size_t)t * W + c) * 32 + lane);
}

// v = band(A) * v, A rows of 2H+1 coefficients (column offsets -H..H).  The
// coefficient tables hold zeros for out-of-range columns and the halos of the
// first/last lanes are zero; a rolling window keeps the H original values that
// the rows after them still need.
template <int C, int H>
__device__ __forceinline__ void matvec_ip(const double *__restrict__ A, const Lane &L, double2 (&v)[C]) {
  double2 lh[H], rh[H];
#pragma unroll
  for (int q = 0; q < H; q++) {
    const double2 tl = L.full ? v[C - H + q] : v[C - 1 - H + q];
    lh[q] = shfl_up2(tl, 1);
    rh[q] = shfl_down2(v[q], 1);
    if (L.lane == 0) lh[q] = czero();
    if (L.lane >= L.lpm - 1) rh[q] = czero();
  }
  double2 win[H];  // win[q] = original v[t-H+q] (left halo at first)
#pragma unroll
  for (int q = 0; q < H; q++) win[q] = lh[q];
#pragma unroll
  for (int t = 0; t < C; t++) {
    const double2 orig = v[t];
    double2 acc = czero();
    if (t < L.n) {
#pragma unroll
      for (int c = 0; c < 2 * H + 1; c++) {
        const int e = t - H + c;
        double2 u;
        if (c < H) u = win[c];
        else if (c == H) u = orig;
        else if (e < C - 1) u = v[e];
        else if (e == C - 1) u = L.full ? v[C - 1] : rh[0];
        else {
          const int i0 = (e - C < H) ? e - C : H - 1, i1 = (e - C + 1 < H) ? e - C + 1 : H - 1;
          u = L.full ? rh[i0] : rh[i1];
        }
        const double w = tab(A, 2 * H + 1, t, c, L.lane);
        acc.x = fma(w, u.x, acc.x);
        acc.y = fma(w, u.y, acc.y);
      }
    }
#pragma unroll
    for (int q = 0; q < H - 1; q++) win[q] = win[q + 1];
    win[H - 1] = orig;
    v[t] = acc;
  }
}

// ---------------------------------------------------------------------
// Band triangular solves (tables chunk-major, see tab()).
//   lower: x_j -= sum_{d=1..B} Lt[j][d-1] x_{j-d}
//   upper: x_i = (x_i - sum_{d=1..B} Ut[i][d] x_{i+d}) * Ut[i][0]
// Scan tables (constant operators): Ks[(s*32 + lane)*B*B] = the lane's
// composed chunk map at Kogge-Stone step s (row-major B x B).
// ---------------------------------------------------------------------
template <int C, int B>
__device__ __forceinline__ void lrun(double2 (&x)[C], const double *__restrict__ Lt, const Lane &L, double2 (&S)[B],
                                     bool write) {
#pragma unroll
  for (int t = 0; t < C; t++)
    if (t < L.n) {
      double2 v = x[t];
#pragma unroll
      for (int d = 0; d < B; d++) {
        const double c = tab(Lt, B, t, d, L.lane);
        v.x = fma(-c, S[d].x, v.x);
        v.y = fma(-c, S[d].y, v.y);
      }
#pragma unroll
      for (int d = B - 1; d > 0; d--) S[d] = S[d - 1];
      S[0] = v;
      if (write) x[t] = v;
    }
}
template <int C, int B>
__device__ __forceinline__ void urun(double2 (&x)[C], const double *__restrict__ Ut, const Lane &L, double2 (&S)[B],
                                     bool write) {
#pragma unroll
  for (int t = C - 1; t >= 0; t--)
    if (t < L.n) {
      double2 v = x[t];
#pragma unroll
      for (int d = 0; d < B; d++) {
        const double c = tab(Ut, B + 1, t, 1 + d, L.lane);
        v.x = fma(-c, S[d].x, v.x);
        v.y = fma(-c, S[d].y, v.y);
      }
      const double r = tab(Ut, B + 1, t, 0, L.lane);
      v.x *= r;
      v.y *= r;
#pragma unroll
      for (int d = B - 1; d > 0; d--) S[d] = S[d - 1];
      S[0] = v;
      if (write) x[t] = v;
    }
}

// scan of the particular responses with precomputed composed maps
template <int B, bool UP>
__device__ __forceinline__ void scan_const(double2 (&S)[B], const double *__restrict__ Ks, int lane) {
#pragma unroll
  for (int s = 0; s < 5; s++) {
    const int off = 1 << s;
    double2 pp[B];
#pragma unroll
    for (int d = 0; d < B; d++) pp[d] = UP ? shfl_up2(S[d], off) : shfl_down2(S[d], off);
    const bool act = UP ? (lane >= off) : (lane + off < 32);
    if (act) {
      const double *A = Ks + (size_t)(s * 32 + lane) * B * B;
#pragma unroll
      for (int r = 0; r < B; r++) {
#pragma unroll
        for (int q = 0; q < B; q++) {
          const double a = __ldg(A + r * B + q);
          S[r].x = fma(a, pp[q].x, S[r].x);
          S[r].y = fma(a, pp[q].y, S[r].y);
        }
      }
    }
  }
}

template <int C, int B>
__device__ __forceinline__ void lsolve_c(double2 (&x)[C], const double *__restrict__ Lt, const double *__restrict__ Ks,
                                         const Lane &L) {
  double2 S[B];
#pragma unroll
  for (int d = 0; d < B; d++) S[d] = czero();
  lrun<C, B>(x, Lt, L, S, false);
  scan_const<B, true>(S, Ks, L.lane);
#pragma unroll
  for (int d = 0; d < B; d++) {
    S[d] = shfl_up2(S[d], 1);
    if (L.lane == 0) S[d] = czero();
  }
  lrun<C, B>(x, Lt, L, S, true);
}
template <int C, int B>
__device__ __forceinline__ void usolve_c(double2 (&x)[C], const double *__restrict__ Ut, const double *__restrict__ Ks,
                                         const Lane &L) {
  double2 S[B];
#pragma unroll
  for (int d = 0; d < B; d++) S[d] = czero();
  urun<C, B>(x, Ut, L, S, false);
  scan_const<B, false>(S, Ks, L.lane);
#pragma unroll
  for (int d = 0; d < B; d++) {
    S[d] = shfl_down2(S[d], 1);
    if (L.lane == 31) S[d] = czero();
  }
  urun<C, B>(x, Ut, L, S, true);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(LMC_FULL, v, off);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(LMC_FULL, v, off));
  return v;
}

// Warp sums of 12 values at once: two exchanges that halve the values a lane
// holds, then three over its last three (36 shuffles in place of 120).  The
// lanes with (lane & 7) == 0 return the sums of values q0 .. q0+2.
__device__ __forceinline__ int warp_sum12(const double (&a)[12], double (&v)[3]) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, g = lane & 8;
  double b[6];
#pragma unroll
  for (int i = 0; i < 6; i++) {
    const double keep = h ? a[6 + i] : a[i], send = h ? a[i] : a[6 + i];
    b[i] = keep + __shfl_xor_sync(LMC_FULL, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double keep = g ? b[3 + i] : b[i], send = g ? b[i] : b[3 + i];
    v[i] = keep + __shfl_xor_sync(LMC_FULL, send, 8);
  }
#pragma unroll
  for (int off = 4; off > 0; off >>= 1)
#pragma unroll
    for (int i = 0; i < 3; i++) v[i] += __shfl_xor_sync(LMC_FULL, v[i], off);
  return (h ? 6 : 0) + (g ? 3 : 0);
}

#ifdef LMC_FFT_TU
// ---------------------------------------------------------------------
// Register DFTs of compile-time size R (natural order in and out):
// y_k = sum_n x_n exp(SIGN 2 pi i nk/R), recursive mixed radix 4/2/3.
// Twiddles exp(-2 pi i e/R) come from a constant table (c_tw), one block
// per size, filled by the host at initialisation.
// ---------------------------------------------------------------------
constexpr int TW_SIZES[] = {4, 6, 8, 9, 12, 16, 18, 24, 32, 36, 48};
__host__ __device__ constexpr int tw_off(int R) {
  int o = 0;
  for (int q : TW_SIZES) {
    if (q == R) return o;
    o += q;
  }
  return -1;
}
constexpr int TW_TOTAL = tw_off(48) + 48;

static __constant__ double2 c_tw[TW_TOTAL];  // one copy per translation unit
static __constant__ float2 c_twf[TW_TOTAL];  // the same, rounded to FP32

template <int R, int SIGN, typename CT>
__device__ __forceinline__ CT ctw(int e) {
  constexpr int o = tw_off(R);
  static_assert(o >= 0, "register DFT size without twiddles");
  CT w;
  if constexpr (sizeof(CT) == sizeof(double2)) w = c_tw[o + e];
  else w = c_twf[o + e];
  return SIGN > 0 ? cconj(w) : w;
}

template <int R, int SIGN, typename CT>
__device__ __forceinline__ void bfly(CT (&x)[R]) {
  using Re = typename CReal<CT>::R;
  if constexpr (R == 2) {
    const CT a = x[0], b = x[1];
    x[0] = cadd(a, b);
    x[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const CT t0 = cadd(x[0], x[2]), t1 = csub(x[0], x[2]), t2 = cadd(x[1], x[3]);
    const CT d = csub(x[1], x[3]);
    const CT t3 = (SIGN > 0) ? cmk<CT>(-d.y, d.x) : cmk<CT>(d.y, -d.x);  // d * (SIGN i)
    x[0] = cadd(t0, t2);
    x[2] = csub(t0, t2);
    x[1] = cadd(t1, t3);
    x[3] = csub(t1, t3);
  } else if constexpr (R == 3) {
    const Re s3 = (Re)0.86602540378443864676;  // sqrt(3)/2
    const CT t = cadd(x[1], x[2]);
    const CT d = csub(x[1], x[2]);
    const CT u = (SIGN > 0) ? cmk<CT>(-s3 * d.y, s3 * d.x) : cmk<CT>(s3 * d.y, -s3 * d.x);
    const CT a = cmk<CT>(x[0].x - (Re)0.5 * t.x, x[0].y - (Re)0.5 * t.y);
    x[0] = cadd(x[0], t);
    x[1] = cadd(a, u);
    x[2] = csub(a, u);
  }
}

// GAP: the middle third of the samples is zero (and not read); the innermost
// stage, radix 3, takes one sample of each third
template <int R, int SIGN, bool GAP = false, typename CT>
__device__ __forceinline__ void rdft(CT (&x)[R]) {
  static_assert(!GAP || R % 3 == 0, "the gap must be whole samples");
  if constexpr (R == 1) {
    return;
  } else if constexpr (R == 3 && GAP) {
    using Re = typename CReal<CT>::R;
    const Re s3 = (Re)0.86602540378443864676;  // sqrt(3)/2
    const CT c = x[2], a = cmk<CT>(x[0].x - (Re)0.5 * c.x, x[0].y - (Re)0.5 * c.y);
    const CT u = (SIGN > 0) ? cmk<CT>(s3 * c.y, -s3 * c.x) : cmk<CT>(-s3 * c.y, s3 * c.x);
    x[0] = cadd(x[0], c);
    x[1] = cadd(a, u);
    x[2] = csub(a, u);
  } else if constexpr (R == 2 || R == 3 || R == 4) {
    bfly<R, SIGN>(x);
  } else {
    constexpr int p = (R % 4 == 0) ? 4 : ((R % 2 == 0) ? 2 : 3);
    constexpr int m = R / p;
    CT sub[p][m];
#pragma unroll
    for (int r = 0; r < p; r++)
#pragma unroll
      for (int j = 0; j < m; j++) sub[r][j] = x[r + p * j];
#pragma unroll
    for (int r = 0; r < p; r++) rdft<m, SIGN, GAP>(sub[r]);
#pragma unroll
    for (int k = 0; k < m; k++) {
      CT t[p];
#pragma unroll
      for (int r = 0; r < p; r++) t[r] = (r == 0 || k == 0) ? sub[r][k] : cmul(sub[r][k], ctw<R, SIGN, CT>(r * k));
      bfly<p, SIGN>(t);
#pragma unroll
      for (int q = 0; q < p; q++) x[k + m * q] = t[q];
    }
  }
}

// The R = 3 Q samples of a first pass whose middle third is zero (the
// 3/2-rule padding), x[0..Q) and x[2Q..3Q): the radix-3 stage comes first and
// sees (a, 0, c).  Natural order in and out.
template <int R, int SIGN, typename CT>
__device__ __forceinline__ void dft_gap(CT (&x)[R]) {
  constexpr int Q = R / 3;
  using Re = typename CReal<CT>::R;
  const Re s3 = (Re)0.86602540378443864676;
  CT y[3][Q];
#pragma unroll
  for (int j = 0; j < Q; j++) {
    const CT a = x[j], c = x[2 * Q + j];
    const CT t = cmk<CT>(a.x - (Re)0.5 * c.x, a.y - (Re)0.5 * c.y);
    const CT u = (SIGN > 0) ? cmk<CT>(s3 * c.y, -s3 * c.x) : cmk<CT>(-s3 * c.y, s3 * c.x);  // -SIGN i s3 c
    y[0][j] = cadd(a, c);
    y[1][j] = cadd(t, u);
    y[2][j] = csub(t, u);
    if constexpr (Q > 1)
      if (j > 0) {
        y[1][j] = cmul(y[1][j], ctw<R, SIGN, CT>(j));
        y[2][j] = cmul(y[2][j], ctw<R, SIGN, CT>(2 * j));
      }
  }
#pragma unroll
  for (int r = 0; r < 3; r++) {
    rdft<Q, SIGN>(y[r]);
#pragma unroll
    for (int k = 0; k < Q; k++) x[r + 3 * k] = y[r][k];
  }
}
// Its transpose: only the outputs 0..Q-1 (lo) and 2Q..3Q-1 (hi) of an R-point
// DFT, the third that the truncation drops not formed.
template <int R, int SIGN, typename CT>
__device__ __forceinline__ void dft_trunc(const CT (&x)[R], CT (&lo)[R / 3], CT (&hi)[R / 3]) {
  constexpr int Q = R / 3;
  using Re = typename CReal<CT>::R;
  const Re s3 = (Re)0.86602540378443864676;
  CT y[3][Q];
#pragma unroll
  for (int r = 0; r < 3; r++) {
#pragma unroll
    for (int k = 0; k < Q; k++) y[r][k] = x[r + 3 * k];
    rdft<Q, SIGN>(y[r]);
  }
#pragma unroll
  for (int j = 0; j < Q; j++) {
    CT a = y[0][j], b = y[1][j], c = y[2][j];
    if constexpr (Q > 1)
      if (j > 0) {
        b = cmul(b, ctw<R, SIGN, CT>(j));
        c = cmul(c, ctw<R, SIGN, CT>(2 * j));
      }
    const CT t = cadd(b, c), e = csub(b, c);
    lo[j] = cadd(a, t);
    // a + w^2 b + w^4 c with w = exp(SIGN 2 pi i / 3)
    hi[j] = (SIGN > 0) ? cmk<CT>(a.x - (Re)0.5 * t.x + s3 * e.y, a.y - (Re)0.5 * t.y - s3 * e.x)
                       : cmk<CT>(a.x - (Re)0.5 * t.x - s3 * e.y, a.y - (Re)0.5 * t.y + s3 * e.x);
  }
}

// The tasks of a pass: K per line, nb lines, T threads.  With T a multiple of
// K a thread keeps its place in the line from round to round.
template <int K, int T, typename Fn>
__device__ __forceinline__ void line_tasks(int nb, Fn &&fn) {
  if constexpr (T % K == 0) {
    const int q = threadIdx.x % K;
    for (int b = threadIdx.x / K; b < nb; b += T / K) fn(b, q);
  } else {
    for (int idx = threadIdx.x; idx < nb * K; idx += T) fn(idx / K, idx % K);
  }
}

// Transform of nb lines of length N = R1 R2 R3 in shared memory, in passes of
// radix R1, R2, R3 (R3 = 1: two passes; R2 = 1: one), a task of a pass being
// one register DFT.  FP64: small radices, as the two-pass form with radices up
// to 48 needs 130 to 255 registers a thread and leaves 8 to 18 warps on an SM.
//
// FP32 (DIT): two passes, every register DFT by decimation in time (rdft)
// whatever is known to be zero or dropped.  The phi equation weights the FP32
// rounding by k^3, and what the rounded twiddles let through to a mode depends
// on the factors that it passes.  Three passes of small radices with the radix
// 3 of the direct transform last (dft_trunc) are further from 64 bits (phi of
// one pass of 512 x 60 x 512 5.6e-6 after 5.0e-6, of 2-D 256 x 60 4.3e-7 after
// 2.9e-7) and put the largest errors at other modes (1.4e-3 of phi's rms).
//
// The inverse ("inv") takes natural order and leaves X[k1 + R1 k2 + R1 R2 k3]
// at position (k1 R2 + k2) R3 + k3; the direct one ("fwd") is its transpose,
// so the samples are never reordered.  Line b starts at sm + b*ld; position n
// is stored at sk(n), one pad slot per P positions (a multiple of the run of
// the last pass), so that its strided tasks hit different banks.
// tw: exp(-2 pi i n k1 / N) at [k1 M + n], M = R2 R3; exp(-2 pi i n k2 / M) at
// [N + k2 R3 + n]; and at FW the factors of the direct transform's first
// twiddled pass, exp(-2 pi i j k / M) (two passes: / N) of task k at
// [FW + j FS + k]: with the tasks fastest the 16-byte loads of eight lanes are
// one line of the L1 instead of eight, which were a quarter of the L1's cycles
// of the FP64 x stage.
// T: the threads of the block.  Every pass ends with a barrier.
__host__ __device__ constexpr int fft_run(int r1, int r2, int r3) { return r3 > 1 ? r3 : r2 > 1 ? r2 : r1; }
template <int R1, int R2, int R3, typename CT = double2, int T = 1, int P = fft_run(R1, R2, R3)>
struct Fft {
  static constexpr int N = R1 * R2 * R3, M = R2 * R3, Q = R1 / 3;
  static constexpr int RUN = fft_run(R1, R2, R3), PR = P / RUN;  // runs per pad slot
  static constexpr int LD = N + (P < N ? N / P : 0);
  static constexpr int FW = N + M, FS = R3 > 1 ? R2 : R1;
  static constexpr bool DIT = sizeof(CT) == sizeof(float2);
  static_assert(R1 % 3 == 0 || DIT, "the 3/2-rule gap must be whole sample rows of the first pass");
  static_assert(R3 == 1 || !DIT, "FP32: two passes");
  // whether sample n is a low one (n < N/3) or a high one (n > 2N/3)
  __host__ __device__ static constexpr bool low(int n) { return n < N / 3; }
  __host__ __device__ static constexpr bool high(int n) { return n > N / 3 * 2; }
  static_assert(P % RUN == 0 && (P == RUN || M % P == 0), "a pad slot follows whole runs");
  __device__ static __forceinline__ int sk(int n) { return P < N ? n + n / P : n; }
  static constexpr int SM = M + (P < N ? M / P : 0);  // sk(k M + n) = k SM + sk(n)
  // natural index of the sample at position n
  __device__ static __forceinline__ int nat(int n) {
    return n / M + R1 * ((n / R3) % R2) + R1 * R2 * (n % R3);
  }
  // and its step along a run of the last pass
  static constexpr int NS = R3 > 1 ? R1 * R2 : R1;
  template <int SIGN>
  __device__ static __forceinline__ CT twd(const CT *__restrict__ tw, int e) {
    const CT w = __ldg(tw + e);
    return SIGN > 0 ? cconj(w) : w;
  }

  // slot of sample j of a second-pass task, from its first
  __host__ __device__ static constexpr int at2(int j) { return R3 > 1 ? j * R3 + j / PR : j; }
  // first pass of the inverse: mk(b, n1) gives the reader of task n1 of line b,
  // rd(o, up) its sample n1 + o (o a multiple of M) in the low (n < N/3) or the
  // high third (up; n > 2N/3: 2N/3 itself is never asked for); the rest is zero
  template <int SIGN, typename L>
  __device__ static __forceinline__ void inv_p1(CT *sm, int nb, int ld, const CT *__restrict__ tw, L &&mk) {
    line_tasks<M, T>(nb, [&](int b, int n1) {
      const auto rd = mk(b, n1);
      CT x[R1];
      if constexpr (R1 % 3 == 0) {
#pragma unroll
        for (int j = 0; j < R1; j++) {
          if (j < Q) x[j] = rd(M * j, false);
          else if (j > 2 * Q || (j == 2 * Q && n1 > 0)) x[j] = rd(M * j, true);
          else x[j] = cz<CT>();
        }
        if constexpr (DIT) rdft<R1, SIGN, true>(x);
        else dft_gap<R1, SIGN>(x);
      } else {  // the ends of the gap lie inside a row of samples
#pragma unroll
        for (int j = 0; j < R1; j++) {
          if (low(M * j) && low(n1 + M * j)) x[j] = rd(M * j, false);
          else if (high(M * j + M - 1) && high(n1 + M * j)) x[j] = rd(M * j, true);
          else x[j] = cz<CT>();
        }
        rdft<R1, SIGN>(x);
      }
      CT *p = sm + (size_t)b * ld + sk(n1);
      const CT *t = tw + n1;
#pragma unroll
      for (int k = 0; k < R1; k++) p[k * SM] = (k > 0 && M > 1) ? cmul(x[k], twd<SIGN>(t, k * M)) : x[k];
    });
    __syncthreads();
  }
  // second pass of the inverse (of the whole transform if R3 = 1)
  template <int SIGN>
  __device__ static __forceinline__ void inv_p2(CT *sm, int nb, int ld, const CT *__restrict__ tw) {
    if constexpr (R2 > 1) {
      line_tasks<R1 * R3, T>(nb, [&](int b, int q) {
        const int k1 = q / R3, n2 = q % R3;
        CT *p = sm + (size_t)b * ld + k1 * SM + n2;
        const CT *t = tw + N + n2;
        CT x[R2];
#pragma unroll
        for (int j = 0; j < R2; j++) x[j] = p[at2(j)];
        rdft<R2, SIGN>(x);
#pragma unroll
        for (int k = 0; k < R2; k++) {
          CT v = x[k];
          if (k > 0 && R3 > 1) v = cmul(v, twd<SIGN>(t, k * R3));
          p[at2(k)] = v;
        }
      });
      __syncthreads();
    }
  }
  // last of three passes of the inverse
  template <int SIGN>
  __device__ static __forceinline__ void inv_p3(CT *sm, int nb, int ld) {
    if constexpr (R3 > 1) {
      line_tasks<R1 * R2, T>(nb, [&](int b, int q) {
        CT *p = sm + (size_t)b * ld + q * R3 + q / PR;
        CT x[R3];
#pragma unroll
        for (int j = 0; j < R3; j++) x[j] = p[j];
        rdft<R3, SIGN>(x);
#pragma unroll
        for (int j = 0; j < R3; j++) p[j] = x[j];
      });
      __syncthreads();
    }
  }
  // the transposes
  template <int SIGN>
  __device__ static __forceinline__ void fwd_p3(CT *sm, int nb, int ld, const CT *__restrict__ tw) {
    if constexpr (R3 > 1) {
      line_tasks<R1 * R2, T>(nb, [&](int b, int q) {
        CT *p = sm + (size_t)b * ld + q * R3 + q / PR;
        const CT *t = tw + FW + q % FS;
        CT x[R3];
#pragma unroll
        for (int j = 0; j < R3; j++) x[j] = p[j];
        rdft<R3, SIGN>(x);
#pragma unroll
        for (int j = 0; j < R3; j++) p[j] = (j > 0) ? cmul(x[j], twd<SIGN>(t, j * FS)) : x[j];
      });
      __syncthreads();
    }
  }
  template <int SIGN>
  __device__ static __forceinline__ void fwd_p2(CT *sm, int nb, int ld, const CT *__restrict__ tw) {
    if constexpr (R2 > 1) {
      line_tasks<R1 * R3, T>(nb, [&](int b, int q) {
        const int k1 = q / R3, n2 = q % R3;
        CT *p = sm + (size_t)b * ld + k1 * SM + n2;
        const CT *t = R3 > 1 ? tw + k1 * M + n2 : tw + FW + k1;
        CT x[R2];
#pragma unroll
        for (int j = 0; j < R2; j++) x[j] = p[at2(j)];
        rdft<R2, SIGN>(x);
#pragma unroll
        for (int j = 0; j < R2; j++) p[at2(j)] = (R3 > 1 || j > 0) ? cmul(x[j], twd<SIGN>(t, j * (R3 > 1 ? R3 : FS))) : x[j];
      });
      __syncthreads();
    }
  }
  // last pass of the direct transform for one task n1 of a line: outputs n1 +
  // M j, lo for j < Q and hi for j >= 2 Q
  template <int SIGN>
  __device__ static __forceinline__ void fwd_p1(const CT *line, int n1, CT (&lo)[Q], CT (&hi)[Q]) {
    static_assert(R1 % 3 == 0, "whole rows of outputs");
    CT x[R1];
    line += sk(n1);
#pragma unroll
    for (int k = 0; k < R1; k++) x[k] = line[k * SM];
    if constexpr (DIT) {
      rdft<R1, SIGN>(x);
#pragma unroll
      for (int j = 0; j < Q; j++) {
        lo[j] = x[j];
        hi[j] = x[2 * Q + j];
      }
    } else {
      dft_trunc<R1, SIGN>(x, lo, hi);
    }
  }
  // the same: put(o, up, v) takes the output v of index n1 + o in the low or
  // (up) the high third
  template <int SIGN, typename W>
  __device__ static __forceinline__ void fwd_out(const CT *line, int n1, W &&put) {
    if constexpr (R1 % 3 == 0) {
      CT lo[Q], hi[Q];
      fwd_p1<SIGN>(line, n1, lo, hi);
#pragma unroll
      for (int j = 0; j < Q; j++) put(M * j, false, lo[j]);
#pragma unroll
      for (int j = 0; j < Q; j++)
        if (j > 0 || n1 > 0) put(M * (2 * Q + j), true, hi[j]);
    } else {
      CT x[R1];
      line += sk(n1);
#pragma unroll
      for (int k = 0; k < R1; k++) x[k] = line[k * SM];
      rdft<R1, SIGN>(x);
#pragma unroll
      for (int j = 0; j < R1; j++) {
        if (low(M * j) && low(n1 + M * j)) put(M * j, false, x[j]);
        else if (high(M * j + M - 1) && high(n1 + M * j)) put(M * j, true, x[j]);
      }
    }
  }
};

#endif  // LMC_FFT_TU

}  // namespace lmcd
