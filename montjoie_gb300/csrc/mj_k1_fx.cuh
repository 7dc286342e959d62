// FP64 element kernel in two-limb fixed point: the same element product as
// k_local_stiffness<double> (mj_k1.cuh), its contractions and factor products
// carried out with 32 x 32 -> 64 bit integer multiply-adds.
//
// Why: a GB300 SM issues 2 FP64 multiply-adds per clock and 32 wide integer
// ones (IMAD.WIDE; both measured), and one 61 x 62 bit product takes three of
// the latter and a short one, so products run several times faster in
// integers.  The FP64 kernel is bound by its FP64 pipe (91% busy).
//
// Numbers.  Every quantity of an element is an integer with one power-of-two
// scale per element, used as two signed 32-bit limbs v = hi 2^32 + lo
// (|lo| <= 2^31), so that every partial product is a signed 32 x 32 one:
//   u : scaled by the element's largest |u| to |u| < 2^60
//   G : the derivative matrix, sums of |G| over a (of the gradient's
//       coefficients G[a][l] and of the divergence's G'[l][a]) < 2^62
//   B': the factors, row sums |B'_a.| < 2^62 over the element, converted when
//       the factors are set (k_fixed_factors)
//   v : the fluxes, shifted by the element's largest |g| to |v| < 2^60
// Point (i, j, k) carries the factor 2^(c_i + c_j + c_k), c from fx_c: B' = 2^c B,
// G'[l][a] = 2^(c_l - c_a) G[l][a], result = 2^-c y.  c roughly undoes the
// quadrature weights, which fall by up to 2^4 per axis towards the faces and
// would otherwise leave few bits there.
// A sum of products keeps hi*hi in one 64-bit accumulator (h) and hi*lo + lo*hi
// in another (m); lo*lo enters m with its upper bits.  Bounds, n = 9 worst:
//   g = sum G u     <= 2^61    h < 2^60, m < 2^62.8
//   v = sum B' g    <= 2^60    h < 2^59, m < 2^62.4
//   y = 3 sums G' v <= 2^62.6  h < 2^60, m < 2^62.8
// so no accumulator overflows for any input in range.
//
// Which elements.  With its one scale per element a value 2^-k below the largest
// keeps 60 - k bits where FP64 keeps 53, and the matrix spends several of the
// 7 to spare (its entries span 2^4.7 at Q4, 2^7 at Q8).  FP64's own error at a
// point hangs on the largest |u| on the three lines through it, each weighted
// by its direction's factor; here the fluxes' unit, which follows the
// element's largest gradient, decides.  So an element takes one scale only if
// that maximum is nowhere more than 2^max(1, sv + X) below the element's
// largest |u|: sv, the bits by which the gradients are below their bound, is
// high (5 to 13) for smooth fields and 1 to 3 for spikes; X = fx_contrast.
// Within this the product is as close to the exact one as FP64's (restated in
// exact integers, 177,000 elements with random, smooth and line-, edge- and
// face-dominated fields, cubic, stretched, curved and skewed: 34 further off in
// relative L2, by at most 3.1 times, nearly all on stretched elements; largest
// error of an entry over its absolute sum in units of 2^-53, in 99.9% of the
// elements and at most: Q4 3.2 and 11, FP64 6.4; Q8 13 and 20, FP64 11; the
// bound of FP64 arithmetic is 16 and 24).  Without it a field that peaks at a
// vertex lost up to 87 times in L2.
// All other elements (spikes, the numerical tail ahead of a front; factors that
// vary by more than 2.5 along an element, which is known when they are
// converted) are computed beside the others of the tile: from Q3 up line by line
// in integers, each line with a scale of its own (fx_lines), at Q1 and Q2 in the
// FP64 arithmetic of k_local_stiffness (fx_exact).  An element out of range (a
// NaN or infinity in u or B, or scales that may leave the normal range) always
// takes the latter.  The choice hangs on the element alone, not on the tile it
// is in.  Of smooth waves 2.5 elements long or more, fewer than 0.04% of the
// elements are chosen.  One such element keeps its tile for 2 us at Q4 and 7 us
// at Q8; spikes everywhere take 43 us per product at 16^3 Q4 (FP64-pipe kernel
// 61, dense field 20), 171 at 15x13x11 Q8 (237, 65).  A run from rest has tails
// in most elements until its waves fill the mesh; in its first hundreds of steps
// a step takes (us; FP64-pipe kernel, dense field) Q4 40^3 460 (610, 178), Q8
// 15^3 264 (366, 102), Q6 24^3 370 (504, 154), Q3 45^3 313 (369, 126), Q2 60^3
// 383 (319, 133), Q1 100^3 374 (354, 170).
//
// Measured (us per launch, FP64-pipe kernel at its best tile -> this kernel):
// Q4 16^3 60 -> 16, 64^3 2300 -> 597; Q8 32^3 3150 -> 750; Q6 40^3 2575 -> 588;
// Q1 64^3 94 -> 41.  What bounds it now (ncu, Q4 48^3): the integer multiply
// pipe (60% busy) behind 16 to 20 warps per SM, which shared memory (the factor
// stage) and registers allow; DRAM is at half of its rate.  Without the lo*lo
// term it takes 15% less and errs up to 3 times more than the FP64 kernel on
// steep fields; with the mirror symmetry it takes 25% less than in the general
// form.
//
// Layout: E elements per CTA, E*n*n threads.  A thread owns a z-line in the
// gather, the z-contractions, the factor products and the result, and an
// x-line and a y-line in the other contractions, whose n results it computes
// from n values held in registers.  So each value crosses shared memory once
// per contraction instead of n times, and no matrix entries are kept in
// registers.  Factors arrive by bulk copy in one stage (free after the factor
// products, refilled during the divergence), Nodle in two; the next tile's u
// is gathered during the divergence and its largest exponent found there too.
//
// SYM: G is antisymmetric under the mirror (a, l) -> (n-1-a, n-1-l), as the
// Gauss-Lobatto matrix is.  Then with e_a = r_a + r_(n-1-a), o_a = r_a - r_(n-1-a)
//   y_l = Q_l + P_l, y_(n-1-l) = Q_l - P_l,  P_l = sum Me e_a, Q_l = sum Mo o_a
// and a line takes n^2/2 products instead of n^2.  A matrix handed in with
// other rounding takes the general form (SYM false, n^2 products).
#pragma once

#include <climits>
#include <cmath>
#include <vector>

#include "mj_internal.cuh"
#include "mj_k1.cuh"

namespace mj {
namespace {

// fac_exp of an element: the scale kb of its factors << 12 | s_z << 8 | s_y << 4 | s_x, s_d the factors' weight of
// direction d against the largest, as a power of two downwards; kFxBad: not finite; kFxUneven: too uneven for one scale.
constexpr int kFxBad = INT_MIN, kFxUneven = INT_MIN + 1;

// Coefficients of the line transforms of every order as (lo, hi, lo >> 17),
// and their scales.  [n][0]: gradient, y_l = sum_a G[a][l] r_a; [n][1]:
// divergence, y_l = sum_a G'[l][a] r_a.  SYM: row l < (n+1)/2 holds Me at
// a < n/2, the middle coefficient at a = n/2 (n odd) and Mo_a at n-1-a;
// general: the matrix.
__constant__ int4 c_fx[kMaxNK + 1][2][kMaxNK * kMaxNK];
__constant__ int2 c_fx_exp[kMaxNK + 1];  // both scales

// Exponent of the similarity scaling at node i of n (see above).
__host__ __device__ constexpr int fx_c(int n, int i) {
  const int d = i < n - 1 - i ? i : n - 1 - i;  // distance from the nearer end
  return d == 0 ? (n == 2 ? 0 : n <= 6 ? 2 : 3) : d == 1 && n >= 6 ? 1 : 0;
}

// X of the contrast rule (see above).
__host__ __device__ constexpr int fx_contrast(int n) {
  return n <= 4 ? 3 - n : n == 5 ? -1 : n <= 7 ? -2 : -3;
}

__device__ __forceinline__ int2 fx_limbs(long long v) {
  const int lo = (int)v;
  return make_int2(lo, (int)(v >> 32) + (int)((unsigned)lo >> 31));
}

// One sum of products, value = h 2^64 + m 2^32, lo*lo to its upper bits in q
// (units of 2^35; at most 9 terms of 2^27).  The wide multiply-adds are
// written out: from 64-bit C++ products the compiler makes about three times
// as many instructions.
struct FxSum {
  long long h, m;
  int q;
  __device__ __forceinline__ FxSum(int2 a, int ahi, int2 b, int bhi) {
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(h) : "r"(a.y), "r"(b.y));
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(m) : "r"(a.y), "r"(b.x));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(m) : "r"(a.x), "r"(b.y));
    q = ahi * bhi;
  }
  __device__ __forceinline__ void mad(int2 a, int ahi, int2 b, int bhi) {
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(h) : "r"(a.y), "r"(b.y));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(m) : "r"(a.y), "r"(b.x));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(m) : "r"(a.x), "r"(b.y));
    q += ahi * bhi;
  }
  // value / 2^(64 - sh), rounded
  __device__ __forceinline__ long long norm(int sh) const {
    long long t;
    asm("mad.wide.s32 %0, %1, 8, %2;" : "=l"(t) : "r"(q), "l"(m));
    return (h << sh) + ((t + (1LL << (31 - sh))) >> (32 - sh));
  }
};
constexpr int kFxLoData = 18, kFxLoCoef = 17;  // lo*lo: (lo >> 18) (lo >> 17) in units of 2^35

constexpr int kFxShG = 3, kFxShY = 3;
constexpr int kFxBitsU = 59, kFxBitsB = 61, kFxBitsG = 61;  // the largest value (sum) in [2^bits, 2^(bits+1))
// y_int = y 2^(c + ku + kb + kg - kFxYBias + sv), sv the shift of the fluxes
constexpr int kFxYBias = (64 - kFxShG) + 64 + (64 - kFxShY);

// One line transform (KIND 0: gradient, 1: divergence).
template <int N, int KIND, bool SYM>
__device__ __forceinline__ void fx_line(const long long (&r)[N], long long (&y)[N]) {
  constexpr int SH = KIND ? kFxShY : kFxShG;
  const int4* c = c_fx[N][KIND];
  auto coef = [&](int at, int2& v, int& hi) {
    const int4 q = c[at];
    v = make_int2(q.x, q.y);
    hi = q.z;
  };
  int2 v;
  int vh;
  if constexpr (SYM) {
    constexpr int H = N / 2, C = N & 1;
    int2 e[H + C], o[H];
    int eh[H + C], oh[H];
#pragma unroll
    for (int a = 0; a < H; a++) {
      e[a] = fx_limbs(r[a] + r[N - 1 - a]);
      o[a] = fx_limbs(r[a] - r[N - 1 - a]);
      eh[a] = e[a].x >> kFxLoData;
      oh[a] = o[a].x >> kFxLoData;
    }
    if (C) {
      e[H] = fx_limbs(r[H]);
      eh[H] = e[H].x >> kFxLoData;
    }
#pragma unroll
    for (int l = 0; l < H + C; l++) {
      coef(l * N + N - 1, v, vh);
      FxSum q(o[0], oh[0], v, vh);
#pragma unroll
      for (int a = 1; a < H; a++) {
        coef(l * N + N - 1 - a, v, vh);
        q.mad(o[a], oh[a], v, vh);
      }
      if (l == H) {  // the middle of an odd line
        y[l] = q.norm(SH);
      } else {
        coef(l * N, v, vh);
        FxSum p(e[0], eh[0], v, vh);
#pragma unroll
        for (int a = 1; a < H + C; a++) {
          coef(l * N + a, v, vh);
          p.mad(e[a], eh[a], v, vh);
        }
        const long long pn = p.norm(SH), qn = q.norm(SH);
        y[l] = qn + pn;
        y[N - 1 - l] = qn - pn;
      }
    }
  } else {
    int2 e[N];
    int eh[N];
#pragma unroll
    for (int a = 0; a < N; a++) {
      e[a] = fx_limbs(r[a]);
      eh[a] = e[a].x >> kFxLoData;
    }
#pragma unroll
    for (int l = 0; l < N; l++) {
      coef(l * N, v, vh);
      FxSum q(e[0], eh[0], v, vh);
#pragma unroll
      for (int a = 1; a < N; a++) {
        coef(l * N + a, v, vh);
        q.mad(e[a], eh[a], v, vh);
      }
      y[l] = q.norm(SH);
    }
  }
}

// Least registers of a thread: at Q1 and Q2 shared memory admits so many CTAs
// that the kernel would spill (us per launch at the registers of all the CTAs
// -> these: Q1 100^3 172 -> 148, Q2 30^3 19.3 -> 17.9, 50^3 67.1 both).
constexpr int fx_regs(int n, int E) { return n == 2 ? 80 : n == 3 ? (E <= 12 ? 96 : 72) : 48; }

template <int N, int E>
struct FxPlan {
  static constexpr int NN = N * N;
  static constexpr int Qp = elem_slots(N);
  static constexpr int RS = N | 1;  // x-lines start an odd number of 8-byte words apart: no bank conflicts
  static constexpr int W = NN * RS;  // work entries per element and array
  static constexpr size_t fac_bytes = sizeof(int2) * 6 * E * Qp;
  static constexpr size_t nod_bytes = sizeof(int) * E * Qp;
  static constexpr size_t work_bytes = ((sizeof(long long) * 3 * E * W + 15) / 16) * 16;
  static constexpr size_t max_bytes = ((sizeof(unsigned) * 4 * E + 15) / 16) * 16;
  static constexpr size_t max_at = fac_bytes + 2 * nod_bytes + work_bytes;
  static constexpr size_t total = max_at + max_bytes + 3 * sizeof(uint64_t);
  static constexpr int threads = E * NN;
  // CTAs per SM that shared memory (228 KB per SM, 1 KB of it per CTA) and fx_regs admit: the register budget
  static constexpr int by_smem = (int)(228 * 1024 / (total + 1024));
  static constexpr int by_regs = 65536 / ((threads + 31) / 32 * 32 * fx_regs(N, E));
  static constexpr int ctas = by_smem < by_regs ? by_smem : by_regs;
  static_assert(fac_bytes % 16 == 0 && nod_bytes % 16 == 0, "bulk copies");
};

// The elements of a tile out of range (s_mode 4) in FP64, the arithmetic of
// k_local_stiffness<double> (compact), their u staged as doubles in s_u;
// scratch: the factor stage, free.  The whole CTA works on their points,
// whichever threads own them: the FP64 pipe takes 16 clocks per warp
// instruction whatever its active lanes, so the points are dealt densely (by
// their element's own threads, 25 or 81 in 2 or 4 warps, one element of a tile
// took 7 us at Q4 and 22 at Q8, dealt so 2 and 13).
template <int N, int E>
__device__ __noinline__ void fx_exact(const double* s_u, double* s_a, double* s_b, const int* s_mode, double* scratch,
                                      const double* __restrict__ fac, double* __restrict__ R,
                                      const int* __restrict__ slot) {
  using P = FxPlan<N, E>;
  constexpr int NN = P::NN, Q = N * NN, Qp = P::Qp, RS = P::RS, W = P::W;
  static_assert(sizeof(double) * E * W + sizeof(int) * E <= P::fac_bytes, "z-fluxes and the list fit the factor stage");
  const double* __restrict__ G = c_gmat64[N];
  int* list = reinterpret_cast<int*>(scratch + E * W);
  int count = 0;
  for (int e = 0; e < E; e++)
    if (s_mode[e] & 4) {
      if (threadIdx.x == 0) list[count] = e;
      count++;
    }
  __syncthreads();
  if (!count) return;
  for (int q = threadIdx.x; q < count * Q; q += P::threads) {
    const int el = list[q / Q], p = q % Q, k = p / NN, ij = p % NN, j = ij / N, i = ij % N;
    const double *rx = s_u + el * W + (k * N + j) * RS, *ry = s_u + el * W + k * N * RS + i;
    const double* rz = s_u + el * W + j * RS + i;
    double gx = 0, gy = 0, gz = 0;
#pragma unroll
    for (int a = 0; a < N; a++) {
      gx += G[a * N + i] * rx[a];
      gy += G[a * N + j] * ry[a * RS];
      gz += G[a * N + k] * rz[a * N * RS];
    }
    const double* f = fac + (size_t)el * 6 * Qp + p;
    const double bxx = f[0], bxy = f[Qp], bxz = f[2 * Qp], byy = f[3 * Qp], byz = f[4 * Qp], bzz = f[5 * Qp];
    const int at = el * W + (k * N + j) * RS + i;
    s_a[at] = fac_dot(bxx, gx, bxy, gy, bxz, gz);
    s_b[at] = fac_dot(bxy, gx, byy, gy, byz, gz);
    scratch[at] = fac_dot(bxz, gx, byz, gy, bzz, gz);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < count * Q; q += P::threads) {
    const int el = list[q / Q], p = q % Q, k = p / NN, ij = p % NN, j = ij / N, i = ij % N;
    const double *rx = s_a + el * W + (k * N + j) * RS, *ry = s_b + el * W + k * N * RS + i;
    const double* rz = scratch + el * W + j * RS + i;
    double y = 0;
#pragma unroll
    for (int a = 0; a < N; a++) {
      y += G[i * N + a] * rx[a];
      y += G[j * N + a] * ry[a * RS];
      y += G[k * N + a] * rz[a * N * RS];
    }
    R[slot[(size_t)el * Qp + p]] = y;
  }
}

// r 2^(59 - e + 1023 + c), truncated: e is at least r's biased exponent + c.
__device__ __forceinline__ long long fx_from_double(double r, int c, int e) {
  const int hi = __double2hiint(r);
  const unsigned mh = (hi & 0xfffff) | ((hi & 0x7ff00000) ? 0x100000 : 0);
  const unsigned long long m = ((unsigned long long)mh << 32 | (unsigned)__double2loint(r)) << (kFxBitsU - 52);
  const long long v = (long long)(m >> min(e - c - max(hi >> 20 & 0x7ff, 1), 63));
  return hi < 0 ? -v : v;
}

// y 2^s, rounded; below the normal range 0.
__device__ __forceinline__ double fx_to_double(long long y, int s) {
  const double d = __ll2double_rn(y);
  const int hi = __double2hiint(d), t = (hi >> 20 & 0x7ff) + s;
  if (y == 0 || t <= 0) return 0.0;
  return t >= 2047 ? copysign(HUGE_VAL, d) : __hiloint2double(hi + s * (1 << 20), __double2loint(d));
}

// A range of global memory (16-byte aligned, a multiple of 16 bytes) into L2.
__device__ __forceinline__ void fx_prefetch(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// One line of doubles transformed in integers, scaled by its own largest value.
template <int N, int KIND, bool SYM>
__device__ __forceinline__ void fx_own_line(const double* in, double* out, int step) {
  double r[N];
  int e = 1;
#pragma unroll
  for (int a = 0; a < N; a++) {
    r[a] = in[a * step];
    e = max(e, max(__double2hiint(r[a]) >> 20 & 0x7ff, 1) + (KIND ? fx_c(N, a) : 0));
  }
  long long v[N], y[N];
#pragma unroll
  for (int a = 0; a < N; a++) v[a] = fx_from_double(r[a], KIND ? fx_c(N, a) : 0, e);
  fx_line<N, KIND, SYM>(v, y);
  const int s = 64 - (KIND ? kFxShY : kFxShG) - kFxBitsU + e - 1023 - (KIND ? c_fx_exp[N].y : c_fx_exp[N].x);
#pragma unroll
  for (int a = 0; a < N; a++) out[a * step] = fx_to_double(y[a], s - (KIND ? fx_c(N, a) : 0));
}

// Orders whose elements outside the contrast rule are transformed line by line:
// 17 FP64 operations per point (the factor rows, six conversions, two sums)
// where FP64 takes 6 n + 9.  At Q1 and Q2 that saves little or nothing, and
// FP64's two or three terms round less than the stages do.
template <int N>
constexpr bool kFxLines = N >= 4;

// The elements of a tile outside the contrast rule (s_mode 2 and not 4): their
// line transforms in integers with a scale for every line, the gradients and
// fluxes doubles in between, the factor rows in FP64.  Rounded once per stage
// it needs no rule: over fields and factors that vary by up to 2^40 within an
// element, entries are closer to the exact product than FP64's (largest error
// over the absolute sum in units of 2^-53, 99% of 96,000 elements: Q1 2.7, FP64
// 2.9; Q4 2.9 and 4.9; Q8 3.4 and 7.6), on the tails ahead of a front too (Q4
// 2.0 and 3.3, Q8 2.1 and 4.8).  Arguments and work distribution as fx_exact.
template <int N, int E, bool SYM>
__device__ __noinline__ void fx_lines(const double* s_u, double* s_a, double* s_b, const int* s_mode, double* scratch,
                                      const double* __restrict__ fac, double* __restrict__ R,
                                      const int* __restrict__ slot) {
  using P = FxPlan<N, E>;
  constexpr int NN = P::NN, Q = N * NN, Qp = P::Qp, RS = P::RS, W = P::W;
  int* list = reinterpret_cast<int*>(scratch + E * W);
  int count = 0;
  for (int e = 0; e < E; e++)
    if ((s_mode[e] & 6) == 2) {
      if (threadIdx.x == 0) list[count] = e;
      count++;
    }
  __syncthreads();
  if (!count) return;
  for (int q = threadIdx.x; q < count * 3 * NN; q += P::threads) {
    const int l = q % NN, d = q / NN % 3, el = list[q / (3 * NN)];
    const int at = el * W + (d == 0 ? l * RS : d == 1 ? l / N * N * RS + l % N : l / N * RS + l % N);
    fx_own_line<N, 0, SYM>(s_u + at, (d == 0 ? s_a : d == 1 ? s_b : scratch) + at,
                           d == 0 ? 1 : d == 1 ? RS : N * RS);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < count * Q; q += P::threads) {
    const int p = q % Q, el = list[q / Q], at = el * W + p / N * RS + p % N;
    const double* f = fac + (size_t)el * 6 * Qp + p;
    const double gx = s_a[at], gy = s_b[at], gz = scratch[at];
    const double bxx = f[0], bxy = f[Qp], bxz = f[2 * Qp], byy = f[3 * Qp], byz = f[4 * Qp], bzz = f[5 * Qp];
    s_a[at] = fac_dot(bxx, gx, bxy, gy, bxz, gz);
    s_b[at] = fac_dot(bxy, gx, byy, gy, byz, gz);
    scratch[at] = fac_dot(bxz, gx, byz, gy, bzz, gz);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < count * 3 * NN; q += P::threads) {
    const int l = q % NN, d = q / NN % 3, el = list[q / (3 * NN)];
    const int at = el * W + (d == 0 ? l * RS : d == 1 ? l / N * N * RS + l % N : l / N * RS + l % N);
    double* v = (d == 0 ? s_a : d == 1 ? s_b : scratch) + at;
    fx_own_line<N, 1, SYM>(v, v, d == 0 ? 1 : d == 1 ? RS : N * RS);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < count * Q; q += P::threads) {
    const int p = q % Q, el = list[q / Q], at = el * W + p / N * RS + p % N;
    R[slot[(size_t)el * Qp + p]] = s_a[at] + s_b[at] + scratch[at];
  }
}

// The contrast rule for the elements of a tile with a thread that is bad (its
// element is out of range) or whose z-line lies low; every thread of the CTA
// calls it, u staged as integers in s_u; scratch: 2 N^2 words per element.
// um: the element's largest |u| (high word), shift: the exponent of the rule.
// s_mode: 2 not by one scale, 4 in FP64.  True: 2 for this thread's element.
template <int N, int E>
__device__ __noinline__ bool fx_choose(const long long* s_u, unsigned* scratch, int* s_mode, bool bad, bool low,
                                       unsigned um, int xp, int shift, int ij) {
  using P = FxPlan<N, E>;
  constexpr int NN = P::NN, RS = P::RS, W = P::W;
  const int el = threadIdx.x / NN, j = ij / N, i = ij - j * N;
  if (bad || low) atomicOr(&s_mode[el], bad ? 6 : xp == kFxUneven ? 2 : 1);
  __syncthreads();
  const bool look = s_mode[el] == 1;
  unsigned* line = scratch + el * 2 * NN;  // largest |u| of the x-lines, then of the y-lines
  unsigned zm = 0u;
  auto mag = [&](int at) {
    const int hi = (int)(s_u[el * W + at] >> 32);
    return (unsigned)(hi ^ (hi >> 31));
  };
  if (look) {
    unsigned xm = 0u, ym = 0u;
#pragma unroll 1
    for (int a = 0; a < N; a++) {
      xm = max(xm, mag(ij * RS + a));
      ym = max(ym, mag((ij / N * N + a) * RS + ij % N));
      zm = max(zm, mag((a * N + j) * RS + i));
    }
    line[ij] = xm >> (xp & 15);
    line[NN + ij] = ym >> (xp >> 4 & 15);
    zm >>= xp >> 8 & 15;
  }
  __syncthreads();
  if (look) {
    const unsigned least = (((um & 0xfffffu) | 0x100000u) << (kFxBitsU - 52)) >> shift;
    bool out = false;
#pragma unroll 1
    for (int k = 0; k < N; k++) out |= max(max(line[k * N + j], line[NN + k * N + i]), zm) < least;
    if (out) atomicOr(&s_mode[el], 2);
  }
  __syncthreads();
  return s_mode[el] & 2;
}

template <int N, int E, bool SYM, long SPIN = kSpinLimit>
__global__ void __launch_bounds__(E* N* N, FxPlan<N, E>::ctas)
    k_local_stiffness_fx(const double* __restrict__ x, const int* __restrict__ nodle_e,
                         const int2* __restrict__ fac_fx, const int* __restrict__ fac_exp,
                         const double* __restrict__ fac_e, double* __restrict__ R, const int* __restrict__ slot_e,
                         int n_tiles, int* __restrict__ err) {
  dependent_wait();
  using P = FxPlan<N, E>;
  constexpr int NN = P::NN, Qp = P::Qp, RS = P::RS, W = P::W;
  extern __shared__ __align__(128) unsigned char smem[];
  int2* s_fac = reinterpret_cast<int2*>(smem);
  auto s_nod = [&](int st) { return reinterpret_cast<int*>(smem + P::fac_bytes + st * P::nod_bytes); };
  long long* s_u = reinterpret_cast<long long*>(smem + P::fac_bytes + 2 * P::nod_bytes);  // [el][k][j][i], rows of RS
  long long* s_a = s_u + E * W;
  long long* s_b = s_a + E * W;
  unsigned* s_max = reinterpret_cast<unsigned*>(smem + P::max_at);  // [2][E]: largest |u| (high word) of the tile's and
  unsigned* s_gmax = s_max + 2 * E;                                 // the next tile's elements; [E]: largest |g|
  int* s_mode = reinterpret_cast<int*>(s_max + 3 * E);  // [E]: 1: a z-line lies low, 2: not by one scale, 4: in FP64
  // bar[0], bar[1]: the Nodle stages; bar[2]: the factor stage
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + P::max_at + P::max_bytes);

  const int t = threadIdx.x;
  const int el = t / NN;
  const int ij = t - el * NN;
  const int j = ij / N;
  const int i = ij - j * N;
  const int lz = el * W + j * RS + i;          // + k*N*RS: the points of z-line (i, j)
  const int lx = el * W + ij * RS;             // + a: x-line (k, j) = (ij / N, ij % N)
  const int ly = el * W + j * N * RS + i;      // + a*RS: y-line (k, i) = (ij / N, ij % N)
  const int pe = el * Qp + ij;

  if (t == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init(&bar[2], 1);
    fence_mbar_init();
  }
  for (int q = t; q < 4 * E; q += P::threads) s_max[q] = 0u;
  __syncthreads();
  auto issue_nod = [&](int st, int tile) {
    if (t == 0 && tile < n_tiles) {
      mbar_expect_tx(&bar[st], (uint32_t)P::nod_bytes);
      bulk_g2s_hint(s_nod(st), nodle_e + (size_t)tile * E * Qp, (uint32_t)P::nod_bytes, &bar[st],
                    l2_evict_first_policy());
    }
  };
  auto issue_fac = [&](int tile) {
    if (t == 0 && tile < n_tiles) {
      mbar_expect_tx(&bar[2], (uint32_t)P::fac_bytes);
      bulk_g2s_hint(s_fac, fac_fx + (size_t)tile * E * 6 * Qp, (uint32_t)P::fac_bytes, &bar[2],
                    l2_evict_first_policy());
    }
  };
  const int g = gridDim.x;
  int tile = blockIdx.x;
  issue_nod(0, tile);
  issue_fac(tile);
  issue_nod(1, tile + g);
  uint32_t ph = 0u;  // bits 0, 1: parity of the next completion of Nodle stage 0, 1; bit 2: of the factor stage
  double u[N];
  unsigned zm = 0u;
  // zm: largest high word of |u| over the thread's line (nonzero for any nonzero u); into the element's maximum
  auto line_max = [&](int par) {
    zm = 0u;
#pragma unroll
    for (int k = 0; k < N; k++)
      zm = max(zm, ((unsigned)__double2hiint(u[k]) & 0x7fffffffu) | (__double2loint(u[k]) != 0 ? 1u : 0u));
    atomicMax(&s_max[par * E + el], zm);
  };
  if (tile < n_tiles) {
    const bool ok = mbar_wait_bounded<SPIN>(&bar[0], 0u);
    if (__syncthreads_or(!ok)) {
      if (t == 0) {  // report; every copy issued above may still be in flight
        atomicExch(err, 1);
        mbar_wait_drain(&bar[0], 0u);
        mbar_wait_drain(&bar[2], 0u);
        if (tile + g < n_tiles) mbar_wait_drain(&bar[1], 0u);
      }
      return;
    }
    ph ^= 1u;
    const int* nd = s_nod(0) + pe;
#pragma unroll
    for (int k = 0; k < N; k++) u[k] = ld_fresh(x + nd[k * NN]);
    line_max(0);
  }
  __syncthreads();
  const int kg = c_fx_exp[N].x + c_fx_exp[N].y;
  for (int it = 0; tile < n_tiles; tile += g, ++it) {
    const int s = it & 1;
    // the element's scales: u 2^ku, B 2^kb, result 2^eo
    const unsigned um = s_max[s * E + el];
    const int xp = __ldg(fac_exp + (size_t)tile * E + el);
    const int eu = (int)(um >> 20) - 1023;
    const int ku = um ? kFxBitsU - eu : 0;
    const int eo = kFxYBias - ku - (xp <= kFxUneven ? 0 : xp >> 12) - kg;
    const bool bad = xp == kFxBad || (um && (eu > 1023 || eu < -900 || eo < -950 || eo > 1000));
    // this thread's z-line below the element's largest |u|, weighted, in units of 2^-20 of a power of two
    const int below = xp == kFxUneven ? INT_MAX : (int)min(um - zm + ((xp >> 8 & 15u) << 20), 0x7fffffffu);
    long long uz[N];
    {
      const double sc = __hiloint2double((1023 + (bad ? 0 : ku)) << 20, 0);
#pragma unroll
      for (int k = 0; k < N; k++) {
        uz[k] = __double2ll_rn(u[k] * sc);
        s_u[lz + k * N * RS] = uz[k];
      }
    }
    __syncthreads();  // u staged, the maxima read
    long long gz[N];
    {
      long long r[N], y[N];
#pragma unroll
      for (int a = 0; a < N; a++) r[a] = s_u[lx + a];
      unsigned gm = 0u;  // largest high word of |g|, one unit low for negative values
      auto top = [&](const long long (&v)[N]) {
#pragma unroll
        for (int a = 0; a < N; a++) {
          const int hi = (int)(v[a] >> 32);
          gm = max(gm, (unsigned)(hi ^ (hi >> 31)));
        }
      };
      fx_line<N, 0, SYM>(r, y);
      top(y);
#pragma unroll
      for (int a = 0; a < N; a++) s_a[lx + a] = y[a];
#pragma unroll
      for (int a = 0; a < N; a++) r[a] = s_u[ly + a * RS];
      fx_line<N, 0, SYM>(r, y);
      top(y);
#pragma unroll
      for (int a = 0; a < N; a++) s_b[ly + a * RS] = y[a];
      fx_line<N, 0, SYM>(uz, gz);
      top(gz);
      atomicMax(&s_gmax[el], gm);
    }
    {  // this tile's factors (the vote is also the barrier after the gradients)
      const bool ok = mbar_wait_bounded<SPIN>(&bar[2], (ph >> 2) & 1u);
      if (__syncthreads_or(!ok)) {
        if (t == 0) {  // report; this tile's factors and the next tile's Nodle may be in flight
          atomicExch(err, 1);
          mbar_wait_drain(&bar[2], (ph >> 2) & 1u);
          if (tile + g < n_tiles) mbar_wait_drain(&bar[s ^ 1], (ph >> (s ^ 1)) & 1u);
        }
        return;
      }
      ph ^= 4u;
    }
    long long vz[N];
    // |g| < 2^(64 - lz) with lz >= 2 leading zeros: |v| < 2^62 2^(64 - lz) / 2^(64 - sv) <= 2^60
    const int sv = min(31, __clz((int)s_gmax[el]) - 2);
    {
      const int2* f = s_fac + el * 6 * Qp + ij;
#pragma unroll
      for (int k = 0; k < N; k++) {
        const int2 gx = fx_limbs(s_a[lz + k * N * RS]), gy = fx_limbs(s_b[lz + k * N * RS]), gk = fx_limbs(gz[k]);
        const int gxh = gx.x >> kFxLoData, gyh = gy.x >> kFxLoData, gkh = gk.x >> kFxLoData;
        const int2* fk = f + k * NN;
        const int2 bxx = fk[0], bxy = fk[Qp], bxz = fk[2 * Qp];
        const int2 byy = fk[3 * Qp], byz = fk[4 * Qp], bzz = fk[5 * Qp];
        const int xyh = bxy.x >> kFxLoCoef, xzh = bxz.x >> kFxLoCoef, yzh = byz.x >> kFxLoCoef;
        FxSum a(gx, gxh, bxx, bxx.x >> kFxLoCoef), b(gx, gxh, bxy, xyh), c(gx, gxh, bxz, xzh);
        a.mad(gy, gyh, bxy, xyh); a.mad(gk, gkh, bxz, xzh);
        b.mad(gy, gyh, byy, byy.x >> kFxLoCoef); b.mad(gk, gkh, byz, yzh);
        c.mad(gy, gyh, byz, yzh); c.mad(gk, gkh, bzz, bzz.x >> kFxLoCoef);
        s_a[lz + k * N * RS] = a.norm(sv);
        s_b[lz + k * N * RS] = b.norm(sv);
        vz[k] = c.norm(sv);
      }
    }
    bool apart = false;  // this thread's element not by one scale
    const int shift = max(1, sv + fx_contrast(N));
    if (__syncthreads_or(bad || below > shift << 20)) {  // also: the factor stage is free, the fluxes are staged
      apart = fx_choose<N, E>(s_u, reinterpret_cast<unsigned*>(s_fac), s_mode, bad, below > shift << 20,
                              s_max[s * E + el], __ldg(fac_exp + (size_t)tile * E + el), shift, ij);
      if (__syncthreads_or(apart)) {
        if (apart) {
          if (ij == 0) {  // read by plain loads in a moment (40^3 Q4 from rest 485 -> 460 us per step, Q8 15^3 290 -> 264)
            fx_prefetch(fac_e + ((size_t)tile * E + el) * 6 * Qp, 6 * Qp * sizeof(double));
            fx_prefetch(slot_e + ((size_t)tile * E + el) * Qp, Qp * sizeof(int));
          }
          bool wide = !kFxLines<N> || eu > 900;  // gradients that may overflow, values that may leave the normal range
#pragma unroll
          for (int k = 0; k < N; k++) {
            s_u[lz + k * N * RS] = __double_as_longlong(u[k]);
            wide |= u[k] != 0.0 && ((unsigned)__double2hiint(u[k]) & 0x7fffffffu) < ((1023u - 960u) << 20);
          }
          if (wide) atomicOr(&s_mode[el], 4);
        }
        __syncthreads();
        double *du = reinterpret_cast<double*>(s_u), *da = reinterpret_cast<double*>(s_a);
        double *db = reinterpret_cast<double*>(s_b), *dz = reinterpret_cast<double*>(s_fac);
        const double* f = fac_e + (size_t)tile * E * 6 * Qp;
        const int* st = slot_e + (size_t)tile * E * Qp;
        if constexpr (kFxLines<N>) {
          fx_lines<N, E, SYM>(du, da, db, s_mode, dz, f, R, st);
          __syncthreads();
        }
        fx_exact<N, E>(du, da, db, s_mode, dz, f, R, st);
        __syncthreads();  // the factor stage and the work arrays are free
      }
      if (t < E) s_mode[t] = 0;
    }
    if (t < E) s_max[s * E + t] = 0u;
    if (t < E) s_gmax[t] = 0u;
    if (t == 0) fence_proxy_async();
    issue_fac(tile + g);  // the next tile's factors, during this divergence

    // gather of the next tile's u, in flight during the divergence
    const int nt = tile + g;
    bool lost = false;
    if (nt < n_tiles) {
      const int so = s ^ 1;
      lost = !mbar_wait_bounded<SPIN>(&bar[so], (ph >> so) & 1u);
      ph ^= 1u << so;
      if (!lost) {
        const int* nd = s_nod(so) + pe;
#pragma unroll
        for (int k = 0; k < N; k++) u[k] = ld_fresh(x + nd[k * NN]);
      }
    }
    long long wz[N];
    if (!apart) {
      long long r[N], y[N];
#pragma unroll
      for (int a = 0; a < N; a++) r[a] = s_a[lx + a];
      fx_line<N, 1, SYM>(r, y);
#pragma unroll
      for (int a = 0; a < N; a++) s_a[lx + a] = y[a];
#pragma unroll
      for (int a = 0; a < N; a++) r[a] = s_b[ly + a * RS];
      fx_line<N, 1, SYM>(r, y);
#pragma unroll
      for (int a = 0; a < N; a++) s_b[ly + a * RS] = y[a];
      fx_line<N, 1, SYM>(vz, wz);
    }
    if (nt < n_tiles && !lost) line_max(s ^ 1);
    if (__syncthreads_or(lost)) {
      if (t == 0) {  // report; Nodle stage s^1 and the factors just issued may be in flight
        atomicExch(err, 1);
        mbar_wait_drain(&bar[s ^ 1], ((ph >> (s ^ 1)) & 1u) ^ 1u);
        mbar_wait_drain(&bar[2], (ph >> 2) & 1u);
      }
      return;
    }
    if (t == 0) fence_proxy_async();
    issue_nod(s, tile + 2 * g);
    if (!apart) {
      const int ex = 1023 + (um ? eo - sv : 9) - fx_c(N, i) - fx_c(N, j);
      const int* st = slot_e + ((size_t)tile * E + el) * Qp + ij;
#pragma unroll
      for (int k = 0; k < N; k++) {
        const long long y = wz[k] + s_a[lz + k * N * RS] + s_b[lz + k * N * RS];
        R[__ldg(st + k * NN)] = __ll2double_rn(y) * __hiloint2double((ex - fx_c(N, k)) << 20, 0);
      }
    }
  }
}

// (n, E): the tile sizes of k1_tile_candidates
#define MJ_FX_VARIANTS(X) \
  X(2, 30) X(2, 60) X(3, 12) X(3, 24) X(4, 8) X(4, 16) X(5, 4) X(5, 5) X(5, 8) X(5, 10) \
  X(6, 3) X(6, 4) X(6, 6) X(7, 2) X(7, 3) X(7, 4) X(7, 5) X(8, 2) X(8, 3) X(8, 4) X(9, 1) X(9, 2) X(9, 3)

template <int N, int E, bool SYM>
int prepare_fx_one(int* ctas) {
  using P = FxPlan<N, E>;
  int dev = 0, optin = 0;
  MJ_CUDA(cudaGetDevice(&dev));
  MJ_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  if ((int)P::total > optin) {
    set_error("element kernel variant does not fit in shared memory");
    return MJ_ERR_ARG;
  }
  MJ_CUDA(cudaFuncSetAttribute(k_local_stiffness_fx<N, E, SYM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)P::total));
  MJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, k_local_stiffness_fx<N, E, SYM>, P::threads, P::total));
  if (*ctas < 1) {
    set_error("element kernel variant cannot be resident");
    return MJ_ERR_ARG;
  }
  return MJ_OK;
}

template <bool SYM>
int prepare_fx(int n, int E, int* ctas) {
#define MJ_X(NV, EV) \
  if (n == NV && E == EV) return prepare_fx_one<NV, EV, SYM>(ctas);
  MJ_FX_VARIANTS(MJ_X)
#undef MJ_X
  set_error("no fixed-point element kernel variant for this order and tile size");
  return MJ_ERR_ARG;
}

template <bool SYM>
void launch_fx(mj_op* op, const void* x, cudaStream_t s) {
#define MJ_X(NV, EV)                                                                                          \
  if (op->n == NV && op->E == EV) {                                                                           \
    launch_dependent(                                                                                         \
        k_local_stiffness_fx<NV, EV, SYM>, op->grid_k1, FxPlan<NV, EV>::threads, FxPlan<NV, EV>::total, s,    \
        static_cast<const double*>(x), op->nodle_e.as<int>(), op->fac_fx.as<int2>(), op->fac_exp.as<int>(),   \
        op->fac_e.as<double>(), op->R.as<double>(), op->slot_e.as<int>(), op->n_tiles, op->err.as<int>());    \
    return;                                                                                                   \
  }
  MJ_FX_VARIANTS(MJ_X)
#undef MJ_X
}
#undef MJ_FX_VARIANTS

// Coefficients of order n into this unit's constant memory.
template <bool SYM>
int set_gmat_fx(int n, const double* g) {
  // gradient y_l = sum_a G[a][l] r_a and divergence y_l = sum_a 2^(c_l - c_a) G[l][a] r_a
  auto coef = [&](int kind, int a, int l) {
    return kind ? std::ldexp(g[l * n + a], fx_c(n, l) - fx_c(n, a)) : g[a * n + l];
  };
  int4 v[2][kMaxNK * kMaxNK] = {};
  int k[2];
  for (int kind = 0; kind < 2; kind++) {
    double m = 0.0;  // largest sum of |coefficients|
    for (int l = 0; l < n; l++) {
      double t = 0.0;
      for (int a = 0; a < n; a++) t += std::fabs(coef(kind, a, l));
      m = std::max(m, t);
    }
    const int kg = kFxBitsG - std::ilogb(m);
    k[kind] = kg;
    auto M = [&](int a, int l) { return std::llrint(std::ldexp(coef(kind, a, l), kg)); };
    auto put = [&](int at, long long x) {
      const int lo = (int)(x & 0xffffffffLL);
      v[kind][at] = make_int4(lo, (int)((x - lo) / 4294967296LL), lo >> kFxLoCoef, 0);
    };
    if (!SYM) {
      for (int l = 0; l < n; l++)
        for (int a = 0; a < n; a++) put(l * n + a, M(a, l));
      continue;
    }
    for (int l = 0; l < (n + 1) / 2; l++) {
      for (int a = 0; a < n / 2; a++) {
        const long long p = M(a, l), q = M(n - 1 - a, l);  // r_a = (e + o) / 2, r_(n-1-a) = (e - o) / 2
        put(l * n + a, (p + q) / 2);
        put(l * n + n - 1 - a, (p - q) / 2);
      }
      if ((n & 1) && l != n / 2) put(l * n + n / 2, M(n / 2, l));
    }
  }
  const size_t per = sizeof(v);
  MJ_CUDA(cudaMemcpyToSymbol(c_fx, v, per, per * n));
  MJ_CUDA(cudaMemcpyToSymbol(c_fx_exp, k, sizeof(int2), sizeof(int2) * n));
  MJ_CUDA(cudaMemcpyToSymbol(c_gmat64, g, sizeof(double) * n * n, sizeof(double) * kMaxNK * kMaxNK * n));
  return MJ_OK;
}

}  // namespace
}  // namespace mj
