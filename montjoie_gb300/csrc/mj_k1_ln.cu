// FP32 element kernel, line-owner layout: the product of k_local_stiffness
// (mj_k1.cuh), term for term and in its order of additions, so the same bits.
//
// A thread owns a z-line (i, j) in the gather, the z-contractions, the factor
// products and the divergence, and an x-line and a y-line (k, .) in the
// gradient: it reads the line's n values once, computes its n derivatives with
// the matrix entries as constant-bank operands, and writes them back.  Per
// point and pass that is 15 + 2 n shared-memory accesses, where the layouts in
// which a thread computes the gradients of its own points take 9 + 4 n (45 at
// Q8, 29 at Q4) and are bound by the shared-memory pipe (Q8: 75% busy at 56%
// of the measured copy bandwidth); and a tile takes three block barriers.
// (Line-owned divergences too, 21 accesses, took Q8 to 152 us, but add each
// point's terms in another order than every other element kernel.)  It stays
// bound by the shared-memory pipe, 70% busy at 20 warps per SM (ncu, Q8 24^3).
// The factors have one stage, refilled during the divergence; Nodle has two.
#include "mj_internal.cuh"
#include "mj_k1.cuh"

namespace mj {
namespace {

template <int N, int E>
struct LnPlan {
  static constexpr int NN = N * N;
  static constexpr int Qp = elem_slots(N);
  static constexpr int RS = N | 1;   // x-lines start an odd number of words apart: no bank conflicts
  static constexpr int W = NN * RS;  // work entries per element and array
  static constexpr size_t fac_bytes = sizeof(float) * 6 * E * Qp;
  static constexpr size_t nod_bytes = sizeof(int) * E * Qp;
  static constexpr size_t work_bytes = ((sizeof(float) * 3 * E * W + 15) / 16) * 16;
  static constexpr size_t total = fac_bytes + 2 * nod_bytes + work_bytes + 3 * sizeof(uint64_t);
  static constexpr int threads = E * NN;
  static constexpr int warps = (threads + 31) / 32;
  // CTAs per SM: what shared memory (228 KB, 1 KB of it per CTA) and the 32 resident CTAs admit, with a floor on the
  // registers of a thread
  static constexpr int by_smem = (int)(228 * 1024 / (total + 1024));
  static constexpr int by_regs = 65536 / (warps * 32 * 72);
  static constexpr int lim = by_smem < 32 ? by_smem : 32;
  static constexpr int ctas = lim < by_regs ? lim : by_regs;
  static_assert(fac_bytes % 16 == 0 && nod_bytes % 16 == 0, "bulk copies");
};

// y_l = sum_a G[a][l] r_a
template <int N>
__device__ __forceinline__ void grad_line(const float (&r)[N], float (&y)[N]) {
#pragma unroll
  for (int l = 0; l < N; l++) {
    float s = 0;
#pragma unroll
    for (int a = 0; a < N; a++) s += c_gmat32[N][a * N + l] * r[a];
    y[l] = s;
  }
}

template <int N, int E, long SPIN = kSpinLimit>
__global__ void __launch_bounds__(E* N* N, LnPlan<N, E>::ctas)
    k_local_stiffness_ln(const float* __restrict__ x, const int* __restrict__ nodle_e,
                         const float* __restrict__ fac_e, float* __restrict__ R, const int* __restrict__ slot_e,
                         int n_tiles, int* __restrict__ err) {
  dependent_wait();
  using P = LnPlan<N, E>;
  constexpr int NN = P::NN, Qp = P::Qp, RS = P::RS, W = P::W;
  extern __shared__ __align__(128) unsigned char smem[];
  float* s_fac = reinterpret_cast<float*>(smem);
  auto s_nod = [&](int st) { return reinterpret_cast<int*>(smem + P::fac_bytes + st * P::nod_bytes); };
  float* s_u = reinterpret_cast<float*>(smem + P::fac_bytes + 2 * P::nod_bytes);  // [el][k][j][i], rows of RS
  float* s_a = s_u + E * W;
  float* s_b = s_a + E * W;
  // bar[0], bar[1]: the Nodle stages; bar[2]: the factor stage
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + P::fac_bytes + 2 * P::nod_bytes + P::work_bytes);

  const int t = threadIdx.x;
  const int el = t / NN;
  const int ij = t - el * NN;
  const int j = ij / N;
  const int i = ij - j * N;
  const int lz = el * W + j * RS + i;      // + k*N*RS: the points of z-line (i, j)
  const int lx = el * W + ij * RS;         // + a: x-line (k, j) = (ij / N, ij % N)
  const int ly = el * W + j * N * RS + i;  // + a*RS: y-line (k, i) = (ij / N, ij % N)
  const int ox = el * W + j * RS;          // + k*N*RS + a: x-line of the points (., j, k)
  const int oy = el * W + i;               // + k*N*RS + a*RS: y-line of the points (i, ., k)
  const int pe = el * Qp + ij;
  float gri[N], grj[N];
#pragma unroll
  for (int a = 0; a < N; a++) {
    gri[a] = c_gmat32[N][i * N + a];
    grj[a] = c_gmat32[N][j * N + a];
  }

  if (t == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init(&bar[2], 1);
    fence_mbar_init();
  }
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
      bulk_g2s_hint(s_fac, fac_e + (size_t)tile * E * 6 * Qp, (uint32_t)P::fac_bytes, &bar[2],
                    l2_evict_first_policy());
    }
  };
  const int g = gridDim.x;
  int tile = blockIdx.x;
  issue_nod(0, tile);
  issue_fac(tile);
  issue_nod(1, tile + g);
  uint32_t ph = 0u;  // bits 0, 1: parity of the next completion of Nodle stage 0, 1; bit 2: of the factor stage
  float u[N];
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
  }
  bool lost = false;  // the wait for this tile's Nodle (done during the previous tile) ran out
  for (int it = 0; tile < n_tiles; tile += g, ++it) {
    const int s = it & 1;
#pragma unroll
    for (int k = 0; k < N; k++) s_u[lz + k * N * RS] = u[k];
    // u staged; every thread is past the previous tile's divergence and past the gather of this tile's u
    if (__syncthreads_or(lost)) {
      if (t == 0) {  // report; this tile's Nodle (parity before the flip below), the next tile's and the factors
        atomicExch(err, 1);
        mbar_wait_drain(&bar[s], ((ph >> s) & 1u) ^ 1u);
        if (tile + g < n_tiles) mbar_wait_drain(&bar[s ^ 1], (ph >> (s ^ 1)) & 1u);
        mbar_wait_drain(&bar[2], (ph >> 2) & 1u);
      }
      return;
    }
    if (t == 0) fence_proxy_async();
    issue_nod(s, tile + 2 * g);
    float z[N];       // along z: gradient, then flux
    {
      float r[N], y[N];
#pragma unroll
      for (int a = 0; a < N; a++) r[a] = s_u[lx + a];
      grad_line<N>(r, y);
#pragma unroll
      for (int a = 0; a < N; a++) s_a[lx + a] = y[a];
#pragma unroll
      for (int a = 0; a < N; a++) r[a] = s_u[ly + a * RS];
      grad_line<N>(r, y);
#pragma unroll
      for (int a = 0; a < N; a++) s_b[ly + a * RS] = y[a];
      grad_line<N>(u, z);
    }
    {  // this tile's factors (the vote is also the barrier after the gradients)
      const bool ok = mbar_wait_bounded<SPIN>(&bar[2], (ph >> 2) & 1u);
      if (__syncthreads_or(!ok)) {
        if (t == 0) {  // report; this tile's factors and the Nodle of the next two tiles may be in flight
          atomicExch(err, 1);
          mbar_wait_drain(&bar[2], (ph >> 2) & 1u);
          if (tile + g < n_tiles) mbar_wait_drain(&bar[s ^ 1], (ph >> (s ^ 1)) & 1u);
          if (tile + 2 * g < n_tiles) mbar_wait_drain(&bar[s], (ph >> s) & 1u);
        }
        return;
      }
      ph ^= 4u;
    }
    const float* f = s_fac + el * 6 * Qp + ij;
#pragma unroll
    for (int k = 0; k < N; k++) {
      const float gx = s_a[lz + k * N * RS], gy = s_b[lz + k * N * RS], gz = z[k];
      const float* fk = f + k * NN;
      const float bxx = fk[0], bxy = fk[Qp], bxz = fk[2 * Qp];
      const float byy = fk[3 * Qp], byz = fk[4 * Qp], bzz = fk[5 * Qp];
      s_a[lz + k * N * RS] = fac_dot(bxx, gx, bxy, gy, bxz, gz);
      s_b[lz + k * N * RS] = fac_dot(bxy, gx, byy, gy, byz, gz);
      z[k] = fac_dot(bxz, gx, byz, gy, bzz, gz);
    }
    __syncthreads();  // the factor stage is free, the fluxes are staged
    if (t == 0) fence_proxy_async();
    issue_fac(tile + g);  // the next tile's factors, during this divergence

    // gather of the next tile's u, in flight during the divergence
    const int nt = tile + g;
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
    const int* st = slot_e + ((size_t)tile * E + el) * Qp + ij;
#pragma unroll
    for (int k = 0; k < N; k++) {
      float y = 0;
#pragma unroll
      for (int a = 0; a < N; a++) {
        y += gri[a] * s_a[ox + k * N * RS + a];
        y += grj[a] * s_b[oy + k * N * RS + a * RS];
        y += c_gmat32[N][k * N + a] * z[a];
      }
      R[__ldg(st + k * NN)] = y;
    }
  }
}

// (n, E).  Compiled for the orders where it is the fastest layout (us per
// launch, best other layout -> this one): Q8 32^3 195 -> 174, Q7 24^3 51 -> 48.
// At Q6 (40^3) it measured 162 against 162, at Q5 47 against 44, at Q4 (64^3)
// 234 against 213.
#define MJ_LN_VARIANTS(X) X(8, 1) X(8, 2) X(9, 1) X(9, 2)

template <int N, int E>
int prepare_ln_one(int* ctas) {
  using P = LnPlan<N, E>;
  MJ_CUDA(cudaFuncSetAttribute(k_local_stiffness_ln<N, E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)P::total));
  MJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, k_local_stiffness_ln<N, E>, P::threads, P::total));
  if (*ctas < 1) {
    set_error("element kernel variant cannot be resident");
    return MJ_ERR_ARG;
  }
  return MJ_OK;
}

}  // namespace

std::vector<int> k1_ln_tile_candidates(int n) {
  std::vector<int> e;
#define MJ_X(NV, EV) \
  if (n == NV) e.push_back(EV);
  MJ_LN_VARIANTS(MJ_X)
#undef MJ_X
  return e;
}

// The derivative matrix of order n in this unit's constant bank.
int k1_set_gmat_ln(int n, const double* g) {
  float v[kMaxNK * kMaxNK];
  for (int a = 0; a < n * n; a++) v[a] = float(g[a]);
  MJ_CUDA(cudaMemcpyToSymbol(c_gmat32, v, sizeof(float) * n * n, sizeof(float) * kMaxNK * kMaxNK * n));
  return MJ_OK;
}

int k1_prepare_ln_f32(int n, int E, int* ctas) {
#define MJ_X(NV, EV) \
  if (n == NV && E == EV) return prepare_ln_one<NV, EV>(ctas);
  MJ_LN_VARIANTS(MJ_X)
#undef MJ_X
  set_error("no line-owner element kernel variant for this order and tile size");
  return MJ_ERR_ARG;
}

// The instance with a bulk-copy wait limit of 0: order 7, 2 elements per CTA.
bool k1_launch_ln_f32_waits_out(int n, int E, int grid, const void* x, const int* nodle_e, const void* fac_e, void* R,
                                const int* slot_e, int n_tiles, int* err, cudaStream_t s) {
  if (n != 8 || E != 2) return false;
  using P = LnPlan<8, 2>;
  auto* k = k_local_stiffness_ln<8, 2, 0>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P::total) != cudaSuccess) return false;
  k<<<grid, P::threads, P::total, s>>>(static_cast<const float*>(x), nodle_e, static_cast<const float*>(fac_e),
                                       static_cast<float*>(R), slot_e, n_tiles, err);
  return true;
}

void k1_launch_ln_f32(int n, int E, int grid, const void* x, const int* nodle_e, const void* fac_e, void* R,
                      const int* slot_e, int n_tiles, int* err, cudaStream_t s) {
#define MJ_X(NV, EV)                                                                                             \
  if (n == NV && E == EV) {                                                                                      \
    launch_dependent(k_local_stiffness_ln<NV, EV>, grid, LnPlan<NV, EV>::threads, LnPlan<NV, EV>::total, s,                   \
        static_cast<const float*>(x), nodle_e, static_cast<const float*>(fac_e), static_cast<float*>(R), slot_e, \
        n_tiles, err);                                                                                           \
    return;                                                                                                      \
  }
  MJ_LN_VARIANTS(MJ_X)
#undef MJ_X
}

}  // namespace mj
