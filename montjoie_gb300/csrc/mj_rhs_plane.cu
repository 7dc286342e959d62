// Launches of the plane form of the one-kernel many-source step
// (mj_rhs_plane.cuh), plain and EN.
#include <cuda_runtime.h>

#include <algorithm>

#include "mj_rhs_plane.cuh"

namespace mj {

namespace {

size_t rp_smem(int base, int E, int S, int n, bool en) {
  return (size_t)base + (en ? (size_t)E * S * n * n * sizeof(float) : 0);
}

template <int N, int E, int LB, int V, bool EN>
int prepare(int S, int* ctas) {
  using P = RpPlan<N, E, LB, V>;
  const size_t smem = rp_smem(P::kSmem, E, S, N, EN);
  size_t limit = 0;
  MJ_CUDA(allow_dynamic_smem(k_rhs_plane<N, E, LB, V, EN>, &limit));
  if (smem > limit) return MJ_OK;
  MJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, k_rhs_plane<N, E, LB, V, EN>, P::T, smem));
  return MJ_OK;
}

template <int N, int E, int LB, int V, bool EN, long SPIN = kSpinLimit>
int launch(int grid, const RsParams& prm, const RpParams& x, SyncState* sync, int par, int* err, cudaStream_t s,
           unsigned long long* stamps) {
  using P = RpPlan<N, E, LB, V>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(P::T);
  cfg.dynamicSmemBytes = rp_smem(P::kSmem, E, prm.S, N, EN);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MJ_CUDA(cudaLaunchKernelEx(&cfg, k_rhs_plane<N, E, LB, V, EN, SPIN>, prm, x, sync, par, err, stamps));
  count_launch();
  return MJ_OK;
}

__global__ void k_mark_interior(const int* __restrict__ nodle_e, const int* __restrict__ ptr, long long items, int n,
                                char* __restrict__ flag, int* __restrict__ bad) {
  const int m = n - 2, Qp = elem_slots(n);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < items;
       t += (long long)gridDim.x * blockDim.x) {
    const int q = (int)(t % (m * m * m));
    const long long e = t / (m * m * m);
    const int i = q % m + 1, j = q / m % m + 1, k = q / (m * m) + 1;
    const int d = nodle_e[e * Qp + (k * n + j) * n + i];
    if (ptr[d + 1] - ptr[d] == 1)
      flag[d] = 1;
    else
      *bad = 1;
  }
}

__global__ void k_interior_mass(const int* __restrict__ nodle_e, const float* __restrict__ m, int n_elt,
                                long long items, int n, float* __restrict__ mi) {
  const int I = n - 2, Qp = elem_slots(n), Ip = (I * I * I + 3) / 4 * 4;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < items;
       t += (long long)gridDim.x * blockDim.x) {
    const int q = (int)(t % Ip);
    const long long e = t / Ip;
    const int i = q % I + 1, j = q / I % I + 1, k = q / (I * I) + 1;
    mi[t] = q < I * I * I && e < n_elt ? m[nodle_e[e * Qp + (k * n + j) * n + i]] : 0.f;
  }
}

}  // namespace

const std::vector<RpVariant>& rp_variants() {
  static const std::vector<RpVariant> v = {
#define MJ_X(N_, E_, LB_, V_) {N_, E_, LB_, V_, RpPlan<N_, E_, LB_, V_>::T, RpPlan<N_, E_, LB_, V_>::kHalf},
      MJ_RP_VARIANTS(MJ_X)
#undef MJ_X
  };
  return v;
}

int rp_prepare(int n, int E, int LB, int V, bool en, int S, int* ctas) {
  *ctas = 0;
#define MJ_X(N_, E_, LB_, V_)                                  \
  if (n == N_ && E == E_ && LB == LB_ && V == V_)              \
    return en ? prepare<N_, E_, LB_, V_, true>(S, ctas) : prepare<N_, E_, LB_, V_, false>(S, ctas);
  MJ_RP_VARIANTS(MJ_X)
#undef MJ_X
  set_error("no many-source step variant");
  return MJ_ERR_ARG;
}

int rp_launch(int n, int E, int LB, int V, bool en, int grid, const RsParams& prm, const RpParams& x,
              SyncState* sync, int par, int* err, cudaStream_t s, unsigned long long* stamps) {
  if (k1_waits_run_out() && n == 5 && E == 4 && LB == 8 && V == 1 && !en) {  // the instance with a wait limit of 0
    size_t limit = 0;
    MJ_CUDA(allow_dynamic_smem(k_rhs_plane<5, 4, 8, 1, false, 0>, &limit));
    return launch<5, 4, 8, 1, false, 0>(grid, prm, x, sync, par, err, s, stamps);
  }
#define MJ_X(N_, E_, LB_, V_)                                                                                    \
  if (n == N_ && E == E_ && LB == LB_ && V == V_)                                                                \
    return en ? launch<N_, E_, LB_, V_, true>(grid, prm, x, sync, par, err, s, stamps)            \
              : launch<N_, E_, LB_, V_, false>(grid, prm, x, sync, par, err, s, stamps);
  MJ_RP_VARIANTS(MJ_X)
#undef MJ_X
  set_error("no many-source step variant");
  return MJ_ERR_ARG;
}

int rp_set_gmat(int n, const float* g) {
  MJ_CUDA(cudaMemcpyToSymbol(c_gmat32, g, sizeof(float) * n * n, sizeof(float) * kMaxNK * kMaxNK * n));
  float2 g2[kMaxNK * kMaxNK];
  for (int a = 0; a < n * n; a++) g2[a] = make_float2(g[a], g[a]);
  MJ_CUDA(cudaMemcpyToSymbol(c_gmat32x2, g2, sizeof(float2) * n * n, sizeof(float2) * kMaxNK * kMaxNK * n));
  return MJ_OK;
}

int rp_mark_interior(const int* nodle_e, const int* ptr, int n_elt, int n, char* flag, int* bad, cudaStream_t s) {
  const long long items = (long long)n_elt * (n - 2) * (n - 2) * (n - 2);
  const int blocks = (int)std::min<long long>((items + 255) / 256, 8 * sm_count());
  k_mark_interior<<<blocks, 256, 0, s>>>(nodle_e, ptr, items, n, flag, bad);
  MJ_CUDA(cudaGetLastError());
  return MJ_OK;
}

int rp_interior_mass(const int* nodle_e, const float* m, int n_elt, int n_elt_pad, int n, float* mi, cudaStream_t s) {
  const int I = n - 2;
  const long long items = (long long)n_elt_pad * ((I * I * I + 3) / 4 * 4);
  const int blocks = (int)std::min<long long>((items + 255) / 256, 8 * sm_count());
  k_interior_mass<<<blocks, 256, 0, s>>>(nodle_e, m, n_elt, items, n, mi);
  MJ_CUDA(cudaGetLastError());
  return MJ_OK;
}

}  // namespace mj
