// Fixed-point FP64 element kernel (mj_k1_fx.cuh) for derivative matrices that
// are antisymmetric under the mirror, the conversion of the factors, and the
// choice between the two forms.
#include "mj_k1_fx.cuh"

namespace mj {

namespace {

// Factors of every element (6 x Qp doubles) as limbs of B' = 2^(c + kb) B and
// the scale kb (largest row sum of |B'| in [2^61, 2^62); kFxBad when a factor
// is not finite).  One warp per element.
__global__ void k_fixed_factors(const double* __restrict__ fac, int2* __restrict__ fx, int* __restrict__ fexp,
                                int n_elt, int n, int Qp) {
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (e >= n_elt) return;
  const double* f = fac + (size_t)e * 6 * Qp;
  auto c_of = [&](int p) { return fx_c(n, p % n) + fx_c(n, p / n % n) + fx_c(n, p / (n * n)); };
  const int Q = n * n * n;
  double m = 0.0;
  bool fin = true;
  for (int p = lane; p < Q; p += 32) {
    double b[6];
    for (int q = 0; q < 6; q++) {
      b[q] = fabs(f[q * Qp + p]);
      fin = fin && isfinite(b[q]);
    }
    const double r = fmax(fmax(b[0] + b[1] + b[2], b[1] + b[3] + b[4]), b[2] + b[4] + b[5]);
    m = fmax(m, scalbn(r, c_of(p)));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  fin = __all_sync(0xffffffffu, fin) && isfinite(m);
  const int kb = fin && m > 0.0 ? kFxBitsB - ilogb(m) : 0;
  for (int t = lane; t < 6 * Qp; t += 32) {
    const int p = t % Qp;
    fx[(size_t)e * 6 * Qp + t] = fx_limbs(fin && p < Q ? __double2ll_rn(scalbn(f[t], kb + c_of(p))) : 0LL);
  }
  if (lane == 0) fexp[e] = fin ? kb : kFxBad;
}

}  // namespace

// The matrix is in the range of the fixed-point forms; *sym: it is exactly
// antisymmetric under the mirror.
bool k1_fx_supports(int n, const double* g, bool* sym) {
  double m = 0.0;
  *sym = true;
  for (int a = 0; a < n * n; a++) {
    m = std::max(m, std::fabs(g[a]));
    *sym = *sym && g[a] == -g[n * n - 1 - a];
  }
  return m > 1e-60 && m < 1e60;
}

int k1_set_gmat_fx_sym(int n, const double* g) { return set_gmat_fx<true>(n, g); }
int k1_prepare_fx_sym(int n, int E, int* ctas) { return prepare_fx<true>(n, E, ctas); }
void k1_launch_fx_sym(mj_op* op, const void* x, cudaStream_t s) { launch_fx<true>(op, x, s); }

int k1_set_gmat_fx(int n, const double* g, bool sym) {
  return sym ? k1_set_gmat_fx_sym(n, g) : k1_set_gmat_fx_gen(n, g);
}
int k1_prepare_fx(const mj_op* op, int E, int* ctas) {
  return op->fx_sym ? k1_prepare_fx_sym(op->n, E, ctas) : k1_prepare_fx_gen(op->n, E, ctas);
}
void k1_launch_fx(mj_op* op, const void* x, cudaStream_t s) {
  if (op->fx_sym) k1_launch_fx_sym(op, x, s);
  else k1_launch_fx_gen(op, x, s);
}

int k1_fixed_factors(mj_op* op, cudaStream_t s) {
  k_fixed_factors<<<(op->n_elt_pad * 32 + 255) / 256, 256, 0, s>>>(
      op->fac_e.as<double>(), op->fac_fx.as<int2>(), op->fac_exp.as<int>(), op->n_elt_pad, op->n, op->Qp);
  count_launch();
  MJ_CUDA(cudaGetLastError());
  return MJ_OK;
}

}  // namespace mj
