// Fixed-point FP64 element kernel (mj_k1_fx.cuh) for derivative matrices that
// are antisymmetric under the mirror, the conversion of the factors, and the
// choice between the two forms.
#include "mj_k1_fx.cuh"

namespace mj {

namespace {

// Factors of every element (6 x Qp doubles) as limbs of B' = 2^(c + kb) B, and
// fac_exp: kb (largest row sum of |B'| in [2^61, 2^62)) and the weights s_d of
// the contrast rule, the smallest with
//   2^s_d beta x (the least, over the lines along d, of the line's largest B'_dd)
//     >= the largest row sum;
// kFxBad when a factor is not finite, kFxUneven when B'_dd varies by more than
// 2 beta between lines.  beta: 1.25 times what the quadrature weights alone make of
// it.  One warp per element.
__global__ void k_fixed_factors(const double* __restrict__ fac, int2* __restrict__ fx, int* __restrict__ fexp,
                                int n_elt, int n, int Qp, double beta) {
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
  double least[3] = {HUGE_VAL, HUGE_VAL, HUGE_VAL}, most[3] = {0, 0, 0};  // of the lines' largest B'_dd
  for (int l = lane; l < n * n; l += 32)
    for (int d = 0; d < 3; d++) {
      const double* fd = f + (d == 0 ? 0 : d == 1 ? 3 : 5) * Qp;
      const int step = d == 0 ? 1 : d == 1 ? n : n * n;
      const int first = d == 0 ? l * n : d == 1 ? l / n * n * n + l % n : l;
      double b = 0.0;
      for (int a = 0; a < n; a++) b = fmax(b, scalbn(fabs(fd[first + a * step]), c_of(first + a * step)));
      least[d] = fmin(least[d], b);
      most[d] = fmax(most[d], b);
    }
  for (int o = 16; o > 0; o >>= 1) {
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    for (int d = 0; d < 3; d++) {
      least[d] = fmin(least[d], __shfl_xor_sync(0xffffffffu, least[d], o));
      most[d] = fmax(most[d], __shfl_xor_sync(0xffffffffu, most[d], o));
    }
  }
  fin = __all_sync(0xffffffffu, fin) && isfinite(m);
  const int kb = fin && m > 0.0 ? kFxBitsB - ilogb(m) : 0;
  for (int t = lane; t < 6 * Qp; t += 32) {
    const int p = t % Qp;
    fx[(size_t)e * 6 * Qp + t] = fx_limbs(fin && p < Q ? __double2ll_rn(scalbn(f[t], kb + c_of(p))) : 0LL);
  }
  if (lane) return;
  int out = kb * 4096;
  bool even = true;
  if (m > 0.0)
    for (int d = 0; d < 3; d++) {
      even = even && most[d] <= 2.0 * beta * least[d];
      int s = 0;
      while (s < 15 && scalbn(beta * least[d], s) < m) s++;
      out |= s << 4 * d;
    }
  fexp[e] = !fin ? kFxBad : even ? out : kFxUneven;
}

// beta of k_fixed_factors: of the weights w 2^c, (largest / smallest)^2 over a
// line's cross-section, and a quarter more.
double fx_beta(int n) {
  double pts[kMaxN], w[kMaxN], lo = HUGE_VAL, hi = 0.0;
  gauss_lobatto(n - 1, pts, w);
  for (int i = 0; i < n; i++) {
    const double v = std::ldexp(w[i], fx_c(n, i));
    lo = std::min(lo, v);
    hi = std::max(hi, v);
  }
  return 1.25 * (hi / lo) * (hi / lo);
}

}  // namespace

// The matrix is one for the fixed-point forms: within 1% (of its largest
// entry) of the Gauss-Lobatto one times a constant, which the contrast rule
// holds for; *sym: it is exactly antisymmetric under the mirror.
bool k1_fx_supports(int n, const double* g, bool* sym) {
  double pts[kMaxN], w[kMaxN], gl[kMaxN * kMaxN], m = 0.0;
  gauss_lobatto(n - 1, pts, w);
  gl_derivative_matrix(n - 1, pts, gl);
  *sym = true;
  for (int a = 0; a < n * n; a++) {
    m = std::max(m, std::fabs(g[a]));
    *sym = *sym && g[a] == -g[n * n - 1 - a];
  }
  const double scale = g[0] / gl[0];
  if (!(m > 1e-60 && m < 1e60) || !std::isfinite(scale)) return false;
  for (int a = 0; a < n * n; a++)
    if (!(std::fabs(g[a] - scale * gl[a]) <= 0.01 * m)) return false;
  return true;
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
// The instance with a bulk-copy wait limit of 0: order 4, 5 elements per CTA.
bool k1_launch_fx_waits_out(mj_op* op, const void* x, cudaStream_t s) {
  if (op->n != 5 || op->E != 5 || !op->fx_sym) return false;
  using P = FxPlan<5, 5>;
  auto* k = k_local_stiffness_fx<5, 5, true, 0>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P::total) != cudaSuccess) return false;
  k<<<op->grid_k1, P::threads, P::total, s>>>(static_cast<const double*>(x), op->nodle_e.as<int>(),
                                              op->fac_fx.as<int2>(), op->fac_exp.as<int>(), op->fac_e.as<double>(),
                                              op->R.as<double>(), op->slot_e.as<int>(), op->n_tiles,
                                              op->err.as<int>());
  return true;
}
void k1_launch_fx(mj_op* op, const void* x, cudaStream_t s) {
  if (op->fx_sym) k1_launch_fx_sym(op, x, s);
  else k1_launch_fx_gen(op, x, s);
}

int k1_fixed_factors(mj_op* op, cudaStream_t s) {
  k_fixed_factors<<<(op->n_elt_pad * 32 + 255) / 256, 256, 0, s>>>(
      op->fac_e.as<double>(), op->fac_fx.as<int2>(), op->fac_exp.as<int>(), op->n_elt_pad, op->n, op->Qp, fx_beta(op->n));
  count_launch();
  MJ_CUDA(cudaGetLastError());
  return MJ_OK;
}

}  // namespace mj
