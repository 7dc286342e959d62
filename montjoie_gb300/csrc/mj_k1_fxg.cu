// Fixed-point FP64 element kernel (mj_k1_fx.cuh) for any derivative matrix.
#include "mj_k1_fx.cuh"

namespace mj {

int k1_set_gmat_fx_gen(int n, const double* g) { return set_gmat_fx<false>(n, g); }
int k1_prepare_fx_gen(int n, int E, int* ctas) { return prepare_fx<false>(n, E, ctas); }
void k1_launch_fx_gen(mj_op* op, const void* x, cudaStream_t s) { launch_fx<false>(op, x, s); }

}  // namespace mj
