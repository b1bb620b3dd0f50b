/*
 * sp_inst_many_exact.cu -- many-step 2D kernels (sp_many2.cuh) of the EXACT
 * form, compiled with --fmad=false as sp_inst_exact.cu is.  In FP32 only models
 * A and AMK: in the sums of a 13-point bilaplacian ptxas fuses packed products
 * with adds (see rmul in sp_common.cuh), other ones here than in the one-step
 * kernels, and a run's bits would depend on how it is cut into calls.
 */
#include "sp_launch.cuh"

#define SP_EXACT_MANY(T, DT, L, G, B)                              \
  SP_REGMANY(SPK_A, SPK_EXACT, MF_A_exact, T, DT, L, G, B);        \
  SP_REGMANY(SPK_AMK, SPK_EXACT, MF_AMK_exact, T, DT, L, G, B);
#define SP_EXACT_MANY64(L, G, B)                                   \
  SP_EXACT_MANY(double, 1, L, G, B)                                \
  SP_REGMANY(SPK_B, SPK_EXACT, MF_B_exact, double, 1, L, G, B);    \
  SP_REGMANY(SPK_C, SPK_EXACT, MF_C_exact, double, 1, L, G, B);    \
  SP_REGMANY(SPK_BMK, SPK_EXACT, MF_BMK_exact, double, 1, L, G, B);

namespace sp {
void register_many_exact_kernels() {
  SP_EXACT_MANY64(5, 6, 13)
  SP_EXACT_MANY64(9, 6, 13)
  SP_EXACT_MANY(float, 0, 5, 6, 13)
  SP_EXACT_MANY(float, 0, 9, 6, 13)
}
}  // namespace sp
