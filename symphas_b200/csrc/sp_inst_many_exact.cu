/*
 * sp_inst_many_exact.cu -- many-step 2D kernels (sp_many2.cuh) of the EXACT
 * form, compiled with --fmad=false as sp_inst_exact.cu is.
 */
#include "sp_launch.cuh"

#define SP_EXACT_MANY(T, DT, L, G, B)                              \
  SP_REGMANY(SPK_A, SPK_EXACT, MF_A_exact, T, DT, L, G, B);        \
  SP_REGMANY(SPK_B, SPK_EXACT, MF_B_exact, T, DT, L, G, B);        \
  SP_REGMANY(SPK_C, SPK_EXACT, MF_C_exact, T, DT, L, G, B);        \
  SP_REGMANY(SPK_AMK, SPK_EXACT, MF_AMK_exact, T, DT, L, G, B);    \
  SP_REGMANY(SPK_BMK, SPK_EXACT, MF_BMK_exact, T, DT, L, G, B);

namespace sp {
void register_many_exact_kernels() {
  SP_EXACT_MANY(double, 1, 5, 6, 13)
  SP_EXACT_MANY(double, 1, 9, 6, 13)
  SP_EXACT_MANY(float, 0, 5, 6, 13)
  SP_EXACT_MANY(float, 0, 9, 6, 13)
}
}  // namespace sp
