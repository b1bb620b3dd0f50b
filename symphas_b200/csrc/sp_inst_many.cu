/*
 * sp_inst_many.cu -- many-step 2D kernels (sp_many2.cuh) of the FUSED form, for
 * the keys of sp_inst_fused.cu, and the warp-strip 2D step (sp_strip2.cuh) of
 * the FP32 models.  (Models B and C on 9 points: sp_inst_points.cu.)
 */
#include "sp_launch.cuh"

#define SP_FUSED_MANY(T, DT)                                       \
  SP_REGMANY(SPK_A, SPK_FUSED, MF_A_fused, T, DT, 5, 6, 13);       \
  SP_REGMANY(SPK_B, SPK_FUSED, MF_B_fused, T, DT, 5, 6, 13);       \
  SP_REGMANY(SPK_C, SPK_FUSED, MF_C_fused, T, DT, 5, 6, 13);       \
  SP_REGMANY(SPK_AMK, SPK_FUSED, MF_AMK_fused, T, DT, 5, 6, 13);   \
  SP_REGMANY(SPK_BMK, SPK_FUSED, MF_BMK_fused, T, DT, 5, 6, 13);   \
  SP_REGMANY(SPK_A, SPK_FUSED, MF_A_fused, T, DT, 9, 6, 13);

#define SP_STRIP2(MODEL, MF0, MF1) SP_REGSTRIP2(MODEL, MF0, MF1, 3, 1);

namespace sp {
void register_many_kernels() {
  SP_STRIP2(SPK_A, MF_A_fused, MF_A_fused)
  SP_STRIP2(SPK_B, MF_B_fused, MF_B_fused)
  SP_STRIP2(SPK_C, MF_C_fused, MF_C_fused)
  SP_STRIP2(SPK_AMK, MF_AMK_fused, MF_AMK_fused)
  SP_STRIP2(SPK_BMK, MF_BMK_fused, MF_BMK_fused)
  SP_STRIP2(SPK_ENS_AB, MF_AMK_fused, MF_BMK_fused)
  SP_FUSED_MANY(float, 0)
  SP_FUSED_MANY(double, 1)
}
}  // namespace sp
