/*
 * sp_inst_points.cu -- kernels of the FUSED form of models B and C on the 9-
 * and 15-point Laplacians, where bilap is not lap o lap and the key runs the
 * exact term order.  Every contraction is spelled out (SP_EXPLICIT_FMA) and the
 * unit is compiled with --fmad=false: left to the compiler, the one-step kernel,
 * the many-step kernel and the tile shapes contract different products, and the
 * bits of a run would depend on how it is cut into calls.
 */
#define SP_EXPLICIT_FMA
#include "sp_launch.cuh"

#define SP_POINTS(T, DT)                                     \
  SP_REG2(SPK_B, SPK_FUSED, MF_B_exact, T, DT, 9, 6, 13);    \
  SP_REG2(SPK_C, SPK_FUSED, MF_C_exact, T, DT, 9, 6, 13);    \
  SP_REG3(SPK_B, SPK_FUSED, MF_B_exact, T, DT, 15, 10, 25);  \
  SP_REG3(SPK_C, SPK_FUSED, MF_C_exact, T, DT, 15, 10, 25);  \
  SP_REGMANY(SPK_B, SPK_FUSED, MF_B_exact, T, DT, 9, 6, 13); \
  SP_REGMANY(SPK_C, SPK_FUSED, MF_C_exact, T, DT, 9, 6, 13);

namespace sp {
namespace {
// narrow tiles where extents fill 64-wide ones badly: two rows a thread, four
// on larger grids (the conditions of sp_inst_wide.cu)
template <class MF, class TC>
void narrow(int model, int pref, long long from) {
  KernelInfo i = Entry3<MF, float, 15, 10, 25, TC, false>::info();
  i.pref = pref;
  i.pref_filled = 0.79;
  i.pref_sites = from;
  register_kernel(KernelKey{model, SPK_FUSED, 3, 0, 15, 10, 25}, i);
}
template <class MF>
void narrow3(int model) {
  narrow<MF, Tiles<float>::D3n1>(model, 1, 400000);
  narrow<MF, Tiles<float>::D3n2>(model, 2, 1500000);
}
}  // namespace

void register_points_kernels() {
  SP_POINTS(float, 0)
  SP_POINTS(double, 1)
  narrow3<MF_B_exact>(SPK_B);
  narrow3<MF_C_exact>(SPK_C);
}
}  // namespace sp
