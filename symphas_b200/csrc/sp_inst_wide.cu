/*
 * sp_inst_wide.cu -- FP32 fused-form kernels with four x-sites per thread
 * (16-byte shared-memory words, two packed FP32x2 instructions per
 * operation).  They evaluate every site exactly as the two-site kernels do
 * and share their field layout, so they are further tile shapes for
 * sp_autotune (registered after the fused set, in their own translation unit
 * so that the build compiles them in parallel), together with the row kernels
 * of the conserved pattern (sp_chrow.cuh) and of any fused 7-point model
 * (sp_row.cuh).
 */
#include "sp_launch.cuh"

// Which shape sp_create starts with, from timing every shape on 48^3 .. 256^3 and
// ragged grids (us a step, default 64 x 16 x 4 against the preferred one):
//   rows of 256 or 128: the row kernels         B 256^3 51.2, 38.5; C 128^3 18.3, 12.8
//   whole groups of four, wider than 64: four sites a thread, 128-wide tiles
//                                               A 200^3 23.0, 17.7; B 100^3 10.7, 8.7
//   whole groups of four, up to 64: 64-wide     B 64^3 4.5, 4.2; A 48^3 3.0, 2.7
//   extents that fill 64-wide tiles badly: 32-wide tiles
//                                               A 75 x 120 x 60 12.3, 8.6; C 150 x 131 x 97 22.0, 17.1
struct Pref {
  int pref = 0, x = 1, xmin = 0;
  double filled = 1.0;
  long long sites = 0;
};
#define SP_WIDE2(MODEL, MF0, MF1)                                                   \
  SP_REG2T(MODEL, SPK_FUSED, MF0, MF1, float, 0, 5, 6, 13, ::sp::Tiles<float>::D2w1); \
  SP_REG2T(MODEL, SPK_FUSED, MF0, MF1, float, 0, 5, 6, 13, ::sp::Tiles<float>::D2w2); \
  SP_REG2T(MODEL, SPK_FUSED, MF0, MF1, float, 0, 5, 6, 13, ::sp::Tiles<float>::D2w3); \
  SP_REG2T(MODEL, SPK_FUSED, MF0, MF1, float, 0, 5, 6, 13, ::sp::Tiles<float>::D2d);  \
  SP_REG2T(MODEL, SPK_FUSED, MF0, MF1, float, 0, 5, 6, 13, ::sp::Tiles<float>::D2e);

namespace sp {
namespace {
KernelInfo with(KernelInfo i, const Pref& p) {
  i.pref = p.pref;
  i.pref_x = p.x;
  i.pref_xmin = p.xmin;
  i.pref_filled = p.filled;
  i.pref_sites = p.sites;
  return i;
}
template <class MF, class TC, int L = 7>
void tile(int model, const Pref& p = {}) {
  register_kernel(KernelKey{model, SPK_FUSED, 3, 0, L, 10, 25},
                  with(Entry3<MF, float, L, 10, 25, TC, false>::info(), p));
}
// the four-site shapes: `best` of them is preferred beyond 64 columns
template <class MF>
void wide3(int model, int best) {
  using T = Tiles<float>;
  const Pref w{2, 4, 65}, none{};
  tile<MF, T::D3w1>(model);
  tile<MF, T::D3w2>(model, best == 2 ? w : none);
  tile<MF, T::D3w3>(model, Pref{1, 4});
  tile<MF, T::D3w4>(model, best == 4 ? w : none);
  tile<MF, T::D3w5>(model);
}
// the narrow shapes, where extents fill 64-wide tiles to at most `filled`: two
// rows a thread on smaller grids, four on larger ones
template <class MF, int L>
void narrow3(int model, double filled, long long from, long long four) {
  tile<MF, Tiles<float>::D3n1, L>(model, Pref{1, 1, 0, filled, from});
  if (four) tile<MF, Tiles<float>::D3n2, L>(model, Pref{2, 1, 0, filled, four});
}
template <class E>
void row(int model, int pref = 0) {
  register_kernel(KernelKey{model, SPK_FUSED, 3, 0, 7, 10, 25}, with(E::info(), Pref{pref}));
}
}  // namespace

void register_wide_kernels() {
  wide3<MF_A_fused>(SPK_A, 2);
  wide3<MF_AMK_fused>(SPK_AMK, 2);
  wide3<MF_B_fused>(SPK_B, 4);
  wide3<MF_BMK_fused>(SPK_BMK, 4);
  wide3<MF_C_fused>(SPK_C, 0);
  narrow3<MF_A_fused, 7>(SPK_A, 0.79, 400000, 0);
  narrow3<MF_AMK_fused, 7>(SPK_AMK, 0.79, 400000, 0);
  narrow3<MF_B_fused, 7>(SPK_B, 0.7, 400000, 0);
  narrow3<MF_BMK_fused, 7>(SPK_BMK, 0.7, 400000, 0);
  tile<MF_C_fused, Tiles<float>::D3n1>(SPK_C, Pref{2, 1, 0, 1.0, 1500000});
  narrow3<MF_A_fused, 15>(SPK_A, 0.79, 400000, 1500000);
  // row kernels of the conserved pattern (x extent 256 or 128, periodic in x)
  row<EntryChRow<MF_B_fused, 256, 10, 1, 2, true, 2>>(SPK_B, 3);
  SP_REGCHROW(SPK_B, MF_B_fused, 256, 10, 1, 2, false, 2);
  SP_REGCHROW(SPK_B, MF_B_fused, 256, 18, 1, 2, true, 1);
  SP_REGCHROW(SPK_B, MF_B_fused, 256, 6, 1, 2, false, 1);
  SP_REGCHROW(SPK_B, MF_B_fused, 256, 6, 1, 2, true, 1);
  SP_REGCHROW(SPK_B, MF_B_fused, 256, 6, 1, 3, false, 1);
  SP_REGCHROW(SPK_B, MF_B_fused, 256, 3, 2, 2, false, 1);
  row<EntryChRow<MF_B_fused, 128, 9, 2, 2, true, 1>>(SPK_B, 3);
  SP_REGCHROW(SPK_B, MF_B_fused, 128, 18, 1, 2, true, 1);
  row<EntryChRow<MF_BMK_fused, 256, 10, 1, 2, true, 2>>(SPK_BMK, 3);
  // row kernels of any fused 7-point model (sp_row.cuh)
  SP_REGROW(SPK_C, MF_C_fused, 256, 6, 1, 1);
  row<EntryRow<MF_C_fused, 256, 6, 2, 1>>(SPK_C, 3);
  SP_REGROW(SPK_C, MF_C_fused, 256, 10, 1, 1);
  row<EntryRow<MF_C_fused, 128, 10, 2, 1>>(SPK_C, 3);
  row<EntryRow<MF_A_fused, 256, 8, 2, 1>>(SPK_A, 3);
  row<EntryRow<MF_A_fused, 128, 16, 2, 1>>(SPK_A, 3);
  SP_REGROW(SPK_B, MF_B_fused, 256, 10, 2, 2);
  row<EntryChRow<MF_BMK_fused, 128, 9, 2, 2, true, 1>>(SPK_BMK, 3);
  SP_WIDE2(SPK_A, MF_A_fused, MF_A_fused)
  SP_WIDE2(SPK_B, MF_B_fused, MF_B_fused)
  SP_WIDE2(SPK_ENS_AB, MF_AMK_fused, MF_BMK_fused)
}
}  // namespace sp
