/*
 * sp_inst_exact3.cu -- further tile shapes of the 3D kernels of the EXACT form
 * in FP64 (compiled with --fmad=false).  Four rows per thread share their
 * neighbour rows' loads (shared memory bounds these kernels: the 25-point
 * bilaplacian reads 17 16-byte words per two sites with two rows a thread);
 * 64-thread CTAs keep enough of them resident.  256^3, B: 122 us with the
 * default 64 x 16 x 2 shape, 108 with 32 x 16 x 4; C: 246 and 229; A: 64 and
 * 60 with 64 x 8 x 4.  Below a million sites the march's latency counts and the
 * default shape is the faster (64^3, B: 7.4 and 8.0).
 */
#include "sp_launch.cuh"

namespace sp {
namespace {
template <class MF, class TC>
void shape(int model, int pref, long long from = 0) {
  KernelInfo i = Entry3<MF, double, 7, 10, 25, TC, true>::info();
  i.pref = pref;
  i.pref_sites = from;
  register_kernel(KernelKey{model, SPK_EXACT, 3, 1, 7, 10, 25}, i);
}
}  // namespace

void register_exact3_kernels() {
  shape<MF_A_exact, Tiles<double>::D3c>(SPK_A, 1);
  shape<MF_AMK_exact, Tiles<double>::D3c>(SPK_AMK, 1);
  shape<MF_B_exact, Tiles<double>::D3d>(SPK_B, 1, 1000000);
  shape<MF_B_exact, Tiles<double>::D3b>(SPK_B, 0);
  shape<MF_C_exact, Tiles<double>::D3d>(SPK_C, 1, 1000000);
  shape<MF_BMK_exact, Tiles<double>::D3d>(SPK_BMK, 1, 1000000);
}
}  // namespace sp
