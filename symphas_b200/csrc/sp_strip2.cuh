/*
 * sp_strip2.cuh -- 2D fused FP32 step as warps that march down the rows, for
 * models lowered onto 5-point Laplacians with at most one staged operand
 * (models A, B, C, AMK, BMK in their fused forms).
 *
 * A warp holds a strip of 128 columns, lane l the four sites 4 l .. 4 l + 3,
 * and marches down `ty` rows: each row is one coalesced 512-byte load, kept in
 * registers while the stencil needs it; the x neighbours come from warp
 * shuffles, the staged operand of a row is computed once and kept for three
 * rows.  The strip's outer lanes only serve as neighbours (a reach of two
 * sites is half a lane), so it writes 120 columns.  No shared memory, no
 * barrier and no copy engine: about half the instructions a site of the tile
 * kernel (k_fd2d), which issue and barriers bound at half of the HBM rate.
 * The halo is read from the field as the tile kernels' boxes read it, and the
 * evaluator forms every sum in the order of the tile kernels, so the fields
 * come out bit-identical.
 *
 * Work items are strips of `ty` rows of an instance, one per warp; their
 * number, not a queue, balances the SMs.
 */
#pragma once

#include "sp_kernels.cuh"

namespace sp {

constexpr int ST2_X = 120, ST2_WARPS = 4;  // columns an item writes; items (warps) per CTA

// the values one row's evaluation reads: rows y - 1, y, y + 1 of the fields and
// of the staged operand
template <int NF, int NS>
struct StripRow {
  using V = Vec<float, 4>;
  V f[NF][3], s[NS > 0 ? NS : 1][3];
};

template <int NF, int NS>
struct StripCtx {
  using scalar_type = float;
  using value_type = Vec<float, 4>;
  using V = value_type;
  static constexpr bool contract = true;
  static constexpr int dim = 2, lap_points = 5, gradlap_points = 6, bilap_points = 13;
  const StripRow<NF, NS>& d;
  V divh2, divh3, divh4;
  const float* cf;
  template <int X, int Y>
  __device__ __forceinline__ V pick(const V (&c)[3]) const {
    static_assert(Y >= -1 && Y <= 1 && (X == 0 || Y == 0), "5-point reach");
    if constexpr (X == 0) {
      return c[Y + 1];
    } else if constexpr (X == -4) {  // the group left: only its last lane is read
      V r = c[1];
      r.v[3] = __shfl_up_sync(0xffffffffu, c[1].v[3], 1);
      return r;
    } else if constexpr (X == 4) {  // the group right: only its first lane is read
      V r = c[1];
      r.v[0] = __shfl_down_sync(0xffffffffu, c[1].v[0], 1);
      return r;
    } else if constexpr (X == -1) {
      V r;
      r.v[0] = __shfl_up_sync(0xffffffffu, c[1].v[3], 1);
      r.v[1] = c[1].v[0];
      r.v[2] = c[1].v[1];
      r.v[3] = c[1].v[2];
      return r;
    } else {
      static_assert(X == 1, "5-point reach");
      V r;
      r.v[0] = c[1].v[1];
      r.v[1] = c[1].v[2];
      r.v[2] = c[1].v[3];
      r.v[3] = __shfl_down_sync(0xffffffffu, c[1].v[0], 1);
      return r;
    }
  }
  template <int I, int X, int Y, int Z>
  __device__ __forceinline__ V var() const {
    static_assert(I >= 1 && I <= NF && Z == 0, "field index");
    return pick<X, Y>(d.f[I - 1]);
  }
  template <int K, int X, int Y, int Z>
  __device__ __forceinline__ V stg() const {
    static_assert(K >= 0 && K < NS && Z == 0, "stage index");
    return pick<X, Y>(d.s[K]);
  }
  __device__ __forceinline__ V coef(int i) const { return V(cf[i - 1]); }
};

template <class M>
struct Strip2 {
  static constexpr int NF = M::nf, NS = M::ns, R = M::R;
  static constexpr int RD = imax(M::r_direct, 0), RS = NS > 0 ? M::RS : 0,
                       RI = imax(M::r_stage, 0);
  static constexpr int U = imax(RD, NS > 0 ? RS + RI : 0);  // newest row read ahead of the output
  static constexpr int NR = U + RD + 1;                     // field rows read
  // the register queues (field rows, staged rows, rows in flight) rotate by
  // static indices with a common period: moving a row that is still being
  // loaded would wait for it
  static constexpr int PER = NR <= 3 ? 3 : 6;
  static constexpr int WARM = 2 * RS;                       // rows that only stage
  static_assert(WARM == 0 || WARM == 2, "staged rows above the first");
  static_assert(NS <= 1 && RS <= 1 && RI <= 1 && RD <= 1 && R <= 2, "5-point reach");
  static_assert(U == R || NS == 0, "reach");
};

// one item: rows y0 .. y1 - 1 of strip `st` of instance ii; RH: depth of the
// periodic images the launch's kernels keep (the largest reach of its models)
template <class M, int PF, int RH>
__device__ __forceinline__ void strip2_march(const Step2Params<float>& p, const M& m,
                                             const Inst2<float>& ip, int ii, int st, int y0,
                                             int y1, double& msum) {
  using K = Strip2<M>;
  using V = Vec<float, 4>;
  constexpr int NF = K::NF, NS = K::NS, R = K::R, RD = K::RD, RS = K::RS, U = K::U, NR = K::NR,
                WARM = K::WARM;
  static_assert(RH >= R && RH <= 4, "image depth");
  const int lane = threadIdx.x & 31;
  const int n0 = ip.n[0], n1 = ip.n[1];
  const long long pitch = ip.pitch;
  const int x = st * ST2_X + 4 * (lane - 1);  // this lane's first column
  const bool ld = x + p.hx + 4 <= pitch;      // inside the padded row
  const bool out = lane >= 1 && lane <= 30 && x < n0;  // n0 is a multiple of 4: whole groups
  float coef[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) coef[i] = ip.coef[i];
  const V divh2(ip.divh2), divh3(ip.divh3), divh4(ip.divh4), vdt(ip.dt);
  const bool rhs = p.rhs_only != 0;

  // rows are loaded PF ahead of the newest row used; row number k (from y0 -
  // WARM - RD on) lives in f[k % PER], staged rows likewise in s
  constexpr int PER = K::PER;
  static_assert(PER % PF == 0, "one period");
  const float* src[NF];
  V f[PER][NF], pre[PF][NF], s[PER];
  int yn = y0 - WARM - RD;  // next row to load; rows before y0 - R are not used
  const int yl = y1 - 1 + U;
#pragma unroll
  for (int q = 0; q < NF; ++q)
    src[q] = p.in[ii * NF + q] + (long long)(yn + p.hy) * pitch + (x + p.hx);
  auto load = [&](V (&v)[NF]) {
    const bool on = ld && yn <= yl && yn >= y0 - R;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      if (on) v[q] = *reinterpret_cast<const V*>(src[q]);
      src[q] += pitch;
    }
    ++yn;
  };
#pragma unroll
  for (int k = 0; k < PER; ++k)
#pragma unroll
    for (int q = 0; q < NF; ++q) f[k][q] = V(0.f);
#pragma unroll
  for (int k = 0; k < PF; ++k)
#pragma unroll
    for (int q = 0; q < NF; ++q) pre[k][q] = V(0.f);
#pragma unroll
  for (int k = 0; k < NR - 1; ++k) load(f[k]);
#pragma unroll
  for (int k = 0; k < PF; ++k) load(pre[k]);
#pragma unroll
  for (int k = 0; k < PER; ++k) s[k] = V(0.f);

  // periodic images along x belong to lanes at a face (xany: some lane of the warp)
  const int xo = out ? int(image_offset(ip.per[0], x, 4, n0, RH, 1)) : 0;
  const bool xany = __any_sync(0xffffffffu, xo != 0);
  float* dst[NF];
#pragma unroll
  for (int q = 0; q < NF; ++q)
    dst[q] = p.out[ii * NF + q] + (long long)(y0 + p.hy) * pitch + (x + p.hx);

  // phase P = number of rows done so far modulo PER
  auto row = [&](int y, auto phase, auto emit) {
    constexpr int P = decltype(phase)::value;
    // field row y - RD + k is f[(P + k) % PER], staged row y - 1 + k is s[(P + k) % PER]
#pragma unroll
    for (int q = 0; q < NF; ++q) f[(P + NR - 1) % PER][q] = pre[P % PF][q];
    load(pre[P % PF]);
    StripRow<NF, NS> d;
    if constexpr (NS > 0) {
#pragma unroll
      for (int q = 0; q < NF; ++q)
#pragma unroll
        for (int k = 0; k < 3; ++k) d.f[q][k] = f[(P + RD + RS - 1 + k) % PER][q];
      s[(P + 2) % PER] = eval(m.s0, StripCtx<NF, NS>{d, divh2, divh3, divh4, coef});
    }
    if constexpr (decltype(emit)::value) {
#pragma unroll
      for (int q = 0; q < NF; ++q) {
        d.f[q][1] = f[(P + RD) % PER][q];
        if constexpr (RD > 0) {
          d.f[q][0] = f[P % PER][q];
          d.f[q][2] = f[(P + 2) % PER][q];
        }
      }
      if constexpr (NS > 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) d.s[0][k] = s[(P + k) % PER];
      }
      const StripCtx<NF, NS> c{d, divh2, divh3, divh4, coef};
      V nv[NF];
      const V r0 = eval(m.r0, c);
      nv[0] = rhs ? r0 : fmadd<true>(vdt, r0, d.f[0][1]);
      if constexpr (NF > 1) {
        const V r1 = eval(m.r1, c);
        nv[1] = rhs ? r1 : fmadd<true>(vdt, r1, d.f[1][1]);
      }
      const long long yo = image_offset(ip.per[1], y, 1, n1, RH, pitch);  // warp-uniform
#pragma unroll
      for (int q = 0; q < NF; ++q) {
        st_if(dst[q], nv[q], out);
        if (xany) st_if(dst[q] + xo, nv[q], xo != 0);
        if (yo != 0) {
          st_if(dst[q] + yo, nv[q], out);
          if (xany) st_if(dst[q] + yo + xo, nv[q], xo != 0);
        }
        dst[q] += pitch;
      }
      if (p.partial && out) msum += vsum<float, 4>(nv[0], x, n0);
    }
  };
  if constexpr (WARM > 0) {
    row(y0 - 2, std::integral_constant<int, 0>{}, std::false_type{});
    row(y0 - 1, std::integral_constant<int, 1>{}, std::false_type{});
  }
  int y = y0;
  auto next = [&](auto phase) -> bool {
    if (y >= y1) return false;
    row(y, std::integral_constant<int, (decltype(phase)::value + WARM) % PER>{}, std::true_type{});
    ++y;
    return true;
  };
  if constexpr (PER == 3) {
    while (next(std::integral_constant<int, 0>{}) && next(std::integral_constant<int, 1>{}) &&
           next(std::integral_constant<int, 2>{})) {
    }
  } else {
    while (next(std::integral_constant<int, 0>{}) && next(std::integral_constant<int, 1>{}) &&
           next(std::integral_constant<int, 2>{}) && next(std::integral_constant<int, 3>{}) &&
           next(std::integral_constant<int, 4>{}) && next(std::integral_constant<int, 5>{})) {
    }
  }
}

template <class M0, class M1, int PF>
__global__ void __launch_bounds__(32 * ST2_WARPS, M0::nf > 1 ? 3 : imax(M0::ns, M1::ns) ? 6 : 7)
    k_fd2w(const __grid_constant__ Step2Params<float> p, const __grid_constant__ M0 m0,
           const __grid_constant__ M1 m1) {
  __shared__ double red[32];
  constexpr int RH = imax(M0::R, M1::R);
  pdl_enter();
  const int item = int(blockIdx.x) * ST2_WARPS + int(threadIdx.x >> 5);
  double msum = 0.0;
  if (item < p.nitems) {
    int2 it = make_int2(0, item);
    if (p.items) it = p.items[item];
    const Inst2<float>& ip = p.inst[it.x];
    const int st = p.items ? it.y & 0xffff : it.y % ip.ntx;
    const int y0 = (p.items ? it.y >> 16 : it.y / ip.ntx) * p.ty;
    const int y1 = min(y0 + p.ty, ip.n[1]);
    if (ip.kind == 0)
      strip2_march<M0, PF, RH>(p, m0, ip, it.x, st, y0, y1, msum);
    else
      strip2_march<M1, PF, RH>(p, m1, ip, it.x, st, y0, y1, msum);
  }
  if (p.partial) {
    const double s = block_sum<32 * ST2_WARPS>(msum, red);
    if (threadIdx.x == 0) p.partial[blockIdx.x] = s;
  }
}

}  // namespace sp
