/*
 * sp_many2.cuh -- many Euler steps per launch for 2D grids that one wave of
 * CTAs covers (SolverFT::step, examples/solvers/solverft.h:46-103, repeated).
 *
 * On such grids a step kernel is bound by its launch and by one trip to memory
 * and back (3 us for 64^2, 4.7 us for 800 x 600, whatever the work).  Here a
 * CTA loads its tile with a margin of (steps x reach) sites around it, runs
 * the steps in shared memory, each on a region smaller than the last, and
 * writes the tile: one launch and one trip for up to `kt` steps.  The margin is
 * work done twice, on SMs that would wait otherwise; tile and depth are chosen
 * for the grid at hand (many_plan in sp_api.cu).  No CTA waits for another.
 *
 * Unlike the temporally blocked tiles of sp_tb2.cuh (compile-time tile and
 * depth, whole 16-byte copies, periodic faces) the tile and the depth are run
 * time values, any x extent is taken (loads are per element, once per launch),
 * and sides may hold a constant: sites beyond such a side keep it in both
 * buffers, no step updates them, and staged operands are evaluated on them as
 * in the one-step kernels.  Sites are evaluated by the same expression code in
 * the same order, so s steps give the bits of s launches of k_fd2d; keys whose
 * products the compiler contracts as it sees fit have no many-step kernel
 * (sp_inst_many_exact.cu) or spell the contractions out (sp_inst_points.cu).
 */
#pragma once

#include "sp_kernels.cuh"

namespace sp {

// threads, columns of a plane, rows of a work item (evaluated together: their
// shared neighbour rows are loaded once)
constexpr int MANY_NT = 512, MANY_PW = 128, MANY_SR = 2;
constexpr int many_w(int esz) { return 16 / esz; }  // sites per thread and row: 16 bytes

struct ManyTile {
  int tx, ty, ntx;   // tile, tiles along x
  int hx, hy;        // margin of this launch (hx rounded to groups, and one more)
  int wall[2];       // 1: constant sides along x, y
  int rows;          // rows of a plane: ty + 2 hy, and SR - 1 that only partial items read
  int cg;            // column groups a row of threads covers: a power of two
};

template <class T>
struct ManyParams {
  Step2Params<T> s;
  ManyTile t;
  T bv[4];  // constants of the sides x-, x+, y-, y+
};

template <class M, class T, int LP, int GP, int BP, bool EXACT>
struct Fd2M {
  static constexpr int W = many_w(sizeof(T)), NT = MANY_NT, PW = MANY_PW, SR = MANY_SR;
  static constexpr int NF = M::nf, NS = M::ns, R = M::R, RS = NS > 0 ? M::RS : 0,
                       RI = imax(M::r_stage, 0);
  static_assert(R <= 2 * W, "margin");
  static constexpr int PLANES = 2 * NF + NS;
};

template <class M, class T, int LP, int GP, int BP, bool EXACT>
__global__ void __launch_bounds__(MANY_NT)
    k_fd2m(const __grid_constant__ ManyParams<T> q, const __grid_constant__ M m) {
  using K = Fd2M<M, T, LP, GP, BP, EXACT>;
  constexpr int W = K::W, NT = K::NT, PW = K::PW, NF = K::NF, NS = K::NS, R = K::R, RS = K::RS,
                SR = K::SR;
  using V = vec_t<T, W>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const Step2Params<T>& p = q.s;
  const ManyTile& t = q.t;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int plane = PW * t.rows;
  T* a = reinterpret_cast<T*>(smem_raw);  // [NF] planes
  T* b = a + NF * plane;                  // [NF]
  T* const sb = b + NF * plane;           // [NS]
  const int ty_ = int(blockIdx.x) / t.ntx, tx_ = int(blockIdx.x) - ty_ * t.ntx;
  const int x0 = tx_ * t.tx, y0 = ty_ * t.ty, gx0 = x0 - t.hx, gy0 = y0 - t.hy;
  const int width = t.tx + 2 * t.hx;
  const int ii = blockIdx.y;

  pdl_enter();
  const Inst2<T>& ip = p.inst[ii];
  const int n0 = ip.n[0], n1 = ip.n[1];

  // ---- the tile and its margin: wrapped around periodic faces, constant
  // beyond the others (the later axis wins in a corner, as in the halo)
  for (int r = warp; r < t.ty + 2 * t.hy; r += NT / 32) {
    int y = gy0 + r;
    const bool oy = t.wall[1] && (y < 0 || y >= n1);
    const T vy = y < 0 ? q.bv[2] : q.bv[3];
    if (!oy) {
      while (y < 0) y += n1;
      while (y >= n1) y -= n1;
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const T* const row =
          p.in[ii * NF + f] + (long long)(oy ? 0 : y + p.hy) * ip.pitch + p.hx;
      T v[PW / 32];
      bool out[PW / 32];
#pragma unroll
      for (int k = 0; k < PW / 32; ++k) {
        const int c = lane + 32 * k;
        int x = gx0 + c;
        out[k] = oy || (t.wall[0] && (x < 0 || x >= n0));
        v[k] = oy ? vy : x < 0 ? q.bv[0] : q.bv[1];
        if (c < width && !out[k]) {
          while (x < 0) x += n0;
          while (x >= n0) x -= n0;
          v[k] = row[x];
        }
      }
#pragma unroll
      for (int k = 0; k < PW / 32; ++k) {
        const int c = lane + 32 * k;
        if (c >= width) continue;
        a[f * plane + r * PW + c] = v[k];
        if (out[k]) b[f * plane + r * PW + c] = v[k];
      }
    }
  }
  T coef[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) coef[i] = ip.coef[i];
  const V vdt(ip.dt), vdivh2(ip.divh2), vdivh3(ip.divh3), vdivh4(ip.divh4);
  // a thread keeps one column group and takes every rstep-th row item of a
  // region (no divisions, whatever the region)
  const int col = (tid & (t.cg - 1)) * W, rr = tid / t.cg, rstep = NT / t.cg;
  __syncthreads();

  for (int j = 0; j < p.tsteps; ++j) {
    const int grow = (p.tsteps - 1 - j) * R;  // the region this step updates: the tile grown by it
    if constexpr (NS > 0) {
      using CS = Ctx<T, W, !EXACT, 2, LP, GP, BP, NF, 1, 0, PW, 1, 1, 0, PW>;
      const int gs = grow + RS, gw = (gs + W - 1) / W * W;
      const int r1 = t.hy + t.ty + gs;
      if (col >= t.hx - gw && col < t.hx + t.tx + gw) {
        CS ctx;
        ctx.divh2 = vdivh2;
        ctx.divh3 = vdivh3;
        ctx.divh4 = vdivh4;
        ctx.cf = coef;
#pragma unroll 1
        for (int r = t.hy - gs + rr * SR; r < r1; r += rstep * SR) {
          const int off = r * PW + col;
          V s0[SR], s1[SR];
#pragma unroll
          for (int k = 0; k < SR; ++k) {
#pragma unroll
            for (int f = 0; f < NF; ++f) ctx.fo[f][0] = a + f * plane + off + k * PW;
            s0[k] = eval(m.s0, ctx);
            if constexpr (NS > 1) s1[k] = eval(m.s1, ctx);
          }
#pragma unroll
          for (int k = 0; k < SR; ++k) {
            if (r + k >= r1) break;
            *reinterpret_cast<V*>(sb + off + k * PW) = s0[k];
            if constexpr (NS > 1) *reinterpret_cast<V*>(sb + plane + off + k * PW) = s1[k];
          }
        }
      }
      __syncthreads();
    }
    using CO = Ctx<T, W, !EXACT, 2, LP, GP, BP, NF, 1, 0, PW, NS, 1, 0, PW>;
    const bool last = j + 1 == p.tsteps;
    // rows and column groups of the region, inside constant sides
    const int gw = (grow + W - 1) / W * W;
    int c0 = t.hx - gw, c1 = t.hx + t.tx + gw, r0 = t.hy - grow, r1 = t.hy + t.ty + grow;
    if (t.wall[0] || last) {
      c0 = max(c0, -gx0);
      c1 = min(c1, n0 - gx0);
    }
    if (t.wall[1] || last) {
      r0 = max(r0, -gy0);
      r1 = min(r1, n1 - gy0);
    }
    if (col >= c0 && col < c1) {
      CO ctx;
      ctx.divh2 = vdivh2;
      ctx.divh3 = vdivh3;
      ctx.divh4 = vdivh4;
      ctx.cf = coef;
      const int x = gx0 + col;
#pragma unroll 1
      for (int r = r0 + rr * SR; r < r1; r += rstep * SR) {
        const int off = r * PW + col;
        V nv[SR][NF];
#pragma unroll
        for (int k = 0; k < SR; ++k) {
#pragma unroll
          for (int f = 0; f < NF; ++f) ctx.fo[f][0] = a + f * plane + off + k * PW;
#pragma unroll
          for (int i = 0; i < NS; ++i) ctx.so[i][0] = sb + i * plane + off + k * PW;
          nv[k][0] = fmadd<!EXACT>(vdt, eval(m.r0, ctx), ctx.template var<1, 0, 0, 0>());
          if constexpr (NF > 1)
            nv[k][1] = fmadd<!EXACT>(vdt, eval(m.r1, ctx), ctx.template var<2, 0, 0, 0>());
        }
#pragma unroll
        for (int k = 0; k < SR; ++k) {
          if (r + k >= r1) break;
          if (!last) {
            // lanes past a constant side keep the constant
            if (t.wall[0] && x + W > n0) {
#pragma unroll
              for (int l = 0; l < W; ++l)
                if (x + l >= n0)
#pragma unroll
                  for (int f = 0; f < NF; ++f) set_lane(nv[k][f], l, q.bv[1]);
            }
#pragma unroll
            for (int f = 0; f < NF; ++f)
              *reinterpret_cast<V*>(b + f * plane + off + k * PW) = nv[k][f];
          } else {
            const int h3[3] = {p.hx, p.hy, 0}, n3[3] = {n0, n1, 1};
            const int per3[3] = {ip.per[0], ip.per[1], 0};
#pragma unroll
            for (int f = 0; f < NF; ++f)
              store_group<T, W, 2, R>(p.out[ii * NF + f], x, gy0 + r + k, 0, nv[k][f], n3, h3, per3,
                                      ip.pitch, 0);
          }
        }
      }
    }
    if (last) break;
    __syncthreads();
    T* const sw = a;
    a = b;
    b = sw;
  }
}

}  // namespace sp
