/*
 * sp_flow.cuh -- the 3x3 circular convolution (forward and data gradient) as a
 * persistent tcgen05 kernel, with the weights resident in shared memory, or, for
 * 128 outputs and more where they do not fit, streamed with the input.  No
 * counterpart in SymPhas.
 *
 * Same operand layout as k_conv3x3_strip (sp_conv.cu): the input is staged as
 * a strip of circularly padded positions, chunk-major (one 16-byte row per
 * position and 8-channel chunk), so the nine taps are nine start addresses of
 * one staged strip.  What differs:
 *
 *   - one CTA per SM walks over the tiles (MT x 128 positions each); resident
 *     weights of its BN output channels are gathered once per CTA, straight
 *     from [cout][3][3][cin] (no re-tiling launch); streamed ones are re-tiled by
 *     k_tile_weights and come with every stage;
 *   - gather, MMAs and epilogue of different tiles overlap: eight producer
 *     warps fill a ring of strips (32 input channels each), one thread issues
 *     the MMAs into one of two tensor-memory accumulators, sixteen warps empty
 *     the other;
 *   - a warp gathers 8 positions x 4 chunks per copy: whole 64-byte segments
 *     of global memory, 128-byte runs of shared memory (16-byte pieces of
 *     different sectors, two lanes a position, read every sector twice); the
 *     epilogue's arithmetic is packed FP32x2 and its stores are 32 bytes a lane.
 */
#pragma once

namespace sp {
namespace conv {

constexpr int FL_PROD = 256, FL_EPI = 512;       // producer and epilogue threads
constexpr int FL_NT = FL_PROD + 32 + FL_EPI;     // and the MMA warp
constexpr int FL_CB = 32;                        // input channels per stage, weights resident
constexpr int FL_CBS = 16;                       // and streamed
constexpr int FL_SMEM = 227 * 1024 - 1024;       // for weights and strips
constexpr int FL_SMAX = 4;                       // stages of the ring

struct FlowParams {
  const __nv_bfloat16* x;    // [N][H][W][Cin]
  const __nv_bfloat16* w;    // [Cout][3][3][Cin]; streamed: as k_tile_weights leaves them
  const float* bias;         // [Cout] or null
  const __nv_bfloat16* res;  // [N][H][W][Cout] or null
  __nv_bfloat16* z;          // pre-activation out, or null
  __nv_bfloat16* a;          // gelu(z) out, or null
  int n, h, wid, cin, cout;
  int P, S;                  // positions of a strip; stages
  int tiles;
  int up;                    // 1: x is [N][H/2][W/2][Cin], read nearest-up-sampled
  int wide;                  // outputs and residual allow 32-byte accesses
};

// a shared-memory descriptor as base (layout) plus start address: the start is
// the low 14 bits in 16-byte units, so an offset is one 32-bit addition
__device__ __forceinline__ uint64_t desc_at(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
template <bool ACCUMULATE>
__device__ __forceinline__ void umma_go(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                        uint32_t idesc) {
  if constexpr (ACCUMULATE)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc));
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc));
}

// one arrival for a warp (an arrival per thread serialises in shared memory:
// 512 of them a tile cost more than the tile's MMAs)
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0)
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

struct U8 {
  uint32_t v[8];
};
__device__ __forceinline__ void st_32b(void* p, const U8& d, bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(d.v[0]),
                 "r"(d.v[1]), "r"(d.v[2]), "r"(d.v[3]), "r"(d.v[4]), "r"(d.v[5]), "r"(d.v[6]),
                 "r"(d.v[7])
                 : "memory");
  } else {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(d.v[0], d.v[1], d.v[2], d.v[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(d.v[4], d.v[5], d.v[6], d.v[7]);
  }
}
__device__ __forceinline__ U8 ld_32b(const void* p, bool wide) {
  U8 d;
  if (wide) {
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(d.v[0]), "=r"(d.v[1]), "=r"(d.v[2]), "=r"(d.v[3]), "=r"(d.v[4]),
                   "=r"(d.v[5]), "=r"(d.v[6]), "=r"(d.v[7])
                 : "l"(p));
  } else {
    const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
    d = U8{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
  }
  return d;
}
__device__ __forceinline__ uint32_t bf2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 f2bf(uint32_t u) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
}
// gelu() of two values (the same function, packed)
__device__ __forceinline__ float2 gelu2(float2 z) {
  const float2 q = __fmul2_rn(z, z);
  const float2 c = __ffma2_rn(q, make_float2(0.7978845608028654f * 0.044715f,
                                             0.7978845608028654f * 0.044715f),
                              make_float2(0.7978845608028654f, 0.7978845608028654f));
  const float2 u = __fmul2_rn(z, c);
  const float2 h = __fmul2_rn(z, make_float2(0.5f, 0.5f));
  return __ffma2_rn(h, make_float2(tanh_fast(u.x), tanh_fast(u.y)), h);
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
        "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
}

// gelu_full() of two values
__device__ __forceinline__ float2 gelu2_full(float2 z) {
  const float k = -2.f * 0.7978845608028654f;
  const float2 c = __ffma2_rn(__fmul2_rn(z, z), make_float2(k * 0.044715f, k * 0.044715f),
                              make_float2(k, k));
  const float2 u = __fmul2_rn(z, c);  // -2 u
  const float2 d = __fadd2_rn(make_float2(__expf(u.x), __expf(u.y)), make_float2(1.f, 1.f));
  return make_float2(__fdividef(z.x, d.x), __fdividef(z.y, d.y));
}

// A padded position: image, row and column of the (H + 2) x (W + 2) grid,
// advanced by a fixed number of positions without divisions.
struct PadPos {
  int n, y, x;
  __device__ __forceinline__ void step(int sy, int sx, int W2, int H2) {
    x += sx;
    y += sy;
    if (x >= W2) {
      x -= W2;
      ++y;
    }
    while (y >= H2) {
      y -= H2;
      ++n;
    }
  }
};

// STREAM: the weights do not fit beside the strips (128 outputs of 128 and more
// inputs: 295 KB) and come with every stage, 16 input channels' share in one
// bulk copy; then a tile is as large as tensor memory allows (MT = 4: one
// accumulator set), so that a stage's 37 KB serve 512 positions, and the next
// tile's first MMAs start as soon as the epilogue has emptied their block.
template <int BN, int MT, bool STREAM>
struct FlowTile {
  static constexpr int M = MT * 128;   // positions per tile
  static constexpr int ACC = MT * BN;  // tensor-memory columns of one accumulator set
  static constexpr int NBUF = 2 * ACC <= 512 ? 2 : 1, COLS = NBUF * ACC;
  static constexpr int CB = STREAM ? FL_CBS : FL_CB, CH = CB / 8;
  static constexpr int WSTAGE = STREAM ? BN * 9 * CB * 2 : 0;  // bytes of a stage's weights
  static constexpr int EWARPS = 4 * (BN / 32 < 4 ? BN / 32 : 4);  // warps that empty a block
  static_assert(COLS <= 512 && (COLS & (COLS - 1)) == 0 && COLS >= 32, "columns");
  static_assert(BN % 32 == 0 && BN <= 128 && MT % 2 == 0 && MT <= 8, "tile");
};

// FULL: the activation by gelu_full (32 -> 32 channels, 16 x 256^2: 75.5 us, and
// 67.8 with tanh.approx; with expf and a divide 109.5, most of it spills)
template <int BN, int MT, bool STREAM, bool FULL>
__global__ void __launch_bounds__(FL_NT, 1) k_conv3x3_flow(const FlowParams p) {
  using TT = FlowTile<BN, MT, STREAM>;
  constexpr int M = TT::M, ACC = TT::ACC, NBUF = TT::NBUF, CB = TT::CB, CH = TT::CH;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int S = p.S, P = p.P, STAGE = CH * P * 16 + TT::WSTAGE;
  const int kch = p.cin / 8;  // 8-channel chunks of the input
  const int nkb = p.cin / CB;
  unsigned char* const wsm = smem;  // [9 * kch chunks][BN rows][16 B]
  unsigned char* const ring = smem + (STREAM ? 0 : 9 * kch * BN * 16);
  float* const bsm = reinterpret_cast<float*>(ring + S * STAGE);  // [BN] bias
  uint64_t* const bars = reinterpret_cast<uint64_t*>(bsm + BN);
  uint64_t *const full = bars, *const empty = bars + FL_SMAX, *const tfull = bars + 2 * FL_SMAX,
           *const tempty = tfull + 2, *const done = tempty + 2 * 8;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int W2 = p.wid + 2, H2 = p.h + 2;
  const uint32_t W2u = uint32_t(W2), HW2u = uint32_t(W2) * uint32_t(H2);
  const int co0 = blockIdx.y * BN;
  constexpr int MMA_WARP = FL_PROD / 32;

  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(TT::COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      tma::mbar_init(&full[s], FL_PROD / 32 + (STREAM ? 1 : 0));
      tma::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < NBUF; ++b) {
      tma::mbar_init(&tfull[b], 1);
      for (int m = 0; m < MT; ++m) tma::mbar_init(&tempty[b * MT + m], TT::EWARPS);
    }
    tma::mbar_init(done, 1);
    tma::fence_barrier_init();
  }
  // the weights, K-major without swizzle: [tap * kch + chunk][output channel]
  if constexpr (!STREAM)
    for (int i = tid; i < 9 * kch * BN; i += FL_NT) {
      const int co = i % BN, kc = i / BN;
      cp_async16(wsm + i * 16, p.w + ((long long)(co0 + co) * 9 * kch + kc) * 8, true);
    }
  for (int i = tid; i < BN; i += FL_NT) bsm[i] = p.bias ? p.bias[co0 + i] : 0.f;
  asm volatile("cp.async.wait_all;" ::: "memory");
  tma::fence_proxy_async();  // generic-proxy writes, read by the tensor core
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  bool bad = false;

  if (warp < MMA_WARP) {
    // ---- producers: a warp copies 32 / CH positions x CH chunks at a time;
    // lane: position lp, chunk j
    constexpr int LP = 32 / CH, STEP = FL_PROD / CH;
    const int j = lane / LP, lp = warp * LP + lane % LP;
    const int sy = STEP / W2, sx = STEP - sy * W2;
    int s = 0, fills = 0;
    uint32_t ph = 1;  // a fresh barrier passes the wait for the phase before its first
    for (int tile = blockIdx.x; tile < p.tiles && !bad; tile += gridDim.x) {
      // strip position 0 is output position tile * M - (W2 + 1); counted from
      // one image earlier, so that it is not negative
      const uint32_t u = uint32_t(tile) * M + HW2u - uint32_t(W2 + 1) + uint32_t(lp);
      const uint32_t nn = u / HW2u, r = u - nn * HW2u, yq = r / W2u;
      const PadPos start{int(nn) - 1, int(yq), int(r - yq * W2u)};
      for (int kb = 0; kb < nkb; ++kb) {
        if (!tma::mbar_wait(&empty[s], ph)) {
          bad = true;
          break;
        }
        unsigned char* dst = ring + s * STAGE + (j * P + lp) * 16;
        const __nv_bfloat16* const xc = p.x + kb * CB + j * 8;
        if (STREAM && tid == 0) {
          tma::mbar_arrive_expect_tx(&full[s], uint32_t(TT::WSTAGE));
          bulk_load(ring + s * STAGE + CH * P * 16,
                    p.w + (long long)(blockIdx.y * nkb + kb) * (TT::WSTAGE / 2),
                    uint32_t(TT::WSTAGE), &full[s]);
        }
        PadPos q = start;
#pragma unroll 4
        for (int pos = lp; pos < P; pos += STEP) {
          int yy = q.y - 1, xx = q.x - 1;
          yy += yy < 0 ? p.h : 0;
          yy -= yy >= p.h ? p.h : 0;
          xx += xx < 0 ? p.wid : 0;
          xx -= xx >= p.wid ? p.wid : 0;
          const bool ok = unsigned(q.n) < unsigned(p.n);
          const int off = p.up ? ((q.n * (p.h >> 1) + (yy >> 1)) * (p.wid >> 1) + (xx >> 1)) * p.cin
                               : ((q.n * p.h + yy) * p.wid + xx) * p.cin;
          cp_async16(dst, xc + (ok ? off : 0), ok);
          dst += STEP * 16;
          q.step(sy, sx, W2, H2);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        tma::fence_proxy_async();
        warp_arrive(&full[s], lane);
        ++fills;
        if (++s == S) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    // the MMA warp waits for every fill it uses; where it gave up, the bulk
    // copies of the last S fills may still be in flight
    if (STREAM && tid == 0) tma::drain(full, S, fills > S ? fills - S : 0, fills - 1);
  } else if (warp == MMA_WARP) {
    if (lane == 0) {
      // ---- MMA issuer: per stage, for every tap and K step of 16 channels,
      // one MMA per 128 positions
      constexpr uint32_t idesc = umma_idesc<BN>();
      // strips: 128 B between 8-row groups (SBO), P x 16 B between chunks (LBO);
      // weights likewise with BN x 16 B, or as k_tile_weights lays them out
      constexpr uint32_t AHI = (128u >> 4) | (1u << 14);
      constexpr uint32_t BHI = (STREAM ? uint32_t(9 * CH * 8) : 128u >> 4) | (1u << 14);
      const uint32_t alo = uint32_t(P) << 16, blo = (STREAM ? 8u : uint32_t(BN)) << 16;
      const uint32_t w0 = blo + (smem_u32(wsm) >> 4), r0 = alo + (smem_u32(ring) >> 4);
      int s = 0, it = 0;
      uint32_t ph = 0;
      for (int tile = blockIdx.x; tile < p.tiles && !bad; tile += gridDim.x, ++it) {
        const int b = it % NBUF;
        const uint32_t eph = uint32_t((it / NBUF) & 1) ^ 1u;
        const uint32_t acc = tmem + uint32_t(b * ACC);
        for (int kb = 0; kb < nkb; ++kb) {
          if (!tma::mbar_wait(&full[s], ph)) {
            bad = true;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a0 = r0 + uint32_t(s * (STAGE / 16));
          const uint32_t b0 = STREAM ? blo + (smem_u32(ring + s * STAGE + CH * P * 16) >> 4)
                                     : w0 + uint32_t(kb * CH * BN);
          auto mma = [&](int t, int kk, int m, auto accumulate) {
            const uint32_t at = a0 + uint32_t((t / 3) * W2 + t % 3 + 2 * kk * P);  // tap's position 0
            const uint32_t bt = b0 + (STREAM ? uint32_t((t * CH + 2 * kk) * 8)
                                             : uint32_t((t * kch + 2 * kk) * BN));
            umma_go<decltype(accumulate)::value>(acc + uint32_t(m * BN), desc_at(at + m * 128, AHI),
                                                 desc_at(bt, BHI), idesc);
          };
          if (NBUF == 1 && kb == 0) {
            // block by block, as the epilogue empties them
#pragma unroll 1
            for (int m = 0; m < MT && !bad; ++m) {
              if (!tma::mbar_wait(&tempty[m], eph)) {
                bad = true;
                break;
              }
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              mma(0, 0, m, std::false_type{});
#pragma unroll
              for (int t = 0; t < 9; ++t)
#pragma unroll
                for (int kk = 0; kk < CB / 16; ++kk)
                  if (t > 0 || kk > 0) mma(t, kk, m, std::true_type{});
            }
          } else {
            // consecutive MMAs go to different blocks
            if (NBUF == 2 && kb == 0) {
              for (int m = 0; m < MT; ++m) bad |= !tma::mbar_wait(&tempty[b * MT + m], eph);
              if (bad) break;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
              for (int m = 0; m < MT; ++m) mma(0, 0, m, std::false_type{});
            } else {
#pragma unroll
              for (int m = 0; m < MT; ++m) mma(0, 0, m, std::true_type{});
            }
#pragma unroll
            for (int kk = 1; kk < CB / 16; ++kk)
#pragma unroll
              for (int m = 0; m < MT; ++m) mma(0, kk, m, std::true_type{});
#pragma unroll 1
            for (int t = 1; t < 9; ++t)
#pragma unroll
              for (int kk = 0; kk < CB / 16; ++kk)
#pragma unroll
                for (int m = 0; m < MT; ++m) mma(t, kk, m, std::true_type{});
          }
          umma_commit(&empty[s]);
          if (++s == S) {
            s = 0;
            ph ^= 1;
          }
        }
        umma_commit(&tfull[b]);
      }
      // every MMA of this CTA done (also after giving up) before it leaves
      umma_commit(done);
      bad |= !tma::mbar_wait(done, 0);
    }
  } else {
    // ---- epilogue: a warp reads lanes 32 (warp % 4) .. + 31 of units (128
    // positions x 32 channels) g, g + G, ...
    constexpr int UNITS = MT * BN / 32, G = FL_EPI / 128;
    static_assert(UNITS % G == 0, "units per warp");
    const int lq = 32 * (warp & 3), g = (warp - MMA_WARP - 1) >> 2;
    const bool wide = p.wide != 0;
    int it = 0;
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, ++it) {
      const int b = it % NBUF;
      bool ok = tma::mbar_wait(&tfull[b], uint32_t((it / NBUF) & 1));
      ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld is warp-collective
      if (!ok) {
        bad = true;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int k = 0; k < UNITS / G; ++k) {
        const int unit = g + k * G, m = unit / (BN / 32), c = unit % (BN / 32);
        const uint32_t q = uint32_t(tile) * M + m * 128 + lq + lane;
        const uint32_t nn = q / HW2u, r = q - nn * HW2u, yq = r / W2u;
        const int yp = int(yq), xp = int(r - yq * W2u);
        const bool store =
            int(nn) < p.n && yp >= 1 && yp <= p.h && xp >= 1 && xp <= p.wid;
        const long long o =
            (((long long)nn * p.h + (yp - 1)) * p.wid + (xp - 1)) * p.cout + co0 + c * 32;
        U8 rr[2];
        if (p.res && store) {
          rr[0] = ld_32b(p.res + o, wide);
          rr[1] = ld_32b(p.res + o + 16, wide);
        }
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(tmem + (uint32_t(lq) << 16) + uint32_t(b * ACC + m * BN + c * 32), v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        // the block's share is in registers: it may be overwritten
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        warp_arrive(&tempty[b * MT + m], lane);
        if (store) {
          const float4* const bias = reinterpret_cast<const float4*>(bsm + c * 32);
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            U8 zz, aa;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float4 bb = bias[hf * 4 + e];
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                float2 f = make_float2(__uint_as_float(v[hf * 16 + 4 * e + 2 * i]),
                                       __uint_as_float(v[hf * 16 + 4 * e + 2 * i + 1]));
                f = __fadd2_rn(f, i ? make_float2(bb.z, bb.w) : make_float2(bb.x, bb.y));
                if (p.res) f = __fadd2_rn(f, f2bf(rr[hf].v[2 * e + i]));
                if (p.z) zz.v[2 * e + i] = bf2(f.x, f.y);
                if (p.a) {
                  const float2 ge = FULL ? gelu2_full(f) : gelu2(f);
                  aa.v[2 * e + i] = bf2(ge.x, ge.y);
                }
              }
            }
            if (p.z) st_32b(p.z + o + hf * 16, zz, wide);
            if (p.a) st_32b(p.a + o + hf * 16, aa, wide);
          }
        }
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(TT::COLS));
  if (bad) atomicExch(&tc_gave_up, 1);
}

// Positions of a strip and stages of the ring that fit beside the weights (0:
// fewer than two do not).
template <int BN, int MT, bool STREAM>
int flow_stages(int cin, int wid, int* P) {
  using TT = FlowTile<BN, MT, STREAM>;
  *P = (TT::M + 2 * (wid + 3) + 7) / 8 * 8;  // M positions and the taps' reach
  const int weights = STREAM ? 0 : 9 * cin * BN * 2;
  const int s = (FL_SMEM - weights) / (TT::CH * *P * 16 + TT::WSTAGE);
  return weights >= FL_SMEM || s < 2 ? 0 : s > FL_SMAX ? FL_SMAX : s;
}

// SP_EINVAL where it does not fit
template <int BN, int MT, bool STREAM = false>
int launch_flow(FlowParams p, cudaStream_t s) {
  using TT = FlowTile<BN, MT, STREAM>;
  if (p.cin % TT::CB != 0) return SP_EINVAL;
  p.S = flow_stages<BN, MT, STREAM>(p.cin, p.wid, &p.P);
  if (p.S == 0) return SP_EINVAL;
  const int smem = (STREAM ? 0 : 9 * p.cin * BN * 2) + p.S * (TT::CH * p.P * 16 + TT::WSTAGE) + 1024;
  auto kern = p.z && p.a ? k_conv3x3_flow<BN, MT, STREAM, true> : k_conv3x3_flow<BN, MT, STREAM, false>;
  const cudaError_t attr =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (attr != cudaSuccess) return SP_ECUDA;
  const long long QN = (long long)(p.h + 2) * (p.wid + 2) * p.n;
  p.tiles = int((QN + TT::M - 1) / TT::M);
  const int ny = p.cout / BN, gx = sms() / ny > 0 ? sms() / ny : 1;
  kern<<<dim3(unsigned(p.tiles < gx ? p.tiles : gx), unsigned(ny)), FL_NT, smem, s>>>(p);
  return cudaGetLastError() == cudaSuccess ? SP_OK : SP_ECUDA;
}

}  // namespace conv
}  // namespace sp
