/*
 * sp_wgrad.cuh -- the weight gradient of the 3x3 circular convolution on
 * tcgen05.  No counterpart in SymPhas.
 *
 *   dw[co][tap][c] += sum over pixels p of dy[p][co] * x[p + offset(tap)][c]
 *
 * as a GEMM with M = output channels, N = input channels and K = pixels.  Both
 * operands keep their channels contiguous in memory (MN-major): staged
 * chunk-major (one 16-byte row of 8 channels per pixel) a run of 8 pixels of a
 * chunk is one 8 x 16-byte core matrix, so the pixel index needs no
 * transposition and a horizontal tap is the x operand's start address moved by
 * whole pixels.
 *
 * Vertical taps come out of the M side.  Rows of dy are staged one after
 * another, so the 128 rows of an MMA span 128 / COB consecutive dy rows of COB
 * channels each: against one row y of x they give the sums for dy rows y - 1,
 * y, y + 1, that is for the three vertical taps.  With COB = 32 one MMA per
 * horizontal tap covers all three (and a fourth row that is dropped); with
 * COB = 64 two do; with COB = 128 a CTA handles one vertical tap and N = 128.
 * One M = 64 or padded M = 128 MMA per tap would run the tensor core at a
 * quarter or half of this.
 *
 * One CTA per SM takes a share of the pixels (split K): eight producer warps
 * gather blocks of R rows x KW columns into a ring of two stages, one thread
 * issues the MMAs into tensor memory, and the sums are added to dw once at the
 * end with 16-byte reductions.  The mma.sync kernel (k_conv3x3_wgrad) gathers
 * x nine times and stays for channel counts outside 32, 64 and multiples of
 * 128.
 */
#pragma once

namespace sp {
namespace conv {

constexpr int WG_PROD = 256, WG_NT = WG_PROD + 32, WG_S = 2;
constexpr int WG_SMEM = 226 * 1024;  // both stages

struct WgParams {
  const __nv_bfloat16* x;   // [N][H][W][Cin]
  const __nv_bfloat16* dy;  // [N][H][W][Cout]
  float* dw;                // [Cout][9][Cin], accumulated
  int n, h, wid, cin, cout;
  int KW, R;       // columns (a multiple of 16) and rows of a block
  int nbx, nby;    // blocks of an image
  int items;       // blocks in all
  int vec;         // dw allows 16-byte reductions
};

template <int COB, int N>
struct WgTile {
  static constexpr int VR = 128 / COB;               // dy rows of an MMA
  static constexpr int NV = COB == 64 ? 2 : 1;       // vertical MMAs per x row
  static constexpr int VSPLIT = COB == 128 ? 3 : 1;  // CTAs that share the vertical taps
  static constexpr int HALO = COB == 128 ? 0 : 2;    // dy rows beyond the x rows
  static constexpr int COLS = NV * 3 * N;            // accumulator columns
  static constexpr int TCOLS = COLS <= 128 ? 128 : COLS <= 256 ? 256 : 512;
  static constexpr int CHO = COB / 8, CHX = N / 8;
  static_assert(COLS <= 512 && N % 32 == 0 && N <= 128, "tile");
};

template <int COB, int N>
__global__ void __launch_bounds__(WG_NT, 1) k_wgrad_tc(const WgParams p) {
  using TT = WgTile<COB, N>;
  constexpr int CHO = TT::CHO, CHX = TT::CHX, HALO = TT::HALO, NV = TT::NV, VR = TT::VR;
  extern __shared__ __align__(1024) unsigned char smem[];
  // a stage: dy rows [(R + HALO) rows][CHO chunks][KW pixels][16 B], then x rows
  // [R][CHX][KW + 8][16 B]; the dy row an MMA reads past the last is x data,
  // and its sums are dropped
  const int KW = p.KW, XP = KW + 8;
  const int DYB = (p.R + HALO) * CHO * KW * 16, STAGE = DYB + p.R * CHX * XP * 16;
  uint64_t* const full = reinterpret_cast<uint64_t*>(smem + WG_S * STAGE);
  uint64_t *const empty = full + WG_S, *const done = empty + WG_S;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ncb = p.cin / N;
  const int vs = blockIdx.y % TT::VSPLIT;  // the vertical tap's dy row, where CTAs share them
  const int c0 = int(blockIdx.y / TT::VSPLIT) % ncb * N;
  const int co0 = int(blockIdx.y / TT::VSPLIT) / ncb * COB;
  constexpr int MMA_WARP = WG_PROD / 32;

  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(TT::TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    for (int s = 0; s < WG_S; ++s) {
      tma::mbar_init(&full[s], WG_PROD / 32);
      tma::mbar_init(&empty[s], 1);
    }
    tma::mbar_init(done, 1);
    tma::fence_barrier_init();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  bool bad = false;
  const int per = p.nbx * p.nby;

  if (warp < MMA_WARP) {
    // ---- producers: a warp copies 8 pixels x 4 chunks (64-byte segments of
    // global memory, conflict-free 128-byte runs of shared memory) at a time
    const int pl = lane & 7, ch = lane >> 3;
    int s = 0;
    uint32_t ph = 1;
    for (int item = blockIdx.x; item < p.items; item += gridDim.x) {
      const int img = item / per, rem = item - img * per, by = rem / p.nbx;
      const int x0 = (rem - by * p.nbx) * KW, y0 = by * p.R;
      const int kw = min(KW, p.wid - x0), rows = min(p.R, p.h - y0);
      if (!tma::mbar_wait(&empty[s], ph)) {
        bad = true;
        break;
      }
      unsigned char* const st = smem + s * STAGE;
      const long long base = (long long)img * p.h;
      for (int pb = warp; pb < XP / 8; pb += WG_PROD / 32) {
        const int px = pb * 8 + pl;
        if (pb < KW / 8) {
          const bool ok = px < kw;  // zeros beyond the row: they add nothing
          const __nv_bfloat16* const src =
              p.dy + (base * p.wid + (ok ? x0 + px : 0)) * p.cout + co0 + ch * 8;
          unsigned char* dst = st + (ch * KW + px) * 16;
          for (int r = 0; r < rows + HALO; ++r) {
            int yy = y0 + r + (HALO ? -1 : vs - 1);
            yy += yy < 0 ? p.h : 0;
            yy -= yy >= p.h ? p.h : 0;
            const __nv_bfloat16* const row = src + (long long)yy * p.wid * p.cout;
#pragma unroll
            for (int g = 0; g < CHO / 4; ++g)
              cp_async16(dst + g * 4 * KW * 16, row + g * 32, ok);
            dst += CHO * KW * 16;
          }
        }
        {
          // x columns x0 - 1 .. x0 + kw, around the row's ends
          const bool ok = px < kw + 2;
          int xx = x0 + px - 1;
          xx += xx < 0 ? p.wid : 0;
          xx -= xx >= p.wid ? p.wid : 0;
          const __nv_bfloat16* row =
              p.x + ((base + y0) * p.wid + (ok ? xx : 0)) * p.cin + c0 + ch * 8;
          unsigned char* dst = st + DYB + (ch * XP + px) * 16;
          for (int r = 0; r < rows; ++r) {
#pragma unroll
            for (int g = 0; g < CHX / 4; ++g)
              cp_async16(dst + g * 4 * XP * 16, row + g * 32, ok);
            row += (long long)p.wid * p.cin;
            dst += CHX * XP * 16;
          }
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      tma::fence_proxy_async();
      warp_arrive(&full[s], lane);
      if (++s == WG_S) {
        s = 0;
        ph ^= 1;
      }
    }
  } else if (lane == 0) {
    // ---- MMA issuer.  M = 128, both operands MN-major (bits 15 and 16); LBO
    // is the distance of 8 pixels (K), SBO that of 8 channels (M or N)
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                               (uint32_t(N >> 3) << 17) | (uint32_t(128 >> 4) << 24);
    const uint32_t ahi = uint32_t(KW) | (1u << 14), bhi = uint32_t(XP) | (1u << 14);
    const uint32_t base = (128u >> 4) << 16;
    int s = 0;
    uint32_t ph = 0;
    bool first = true;
    for (int item = blockIdx.x; item < p.items && !bad; item += gridDim.x) {
      const int rem = item % per, by = rem / p.nbx;
      const int rows = min(p.R, p.h - by * p.R);
      if (!tma::mbar_wait(&full[s], ph)) {
        bad = true;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a0 = base + (smem_u32(smem + s * STAGE) >> 4);
      const uint32_t b0 = base + (smem_u32(smem + s * STAGE + DYB) >> 4);
      for (int r = 0; r < rows; ++r)
        for (int k = 0; k < KW; k += 16) {
          const uint32_t ar = a0 + uint32_t(r * CHO * KW + k);
          const uint32_t br = b0 + uint32_t(r * CHX * XP + k);
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            const uint64_t ad = desc_at(ar + uint32_t(v * VR * CHO * KW), ahi);
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
              const uint32_t d = tmem + uint32_t((v * 3 + dx) * N);
              if (first)
                umma_go<false>(d, ad, desc_at(br + dx, bhi), idesc);
              else
                umma_go<true>(d, ad, desc_at(br + dx, bhi), idesc);
            }
          }
          first = false;
        }
      umma_commit(&empty[s]);
      if (++s == WG_S) {
        s = 0;
        ph ^= 1;
      }
    }
    umma_commit(done);
    bad |= !tma::mbar_wait(done, 0);
  }
  if (warp < MMA_WARP) {
    // ---- the sums: lane = M row = (dy row d, output channel), columns = input
    // channels; dy row d against x row y is the tap with vertical index 2 - d
    bad |= !tma::mbar_wait(done, 0);
    const bool ok = __all_sync(0xffffffffu, !bad);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int quarter = warp & 3, row = 32 * quarter + lane;
    for (int blk = warp >> 2; blk < TT::COLS / 32; blk += WG_PROD / 128) {
      uint32_t v[32];
      __syncwarp();
      tmem_ld32(tmem + (uint32_t(32 * quarter) << 16) + uint32_t(blk * 32), v);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      const int col = blk * 32, vd = col / N, c = col - vd * N;
      const int d = COB == 128 ? vs : (vd / 3) * VR + row / COB;
      if (!ok || d > 2) continue;
      float* const o = p.dw + ((long long)(co0 + row % COB) * 9 + (2 - d) * 3 + vd % 3) * p.cin +
                       c0 + c;
      if (p.vec) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o + 4 * i),
                       "f"(__uint_as_float(v[4 * i])), "f"(__uint_as_float(v[4 * i + 1])),
                       "f"(__uint_as_float(v[4 * i + 2])), "f"(__uint_as_float(v[4 * i + 3]))
                       : "memory");
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) atomicAdd(o + i, __uint_as_float(v[i]));
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(TT::TCOLS));
  if (bad) atomicExch(&tc_gave_up, 1);
}

template <int COB, int N>
int launch_wgrad(WgParams p, cudaStream_t s) {
  using TT = WgTile<COB, N>;
  // columns: blocks of at most 128, of equal width up to the 16 pixels of an
  // MMA's K; rows: as many as two stages hold, at most 8 (more rows read the
  // dy rows above and below less often, and leave fewer blocks to share out)
  p.nbx = (p.wid + 127) / 128;
  p.KW = ((p.wid + p.nbx - 1) / p.nbx + 15) / 16 * 16;
  p.nbx = (p.wid + p.KW - 1) / p.KW;
  const int dyrow = TT::CHO * p.KW * 16, xrow = TT::CHX * (p.KW + 8) * 16;
  p.R = (WG_SMEM / WG_S - TT::HALO * dyrow) / (dyrow + xrow);
  // the dy row an MMA reads past a stage's last lies in its x rows, or in the
  // next stage, or (the last stage) in the barriers' slack below
  if (p.R < 1) return SP_EINVAL;
  p.R = p.R < 8 ? p.R : 8;
  p.R = p.R < p.h ? p.R : p.h;
  p.nby = (p.h + p.R - 1) / p.R;
  const long long items = (long long)p.n * p.nbx * p.nby;
  if (items >= (1LL << 31)) return SP_EINVAL;
  p.items = int(items);
  const int stage = (p.R + TT::HALO) * dyrow + p.R * xrow;
  int smem = WG_S * stage + 64;
  // the spare dy row of the last stage's last x row must lie inside
  const int need = stage * (WG_S - 1) + (p.R + TT::HALO + (TT::HALO ? 1 : 0)) * dyrow;
  if (smem < need) smem = need;
  if (smem > 227 * 1024) return SP_EINVAL;
  const cudaError_t attr = cudaFuncSetAttribute(
      k_wgrad_tc<COB, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (attr != cudaSuccess) return SP_ECUDA;
  const int ny = TT::VSPLIT * (p.cin / N) * (p.cout / COB);
  const int gx = sms() / ny > 0 ? sms() / ny : 1;
  k_wgrad_tc<COB, N><<<dim3(unsigned(p.items < gx ? p.items : gx), unsigned(ny)), WG_NT, smem, s>>>(
      p);
  return cudaGetLastError() == cudaSuccess ? SP_OK : SP_ECUDA;
}

// the tensor-memory kernel where its tiles fit the channels, else SP_EINVAL
inline int wgrad_tc(const WgParams& p, cudaStream_t s) {
  const int n = p.cin % 128 == 0 ? 128 : p.cin % 64 == 0 ? 64 : 32;
  if (p.cout == 32)
    return n == 128 ? launch_wgrad<32, 128>(p, s)
           : n == 64 ? launch_wgrad<32, 64>(p, s)
                     : launch_wgrad<32, 32>(p, s);
  if (p.cout == 64)
    return n >= 64 ? launch_wgrad<64, 64>(p, s) : launch_wgrad<64, 32>(p, s);
  if (p.cout % 128 == 0)
    return n == 128 ? launch_wgrad<128, 128>(p, s)
           : n == 64 ? launch_wgrad<128, 64>(p, s)
                     : launch_wgrad<128, 32>(p, s);
  return SP_EINVAL;
}

}  // namespace conv
}  // namespace sp
