/*
 * sp_ends.cuh -- the jump network's first and last convolutions at inference,
 * and the element-wise backward of a layer in training.  No counterpart in
 * SymPhas.
 *
 * The first layer's input has one channel that is not zero and the last
 * layer's output one channel that is used, so as 32-channel convolutions they
 * move and multiply 32 times what they need.  Here the first reads the fp32
 * field and writes its activations, the last reads activations and writes the
 * fp32 field: both are bound by the one 64-byte-per-pixel side (0.27 GB for 64
 * fields of 256^2: 42 us at 6460 GB/s).
 */
#pragma once

namespace sp {
namespace conv {

// a[n][y][x][co] = gelu(bias[co] + sum over the taps of w[co][tap][0] *
// bf16(psi)), circular.  A CTA takes 64 columns x 32 output channels and
// marches down R rows: four lanes a pixel, each with the 72 weights of its 8
// channels in registers and the 3 x 3 window of psi, of which a row adds three.
constexpr int IN1_NT = 256, IN1_X = 64, IN1_R = 32;
__global__ void __launch_bounds__(IN1_NT, 2)
    k_conv3x3_in1(const float* __restrict__ psi, const __nv_bfloat16* __restrict__ w,
                  const float* __restrict__ bias, __nv_bfloat16* __restrict__ a, int h, int wid,
                  int cin, int cout) {
  const int co = blockIdx.z % (cout / 32) * 32 + (threadIdx.x & 3) * 8;
  const long long img = blockIdx.z / (cout / 32);
  const int x = blockIdx.x * IN1_X + (threadIdx.x >> 2), y0 = blockIdx.y * IN1_R;
  __shared__ __align__(16) float ws[10][32];  // taps and bias of the 32 channels
  for (int i = threadIdx.x; i < 320; i += IN1_NT) {
    const int t = i >> 5, c = co - (threadIdx.x & 3) * 8 + (i & 31);
    ws[t][i & 31] = t == 9 ? (bias ? bias[c] : 0.f) : __bfloat162float(w[((long long)c * 9 + t) * cin]);
  }
  __syncthreads();
  float2 wt[9][4], b[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    b[e] = *reinterpret_cast<const float2*>(&ws[9][(threadIdx.x & 3) * 8 + 2 * e]);
#pragma unroll
    for (int t = 0; t < 9; ++t)
      wt[t][e] = *reinterpret_cast<const float2*>(&ws[t][(threadIdx.x & 3) * 8 + 2 * e]);
  }
  if (x >= wid) return;
  const int xl = x == 0 ? wid - 1 : x - 1, xr = x == wid - 1 ? 0 : x + 1;
  const float* const f = psi + img * h * wid;
  const int ye = min(y0 + IN1_R, h);
  auto row = [&](int y, float (&v)[3]) {
    y = min(y, ye);  // (rows past the last one needed are not used)
    const float* const r = f + (long long)(y < 0 ? y + h : y >= h ? y - h : y) * wid;
    v[0] = __ldg(r + xl);
    v[1] = __ldg(r + x);
    v[2] = __ldg(r + xr);
  };
  auto put = [&](float (&d)[3], const float (&s)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) d[i] = __bfloat162float(__float2bfloat16_rn(s[i]));
  };
  // one row in flight; a row is rounded where it is used, not where it is loaded
  float v[3][3], n1[3];
  {
    float r0[3], r1[3];
    row(y0 - 1, r0);
    row(y0, r1);
    row(y0 + 1, n1);
    put(v[0], r0);
    put(v[1], r1);
  }
  __nv_bfloat16* o = a + ((img * h + y0) * wid + x) * cout + co;
  for (int y = y0; y < ye; ++y) {
    put(v[2], n1);
    row(y + 2, n1);
    float2 z[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      z[e] = b[e];
#pragma unroll
      for (int t = 0; t < 9; ++t)
        z[e] = __ffma2_rn(wt[t][e], make_float2(v[t / 3][t % 3], v[t / 3][t % 3]), z[e]);
      z[e] = gelu2(z[e]);
    }
    *reinterpret_cast<uint4*>(o) = make_uint4(bf2(z[0].x, z[0].y), bf2(z[1].x, z[1].y),
                                              bf2(z[2].x, z[2].y), bf2(z[3].x, z[3].y));
    o += (long long)wid * cout;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      v[0][i] = v[1][i];
      v[1][i] = v[2][i];
    }
  }
}

// out[n][y][x] = bias[0] + sum over taps and channels of w[0][tap][c] * x,
// circular, fp32.  A CTA holds 64 columns (62 outputs) and marches down R
// rows: lane group of cin / 8 lanes a pixel, each with the 72 weights of its 8
// channels.  A row of x adds to three output rows and three horizontal taps,
// nine sums a lane; an output row that has its three rows is summed over the
// group by shuffles and over its three columns through shared memory.
constexpr int OUT1_NT = 256, OUT1_R = 64;
template <int CIN>
__global__ void __launch_bounds__(OUT1_NT, 2)
    k_conv3x3_out1(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   const float* __restrict__ bias, float* __restrict__ out, int h, int wid) {
  constexpr int GL = CIN / 8, COLS = OUT1_NT / GL;  // lanes a pixel, columns of a CTA
  constexpr int RB = 4;  // rows between barriers
  __shared__ float vs[2][RB][3][COLS];
  const int c0 = (threadIdx.x % GL) * 8, col = threadIdx.x / GL;
  const int x0 = blockIdx.x * (COLS - 2), y0 = blockIdx.y * OUT1_R;
  const long long img = blockIdx.z;
  int xx = x0 - 1 + col;  // the column this group reads; columns past the edge wrap
  xx += xx < 0 ? wid : 0;
  xx %= wid;
  float2 wt[9][4];
#pragma unroll
  for (int t = 0; t < 9; ++t) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(w + t * CIN + c0));
    wt[t][0] = f2bf(u.x);
    wt[t][1] = f2bf(u.y);
    wt[t][2] = f2bf(u.z);
    wt[t][3] = f2bf(u.w);
  }
  const float b = bias ? bias[0] : 0.f;
  const __nv_bfloat16* const f = x + (img * h * wid + xx) * CIN + c0;
  const int ye = min(y0 + OUT1_R, h);
  auto load = [&](int y) {
    y = min(y, ye);  // (rows past the last one needed are not used)
    y += y < 0 ? h : 0;
    y -= y >= h ? h : 0;
    return __ldg(reinterpret_cast<const uint4*>(f + (long long)y * wid * CIN));
  };
  float2 s[3][3];  // [output row y - 1, y, y + 1][horizontal tap]
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int d = 0; d < 3; ++d) s[i][d] = make_float2(0.f, 0.f);
  // one row of x: it adds to three output rows; `t`, if not null, gets the column
  // sums of output row y - 1, which is then complete
  auto row = [&](const uint4& cur, float* t) {
    const float2 v[4] = {f2bf(cur.x), f2bf(cur.y), f2bf(cur.z), f2bf(cur.w)};
    // row y is the lower row (dy = +1) of output y - 1, the centre of y, the
    // upper row (dy = -1) of y + 1
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[i][d] = __ffma2_rn(wt[(2 - i) * 3 + d][e], v[e], s[i][d]);
    if (t) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        float u = s[0][d].x + s[0][d].y;
#pragma unroll
        for (int m = GL / 2; m > 0; m >>= 1) u += __shfl_xor_sync(0xffffffffu, u, m);
        if (threadIdx.x % GL == 0) t[d * COLS + col] = u;
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      s[0][d] = s[1][d];
      s[1][d] = s[2][d];
      s[2][d] = make_float2(0.f, 0.f);
    }
  };
  row(load(y0 - 1), nullptr);
  row(load(y0), nullptr);
  uint4 nx[RB];  // the next rows, in flight
#pragma unroll
  for (int k = 0; k < RB; ++k) nx[k] = load(y0 + 1 + k);
  int buf = 0;
  for (int o = y0; o < ye; o += RB, buf ^= 1) {
    uint4 cur[RB];
#pragma unroll
    for (int k = 0; k < RB; ++k) cur[k] = nx[k];
#pragma unroll
    for (int k = 0; k < RB; ++k) nx[k] = load(o + RB + 1 + k);
#pragma unroll
    for (int k = 0; k < RB; ++k) row(cur[k], &vs[buf][k][0][0]);
    // one barrier: the other buffer's readers passed the one before
    __syncthreads();
#pragma unroll
    for (int k = 0; k < (RB * COLS + OUT1_NT - 1) / OUT1_NT; ++k) {
      const int i = threadIdx.x + k * OUT1_NT, r = i / COLS, c = i - r * COLS;
      if (r < RB && c < COLS - 2 && x0 + c < wid && o + r < ye)
        out[(img * h + o + r) * wid + x0 + c] =
            b + ((vs[buf][r][0][c] + vs[buf][r][1][c + 1]) + vs[buf][r][2][c + 2]);
    }
  }
}

// The derivative of gelu (tanh form) at z, from one exponential of a
// non-positive argument (no overflow, no cancellation in 1 - tanh^2):
// with s = sigmoid(2 u), 0.5 (1 + tanh u) = s and 0.5 (1 - tanh^2 u) = 2 s (1 - s).
__device__ __forceinline__ float gelu_grad(float z) {
  const float k = 0.7978845608028654f, q = 0.044715f;
  const float z2 = z * z, u = k * z * fmaf(q, z2, 1.f);
  const float e = __expf(-2.f * fabsf(u)), r = __fdividef(1.f, 1.f + e);
  const float s = u >= 0.f ? r : e * r, ss = e * r * r;
  return fmaf(2.f * z * ss, k * fmaf(3.f * q, z2, 1.f), s);
}

// dz = da * gelu'(z) (bf16) and the column sums of dz as stored; with z null
// only the sums of da.  One pass over memory where torch took four (the
// derivative, a cast to fp32, a reduction, an addition).  A thread owns 8
// channels of every (blockDim / groups)-th pixel.  A CTA's sums go to its row
// of `part` ([CTA][c], added up by k_bias_sum: the same bits in every run), or,
// where there is none, to db in the order in which the CTAs end.
constexpr int GB_NT = 256;
template <bool Z>
__global__ void __launch_bounds__(GB_NT)
    k_gelu_bwd(const __nv_bfloat16* __restrict__ z, const __nv_bfloat16* __restrict__ da,
               __nv_bfloat16* __restrict__ dz, float* __restrict__ db, float* __restrict__ part,
               long long npix, int cs) {
  extern __shared__ float sums[];  // [rows of a block][c]
  const int c0 = blockIdx.y * 8 * GB_NT, c = min(cs - c0, 8 * GB_NT);  // this CTA's channels
  const int cg = c / 8, rows = GB_NT / cg;
  const int g = threadIdx.x % cg, r = threadIdx.x / cg;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  if (r < rows) {
    const long long step = (long long)gridDim.x * rows;
    constexpr int U = 4;  // pixels whose loads are issued together
    for (long long p = (long long)blockIdx.x * rows + r; p < npix; p += U * step) {
      uint4 d[U], zz[U];
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (p + k * step < npix) {
          const long long o = (p + k * step) * cs + c0 + g * 8;
          d[k] = __ldg(reinterpret_cast<const uint4*>(da + o));
          if constexpr (Z) zz[k] = __ldg(reinterpret_cast<const uint4*>(z + o));
        }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        if (p + k * step >= npix) break;
        uint32_t* const dv = reinterpret_cast<uint32_t*>(&d[k]);
        if constexpr (Z) {
          const uint32_t* const zv = reinterpret_cast<const uint32_t*>(&zz[k]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = f2bf(zv[e]), y = f2bf(dv[e]);
            dv[e] = bf2(y.x * gelu_grad(f.x), y.y * gelu_grad(f.y));
          }
          *reinterpret_cast<uint4*>(dz + (p + k * step) * cs + c0 + g * 8) = d[k];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 y = f2bf(dv[e]);
          acc[2 * e] += y.x;
          acc[2 * e + 1] += y.y;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) sums[r * c + g * 8 + e] = acc[e];
  }
  __syncthreads();
  if (!db && !part) return;
  for (int i = threadIdx.x; i < c; i += GB_NT) {
    float t = 0.f;
    for (int k = 0; k < rows; ++k) t += sums[k * c + i];
    if (part)
      part[(long long)blockIdx.x * cs + c0 + i] = t;
    else
      atomicAdd(db + c0 + i, t);
  }
}

// db[c] += the sum of part[0 .. rows - 1][c], in a fixed order: 32 channels a
// CTA, each by 32 lanes over every 32nd row.  A launch and the latency of a lane's
// up to 28 rows (6 CTAs on each of 148 SMs), of which 14 are in flight: with
// k_gelu_bwd 55.4 us for 32 channels of 16 x 256^2 pixels (57.4 with 4 in flight;
// 49.3 with the CTAs' atomics, whose order differs from run to run).
__global__ void __launch_bounds__(1024)
    k_bias_sum(const float* part, float* __restrict__ db, int rows, int cs) {
  __shared__ float s[32][33];
  constexpr int U = 14;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, c = blockIdx.x * 32 + x;
  float t = 0.f;
  for (int r = y; r < rows; r += 32 * U) {
    float v[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      v[k] = c < cs && r + 32 * k < rows ? part[(long long)(r + 32 * k) * cs + c] : 0.f;
#pragma unroll
    for (int k = 0; k < U; ++k) t += v[k];
  }
  s[y][x] = t;
  __syncthreads();
  t = s[x][y];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if (x == 0 && blockIdx.x * 32 + y < cs) db[blockIdx.x * 32 + y] += t;
}

inline bool al16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace conv
}  // namespace sp

extern "C" int sp_conv3x3_in1(const float* psi, const void* w, const float* bias, void* a, int n,
                              int h, int w_, int cin, int cout, void* stream) {
  using namespace sp::conv;
  if (!psi || !w || !a || n < 1 || h < 1 || w_ < 1 || cin < 1 || cout < 32 || cout % 32 != 0 ||
      !al16(a))
    return SP_EINVAL;
  const long long gz = (long long)n * (cout / 32), gy = (h + IN1_R - 1) / IN1_R;
  if (gz > 65535 || gy > 65535) return SP_EINVAL;
  k_conv3x3_in1<<<dim3(unsigned((w_ + IN1_X - 1) / IN1_X), unsigned(gy), unsigned(gz)), IN1_NT, 0,
                  static_cast<cudaStream_t>(stream)>>>(
      psi, static_cast<const __nv_bfloat16*>(w), bias, static_cast<__nv_bfloat16*>(a), h, w_, cin,
      cout);
  return cudaGetLastError() == cudaSuccess ? SP_OK : SP_ECUDA;
}

extern "C" int sp_conv3x3_out1(const void* x, const void* w, const float* bias, float* out, int n,
                               int h, int w_, int cin, void* stream) {
  using namespace sp::conv;
  if (!x || !w || !out || n < 1 || h < 1 || w_ < 1 || !(cin == 32 || cin == 64) || !al16(x) ||
      !al16(w))
    return SP_EINVAL;
  const int cols = OUT1_NT / (cin / 8) - 2;
  const long long gy = (h + OUT1_R - 1) / OUT1_R;
  if (n > 65535 || gy > 65535) return SP_EINVAL;
  const dim3 grid(unsigned((w_ + cols - 1) / cols), unsigned(gy), unsigned(n));
  auto kern = cin == 32 ? k_conv3x3_out1<32> : k_conv3x3_out1<64>;
  kern<<<grid, OUT1_NT, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), bias, out, h, w_);
  return cudaGetLastError() == cudaSuccess ? SP_OK : SP_ECUDA;
}

namespace {
// CTAs along the pixels: 6 an SM, each of which adds its c sums once
long long gelu_bwd_rows(long long npix, int c) {
  using namespace sp::conv;
  const int rows = GB_NT / ((c < 8 * GB_NT ? c : 8 * GB_NT) / 8);
  const long long want = (npix + rows - 1) / rows, most = 6LL * sms();
  return want < most ? want : most;
}

int gelu_bwd(const void* z, const void* da, void* dz, float* db, float* part, long long npix, int c,
             void* stream) {
  using namespace sp::conv;
  if (!da || npix < 1 || c < 8 || c % 8 != 0 || !al16(da) || !al16(z) ||
      !al16(dz) || (z ? !dz : !db))
    return SP_EINVAL;
  // blocks of at most 2048 channels (one lane group of 8 a thread)
  const int ny = (c + 8 * GB_NT - 1) / (8 * GB_NT);
  if (ny > 65535) return SP_EINVAL;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int rows = int(gelu_bwd_rows(npix, c));
  if (!db) part = nullptr;
  auto kern = z ? k_gelu_bwd<true> : k_gelu_bwd<false>;
  // a row of sums per pixel lane: 8 KB at most, whatever the channel count
  kern<<<dim3(unsigned(rows), unsigned(ny)), GB_NT, 8 * GB_NT * int(sizeof(float)), s>>>(
      static_cast<const __nv_bfloat16*>(z), static_cast<const __nv_bfloat16*>(da),
      static_cast<__nv_bfloat16*>(dz), db, part, npix, c);
  if (part) k_bias_sum<<<unsigned((c + 31) / 32), 1024, 0, s>>>(part, db, rows, c);
  return cudaGetLastError() == cudaSuccess ? SP_OK : SP_ECUDA;
}
}  // namespace

extern "C" int sp_gelu_bwd_bf16(const void* z, const void* da, void* dz, float* db, long long npix,
                                int c, void* stream) {
  return gelu_bwd(z, da, dz, db, nullptr, npix, c, stream);
}

extern "C" int sp_gelu_bwd_scratch(long long npix, int c, long long* floats) {
  if (npix < 1 || c < 8 || c % 8 != 0 || !floats) return SP_EINVAL;
  *floats = gelu_bwd_rows(npix, c) * c;
  return SP_OK;
}

extern "C" int sp_gelu_bwd_ordered_bf16(const void* z, const void* da, void* dz, float* db,
                                        float* scratch, long long npix, int c, void* stream) {
  if (!db || !scratch) return SP_EINVAL;
  return gelu_bwd(z, da, dz, db, scratch, npix, c, stream);
}
