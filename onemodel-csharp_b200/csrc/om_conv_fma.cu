// Convolution on the fp32 FMA pipe straight from NCHW tensors, for the shapes whose product is too small for its unfolded matrix:
// the first layer of a network (1 or 3 input channels), and the few-channel layers whose pitches keep them off the tensor pipe.
// Unfolding wrote and read 9 times the input, the products then ran as one small matrix per image, and the bias was a pass of
// its own: 256 images of 3 x 32 x 32 to 64 channels took 157 us forward (67 MB written: 10 us), 69 now.
//
// Every forward value is one accumulator over k = (c, ky, kx) in increasing order; every input gradient is, tap by tap in
// increasing (ky, kx), one accumulator over the output channels, the taps' sums added in order: the bits of the product on the
// unfolded matrix and of its fold. What bounds the kernels is the load/store unit (4 loads and 8 broadcast words of the weights
// for 32 multiply-adds of a thread), and at a few hundred CTAs the latency of the loads.
#include "om_conv.cuh"

namespace om {

constexpr int CF_CH = 32;              // channels of a CTA: 8 for each of its four warps
constexpr int CF_PX = 4;               // pixels of a thread, 32 apart: a warp's load is one row segment
constexpr int CF_TILE = 32 * CF_PX;    // pixels of a CTA
constexpr int CF_CHUNK = 64;           // k's (channels, for the input gradient) of weights in shared memory at a time
constexpr int CF_MAX_TAPS = 32;

// The taps (bits in (ky, kx) order) of a window with its first tap at (y0, x0) that lie inside the image.
__device__ __forceinline__ uint32_t taps_inside(const ConvGeom& g, int y0, int x0) {
  uint32_t row = 0, mask = 0;
  for (int kx = 0; kx < g.kw; kx++)
    if ((unsigned)(x0 + kx * g.dw) < (unsigned)g.w) row |= 1u << kx;
  for (int ky = 0; ky < g.kh; ky++)
    if ((unsigned)(y0 + ky * g.dh) < (unsigned)g.h) mask |= row << (ky * g.kw);
  return mask;
}

__global__ void __launch_bounds__(128)
conv_fma_fwd_kernel(const ConvGeom g, const float* x, const float* w, const float* bias, float* __restrict__ y) {
  pdl_enter();
  __shared__ __align__(16) float ws[CF_CHUNK][CF_CH];
  __shared__ int2 ks[CF_CHUNK];        // offset of k in the image, its tap's bit
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int plane = g.oh * g.ow, hw = g.h * g.w, taps = g.kh * g.kw, kk = g.cin * taps;
  const int pixels = g.n * plane, co0 = blockIdx.y * CF_CH;
  const float* base[CF_PX];
  uint32_t mask[CF_PX];
#pragma unroll
  for (int j = 0; j < CF_PX; j++) {
    const int q = blockIdx.x * CF_TILE + j * 32 + lane;
    mask[j] = 0;
    base[j] = x;
    if (q < pixels) {
      const int n = q / plane, r = q - n * plane;
      const int y0 = (r / g.ow) * g.sh - g.pt, x0 = (r % g.ow) * g.sw - g.pl;
      mask[j] = taps_inside(g, y0, x0);
      base[j] = x + (long long)n * g.cin * hw + (long long)y0 * g.w + x0;
    }
  }
  float acc[8][CF_PX];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < CF_PX; j++) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < kk; k0 += CF_CHUNK) {
    const int kn = min(CF_CHUNK, kk - k0);
    __syncthreads();
    for (int i = threadIdx.x; i < CF_CHUNK * CF_CH; i += 128) {
      const int k = i % CF_CHUNK, c = i / CF_CHUNK;
      if (k < kn) ws[k][c] = co0 + c < g.cout ? ld_global(w + (long long)(co0 + c) * kk + k0 + k) : 0.f;
    }
    if (threadIdx.x < kn) {
      const int k = k0 + threadIdx.x, c = k / taps, t = k - c * taps;
      ks[threadIdx.x] = make_int2(c * hw + (t / g.kw) * g.dh * g.w + (t % g.kw) * g.dw, (int)(1u << t));
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < kn; k++) {
      const int2 e = ks[k];
      float v[CF_PX];
#pragma unroll
      for (int j = 0; j < CF_PX; j++) v[j] = (mask[j] & (uint32_t)e.y) ? ld_global(base[j] + e.x) : 0.f;
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&ws[k][warp * 8 + i]);
#pragma unroll
        for (int j = 0; j < CF_PX; j++) {
          acc[i][j] = fmaf(a.x, v[j], acc[i][j]);
          acc[i + 1][j] = fmaf(a.y, v[j], acc[i + 1][j]);
          acc[i + 2][j] = fmaf(a.z, v[j], acc[i + 2][j]);
          acc[i + 3][j] = fmaf(a.w, v[j], acc[i + 3][j]);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < CF_PX; j++) {
    const int q = blockIdx.x * CF_TILE + j * 32 + lane;
    if (q >= pixels) break;
    const int n = q / plane, r = q - n * plane;
    float* out = y + ((long long)n * g.cout + co0 + warp * 8) * plane + r;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int co = co0 + warp * 8 + i;
      if (co < g.cout) out[(long long)i * plane] = bias ? acc[i][j] + ld_global(bias + co) : acc[i][j];
    }
  }
}

__global__ void __launch_bounds__(128)
conv_fma_dgrad_kernel(const ConvGeom g, const float* gr, const float* w, float* __restrict__ dx) {
  pdl_enter();
  __shared__ __align__(16) float ws[CF_CHUNK][CF_CH];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int plane = g.oh * g.ow, hw = g.h * g.w, taps = g.kh * g.kw, kk = g.cin * taps;
  const int pixels = g.n * hw, c0 = blockIdx.y * CF_CH;
  int py[CF_PX], pxx[CF_PX];
  const float* image[CF_PX];
#pragma unroll
  for (int j = 0; j < CF_PX; j++) {
    const int q = blockIdx.x * CF_TILE + j * 32 + lane;
    const int n = q < pixels ? q / hw : 0, r = q < pixels ? q - n * hw : 0;
    py[j] = q < pixels ? r / g.w + g.pt : -1;      // (a row above every tap's reach: no tap lands on it)
    pxx[j] = r % g.w + g.pl;
    image[j] = gr + (long long)n * g.cout * plane;
  }
  float total[8][CF_PX];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < CF_PX; j++) total[i][j] = 0.f;
  for (int t = 0; t < taps; t++) {
    const int ky = t / g.kw, kx = t % g.kw;
    bool on[CF_PX];
    const float* src[CF_PX];
#pragma unroll
    for (int j = 0; j < CF_PX; j++) {
      const int ty = py[j] - ky * g.dh, tx = pxx[j] - kx * g.dw;
      const int oy = ty / g.sh, ox = tx / g.sw;
      on[j] = ty >= 0 && tx >= 0 && oy * g.sh == ty && ox * g.sw == tx && oy < g.oh && ox < g.ow;
      src[j] = image[j] + (on[j] ? oy * g.ow + ox : 0);
    }
    float acc[8][CF_PX];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int j = 0; j < CF_PX; j++) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < g.cout; k0 += CF_CHUNK) {
      const int kn = min(CF_CHUNK, g.cout - k0);
      __syncthreads();
      for (int i = threadIdx.x; i < CF_CHUNK * CF_CH; i += 128) {
        const int c = i % CF_CH, k = i / CF_CH;
        if (k < kn) ws[k][c] = c0 + c < g.cin ? ld_global(w + (long long)(k0 + k) * kk + (c0 + c) * taps + t) : 0.f;
      }
      __syncthreads();
#pragma unroll 4
      for (int k = 0; k < kn; k++) {
        float v[CF_PX];
#pragma unroll
        for (int j = 0; j < CF_PX; j++) v[j] = on[j] ? ld_global(src[j] + (long long)(k0 + k) * plane) : 0.f;
        const float4 a = *reinterpret_cast<const float4*>(&ws[k][warp * 8]), b = *reinterpret_cast<const float4*>(&ws[k][warp * 8 + 4]);
        const float wv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int j = 0; j < CF_PX; j++) acc[i][j] = fmaf(wv[i], v[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int j = 0; j < CF_PX; j++)
        if (on[j]) total[i][j] += acc[i][j];
  }
#pragma unroll
  for (int j = 0; j < CF_PX; j++) {
    const int q = blockIdx.x * CF_TILE + j * 32 + lane;
    if (q >= pixels) break;
    const int n = q / hw, r = q - n * hw;
    float* out = dx + ((long long)n * g.cin + c0 + warp * 8) * hw + r;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (c0 + warp * 8 + i < g.cin) out[(long long)i * hw] = total[i][j];
  }
}

// part[slice][co][k] = sum over the slice's pixels of g[co, pixel] x[k's channel, pixel's input position of k's tap]. A CTA: 32 output
// channels (8 a warp) x 128 k's (lane + 32 j) over its slice, 32 pixels at a time turned through shared memory: both
// operands as rows of pixels, read four pixels at a time (rows of 36 floats: no bank conflicts).
constexpr int CF_COLS = 128, CF_LD = 36;
__global__ void __launch_bounds__(128)
conv_fma_wgrad_kernel(const ConvGeom g, const float* gr, const float* x, int per_slice, float* __restrict__ part) {
  pdl_enter();
  __shared__ __align__(16) float gs[CF_CH][CF_LD];
  __shared__ __align__(16) float xs[CF_COLS][CF_LD];
  __shared__ int2 ks[CF_COLS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int plane = g.oh * g.ow, hw = g.h * g.w, taps = g.kh * g.kw, kk = g.cin * taps;
  const int pixels = g.n * plane, k0 = blockIdx.x * CF_COLS, co0 = blockIdx.y * CF_CH;
  const int q_begin = blockIdx.z * per_slice, q_end = min(pixels, q_begin + per_slice);
  {
    const int k = k0 + threadIdx.x, c = k / taps, t = k - c * taps;
    ks[threadIdx.x] = k < kk ? make_int2(c * hw + (t / g.kw) * g.dh * g.w + (t % g.kw) * g.dw, (int)(1u << t)) : make_int2(0, 0);
  }
  const int cols = min(CF_COLS, kk - k0);
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
  for (int q0 = q_begin; q0 < q_end; q0 += 32) {
    const int q = q0 + lane;
    const bool inside = q < q_end;
    uint32_t mask = 0;
    const float *xb = x, *gb = gr;
    if (inside) {
      const int n = q / plane, r = q - n * plane;
      const int y0 = (r / g.ow) * g.sh - g.pt, x0 = (r % g.ow) * g.sw - g.pl;
      mask = taps_inside(g, y0, x0);
      xb = x + (long long)n * g.cin * hw + (long long)y0 * g.w + x0;
      gb = gr + ((long long)n * g.cout + co0) * plane + r;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < CF_CH / 4; i++) {
      const int c = warp + 4 * i;
      gs[c][lane] = inside && co0 + c < g.cout ? ld_global(gb + (long long)c * plane) : 0.f;
    }
#pragma unroll 8
    for (int k = warp; k < cols; k += 4) {
      const int2 e = ks[k];
      xs[k][lane] = (mask & (uint32_t)e.y) ? ld_global(xb + e.x) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 32; p += 4) {
      float4 xv[4];
#pragma unroll
      for (int j = 0; j < 4; j++) xv[j] = lane + 32 * j < cols ? *reinterpret_cast<const float4*>(&xs[lane + 32 * j][p]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float4 a = *reinterpret_cast<const float4*>(&gs[warp * 8 + i][p]);
#pragma unroll
        for (int j = 0; j < 4; j++) {
          acc[i][j] = fmaf(a.x, xv[j].x, acc[i][j]);
          acc[i][j] = fmaf(a.y, xv[j].y, acc[i][j]);
          acc[i][j] = fmaf(a.z, xv[j].z, acc[i][j]);
          acc[i][j] = fmaf(a.w, xv[j].w, acc[i][j]);
        }
      }
    }
  }
  float* out = part + (long long)blockIdx.z * g.cout * kk;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int co = co0 + warp * 8 + i;
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (co < g.cout && lane + 32 * j < cols) out[(long long)co * kk + k0 + lane + 32 * j] = acc[i][j];
  }
}

// dw (+)= the slices in a fixed order: eight shares of a value's slices, each in increasing order, then the shares.
__global__ void __launch_bounds__(256) conv_fma_finish_kernel(const float* part, int slices, int len, float* dw, int accumulate) {
  pdl_enter();
  __shared__ float sums[8][32];
  const int lane = threadIdx.x & 31, share = threadIdx.x >> 5, at = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (at < len) {
#pragma unroll 8
    for (int s = share; s < slices; s += 8) acc += part[(long long)s * len + at];
  }
  sums[share][lane] = acc;
  __syncthreads();
  if (share == 0 && at < len) {
    for (int y = 1; y < 8 && y < slices; y++) acc += sums[y][lane];
    dw[at] = accumulate ? dw[at] + acc : acc;
  }
}

// Offsets inside an image are 32-bit, pixels (with a tile's overhang) 31-bit numbers, taps a 32-bit mask.
static bool sizes_fit(const ConvGeom& g) {
  const long long reach = (long long)(g.kh - 1) * g.dh * g.w + (long long)g.kw * g.dw + (long long)g.pt * g.w + g.pl;
  return g.groups == 1 && (long long)g.kh * g.kw <= CF_MAX_TAPS && (long long)g.cin * g.h * g.w + reach < (1ll << 30) &&
         (long long)g.n * g.oh * g.ow < (1ll << 30) && (long long)g.n * g.h * g.w < (1ll << 30) && g.n <= 65535 &&
         (long long)g.cin * g.kh * g.kw <= 65535 && (long long)g.cout * g.kh * g.kw <= (1 << 20);
}

// The lines between these kernels and the product on an unfolded matrix, 3 x 3 windows, fp32 tier, us before / now:
//   forward        256 x 3 x 32 x 32 to 64: 161 / 69, 64 x 1 x 32 x 256 to 64: 222 / 92, 37 x 24 x 22 x 25 to 48: 113 / 52, 64 x 32 x 31 x 31 to
//                  64: 345 / 142. Up to 288 terms a value; with more than 72 the latency of the loads shows where there are few CTAs
//                  (8 x 16 x 24 x 24 to 32, 36 CTAs: 31 / 34).
//   input gradient 64 x 32 x 31 x 31: 190 / 151 (64 to 32: 138 / 80), 128 x 64 x 31 x 31 from 64: 641 / 550; not with few channels, or channels
//                  that leave a part of the CTA's 32 idle (3 of 64: 167 / 460, 24 of 48: 59 / 78), or few CTAs (15 / 50 at 36).
//   weight gradient 256 x 3 x 32 x 32 by 64: 265 / 138, 64 x 1 x 32 x 256 by 64: 1538 / 273, 37 x 24 x 22 x 25 by 48: 144 / 45, 64 x 32 x 31 x 31
//                  by 64: 562 / 145, 8 x 16 x 24 x 24 by 32: 89 / 19.
static int64_t ctas(int64_t pixels, int channels) { return ceil_div(pixels, CF_TILE) * ceil_div(channels, CF_CH); }
bool conv_fma_fwd_fits(const ConvGeom& g) {
  const int kk = g.cin * g.kh * g.kw;
  return sizes_fit(g) && kk <= 288 && (kk <= 72 || ctas((int64_t)g.n * g.oh * g.ow, g.cout) >= 120);
}
bool conv_fma_dgrad_fits(const ConvGeom& g) {
  return sizes_fit(g) && g.cin <= 64 && g.cout <= 64 && 8 * g.cin >= 7 * (int)ceil_div(g.cin, CF_CH) * CF_CH && ctas((int64_t)g.n * g.h * g.w, g.cin) >= 120;
}
bool conv_fma_wgrad_fits(const ConvGeom& g) { return sizes_fit(g) && g.cin * g.kh * g.kw <= 288 && g.cout <= 64; }

int32_t conv_fma_fwd(om_ctx* ctx, const ConvGeom& g, const float* x, const float* w, const float* bias, float* y) {
  const dim3 grid((unsigned)ceil_div((int64_t)g.n * g.oh * g.ow, CF_TILE), (unsigned)ceil_div(g.cout, CF_CH));
  launch_chained(ctx, conv_fma_fwd_kernel, grid, 128, 0, g, x, w, bias, y);
  OM_LAUNCH_CHECK(ctx, "conv_fma_fwd");
  return OM_OK;
}

int32_t conv_fma_dgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* w, float* dx) {
  const dim3 grid((unsigned)ceil_div((int64_t)g.n * g.h * g.w, CF_TILE), (unsigned)ceil_div(g.cin, CF_CH));
  launch_chained(ctx, conv_fma_dgrad_kernel, grid, 128, 0, g, gr, w, dx);
  OM_LAUNCH_CHECK(ctx, "conv_fma_dgrad");
  return OM_OK;
}

int32_t conv_fma_wgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* x, float* dw, int accumulate) {
  const int kk = g.cin * g.kh * g.kw, len = g.cout * kk;
  const int64_t pixels = (int64_t)g.n * g.oh * g.ow, tiles = ceil_div(kk, CF_COLS) * ceil_div(g.cout, CF_CH);
  // Slices for four CTAs an SM on 148 SMs, whole steps of 32 pixels: a function of the shape alone.
  const int per_slice = (int)std::max<int64_t>(64, ceil_div(ceil_div(pixels, std::max<int64_t>(1, 4 * 148 / tiles)), 32) * 32);
  const int slices = (int)ceil_div(pixels, per_slice);
  float* part = nullptr;
  OM_TRY(pool_alloc(ctx, sizeof(float) * (size_t)slices * len, false, (void**)&part));
  launch_chained(ctx, conv_fma_wgrad_kernel, dim3((unsigned)ceil_div(kk, CF_COLS), (unsigned)ceil_div(g.cout, CF_CH), (unsigned)slices), 128, 0, g, gr, x, per_slice, part);
  launch_chained(ctx, conv_fma_finish_kernel, (unsigned)ceil_div(len, 32), 256, 0, part, slices, len, dw, accumulate);
  pool_free(ctx, part);
  OM_LAUNCH_CHECK(ctx, "conv_fma_wgrad");
  return OM_OK;
}

}  // namespace om
