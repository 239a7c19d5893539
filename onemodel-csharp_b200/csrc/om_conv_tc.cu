// Convolution on the tensor pipe without an unfolded matrix: implicit products over NCHW tensors (ConvBackward and its forward,
// BackwardNn.cs:317-462 of the reference), TF32 operands, fp32 accumulators in tensor memory.
//
//   forward  y[co, pixel]  = sum over k = (c, tap)    W[co, k]          x[c, pixel's input position of the tap]
//   dgrad    dx[c, pixel]  = sum over taps of the sum over co of   W[co, c, tap]     g[co, pixel's output position of the tap]
//   wgrad    dW[co, n]     = sum over k = pixels      g[co, pixel]      x[n's channel, pixel's input position of n's tap]
//
// The operand that an unfolded matrix would hold is gathered by eight warps straight into the K-major, 128-byte-swizzled
// operand tile, rounded to TF32 (nearest even, as TMA rounds) on the way. Lanes own consecutive pixels, so a load is one or
// two row segments. k runs in units of eight channels of one tap: inside a unit the source position moves by whole planes
// and lies inside the image or outside for all eight, so an element costs an addition, a load, a rounding and a quarter of a
// 16-byte store. (With k in the weights' own order, channel by channel, each element looked its offset and its tap up in a table:
// 17 instructions and 12 load/store wavefronts, 202 us for 256 images of 64 x 32 x 32 through a 3 x 3 window to 64
// channels; the unfolded form took 455.) Units of four neighbouring channel groups share a tap before the next tap comes, so the
// taps of a window find each other's lines in L1. The weights are turned into the order of the units by a small kernel.
// What bounds the kernels is the load/store unit: 128 x 32 gathered elements a 128 x 128 x 32 product.
//
// dgrad (channels-last only) with stride s works on the s * s classes of input positions modulo the stride (grid z): each is a stride-1
// problem over the taps that reach it, so no product is formed with the zeros between the strides.
#include "om_conv.cuh"
#include "om_tc.cuh"

namespace om {

constexpr int CV_TILE = 128;                      // channels (accumulator rows) and pixels / unit columns (columns) of a tile
constexpr int CV_BK = 32;                         // one 128-byte swizzle row of k
constexpr int CV_UNIT = 8;                        // channels of one tap
constexpr int CV_GROUP = 4;                       // units of one tap that follow one another
constexpr int CV_BLOCK = CV_TILE * 128;           // one operand block: 16 KiB
constexpr int CV_PRODUCERS = 8;                   // gathering warps, also the epilogue
constexpr int CV_THREADS = 32 * (CV_PRODUCERS + 2);   // + one warp issuing products, one issuing TMA loads
constexpr int CV_MAX_TAPS = 32;                   // a thread keeps the taps that lie inside the image as a bit mask
constexpr int CV_MAX_PHASES = 4;
constexpr int CV_STG_LD = CV_TILE + 4;            // floats per staged result row

// n / d for 0 <= n < 2^31 by a multiplication (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994): s = ceil(log2 d), mul = floor(2^32 (2^s - d) / d) + 1, n / d = (mulhi(n, mul) + n) >> s.
struct CvDiv {
  uint32_t mul, shift;
};
static CvDiv cv_div(uint32_t d) {
  CvDiv r;
  r.shift = 0;
  while ((1ull << r.shift) < d) r.shift++;
  r.mul = (uint32_t)(((1ull << 32) * ((1ull << r.shift) - d)) / d + 1);
  return r;
}
__device__ __forceinline__ int cv_quot(int n, CvDiv d) { return (int)((__umulhi((uint32_t)n, d.mul) + (uint32_t)n) >> d.shift); }

// Unit u of channels x taps (UNIT channels of a tap, GROUP neighbouring channel blocks of a tap before the next tap): its tap, and its
// first channel.
template <int UNIT, int GROUP>
__host__ __device__ __forceinline__ void cv_unit(int u, int channels, int taps, int* tap, int* c0) {
  const int blocks = (channels + UNIT - 1) / UNIT;
  const int sg = u / (GROUP * taps), r = u - sg * GROUP * taps;
  const int width = blocks - sg * GROUP < GROUP ? blocks - sg * GROUP : GROUP;
  *tap = r / width;
  *c0 = (sg * GROUP + r % width) * UNIT;
}
static int cv_units(int channels, int taps, int unit) { return (channels + unit - 1) / unit * taps; }

struct ConvTcParams {
  const float* src;
  float* out;
  const float* bias;
  int32_t* status;
  int images, m;               // output channels
  int sc, sh, sw;              // source channels and plane
  int pw, plane;               // width and size of the output plane
  CvDiv div_plane, div_w;
  int step_y, step_x, base_y, base_x;   // source position of pixel (y, x) and tap t: y * step_y + base_y + dy[t], likewise x
  int vec;                     // four consecutive pixels are 16 aligned bytes of the output
  int taps, units;
  int dy[CV_MAX_TAPS], dx[CV_MAX_TAPS];
};

__device__ __forceinline__ uint32_t rn_tf32(float x) {
  uint32_t r;
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void cv_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__host__ __device__ constexpr uint32_t cv_idesc() {   // kind::tf32, fp32 accumulator, both operands K-major, N = M = 128
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(CV_TILE >> 3) << 17) | ((uint32_t)(CV_TILE >> 4) << 24);
}

// The products of one stage: MT accumulators of 128 rows share the gathered tile.
template <int MT>
__device__ __forceinline__ void cv_issue(uint32_t tmem, uint32_t a_addr, uint32_t b_addr, int mts, bool first) {
#pragma unroll
  for (int mt = 0; mt < MT; mt++) {
    if (mt >= mts) break;
#pragma unroll
    for (int ks = 0; ks < CV_BK / 8; ks++)
      umma_tf32(tmem + mt * CV_TILE, make_desc(a_addr + mt * CV_BLOCK + ks * 32, 16, 1024, 2), make_desc(b_addr + ks * 32, 16, 1024, 2), cv_idesc(),
                (!first || ks > 0) ? 1u : 0u);
  }
}

// Turns this CTA's 128 x 128 accumulator into rows of CV_STG_LD floats in shared memory (the dead operand stages).
__device__ __forceinline__ void cv_stage_rows(float* stg, uint32_t tmem, int warp, int lane) {
  const int quad = warp & 3, half = warp >> 2;
#pragma unroll
  for (int c = 0; c < 2; c++) {
    uint32_t r[32];
    const int col = half * 64 + c * 32;
    tmem_ld_32x32b_x32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)col, r);
    tmem_ld_wait();
    float* dst = stg + (quad * 32 + lane) * CV_STG_LD + col;
#pragma unroll
    for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(dst + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
  }
}

// Eight channels of one tap for this lane's pixel. o: byte offset of the first (modulo 2^32), step: bytes of a plane.
__device__ __forceinline__ void cv_load_unit(float* v, const float* src, uint32_t o, uint32_t step, int count) {
#pragma unroll
  for (int j = 0; j < CV_UNIT; j++) v[j] = 0.f;
  const char* base = reinterpret_cast<const char*>(src);
  if (count == CV_UNIT) {
#pragma unroll
    for (int j = 0; j < CV_UNIT; j++) {
      v[j] = ld_global(reinterpret_cast<const float*>(base + o));
      o += step;
    }
  } else if (count > 0) {        // the last channels
#pragma unroll
    for (int j = 0; j < CV_UNIT; j++) {
      if (j < count) v[j] = ld_global(reinterpret_cast<const float*>(base + o));
      o += step;
    }
  }
}

// ---- forward ---------------------------------------------------------------------------------------------------------------
// MT: 128-row accumulators per CTA; two (three stages become two, so that two CTAs still share an SM) halve the gathering
// per product where there are more than 128 output channels and pixels enough to fill the device.
template <int MT>
__global__ void __launch_bounds__(CV_THREADS, 2)
conv_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ ConvTcParams p) {
  constexpr int STAGES = MT == 1 ? 3 : 2;
  constexpr int STAGE_BYTES = (MT + 1) * CV_BLOCK;
  constexpr uint32_t TMEM_COLS = MT * CV_TILE;
  const int plane = p.plane;
  const int pixels = p.images * plane;
  const int q0 = blockIdx.x * CV_TILE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int2* units = reinterpret_cast<int2*>(smem + STAGES * STAGE_BYTES + 128);   // byte offset; tap | channels << 8

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * (MT * CV_TILE);
  const int mts = min(MT, (p.m - m0 + CV_TILE - 1) / CV_TILE);
  const int k_blocks = (p.units * CV_UNIT + CV_BK - 1) / CV_BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], 1 + CV_PRODUCERS);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int u = threadIdx.x; u < k_blocks * (CV_BK / CV_UNIT); u += CV_THREADS) {
    int2 e = make_int2(0, 0);
    if (u < p.units) {
      int t, c0;
      cv_unit<CV_UNIT, CV_GROUP>(u, p.sc, p.taps, &t, &c0);
      e.x = (int)(4u * (uint32_t)(c0 * p.sh * p.sw + p.dy[t] * p.sw + p.dx[t]));
      e.y = t | (min(CV_UNIT, p.sc - c0) << 8);
    }
    units[u] = e;
  }
  if (warp == CV_PRODUCERS) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();   // tensor memory is held: later kernels may become resident
  pdl_wait();      // everything below may depend on the previous kernel

  if (warp < CV_PRODUCERS) {
    // ---- gather: a thread owns a pixel and two of a stage's four units ----
    const int half = warp >> 2;
    const int px = (warp & 3) * 32 + lane;
    const int q = q0 + px;
    uint32_t mask = 0, base = 0;
    if (q < pixels) {
      const int n = cv_quot(q, p.div_plane), r = q - n * plane;
      const int y = cv_quot(r, p.div_w), x = r - y * p.pw;
      const int y0 = y * p.step_y + p.base_y, x0 = x * p.step_x + p.base_x;
      for (int t = 0; t < p.taps; t++)
        if ((unsigned)(y0 + p.dy[t]) < (unsigned)p.sh && (unsigned)(x0 + p.dx[t]) < (unsigned)p.sw) mask |= 1u << t;
      base = 4u * ((uint32_t)n * (uint32_t)(p.sc * p.sh * p.sw) + (uint32_t)(y0 * p.sw + x0));
    }
    const uint32_t step = 4u * (uint32_t)(p.sh * p.sw);
    auto fetch = [&](float (&v)[16], int kb) {
      if (kb >= k_blocks) return;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int2 e = units[kb * 4 + half * 2 + i];
        cv_load_unit(v + 8 * i, p.src, base + (uint32_t)e.x, step, (mask >> (e.y & 31)) & 1 ? e.y >> 8 : 0);
      }
    };
    bool ok = true;
    auto deposit = [&](const float (&v)[16], int kb) {
      if (!ok || kb >= k_blocks) return;
      const int s = kb % STAGES;
      const uint32_t round = kb / STAGES;
      if (round > 0) ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], (round - 1) & 1, abort_flag, p.status, 71));
      if (!ok) return;
      uint8_t* row = smem + (size_t)s * STAGE_BYTES + MT * CV_BLOCK + px * 128;
#pragma unroll
      for (int c = 0; c < 4; c++)
        *reinterpret_cast<uint4*>(row + (((half * 4 + c) ^ (px & 7)) << 4)) =
            make_uint4(rn_tf32(v[4 * c]), rn_tf32(v[4 * c + 1]), rn_tf32(v[4 * c + 2]), rn_tf32(v[4 * c + 3]));
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) cv_arrive(&full[s]);
    };
    float v0[16], v1[16], v2[16];     // the loads of two blocks are in flight while one is stored
    fetch(v0, 0);
    fetch(v1, 1);
    for (int kb = 0; kb < k_blocks && ok; kb += 3) {
      fetch(v2, kb + 2);
      deposit(v0, kb);
      fetch(v0, kb + 3);
      deposit(v1, kb + 1);
      fetch(v1, kb + 4);
      deposit(v2, kb + 2);
    }
    // ---- results: accumulator rows through shared memory to rows of consecutive pixels ----
    ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, p.status, 72)) && ok;
    tc_fence_after();
    float* stg = reinterpret_cast<float*>(smem);
    long long at[4];               // output positions of this lane's pixels relative to their image's first channel; -1 past the end
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int qi = q0 + (p.vec ? 4 * lane : lane + 32 * i);
      at[i] = -1;
      if (qi < pixels) {
        const int n = cv_quot(qi, p.div_plane);
        at[i] = (long long)n * p.m * plane + (qi - n * plane);
      }
    }
    for (int mt = 0; mt < mts; mt++) {
      if (ok) cv_stage_rows(stg, tmem_base + mt * CV_TILE, warp, lane);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (ok) {
#pragma unroll 4
        for (int i = 0; i < 16; i++) {
          const int row = warp * 16 + i, co = m0 + mt * CV_TILE + row;
          if (co >= p.m) break;
          const float bv = p.bias ? ld_global(p.bias + co) : 0.f;
          float* out = p.out + (long long)co * plane;
          const float* sr = stg + row * CV_STG_LD;
          if (p.vec) {
            if (at[0] >= 0) {
              float4 v = *reinterpret_cast<const float4*>(sr + 4 * lane);
              if (p.bias) { v.x += bv; v.y += bv; v.z += bv; v.w += bv; }
              *reinterpret_cast<float4*>(out + at[0]) = v;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
              if (at[j] >= 0) out[at[j]] = p.bias ? sr[lane + 32 * j] + bv : sr[lane + 32 * j];
          }
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
  } else if (warp == CV_PRODUCERS) {
    if (lane == 0) {
      for (int kb = 0; kb < k_blocks; kb++) {
        const int s = kb % STAGES;
        if (!mbar_wait(&full[s], (kb / STAGES) & 1, abort_flag, p.status, 73)) break;
        tc_fence_after();
        const uint32_t a = smem_u32(smem + (size_t)s * STAGE_BYTES);
        cv_issue<MT>(tmem_base, a, a + MT * CV_BLOCK, mts, kb == 0);
        umma_commit(&empty[s]);
      }
      umma_commit(acc_full);
    }
  } else if (lane == 0) {
    for (int kb = 0; kb < k_blocks; kb++) {
      const int s = kb % STAGES;
      const uint32_t round = kb / STAGES;
      if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1, abort_flag, p.status, 74)) break;
      mbar_expect_tx(&full[s], (uint32_t)(mts * CV_BLOCK));
      for (int mt = 0; mt < mts; mt++)
        tma_load_4d(smem + (size_t)s * STAGE_BYTES + mt * CV_BLOCK, &map_a, kb * CV_BK, m0 + mt * CV_TILE, 0, 0, &full[s]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == CV_PRODUCERS) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// The weights in the order of the units, one K-major row per output channel: wt[m][CV_UNIT u + i] is the weight of tap(u) and source channel
// c0(u) + i, zero past the last channel.
__global__ void __launch_bounds__(256) conv_turn_weights_kernel(const float* w, float* __restrict__ wt, int channels, int taps, int ld) {
  pdl_enter();
  const int m = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ld; i += gridDim.x * blockDim.x) {
    int tap, c0;
    cv_unit<CV_UNIT, CV_GROUP>(i / CV_UNIT, channels, taps, &tap, &c0);
    const int c = c0 + i % CV_UNIT;
    wt[(long long)m * ld + i] = c < channels ? ld_global(w + ((long long)m * channels + c) * taps + tap) : 0.f;
  }
}

// ---- weight gradient -------------------------------------------------------------------------------------------------------
struct ConvWgradParams {
  const float* gr;
  const float* x;
  float* part;                 // [splits][cout][8 * units]
  int32_t* status;
  int cout, units, cin, h, w, kw, taps, sh, sw, pt, pl, dh, dw, ow, plane;
  CvDiv div_plane, div_w;
  int pixels;
  int blocks_per_split;
};

// One CTA: 128 output channels x 128 columns (16 units of eight channels of a tap) over a slice of the pixels, 32 of them a stage. A lane
// owns a pixel and a warp two units, so both operands are loaded along rows and written as whole 128-byte operand rows.
// A_TMA: whole stages of the gradient come by TMA (planes of a multiple of 32 pixels); otherwise the warps load its rows too.
template <bool A_TMA>
__global__ void __launch_bounds__(CV_THREADS, 2)
conv_wgrad_tc_kernel(const __grid_constant__ CUtensorMap map_g, const __grid_constant__ ConvWgradParams p) {
  constexpr int STAGES = 3;
  constexpr int STAGE_BYTES = 2 * CV_BLOCK;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * CV_TILE, m0 = blockIdx.y * CV_TILE;
  const int all_blocks = (p.pixels + CV_BK - 1) / CV_BK;
  const int b0 = blockIdx.z * p.blocks_per_split;
  const int k_blocks = min(p.blocks_per_split, all_blocks - b0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], CV_PRODUCERS + (A_TMA ? 1 : 0));
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == CV_PRODUCERS) {
    tmem_alloc(tmem_slot, CV_TILE);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();   // tensor memory is held: later kernels may become resident
  pdl_wait();      // everything below may depend on the previous kernel

  if (warp < CV_PRODUCERS) {
    bool ok = true;
    const int row0 = warp * 16;
    // This warp's two units (columns) and 16 output channels (rows): the same for every stage.
    int dy[2] = {0, 0}, dx[2] = {0, 0}, count[2] = {0, 0};
    uint32_t off[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int u = (n0 + row0) / CV_UNIT + i;
      if (u < p.units) {
        int t, c0;
        cv_unit<CV_UNIT, CV_GROUP>(u, p.cin, p.taps, &t, &c0);
        dy[i] = (t / p.kw) * p.dh - p.pt;
        dx[i] = (t % p.kw) * p.dw - p.pl;
        count[i] = min(CV_UNIT, p.cin - c0);
        off[i] = 4u * (uint32_t)(c0 * p.h * p.w);
      }
    }
    const uint32_t step = 4u * (uint32_t)(p.h * p.w), gstep = 4u * (uint32_t)p.plane;
    const int rows = min(16, p.cout - m0 - row0);
    auto fetch = [&](float (&vb)[16], float (&va)[A_TMA ? 1 : 16], int kb) {
      if (kb >= k_blocks) return;
      const int q = (b0 + kb) * CV_BK + lane;
      const bool inside = q < p.pixels;
      const int n = cv_quot(inside ? q : 0, p.div_plane), r = (inside ? q : 0) - n * p.plane;
      const int oy = cv_quot(r, p.div_w), ox = r - oy * p.ow;
      const uint32_t image = (uint32_t)n * (uint32_t)(p.cin * p.h * p.w);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int y = oy * p.sh + dy[i], x = ox * p.sw + dx[i];
        const bool in = inside && (unsigned)y < (unsigned)p.h && (unsigned)x < (unsigned)p.w;
        cv_load_unit(vb + 8 * i, p.x, off[i] + 4u * (image + (uint32_t)(y * p.w + x)), step, in ? count[i] : 0);
      }
      if (!A_TMA) {
        const uint32_t o = 4u * (((uint32_t)n * (uint32_t)p.cout + (uint32_t)(m0 + row0)) * (uint32_t)p.plane + (uint32_t)r);
        cv_load_unit(va, p.gr, o, gstep, inside ? max(0, min(CV_UNIT, rows)) : 0);
        cv_load_unit(va + (A_TMA ? 0 : 8), p.gr, o + 8u * gstep, gstep, inside ? max(0, min(CV_UNIT, rows - CV_UNIT)) : 0);
      }
    };
    auto deposit = [&](const float (&vb)[16], const float (&va)[A_TMA ? 1 : 16], int kb) {
      if (!ok || kb >= k_blocks) return;
      const int s = kb % STAGES;
      const uint32_t round = kb / STAGES;
      if (round > 0) ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], (round - 1) & 1, abort_flag, p.status, 75));
      if (!ok) return;
      uint8_t* a = smem + (size_t)s * STAGE_BYTES;
#pragma unroll
      for (int i = 0; i < 16; i++) {
        const int at = (row0 + i) * 128 + (((lane >> 2) ^ (i & 7)) << 4) + (lane & 3) * 4;      // (row0 is a multiple of 8)
        *reinterpret_cast<uint32_t*>(a + CV_BLOCK + at) = rn_tf32(vb[i]);
        if (!A_TMA) *reinterpret_cast<uint32_t*>(a + at) = rn_tf32(va[A_TMA ? 0 : i]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) cv_arrive(&full[s]);
    };
    float vb0[16], vb1[16], va0[A_TMA ? 1 : 16], va1[A_TMA ? 1 : 16];
    fetch(vb0, va0, 0);
    for (int kb = 0; kb < k_blocks && ok; kb += 2) {
      fetch(vb1, va1, kb + 1);
      deposit(vb0, va0, kb);
      fetch(vb0, va0, kb + 2);
      deposit(vb1, va1, kb + 1);
    }
    ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, p.status, 76)) && ok;
    tc_fence_after();
    float* stg = reinterpret_cast<float*>(smem);
    if (ok) cv_stage_rows(stg, tmem_base, warp, lane);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (ok) {
      const int ld = p.units * CV_UNIT, col = n0 + 4 * lane;
      float* out = p.part + (long long)blockIdx.z * p.cout * ld + col;
      if (col < ld) {
#pragma unroll 4
        for (int i = 0; i < rows; i++)
          *reinterpret_cast<float4*>(out + (long long)(m0 + row0 + i) * ld) = *reinterpret_cast<const float4*>(stg + (row0 + i) * CV_STG_LD + 4 * lane);
      }
    }
  } else if (warp == CV_PRODUCERS) {
    if (lane == 0) {
      for (int kb = 0; kb < k_blocks; kb++) {
        const int s = kb % STAGES;
        if (!mbar_wait(&full[s], (kb / STAGES) & 1, abort_flag, p.status, 77)) break;
        tc_fence_after();
        const uint32_t a = smem_u32(smem + (size_t)s * STAGE_BYTES);
        cv_issue<1>(tmem_base, a, a + CV_BLOCK, 1, kb == 0);
        umma_commit(&empty[s]);
      }
      umma_commit(acc_full);
    }
  } else if (lane == 0 && A_TMA) {
    for (int kb = 0; kb < k_blocks; kb++) {
      const int s = kb % STAGES;
      const uint32_t round = kb / STAGES;
      if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1, abort_flag, p.status, 78)) break;
      const int q = (b0 + kb) * CV_BK, n = cv_quot(q, p.div_plane);
      mbar_expect_tx(&full[s], CV_BLOCK);
      tma_load_4d(smem + (size_t)s * STAGE_BYTES, &map_g, q - n * p.plane, m0, n, 0, &full[s]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == CV_PRODUCERS) {
    tc_fence_after();
    tmem_dealloc(tmem_base, CV_TILE);
  }
}

// dW[co][c][tap] (+)= the slices' sums. A CTA: 256 / SHARES unit columns of an output channel x SHARES shares of the slices (share y
// takes slices y, y + SHARES, ... in order), the shares added in order. Eight shares for many slices: with up to 296 of them one
// thread a value is a chain of as many loads (21 us against 5). One share for a few: 512 x 4608 weights in two slices took 67 us
// with eight, most of whose threads had nothing to add.
template <int SHARES, int UNIT, int GROUP>
__global__ void __launch_bounds__(256)
conv_wgrad_finish_kernel(const float* part, int splits, int cout, int units, int cin, int taps, float* dw, int accumulate) {
  pdl_enter();
  constexpr int COLS = 256 / SHARES;
  __shared__ float sums[SHARES][COLS];
  const int ld = units * UNIT, lane = threadIdx.x % COLS, share = threadIdx.x / COLS;
  const int col = blockIdx.x * COLS + lane, co = blockIdx.y;
  float acc = 0.f;
  if (col < ld) {
    const float* src = part + (long long)co * ld + col;
    const long long stride = (long long)cout * ld;
#pragma unroll 4
    for (int s = share; s < splits; s += SHARES) acc += src[s * stride];
  }
  if (SHARES > 1) {
    sums[share][lane] = acc;
    __syncthreads();
  }
  if (share == 0 && col < ld) {
    int t, c0;
    cv_unit<UNIT, GROUP>(col / UNIT, cin, taps, &t, &c0);
    const int c = c0 + col % UNIT;
    if (c >= cin) return;
    for (int y = 1; y < SHARES && y < splits; y++) acc += sums[y][lane];
    float* dst = dw + ((long long)co * cin + c) * taps + t;
    *dst = accumulate ? *dst + acc : acc;
  }
}

// ---- channels last ---------------------------------------------------------------------------------------------------------
// Where pixels tile well, the source is first turned to [n][h][w][c] (one pass over the activation), and everything the products read
// comes by TMA: 128 pixels are a box of the turned tensor, a tap moves the box by whole pixels, and what lies outside the image
// reads as zero. No warp touches an operand, so the pace is that of operand delivery to shared memory, as for the plain products
// (the gathering kernels above are held up by the load/store unit).
//   forward, dgrad   D [128 pixels, NT channels] += x [pixels + tap, 32 c] W [NT, (32 c, tap)]      both K-major
//   wgrad            D [128 co, 4 x (32 c, tap)] += g [32 pixels, co] x [32 pixels + tap, 32 c]      both MN-major
// Accumulator rows are pixels, so a warp's store of one channel is 32 neighbouring pixels of the NCHW result.
struct ConvTurn {               // weights addressed by their strides over (m, source channel)
  int m, sc;
  long long stride_m, stride_sc;
  int by_tap;                  // all channels of a tap before the next tap
  int taps[CV_MAX_PHASES], ld[CV_MAX_PHASES];
  long long start[CV_MAX_PHASES];
  int tap[CV_MAX_PHASES][CV_MAX_TAPS];
};
// The weights for these kernels: wt[phase][m][(32-channel block, tap), 32], or (tap, 32-channel block) for dgrad, by tiles of
// 8 m x 32 source channels through shared memory. Read and written in runs (element by element, the reads were 4 bytes a line:
// 512 x 512 x 3 x 3 took 14 us).
constexpr int CN_PACK_M = 8;
__global__ void __launch_bounds__(256) conv_pack_weights_kernel(const float* w, float* __restrict__ wt, const __grid_constant__ ConvTurn t, int taps_all, int phases) {
  pdl_enter();
  extern __shared__ float pack[];       // [8 m][32 channels][taps, to an odd number]
  const int m0 = blockIdx.y * CN_PACK_M, c0 = blockIdx.x * CV_BK, tp = taps_all | 1;
  const bool by_m = t.stride_sc < t.stride_m;          // a run of memory is (channel, tap) of one m, or (m, tap) of one channel
  const int run = (by_m ? CV_BK : CN_PACK_M) * taps_all;
  for (int e = threadIdx.x; e < CN_PACK_M * CV_BK * taps_all; e += 256) {
    const int outer = e / run, rem = e - outer * run, inner = rem / taps_all, tap = rem - inner * taps_all;
    const int m = by_m ? outer : inner, c = by_m ? inner : outer;
    pack[(m * CV_BK + c) * tp + tap] = m0 + m < t.m && c0 + c < t.sc ? ld_global(w + (m0 + m) * t.stride_m + (c0 + c) * t.stride_sc + tap) : 0.f;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (m0 + warp >= t.m) return;
  for (int z = 0; z < phases; z++) {
    float* out = wt + t.start[z] + (long long)(m0 + warp) * t.ld[z] + lane;
    for (int j = 0; j < t.taps[z]; j++) {
      const int block = t.by_tap ? j * (int)gridDim.x + (int)blockIdx.x : (int)blockIdx.x * t.taps[z] + j;
      out[(long long)block * CV_BK] = pack[(warp * CV_BK + lane) * tp + t.tap[z][j]];
    }
  }
}

struct ConvBox {
  int w, h, n;                 // a tile of w x h x n pixels (powers of two)
  int tw, th, tn;              // tiles along each
};
struct ConvNhwcPhase {
  int ph, pw, oy0, ox0, taps, k_blocks, chain;
  ConvBox box;
  int dy[CV_MAX_TAPS], dx[CV_MAX_TAPS];
};
struct ConvNhwcParams {
  float* out;
  const float* bias;
  int32_t* status;
  int images, m, out_w, out_plane;
  int step_y, step_x, base_y, base_x, ostep_y, ostep_x;
  int by_tap, sh, sw;          // by_tap: chain t is tap t, and counts for the pixels whose position of it lies in the sh x sw source plane
  ConvNhwcPhase phase[CV_MAX_PHASES];
};
struct ConvNhwcMaps {
  CUtensorMap src[CV_MAX_PHASES], w[CV_MAX_PHASES];
};

// t[q][c] = s[n][c][p] for pixel q = n * plane + p; rows of cp floats (c rounded up to a multiple of four, zero there). SUMS: the pass also
// leaves the channels' sums over this CTA's pixels in sums[blockIdx.x][c], in double (the bias gradient, which would otherwise be
// another pass over the gradient: 118 us a step for the eight layers of the convolutional network).
constexpr int CN_PX = 64, CN_SUM_CTAS = 512;
template <bool SUMS>
__global__ void __launch_bounds__(256) conv_channels_last_kernel(const float* src, float* __restrict__ t, int pixels, int plane, CvDiv div_plane, int c, int cp,
                                                                 double* __restrict__ sums) {
  pdl_enter();
  __shared__ float tile[32][CN_PX + 1];
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int c0 = blockIdx.y * 32;
  double acc = 0.0;
  for (int q0 = blockIdx.x * CN_PX; q0 < pixels; q0 += gridDim.x * CN_PX) {
#pragma unroll
    for (int i = 0; i < CN_PX / 32; i++) {
      const int q = q0 + 32 * i + lane;
      const int n = cv_quot(q < pixels ? q : 0, div_plane), p = (q < pixels ? q : 0) - n * plane;
      const float* base = src + (long long)n * c * plane + p;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int ch = c0 + row + 8 * j;
        tile[row + 8 * j][32 * i + lane] = q < pixels && ch < c ? ld_global(base + (long long)ch * plane) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < CN_PX / 8; i++) {
      const int q = q0 + row + 8 * i;
      const float v = tile[lane][row + 8 * i];
      if (SUMS) acc += (double)v;
      if (c0 + lane < cp && q < pixels) t[(long long)q * cp + c0 + lane] = v;
    }
    __syncthreads();
  }
  if (SUMS) {
    __shared__ double part[8][32];
    part[row][lane] = acc;
    __syncthreads();
    if (row == 0 && c0 + lane < c) {
      for (int i = 1; i < 8; i++) acc += part[i][lane];
      sums[(long long)blockIdx.x * c + c0 + lane] = acc;
    }
  }
}
// dbias[co] (+)= the CTAs' sums: eight shares of them in increasing order, then the shares, in double.
__global__ void __launch_bounds__(256) conv_sums_finish_kernel(const double* sums, int ctas, int c, float* dbias, int accumulate) {
  pdl_enter();
  __shared__ double part[8][32];
  const int lane = threadIdx.x & 31, share = threadIdx.x >> 5, ch = blockIdx.x * 32 + lane;
  double acc = 0.0;
  if (ch < c) {
#pragma unroll 8
    for (int i = share; i < ctas; i += 8) acc += sums[(long long)i * c + ch];
  }
  part[share][lane] = acc;
  __syncthreads();
  if (share == 0 && ch < c) {
    for (int i = 1; i < 8; i++) acc += part[i][lane];
    dbias[ch] = accumulate ? dbias[ch] + (float)acc : (float)acc;
  }
}

// Warp 0: TMA, warp 1: products, the others: results. With chains there are two result warps for a quarter of the rows, half of the columns each.
constexpr int CN_THREADS = 192, CN_CHAIN_THREADS = 320;
__host__ __device__ constexpr int cn_threads(bool chains) { return chains ? CN_CHAIN_THREADS : CN_THREADS; }
// What the result warps do with a tile that arrives in chains of `chain` k blocks (see conv_nhwc_kernel): add chain c, in accumulator c % 2 (`pitch` columns
// apart), to their registers while the other accumulator is being filled. `take(c)`: whether the lane's row counts it.
template <int COLS, typename Take>
__device__ __forceinline__ bool cn_add_chains(float (&acc)[COLS], uint32_t tmem, int pitch, int chains, uint64_t* full, uint64_t* empty, volatile int* abort_flag,
                                              int32_t* status, int where, Take take) {
#pragma unroll
  for (int j = 0; j < COLS; j++) acc[j] = 0.f;
  for (int c = 0; c < chains; c++) {
    const bool on = take(c);
    if (!__all_sync(0xffffffffu, mbar_wait(&full[c & 1], (uint32_t)(c >> 1) & 1, abort_flag, status, where))) return false;
    tc_fence_after();
#pragma unroll
    for (int col = 0; col < COLS; col += 16) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(tmem + (uint32_t)((c & 1) * pitch + col), r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; j++) acc[col + j] += on ? __uint_as_float(r[j]) : 0.f;
    }
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) cv_arrive(&empty[c & 1]);
  }
  return true;
}
// CHAINS: the sum over k in several accumulator chains that are added in fp32 in increasing order. The tensor core cuts what a step of its accumulator
// cannot hold instead of rounding it, an error that grows with the number of steps (1.8e-8 of the result a step of eight k's: 4.9e-6 at k
// = 2304). With a chain a tap, dx has the bits of the product on the unfolded matrix and its fold, and a tap outside the gradient's plane
// is left out whatever its weight is; in one chain over all taps it was 7 times as far from the exact sums (128 channels
// 2.6e-6 against 3.4e-7). Two accumulators, so that one is read back while the other is filled; us in one chain / a chain a tap: 256 x 64 x 32 x 32 from 128 with
// stride 2 83 / 95, 64 x 64 x 16 x 128 from 128 99 / 119, 32 x 256 x 14 x 14 from 256 44 / 52.
template <int NT, int STAGES, bool CHAINS>
__global__ void __launch_bounds__(cn_threads(CHAINS), STAGES > 4 ? 1 : 2)
conv_nhwc_kernel(const __grid_constant__ ConvNhwcMaps maps, const __grid_constant__ ConvNhwcParams p) {
  constexpr int STAGE_BYTES = CV_BLOCK + NT * 128;
  constexpr int ACCS = CHAINS ? 2 : 1;
  const ConvNhwcPhase& ph = p.phase[blockIdx.z];
  const ConvBox& box = ph.box;
  const int tile = blockIdx.x;
  if (tile >= box.tw * box.th * box.tn) return;       // the classes of a strided gradient differ in size
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint64_t* acc_empty = acc_full + ACCS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + ACCS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * NT, k_blocks = ph.k_blocks;
  const int tx = tile % box.tw, ty = tile / box.tw % box.th, tn = tile / (box.tw * box.th);
  const int x0 = tx * box.w, y0 = ty * box.h, n0 = tn * box.n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < ACCS; a++) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 8);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, ACCS * NT);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();   // tensor memory is held: later kernels may become resident
  pdl_wait();      // everything below may depend on the previous kernel

  if (warp == 0) {
    if (lane == 0) {
      const int blocks = ph.taps > 0 ? k_blocks / ph.taps : 0;
      int t = 0, c0 = 0;
      for (int kb = 0; kb < k_blocks; kb++) {
        const int s = kb % STAGES;
        const uint32_t round = kb / STAGES;
        if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1, abort_flag, p.status, 81)) break;
        uint8_t* a = smem + (size_t)s * STAGE_BYTES;
        mbar_expect_tx(&full[s], STAGE_BYTES);
        tma_load_4d(a, &maps.src[blockIdx.z], c0, x0 * p.step_x + p.base_x + ph.dx[t], y0 * p.step_y + p.base_y + ph.dy[t], n0, &full[s]);
        tma_load_4d(a + CV_BLOCK, &maps.w[blockIdx.z], kb * CV_BK, m0, 0, 0, &full[s]);
        if (p.by_tap) {
          c0 += CV_BK;
          if (c0 == blocks * CV_BK) {
            c0 = 0;
            t++;
          }
        } else if (++t == ph.taps) {
          t = 0;
          c0 += CV_BK;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && k_blocks > 0) {
      constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(CV_TILE >> 4) << 24);
      int c = 0, at = 0;           // the chain, and the block of it
      for (int kb = 0; kb < k_blocks; kb++) {
        const int s = kb % STAGES;
        if (CHAINS && at == 0 && c >= ACCS && !mbar_wait(&acc_empty[c & 1], (uint32_t)((c >> 1) - 1) & 1, abort_flag, p.status, 87)) break;
        if (!mbar_wait(&full[s], (kb / STAGES) & 1, abort_flag, p.status, 82)) break;
        tc_fence_after();
        const uint32_t a = smem_u32(smem + (size_t)s * STAGE_BYTES), b = a + CV_BLOCK;
#pragma unroll
        for (int ks = 0; ks < CV_BK / 8; ks++)
          umma_tf32(tmem_base + (CHAINS ? (c & 1) * NT : 0), make_desc(a + ks * 32, 16, 1024, 2), make_desc(b + ks * 32, 16, 1024, 2), idesc,
                    ((CHAINS ? at : kb) > 0 || ks > 0) ? 1u : 0u);
        umma_commit(&empty[s]);
        if (CHAINS && (++at == ph.chain || kb == k_blocks - 1)) {
          umma_commit(&acc_full[c & 1]);
          at = 0;
          c++;
        }
      }
      if (!CHAINS) umma_commit(acc_full);
    }
  } else {
    const int quad = warp & 3, slot = quad * 32 + lane;
    const int ix = slot % box.w, iy = slot / box.w % box.h, in = slot / (box.w * box.h);
    const int x = x0 + ix, y = y0 + iy, n = n0 + in;
    const bool valid = x < ph.pw && y < ph.ph && n < p.images;
    float* out = p.out + ((long long)n * p.m + m0) * p.out_plane + (long long)(y * p.ostep_y + ph.oy0) * p.out_w + x * p.ostep_x + ph.ox0;
    const uint32_t rows = tmem_base + ((uint32_t)(quad * 32) << 16);
    if constexpr (CHAINS) {
      const int sy = y * p.step_y + p.base_y, sx = x * p.step_x + p.base_x;
      constexpr int COLS = NT / 2;
      const int col0 = (warp - 2) / 4 * COLS;
      float acc[COLS];
      const bool ok = cn_add_chains<COLS>(acc, rows + (uint32_t)col0, NT, (k_blocks + ph.chain - 1) / ph.chain, acc_full, acc_empty, abort_flag, p.status, 83, [&](int c) {
        return !p.by_tap || ((unsigned)(sy + ph.dy[c]) < (unsigned)p.sh && (unsigned)(sx + ph.dx[c]) < (unsigned)p.sw);
      });
      if (ok && valid) {
#pragma unroll
        for (int j = 0; j < COLS; j++)
          if (m0 + col0 + j < p.m) out[(long long)(col0 + j) * p.out_plane] = p.bias ? acc[j] + ld_global(p.bias + m0 + col0 + j) : acc[j];
      }
    } else {
      const bool ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, p.status, 83));
      tc_fence_after();
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < NT && m0 + c < p.m; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(rows + (uint32_t)c, r);
          tmem_ld_wait();
          if (p.bias) add_bias32(r, p.bias, m0 + c, p.m);
          if (valid) {
#pragma unroll
            for (int j = 0; j < 32; j++)
              if (m0 + c + j < p.m) out[(long long)(c + j) * p.out_plane] = __uint_as_float(r[j]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, ACCS * NT);
  }
}

struct ConvNhwcWgradParams {
  float* part;                 // [splits][cout][32 * units]
  int32_t* status;
  int cout, units, cin, kw, taps, sh, sw, pt, pl, dh, dw;
  ConvBox box;                 // 32 pixels, tiling the output exactly
  int blocks, blocks_per_split;
  int chain;                   // pixel boxes an accumulator adds up
};
// One CTA: 128 output channels x four units of 32 channels of a tap, over a slice of the pixel boxes. CHAINS: a slice in several accumulator
// chains, as in conv_nhwc_kernel, where the product on the unfolded matrix has shorter slices.
template <bool CHAINS>
__global__ void __launch_bounds__(cn_threads(CHAINS), 2)
conv_nhwc_wgrad_kernel(const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ ConvNhwcWgradParams p) {
  constexpr int STAGES = 3, ACCS = CHAINS ? 2 : 1;
  constexpr int STAGE_BYTES = 2 * CV_BLOCK, CHUNK = CV_BK * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint64_t* acc_empty = acc_full + ACCS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + ACCS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int u0 = blockIdx.x * 4, m0 = blockIdx.y * CV_TILE;
  const int b0 = blockIdx.z * p.blocks_per_split;
  const int k_blocks = min(p.blocks_per_split, p.blocks - b0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < ACCS; a++) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 8);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, ACCS * CV_TILE);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();   // tensor memory is held: later kernels may become resident
  pdl_wait();      // everything below may depend on the previous kernel

  if (warp == 0) {
    if (lane == 0) {
      int dy[4], dx[4], c0[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        int t;
        cv_unit<CV_BK, 1>(min(u0 + j, p.units - 1), p.cin, p.taps, &t, &c0[j]);    // (past the last unit: its columns are not stored)
        dy[j] = (t / p.kw) * p.dh - p.pt;
        dx[j] = (t % p.kw) * p.dw - p.pl;
      }
      for (int kb = 0; kb < k_blocks; kb++) {
        const int s = kb % STAGES;
        const uint32_t round = kb / STAGES;
        if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1, abort_flag, p.status, 84)) break;
        const int b = b0 + kb;
        const int x0 = b % p.box.tw * p.box.w, y0 = b / p.box.tw % p.box.th * p.box.h, n0 = b / (p.box.tw * p.box.th) * p.box.n;
        uint8_t* a = smem + (size_t)s * STAGE_BYTES;
        // Channels past the last 32-channel block of the gradient are outside the tensor (zero), as are taps outside the image.
        int rows = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) rows += m0 + 32 * j < p.cout;
        mbar_expect_tx(&full[s], (uint32_t)((rows + 4) * CHUNK));
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (j < rows) tma_load_4d(a + j * CHUNK, &map_g, m0 + 32 * j, x0, y0, n0, &full[s]);
          tma_load_4d(a + CV_BLOCK + j * CHUNK, &map_x, c0[j], x0 * p.sw + dx[j], y0 * p.sh + dy[j], n0, &full[s]);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(CV_TILE >> 3) << 17) | ((uint32_t)(CV_TILE >> 4) << 24);
      int c = 0, at = 0;           // the chain, and the box of it
      for (int kb = 0; kb < k_blocks; kb++) {
        const int s = kb % STAGES;
        if (CHAINS && at == 0 && c >= ACCS && !mbar_wait(&acc_empty[c & 1], (uint32_t)((c >> 1) - 1) & 1, abort_flag, p.status, 88)) break;
        if (!mbar_wait(&full[s], (kb / STAGES) & 1, abort_flag, p.status, 85)) break;
        tc_fence_after();
        const uint32_t a = smem_u32(smem + (size_t)s * STAGE_BYTES), b = a + CV_BLOCK;
#pragma unroll
        for (int ks = 0; ks < CV_BK / 8; ks++)
          umma_tf32(tmem_base + (CHAINS ? (c & 1) * CV_TILE : 0), make_desc(a + ks * 1024, CHUNK, 512, 1), make_desc(b + ks * 1024, CHUNK, 512, 1), idesc,
                    ((CHAINS ? at : kb) > 0 || ks > 0) ? 1u : 0u);
        umma_commit(&empty[s]);
        if (CHAINS && (++at == p.chain || kb == k_blocks - 1)) {
          umma_commit(&acc_full[c & 1]);
          at = 0;
          c++;
        }
      }
      if (!CHAINS) umma_commit(acc_full);
    }
  } else {
    const int quad = warp & 3;
    const uint32_t rows = tmem_base + ((uint32_t)(quad * 32) << 16);
    // Accumulator rows through shared memory, then rows of whole 128-byte lines (COLS columns a warp). The last chain is complete only after every product,
    // and nothing more is loaded: the operand stages are dead.
    constexpr int COLS = CHAINS ? CV_TILE / 2 : CV_TILE, LD = COLS + 4;
    float* stg = reinterpret_cast<float*>(smem) + (warp - 2) * 32 * LD;
    const int col0 = (warp - 2) / 4 * COLS;
    bool ok;
    if constexpr (CHAINS) {
      float acc[COLS];
      ok = cn_add_chains<COLS>(acc, rows + (uint32_t)col0, CV_TILE, (k_blocks + p.chain - 1) / p.chain, acc_full, acc_empty, abort_flag, p.status, 86,
                               [](int) { return true; });
      if (ok) {
#pragma unroll
        for (int j = 0; j < COLS; j += 4) *reinterpret_cast<float4*>(stg + lane * LD + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
      }
    } else {
      ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, p.status, 86));
      tc_fence_after();
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < 4; c++) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(rows + (uint32_t)(c * 32), r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(stg + lane * LD + c * 32 + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
        }
      }
    }
    if (ok) {
      __syncwarp();
      constexpr int LANES = COLS / 4;                  // of a row
      const int ld = p.units * CV_BK, col = u0 * CV_BK + col0 + 4 * (lane % LANES);
      float* out = p.part + (long long)blockIdx.z * p.cout * ld + col;
      if (col < ld) {
#pragma unroll 4
        for (int i = lane / LANES; i < 32; i += 32 / LANES) {
          const int co = m0 + quad * 32 + i;
          if (co >= p.cout) break;
          *reinterpret_cast<float4*>(out + (long long)co * ld) = *reinterpret_cast<const float4*>(stg + i * LD + 4 * (lane % LANES));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, ACCS * CV_TILE);
  }
}

// ---- host side -------------------------------------------------------------------------------------------------------------
// K-major TF32 operand [rows, inner] (planes of them) with boxes of 32 x 128.
static bool cv_map(CUtensorMap* map, const float* base, long long inner, long long rows, long long ld, long long count, long long stride) {
  cuuint64_t dims[4] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)count, 1};
  const cuuint64_t filler = (((cuuint64_t)ld * rows * 4) + 15) & ~(cuuint64_t)15;
  cuuint64_t strides[3] = {(cuuint64_t)ld * 4, count > 1 ? (cuuint64_t)stride * 4 : filler, filler};
  cuuint32_t box[4] = {CV_BK, CV_TILE, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_TFLOAT32, 4, const_cast<float*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Byte offsets into a tensor are 32-bit and pixels (with a tile's or a slice's overhang) 31-bit numbers, taps a 32-bit mask.
static bool cv_sizes_fit(const ConvGeom& g) {
  const long long in = (long long)g.n * g.cin * g.h * g.w, out = (long long)g.n * g.cout * g.oh * g.ow;
  return g.groups == 1 && (long long)g.kh * g.kw <= CV_MAX_TAPS && in < (1ll << 30) && out < (1ll << 30) &&
         (long long)g.n * g.oh * g.ow < (1ll << 30) && (long long)g.n * g.h * g.w < (1ll << 30) &&
         (long long)g.cin * g.kh * g.kw <= 65535 && (long long)g.cout * g.kh * g.kw <= 65535 && g.n <= 65535 &&
         (long long)(g.kh - 1) * g.dh * g.w + (long long)g.kw * g.dw + (long long)g.pt * g.w + g.pl < (1ll << 28);
}

template <int MT>
static int32_t launch_conv_as(om_ctx* ctx, const CUtensorMap& map, const ConvTcParams& p, dim3 grid) {
  constexpr int STAGES = MT == 1 ? 3 : 2;
  constexpr size_t stages = (size_t)STAGES * (MT + 1) * CV_BLOCK;
  constexpr int most = 227 * 1024;
  static_assert(stages >= (size_t)CV_TILE * CV_STG_LD * 4, "the result rows are staged in the operand stages");
  static_assert(stages + 1024 + 128 + (65535 + CV_MAX_TAPS * CV_UNIT) / CV_UNIT * sizeof(int2) + 64 <= most, "every table of units fits");
  const size_t smem = stages + 1024 + 128 + (size_t)((p.units + 3) & ~3) * sizeof(int2);
  static bool set = false;
  if (!set) {
    OM_CUDA(ctx, cudaFuncSetAttribute(conv_tc_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    set = true;
  }
  launch_chained(ctx, conv_tc_kernel<MT>, grid, CV_THREADS, smem, map, p);
  OM_LAUNCH_CHECK(ctx, "conv_tc");
  return OM_OK;
}

// Where the product on the unfolded matrix would add up k in several slices, one accumulator for all of it would lose bits.
bool conv_tc_fwd_fits(const ConvGeom& g) {
  const int kk = g.cin * g.kh * g.kw;
  return encode_fn() && cv_sizes_fit(g) && product_chain_blocks(g.cout, g.n * g.oh * g.ow, kk) >= (int)ceil_div(kk, CV_BK);
}

int32_t conv_tc_fwd(om_ctx* ctx, const ConvGeom& g, const float* x, const float* w, const float* bias, float* y) {
  ConvTcParams p = {};
  p.src = x; p.out = y; p.bias = bias; p.status = ctx->status_dev;
  p.images = g.n; p.m = g.cout; p.sc = g.cin; p.sh = g.h; p.sw = g.w;
  p.pw = g.ow; p.plane = g.oh * g.ow;
  p.div_plane = cv_div((uint32_t)p.plane);
  p.div_w = cv_div((uint32_t)p.pw);
  p.step_y = g.sh; p.step_x = g.sw; p.base_y = -g.pt; p.base_x = -g.pl;
  p.vec = (p.plane & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
  p.taps = g.kh * g.kw;
  p.units = cv_units(g.cin, p.taps, CV_UNIT);
  for (int t = 0; t < p.taps; t++) {
    p.dy[t] = (t / g.kw) * g.dh;
    p.dx[t] = (t % g.kw) * g.dw;
  }
  const int ld = p.units * CV_UNIT;
  float* wt = nullptr;
  CUtensorMap map;
  OM_TRY(pool_alloc(ctx, sizeof(float) * (size_t)ld * p.m, false, (void**)&wt));
  int32_t st = cv_map(&map, wt, ld, p.m, ld, 1, 0) ? OM_OK : fail(ctx, OM_ERR_CUDA, "cuTensorMapEncodeTiled failed for a convolution's turned weights");
  if (st == OM_OK) {
    launch_chained(ctx, conv_turn_weights_kernel, dim3((unsigned)std::min<int64_t>(ceil_div(ld, 256), 64), (unsigned)p.m), 256, 0, w, wt, g.cin, p.taps, ld);
    // Two accumulators once that still leaves a CTA for every SM.
    const int64_t tiles = ceil_div((int64_t)g.n * p.plane, CV_TILE);
    const bool two = p.m > CV_TILE && tiles * ceil_div(p.m, 2 * CV_TILE) >= 148;
    const dim3 grid((unsigned)tiles, (unsigned)ceil_div(p.m, two ? 2 * CV_TILE : CV_TILE));
    st = two ? launch_conv_as<2>(ctx, map, p, grid) : launch_conv_as<1>(ctx, map, p, grid);
  }
  pool_free(ctx, wt);
  return st;
}

template <int UNIT, int GROUP>
static void launch_finish(om_ctx* ctx, const float* part, int splits, const ConvGeom& g, int units, float* dw, int accumulate) {
  const int ld = units * UNIT;
  if (splits <= 8)
    launch_chained(ctx, conv_wgrad_finish_kernel<1, UNIT, GROUP>, dim3((unsigned)ceil_div(ld, 256), (unsigned)g.cout), 256, 0, part, splits, g.cout, units, g.cin,
                                                                                                                        g.kh * g.kw, dw, accumulate);
  else
    launch_chained(ctx, conv_wgrad_finish_kernel<8, UNIT, GROUP>, dim3((unsigned)ceil_div(ld, 32), (unsigned)g.cout), 256, 0, part, splits, g.cout, units, g.cin,
                                                                                                                       g.kh * g.kw, dw, accumulate);
}

// Planes of whole stages always. With others the warps gather both operands, and the few pixels of a small product are too long a chain of loads; us
// unfolded / here: 37 x 64 x 11 x 12 by 64 (4884 pixels, 2.8 M floats unfolded) 26 / 34, 37 x 256 x 11 x 12 by 256 (4884, 11 M) 63 / 75, 32 x 256 x 14 x 14 by
// 256 (6272, 14 M) 77 / 89, 37 x 16 x 22 x 28 by 32 (22792, 3.3 M) 32 / 38, 128 x 32 x 24 x 24 by 32 with stride 2 (18432, 5.3 M) 34 / 38; 37 x 32 x 22 x 28
// by 32 (22792, 6.6 M) 40 / 38, 16 x 32 x 30 x 30 by 32 with 5 x 5 (14400, 11.5 M) 56 / 42.
bool conv_tc_wgrad_fits(const ConvGeom& g) {
  const long long pixels = (long long)g.n * g.oh * g.ow;
  return encode_fn() && cv_sizes_fit(g) && ((g.oh * g.ow) % CV_BK == 0 || (pixels >= 12288 && pixels * g.cin * g.kh * g.kw >= 6500000));
}

template <bool A_TMA>
static int32_t launch_wgrad(om_ctx* ctx, const CUtensorMap& map, const ConvWgradParams& p, dim3 grid) {
  constexpr size_t smem = (size_t)3 * 2 * CV_BLOCK + 1024 + 128;
  static bool set = false;
  if (!set) {
    OM_CUDA(ctx, cudaFuncSetAttribute(conv_wgrad_tc_kernel<A_TMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set = true;
  }
  launch_chained(ctx, conv_wgrad_tc_kernel<A_TMA>, grid, CV_THREADS, smem, map, p);
  return OM_OK;
}

int32_t conv_tc_wgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* x, float* dw, int accumulate) {
  ConvWgradParams p = {};
  p.gr = gr; p.x = x; p.status = ctx->status_dev;
  p.cout = g.cout; p.cin = g.cin; p.h = g.h; p.w = g.w; p.kw = g.kw; p.taps = g.kh * g.kw; p.sh = g.sh; p.sw = g.sw;
  p.pt = g.pt; p.pl = g.pl; p.dh = g.dh; p.dw = g.dw; p.ow = g.ow; p.plane = g.oh * g.ow;
  p.units = cv_units(g.cin, p.taps, CV_UNIT);
  p.div_plane = cv_div((uint32_t)p.plane);
  p.div_w = cv_div((uint32_t)g.ow);
  p.pixels = g.n * p.plane;
  const bool a_tma = (p.plane & 31) == 0 && (reinterpret_cast<uintptr_t>(gr) & 15) == 0;
  CUtensorMap map = {};
  if (a_tma && !cv_map(&map, gr, p.plane, g.cout, p.plane, g.n, (long long)g.cout * p.plane))
    return fail(ctx, OM_ERR_CUDA, "cuTensorMapEncodeTiled failed for a convolution's gradient");
  // Slices of the pixels for one round of two CTAs an SM, each at least eight stages long, and none longer than those of the product on the
  // unfolded matrix (what one accumulator adds up loses bits with its length): a function of the shape alone.
  const int ld = p.units * CV_UNIT;
  const int tn = (int)ceil_div(ld, CV_TILE), tm = (int)ceil_div(g.cout, CV_TILE);
  const long long blocks = ceil_div(p.pixels, CV_BK);
  int splits = (int)std::max<long long>(1, std::min<long long>(kSplitSlots / ((long long)tn * tm), blocks / 8));
  p.blocks_per_split = std::min((int)ceil_div(blocks, splits), product_chain_blocks(g.cout, g.cin * p.taps, p.pixels));
  splits = (int)ceil_div(blocks, p.blocks_per_split);
  OM_TRY(pool_alloc(ctx, sizeof(float) * (size_t)splits * g.cout * ld, false, (void**)&p.part));
  const dim3 grid((unsigned)tn, (unsigned)tm, (unsigned)splits);
  int32_t st = a_tma ? launch_wgrad<true>(ctx, map, p, grid) : launch_wgrad<false>(ctx, map, p, grid);
  if (st == OM_OK) launch_finish<CV_UNIT, CV_GROUP>(ctx, p.part, splits, g, p.units, dw, accumulate);
  pool_free(ctx, p.part);
  OM_TRY(st);
  OM_LAUNCH_CHECK(ctx, "conv_wgrad_tc");
  return OM_OK;
}

// ---- channels last, host side ----------------------------------------------------------------------------------------------
// The box of `size` pixels (a power of two) that covers a grid of w x h x n pixels in the fewest tiles, the widest of those.
static ConvBox cn_box(int size, int w, int h, int n) {
  ConvBox best = {};
  long long fewest = -1;
  for (int bw = size; bw >= 1; bw /= 2)
    for (int bh = size / bw; bh >= 1; bh /= 2) {
      const ConvBox b = {bw, bh, size / bw / bh, (int)ceil_div(w, bw), (int)ceil_div(h, bh), (int)ceil_div(n, size / bw / bh)};
      const long long tiles = (long long)b.tw * b.th * b.tn;
      if (fewest < 0 || tiles < fewest) {
        fewest = tiles;
        best = b;
      }
    }
  return best;
}
static int cn_pitch(int c) { return (c + 3) & ~3; }

// The turned tensor [n][h][w][c] with boxes of 32 channels x `box`, taken every (sy, sx) pixels.
static bool cn_map(CUtensorMap* map, const float* base, int c, int w, int h, int n, const ConvBox& box, int sx, int sy, bool mn_major) {
  const cuuint64_t row = (cuuint64_t)cn_pitch(c) * 4;
  cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
  cuuint64_t strides[3] = {row, row * w, row * w * h};
  cuuint32_t bx[4] = {CV_BK, (cuuint32_t)(box.w * sx), (cuuint32_t)(box.h * sy), (cuuint32_t)box.n};
  cuuint32_t estr[4] = {1, (cuuint32_t)sx, (cuuint32_t)sy, 1};
  return encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_TFLOAT32, 4, const_cast<float*>(base), dims, strides, bx, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int32_t cn_turn(om_ctx* ctx, const float* src, int n, int c, int plane, float** out) {
  const int pixels = n * plane, cp = cn_pitch(c);
  OM_TRY(pool_alloc(ctx, sizeof(float) * (size_t)pixels * cp, false, (void**)out));
  launch_chained(ctx, conv_channels_last_kernel<false>, dim3((unsigned)ceil_div(pixels, CN_PX), (unsigned)ceil_div(cp, 32)), 256, 0, src, *out, pixels, plane,
                 cv_div((uint32_t)plane), c, cp, nullptr);
  return OM_OK;
}

// A block of 32 channels may be partly empty, and a box partly outside the grid: at least two thirds of the work has to be real.
static bool cn_channels_fit(int c) { return 3 * c >= 2 * (int)ceil_div(c, 32) * 32; }
static bool cn_sizes_fit(const ConvGeom& g) {
  return encode_fn() && cv_sizes_fit(g) && g.sh <= 2 && g.sw <= 2 && (long long)g.n * g.h * g.w * cn_pitch(g.cin) < (1ll << 30) &&
         (long long)g.n * g.oh * g.ow * cn_pitch(g.cout) < (1ll << 30);
}
// The lines between the channels-last form and the others, 3 x 3 windows, us channels last / unfolded / gathered:
//   forward         against the unfolded matrix by its size, np x k floats: 16 x 256 x 12 x 12 to 256 (5.3 M) 52 / 38, 8 x 512 x 8 x 8 to 512 (2.4 M)
//                   83 / 32, 37 x 64 x 11 x 12 to 64 (2.8 M) 28 / 26; 37 x 128 x 11 x 12 to 128 (5.6 M) 39 / 38, 32 x 96 x 16 x 16 to 96 (7.1 M)
//                   34 / 40, 37 x 256 x 11 x 12 to 256 (11 M) 54 / 63. Against the gathering kernel by its products: 64 x 40 x 20 x 32 to 40
//                   (1.2 GFLOP) 38 / 65 / 34, 64 x 24 x 20 x 32 to 48 (0.8) 30 / 46 / 26, 37 x 64 x 22 x 28 to 64 (1.7) 26 / 52.
//   input gradient  by the size of the unfolded matrix, the zeros between strides counted: 37 x 24 x 22 x 28 from 48 (4.9 M) 32 / 32, 16 x 256 x 12 x 12
//                   from 256 (5.3 M) 50 / 36, 8 x 512 x 8 x 8 from 512 (2.4 M) 79 / 36; 37 x 128 x 11 x 12 from 128 (5.6 M) 36 / 40, 64 x 16 x 20 x 32
//                   from 16 (5.9 M) 30 / 34, 37 x 132 x 11 x 12 from 36 (5.8 M) 30 / 36, 128 x 16 x 24 x 24 from 16 (10.6 M) 36 / 50, with stride 2 24 / 36.
//                   A deep k makes the few CTAs of a small plane long: 32 x 512 x 7 x 7 from 512 (7.2 M, 144 blocks of k) 81 / 56, 256 x 512 x 4 x 4 from
//                   512 (18.9 M) 83 / 104. 1 x 1 windows always: 64 x 64 x 16 x 16 15 / 22, 16 x 128 x 14 x 14 from 256 17 / 22.
constexpr long long CN_MIN_UNFOLDED = 5500000, CN_MIN_UNFOLDED_A_BLOCK = 80000;
constexpr double CN_MIN_FLOPS = 1e9;
static double cn_flops(const ConvGeom& g) { return 2.0 * g.n * g.oh * g.ow * (double)g.cout * g.cin * g.kh * g.kw; }

template <int NT, int STAGES, bool CHAINS>
static int32_t launch_nhwc(om_ctx* ctx, const ConvNhwcMaps& maps, const ConvNhwcParams& p, dim3 grid) {
  constexpr size_t smem = (size_t)STAGES * (CV_BLOCK + NT * 128) + 1024 + 256;
  static bool set = false;
  if (!set) {
    OM_CUDA(ctx, cudaFuncSetAttribute(conv_nhwc_kernel<NT, STAGES, CHAINS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set = true;
  }
  launch_chained(ctx, conv_nhwc_kernel<NT, STAGES, CHAINS>, grid, cn_threads(CHAINS), smem, maps, p);
  return check_cuda(ctx, cudaGetLastError(), "conv_nhwc");
}

// Runs the product of every phase from the turned source (turned here when none is given); the phases' grids, taps and output
// positions are set.
static int32_t run_conv_nhwc(om_ctx* ctx, ConvNhwcParams& p, ConvTurn& turn, int phases, int taps_all, const float* src, const float* turned, int sc, int sh, int sw,
                             const float* w) {
  ConvNhwcMaps maps = {};
  float *own = nullptr, *wt = nullptr;
  if (!turned) OM_TRY(cn_turn(ctx, src, p.images, sc, sh * sw, &own));
  const float* t = turned ? turned : own;
  const int nt = p.m <= 64 ? 64 : 128;
  long long floats = 0, most = 0;
  int most_ld = 0;
  bool chains = false;
  turn.by_tap = p.by_tap;
  p.sh = sh;
  p.sw = sw;
  for (int z = 0; z < phases; z++) {
    ConvNhwcPhase& f = p.phase[z];
    f.box = cn_box(CV_TILE, f.pw, f.ph, p.images);
    const int units = cv_units(sc, f.taps, CV_BK);
    f.k_blocks = units;
    if (p.by_tap) f.chain = units / std::max(1, f.taps);
    f.chain = std::max(1, f.chain);
    chains = chains || f.chain < units || units == 0;
    turn.taps[z] = f.taps;
    turn.ld[z] = units * CV_BK;
    turn.start[z] = floats;
    floats += (long long)turn.ld[z] * p.m;
    most_ld = std::max(most_ld, turn.ld[z]);
    most = std::max(most, (long long)f.box.tw * f.box.th * f.box.tn);
  }
  int32_t st = pool_alloc(ctx, sizeof(float) * (size_t)std::max<long long>(floats, 4), false, (void**)&wt);
  for (int z = 0; z < phases && st == OM_OK; z++) {
    const ConvNhwcPhase& f = p.phase[z];
    if (f.k_blocks == 0) continue;
    bool ok = cn_map(&maps.src[z], t, sc, sw, sh, p.images, f.box, p.step_x, p.step_y, false);
    cuuint64_t dims[4] = {(cuuint64_t)turn.ld[z], (cuuint64_t)p.m, 1, 1};
    const cuuint64_t row = (cuuint64_t)turn.ld[z] * 4;
    cuuint64_t strides[3] = {row, row * p.m, row * p.m};
    cuuint32_t bx[4] = {CV_BK, (cuuint32_t)nt, 1, 1}, estr[4] = {1, 1, 1, 1};
    ok = ok && encode_fn()(&maps.w[z], CU_TENSOR_MAP_DATA_TYPE_TFLOAT32, 4, wt + turn.start[z], dims, strides, bx, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    if (!ok) st = fail(ctx, OM_ERR_CUDA, "cuTensorMapEncodeTiled failed for a convolution's operands");
  }
  if (st == OM_OK && most > 0) {
    if (most_ld > 0)
      launch_chained(ctx, conv_pack_weights_kernel, dim3((unsigned)ceil_div(sc, CV_BK), (unsigned)ceil_div(p.m, CN_PACK_M)), 256,
                     sizeof(float) * CN_PACK_M * CV_BK * (taps_all | 1), w, wt, turn, taps_all, phases);
    const dim3 grid((unsigned)most, (unsigned)ceil_div(p.m, nt), (unsigned)phases);
    // Twice the stages where the grid gives an SM one CTA at most.
    const bool alone = (int64_t)grid.x * grid.y * grid.z <= 148;
    if (chains && nt == 64) st = alone ? launch_nhwc<64, 8, true>(ctx, maps, p, grid) : launch_nhwc<64, 4, true>(ctx, maps, p, grid);
    else if (chains) st = alone ? launch_nhwc<128, 6, true>(ctx, maps, p, grid) : launch_nhwc<128, 3, true>(ctx, maps, p, grid);
    else if (nt == 64) st = alone ? launch_nhwc<64, 8, false>(ctx, maps, p, grid) : launch_nhwc<64, 4, false>(ctx, maps, p, grid);
    else st = alone ? launch_nhwc<128, 6, false>(ctx, maps, p, grid) : launch_nhwc<128, 3, false>(ctx, maps, p, grid);
  }
  if (own) pool_free(ctx, own);
  if (wt) pool_free(ctx, wt);
  return st;
}

// The taps that reach the input positions (oy0, ox0) modulo the stride, and where in the gradient from a pixel of that class.
static int class_taps(const ConvGeom& g, int oy0, int ox0, int* dy, int* dx, int* tap) {
  int n = 0;
  for (int t = 0; t < g.kh * g.kw; t++) {
    const int ty = oy0 + g.pt - (t / g.kw) * g.dh, tx = ox0 + g.pl - (t % g.kw) * g.dw;
    if (ty % g.sh || tx % g.sw) continue;      // (exact for negative values too)
    dy[n] = ty / g.sh;
    dx[n] = tx / g.sw;
    tap[n++] = t;
  }
  return n;
}

static bool cn_grid_fits(int w, int h, int n) {
  const ConvBox b = cn_box(CV_TILE, w, h, n);
  return 3 * (long long)w * h * n >= 2 * (long long)b.tw * b.th * b.tn * CV_TILE;
}
bool conv_nhwc_fwd_fits(const ConvGeom& g) {
  return cn_sizes_fit(g) && cn_channels_fit(g.cin) && cn_grid_fits(g.ow, g.oh, g.n) && (long long)g.n * g.oh * g.ow * g.cin * g.kh * g.kw >= CN_MIN_UNFOLDED &&
         (cn_flops(g) >= CN_MIN_FLOPS || !conv_tc_fwd_fits(g));
}

int32_t conv_nhwc_fwd(om_ctx* ctx, const ConvGeom& g, const float* x, const float* w, const float* bias, float* y) {
  ConvNhwcParams p = {};
  ConvTurn turn = {};
  p.out = y; p.bias = bias; p.status = ctx->status_dev;
  p.images = g.n; p.m = g.cout; p.out_w = g.ow; p.out_plane = g.oh * g.ow;
  p.step_y = g.sh; p.step_x = g.sw; p.base_y = -g.pt; p.base_x = -g.pl; p.ostep_y = p.ostep_x = 1;
  ConvNhwcPhase& f = p.phase[0];
  f.ph = g.oh; f.pw = g.ow; f.taps = g.kh * g.kw;
  f.chain = cv_units(g.cin, f.taps, CV_BK);
  const int plain = product_chain_blocks(g.cout, g.n * g.oh * g.ow, g.cin * f.taps);
  if (plain < (int)ceil_div(g.cin * f.taps, CV_BK)) f.chain = plain;     // (a chain no longer than the product on the unfolded matrix has)
  for (int t = 0; t < f.taps; t++) {
    f.dy[t] = (t / g.kw) * g.dh;
    f.dx[t] = (t % g.kw) * g.dw;
    turn.tap[0][t] = t;
  }
  turn.m = g.cout; turn.sc = g.cin;
  turn.stride_m = (long long)g.cin * f.taps; turn.stride_sc = f.taps;
  return run_conv_nhwc(ctx, p, turn, 1, f.taps, x, nullptr, g.cin, g.h, g.w, w);
}

// (what a box holds outside the grid counts against the size of the unfolded matrix: three times the time, at a quarter of the pixels)
bool conv_nhwc_dgrad_fits(const ConvGeom& g) {
  if (!cn_sizes_fit(g)) return false;
  if (g.kh * g.kw == 1) return true;
  const int cw = (int)ceil_div(g.w, g.sw), ch = (int)ceil_div(g.h, g.sh);
  const ConvBox b = cn_box(CV_TILE, cw, ch, g.n);
  const double unfolded = (double)g.n * g.oh * g.ow * g.sh * g.sw * g.cin * g.kh * g.kw, filled = (double)cw * ch * g.n / ((double)b.tw * b.th * b.tn * CV_TILE);
  return unfolded * filled >= (double)std::max(CN_MIN_UNFOLDED, CN_MIN_UNFOLDED_A_BLOCK * cv_units(g.cout, g.kh * g.kw, CV_BK));
}

int32_t conv_nhwc_dgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* w, float* dx, const float* gt) {
  ConvNhwcParams p = {};
  ConvTurn turn = {};
  p.out = dx; p.status = ctx->status_dev;
  p.images = g.n; p.m = g.cin; p.out_w = g.w; p.out_plane = g.h * g.w;
  p.step_y = p.step_x = 1; p.by_tap = 1; p.ostep_y = g.sh; p.ostep_x = g.sw;
  for (int z = 0; z < g.sh * g.sw; z++) {
    ConvNhwcPhase& f = p.phase[z];
    f.oy0 = z / g.sw;
    f.ox0 = z % g.sw;
    f.ph = f.oy0 < g.h ? (g.h - f.oy0 + g.sh - 1) / g.sh : 0;
    f.pw = f.ox0 < g.w ? (g.w - f.ox0 + g.sw - 1) / g.sw : 0;
    f.taps = class_taps(g, f.oy0, f.ox0, f.dy, f.dx, turn.tap[z]);
  }
  turn.m = g.cin; turn.sc = g.cout;
  turn.stride_m = g.kh * g.kw; turn.stride_sc = (long long)g.cin * g.kh * g.kw;
  return run_conv_nhwc(ctx, p, turn, g.sh * g.sw, g.kh * g.kw, gr, gt, g.cout, g.oh, g.ow, w);
}

// The pixel boxes have to tile the output exactly: a slot outside it would multiply its zero gradient with values of the input, which may
// be infinite.
bool conv_nhwc_wgrad_fits(const ConvGeom& g) {
  if (!cn_sizes_fit(g) || !cn_channels_fit(g.cin) || cn_flops(g) < CN_MIN_FLOPS) return false;
  const ConvBox b = cn_box(CV_BK, g.ow, g.oh, g.n);
  return g.ow % b.w == 0 && g.oh % b.h == 0 && g.n % b.n == 0;
}

template <bool CHAINS>
static int32_t launch_nhwc_wgrad(om_ctx* ctx, const CUtensorMap& map_g, const CUtensorMap& map_x, const ConvNhwcWgradParams& p, dim3 grid) {
  constexpr size_t smem = (size_t)3 * 2 * CV_BLOCK + 1024 + 128;
  static_assert(3 * 2 * CV_BLOCK >= (cn_threads(CHAINS) - 64) * (CV_TILE / (CHAINS ? 2 : 1) + 4) * 4, "the result rows are staged in the operand stages");
  static bool set = false;
  if (!set) {
    OM_CUDA(ctx, cudaFuncSetAttribute(conv_nhwc_wgrad_kernel<CHAINS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set = true;
  }
  launch_chained(ctx, conv_nhwc_wgrad_kernel<CHAINS>, grid, cn_threads(CHAINS), smem, map_g, map_x, p);
  return OM_OK;
}

int32_t conv_nhwc_wgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* x, float* dw, int accumulate, const float* turned) {
  ConvNhwcWgradParams p = {};
  p.status = ctx->status_dev;
  p.cout = g.cout; p.cin = g.cin; p.kw = g.kw; p.taps = g.kh * g.kw; p.sh = g.sh; p.sw = g.sw; p.pt = g.pt; p.pl = g.pl; p.dh = g.dh; p.dw = g.dw;
  p.units = cv_units(g.cin, p.taps, CV_BK);
  p.box = cn_box(CV_BK, g.ow, g.oh, g.n);
  p.blocks = p.box.tw * p.box.th * p.box.tn;
  const int ld = p.units * CV_BK;
  const int tn = (int)ceil_div(p.units, 4), tm = (int)ceil_div(g.cout, CV_TILE);
  // Slices of the pixels for one round of two CTAs an SM, each at least eight stages long: a function of the shape alone.
  int splits = (int)std::max<long long>(1, std::min<long long>(kSplitSlots / ((long long)tn * tm), p.blocks / 8));
  p.blocks_per_split = (int)ceil_div(p.blocks, splits);
  splits = (int)ceil_div(p.blocks, p.blocks_per_split);
  // No longer than the chains of the product on the unfolded matrix, and half of them where the boxes walk the pixels in another order than it does: of 90
  // geometries three were 6 to 8 % further from float64 than that product with its length (60 x 128 x 8 x 54 by 256: 3.41e-6 / 3.66e-6).
  const int plain = product_chain_blocks(g.cout, g.cin * p.taps, g.n * g.oh * g.ow);
  const bool in_order = (p.box.w == g.ow && (p.box.h == g.oh || p.box.n == 1)) || (p.box.h == 1 && p.box.n == 1);
  p.chain = std::min(p.blocks_per_split, in_order ? plain : (plain + 1) / 2);
  float *own = nullptr, *xt = nullptr;
  CUtensorMap map_g = {}, map_x = {};
  int32_t st = turned ? OM_OK : cn_turn(ctx, gr, g.n, g.cout, g.oh * g.ow, &own);
  const float* gt = turned ? turned : own;
  if (st == OM_OK) st = cn_turn(ctx, x, g.n, g.cin, g.h * g.w, &xt);
  if (st == OM_OK) st = pool_alloc(ctx, sizeof(float) * (size_t)splits * g.cout * ld, false, (void**)&p.part);
  if (st == OM_OK && (!cn_map(&map_g, gt, g.cout, g.ow, g.oh, g.n, p.box, 1, 1, true) || !cn_map(&map_x, xt, g.cin, g.w, g.h, g.n, p.box, g.sw, g.sh, true)))
    st = fail(ctx, OM_ERR_CUDA, "cuTensorMapEncodeTiled failed for a convolution's operands");
  if (st == OM_OK) {
    const dim3 grid((unsigned)tn, (unsigned)tm, (unsigned)splits);
    st = p.chain < p.blocks_per_split ? launch_nhwc_wgrad<true>(ctx, map_g, map_x, p, grid) : launch_nhwc_wgrad<false>(ctx, map_g, map_x, p, grid);
    if (st == OM_OK) {
      launch_finish<CV_BK, 1>(ctx, p.part, splits, g, p.units, dw, accumulate);
      st = check_cuda(ctx, cudaGetLastError(), "conv_nhwc_wgrad");
    }
  }
  if (own) pool_free(ctx, own);
  if (xt) pool_free(ctx, xt);
  if (p.part) pool_free(ctx, p.part);
  return st;
}

long long conv_nhwc_turned_floats(const ConvGeom& g) { return (long long)g.n * g.oh * g.ow * cn_pitch(g.cout); }

int32_t conv_nhwc_turn_gradient(om_ctx* ctx, const ConvGeom& g, const float* gr, float* turned, float* dbias, int accumulate_b) {
  const int plane = g.oh * g.ow, pixels = g.n * plane, cp = cn_pitch(g.cout);
  const unsigned columns = (unsigned)ceil_div(cp, 32), tiles = (unsigned)ceil_div(pixels, CN_PX);
  if (!dbias) {
    launch_chained(ctx, conv_channels_last_kernel<false>, dim3(tiles, columns), 256, 0, gr, turned, pixels, plane, cv_div((uint32_t)plane), g.cout, cp, nullptr);
  } else {
    const int ctas = std::min((int)tiles, CN_SUM_CTAS);
    double* sums = nullptr;
    OM_TRY(pool_alloc(ctx, sizeof(double) * (size_t)ctas * g.cout, false, (void**)&sums));
    launch_chained(ctx, conv_channels_last_kernel<true>, dim3((unsigned)ctas, columns), 256, 0, gr, turned, pixels, plane, cv_div((uint32_t)plane), g.cout, cp, sums);
    launch_chained(ctx, conv_sums_finish_kernel, (unsigned)ceil_div(g.cout, 32), 256, 0, sums, ctas, g.cout, dbias, accumulate_b);
    pool_free(ctx, sums);
  }
  OM_LAUNCH_CHECK(ctx, "conv_nhwc_turn_gradient");
  return OM_OK;
}

}  // namespace om
