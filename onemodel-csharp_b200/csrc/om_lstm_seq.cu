// Whole-sequence LSTM kernels: all T time steps of one or two directions in ONE cooperative launch.
//
// The step-by-step path (om_recurrent.cu) launches a recurrent product and a gate kernel per time step: at the sizes
// of a text-line recogniser (batch 64, hidden 256, 64 frames) each of those ~1000 launches per training step does a
// few microseconds of work and the sequence is bound by launch and dependency latency. Here the work of a step is
// tiled over CTAs as (16 hidden units) x (a group of batch rows): a CTA keeps the rows (forward) or columns (backward)
// of W_hh that belong to its units in shared memory for the whole sequence, and per step brings in only the previous
// state (forward: h, 16 rows x H) or the shares of its units' state gradient (backward: 16 rows x 16 units from H / 16
// slices) of its own batch rows, computes with fp32 FMAs from shared memory, applies the cell, and meets the CTAs that
// share its batch rows (the other unit slices) at a barrier, once per time step. CTAs of different row groups and directions never wait for one another.
//
// Arithmetic: fp32 throughout (more accurate than the TF32 product of the step-by-step fast path). A dot product is
// split in eight (forward) or 2 H / 16 (backward) k ranges summed in a fixed order, so results do not depend on scheduling;
// they are not the one-accumulator order of the reference's exact tier, which stays on the step-by-step path.
//
// CTAs wait on one another, so the launch is cooperative (all CTAs resident at once; the host checks the occupancy
// first) and every wait at the barrier is bounded: after about a second a CTA raises OM_ERR_TIMEOUT in the context's
// status word and returns, and the others follow at their own bound.
#include "om_lstm_seq.cuh"

namespace om {

constexpr int kSeqThreads = 256;
constexpr int kSeqRows = 16;          // batch rows per pass
constexpr int kSeqUnits = 16;         // hidden units per CTA
constexpr int kSeqMaxGroups = 16;     // row groups (barrier counters) per direction
constexpr int kSeqPad = 4;            // floats of padding per shared-memory row: rows land on different banks
constexpr long long kSeqWaitCycles = 2000000000LL;

__device__ __forceinline__ float seq_sigm(float x) { return 1.0f / (1.0f + expf(-x)); }

// Barrier of one (direction, row group): arrival number `target` completes it. Returns false when the wait ran out.
__device__ __forceinline__ bool seq_barrier(unsigned* counter, unsigned target, int32_t* status, int* failed, int where) {
  __syncthreads();
  if (threadIdx.x == 0) {
    // Release at device scope: the CTA's writes (ordered before this thread by the barrier above) are visible to whoever
    // observes the count.
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    const long long t0 = clock64();
    for (;;) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      if (v >= target) break;
      if (clock64() - t0 > kSeqWaitCycles) {
        *failed = 1;
        if (atomicCAS(status, 0, (int32_t)OM_ERR_TIMEOUT) == 0) status[1] = where;
        break;
      }
    }
  }
  __syncthreads();
  return *failed == 0;
}

// Copies rows r0 .. r0 + 15 of src [B, 4 * q4] (written by other CTAs of this launch: past L1) into rows of ld floats, zero beyond B; the loads
// of four rounds are in flight together.
__device__ __forceinline__ void seq_stage_rows(float* dst, int ld, const float* src, int r0, int B, int q4, int tid) {
  for (int base = tid; base < kSeqRows * q4; base += 4 * kSeqThreads) {
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int idx = base + i * kSeqThreads, r = idx / q4, b = r0 + r;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (idx < kSeqRows * q4 && b < B) v[i] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)b * 4 * q4) + (idx - r * q4));
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int idx = base + i * kSeqThreads, r = idx / q4;
      if (idx < kSeqRows * q4) *reinterpret_cast<float4*>(dst + (size_t)r * ld + 4 * (idx - r * q4)) = v[i];
    }
  }
}

// Forward. Grid (H / 16, row groups, directions). Shared memory: ws [64][H + 4] (row q * 16 + j = W_hh[q * H + j0 + j, :]),
// hs [16][H + 4] (previous h of the pass's rows).
// Threads: k lane = tid % 8, unit = tid / 8 % 16, row half = tid / 128: a thread forms the four gate dot products of one unit for eight
// batch rows over every eighth float4 of k (12 shared-memory reads for 128 multiply-adds: the reads bound the product, and
// with two rows a thread they were 6 for 32); the eight k lanes then fold their sums by halves, each keeping half of the rows
// it holds, so that every thread ends with the four gates of one (row, unit) and applies the cell to it.
__global__ void __launch_bounds__(kSeqThreads) lstm_seq_fwd_kernel(const LstmSeqFwdParams p) {
  extern __shared__ __align__(16) float seq_smem[];
  __shared__ int failed;
  const LstmSeqFwdDir& D = p.d[blockIdx.z];
  const int H = p.h, B = p.b, T = p.t, H4 = 4 * p.h, ldw = p.h + kSeqPad;
  const int j0 = blockIdx.x * kSeqUnits, tid = threadIdx.x;
  const int group_rows = p.passes * kSeqRows, row_base = blockIdx.y * group_rows;
  float* ws = seq_smem;
  float* hs = ws + (size_t)64 * ldw;
  const int hq = H / 4;
  for (int idx = tid; idx < 64 * hq; idx += kSeqThreads) {
    const int row = idx / hq, k4 = idx % hq, q = row / kSeqUnits, j = row % kSeqUnits;
    *reinterpret_cast<float4*>(ws + (size_t)row * ldw + 4 * k4) = __ldg(reinterpret_cast<const float4*>(D.w_hh + (size_t)(q * H + j0 + j) * H) + k4);
  }
  if (tid == 0) failed = 0;
  __syncthreads();
  const int kl = tid & 7, un = (tid >> 3) & 15, rh = tid >> 7;
  const size_t bh = (size_t)B * H;
  unsigned* counter = D.counter + blockIdx.y;
  const int jg = j0 + un;
  float bias[4] = {0.f, 0.f, 0.f, 0.f};
  if (D.bias != nullptr)
    for (int q = 0; q < 4; q++) bias[q] = D.bias[q * H + jg];
  // With one pass a CTA the thread's (row, unit) is the same at every step: its cell state stays in a register and the next step's
  // pre-activations are fetched ahead of the barrier (they do not depend on the other CTAs).
  float pre[4] = {0.f, 0.f, 0.f, 0.f}, c_own = 0.f;
  for (int f = 0; f < T; f++) {
    const int tt = D.reverse ? T - 1 - f : f;
    const int pt = D.reverse ? tt + 1 : tt - 1;
    const float* hp = f == 0 ? D.h0 : D.y + (size_t)pt * bh;
    const float* cp = f == 0 ? D.c0 : D.c + (size_t)pt * bh;
    float* gates_t = D.gates + (size_t)tt * B * H4;
    for (int pass = 0; pass < p.passes; pass++) {
      const int r0 = row_base + pass * kSeqRows;
      if (r0 >= B) break;
      const int b = r0 + rh * 8 + kl;
      float cprev = c_own;
      if (b < B && (p.passes > 1 || f == 0)) {
#pragma unroll
        for (int q = 0; q < 4; q++) pre[q] = gates_t[(size_t)b * H4 + q * H + jg];
        cprev = cp != nullptr ? __ldcg(cp + (size_t)b * H + jg) : 0.f;
      }
      float acc[8][4];
#pragma unroll
      for (int r = 0; r < 8; r++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[r][q] = 0.f;
      if (hp != nullptr) {
        seq_stage_rows(hs, ldw, hp, r0, B, hq, tid);
        __syncthreads();
        const float* hrow = hs + (size_t)rh * 8 * ldw;
        const float* wrow = ws + (size_t)un * ldw;
#pragma unroll 2
        for (int k4 = kl; k4 < hq; k4 += 8) {
          float4 w[4];
#pragma unroll
          for (int q = 0; q < 4; q++) w[q] = *reinterpret_cast<const float4*>(wrow + (size_t)q * kSeqUnits * ldw + 4 * k4);
#pragma unroll
          for (int r = 0; r < 8; r++) {
            const float4 a = *reinterpret_cast<const float4*>(hrow + (size_t)r * ldw + 4 * k4);
#pragma unroll
            for (int q = 0; q < 4; q++) {
              acc[r][q] = fmaf(a.x, w[q].x, acc[r][q]);
              acc[r][q] = fmaf(a.y, w[q].y, acc[r][q]);
              acc[r][q] = fmaf(a.z, w[q].z, acc[r][q]);
              acc[r][q] = fmaf(a.w, w[q].w, acc[r][q]);
            }
          }
        }
      }
      // fold the eight k lanes: after the step of width w a lane holds w rows, the last one is row rh * 8 + kl
#pragma unroll
      for (int w = 4; w > 0; w >>= 1) {
        const bool high = (kl & w) != 0;
#pragma unroll
        for (int r = 0; r < 4; r++) {
          if (r >= w) break;
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const float keep = high ? acc[r + w][q] : acc[r][q], send = high ? acc[r][q] : acc[r + w][q];
            acc[r][q] = keep + __shfl_xor_sync(0xffffffffu, send, w);
          }
        }
      }
      if (b < B) {
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          float tv = pre[q] + acc[0][q];
          if (D.bias != nullptr) tv = tv + bias[q];
          v[q] = tv;
        }
        const float gi = seq_sigm(v[0]), gf = seq_sigm(v[1]), gg = tanhf(v[2]), go = seq_sigm(v[3]);
        const size_t idx = (size_t)b * H + jg;
        const float fc = gf * cprev;
        const float ig = gi * gg;
        const float cn = fc + ig;
        const float tc = tanhf(cn);
        D.y[(size_t)tt * bh + idx] = go * tc;
        float* g = gates_t + (size_t)b * H4;
        g[jg] = gi;
        g[H + jg] = gf;
        g[2 * H + jg] = gg;
        g[3 * H + jg] = go;
        D.c[(size_t)tt * bh + idx] = cn;
        D.tanh_c[(size_t)tt * bh + idx] = tc;
        c_own = cn;
        if (p.passes == 1 && f + 1 < T) {
          const float* next = D.gates + (size_t)(D.reverse ? tt - 1 : tt + 1) * B * H4 + (size_t)b * H4 + jg;
#pragma unroll
          for (int q = 0; q < 4; q++) pre[q] = next[q * H];
        }
      }
      __syncthreads();   // hs is reused by the next pass
    }
    if (f + 1 < T && !seq_barrier(counter, (unsigned)(f + 1) * gridDim.x, p.status, &failed, 9100 + (int)blockIdx.z)) return;
  }
}

// Backward. Grid as forward. dh of the previous step is dG_t W_hh, a sum over all 4 H gate columns. A CTA owns 64 of them (its 16 units'
// gates): it forms their share of the sum for ALL units and leaves it in `part`, and after the barrier every CTA adds the
// shares of its own units in the order of the slices. (Exchanging dG_t itself instead, every CTA read 16 rows x 4 H a step,
// four times what the shares of its units are.) Shares of even and odd steps lie apart: a CTA may write step s + 1's while another still
// reads step s's, and all have read step s's before anyone passes the barrier of s + 1.
// Shared memory: ws [64][H] (row q * 16 + j = W_hh[q * H + j0 + j, :]), ds [64][16] (the gate gradients of the pass's rows, turned), red
// [128][36] (the second k half's sums), dh_s and dc_s [group rows][16] (the state gradients of this CTA's units).
// Threads of the product: k half = tid / 128, row half = tid / 64 % 2, column quad = tid % 64 (+ 64 a round): eight rows x four columns
// over 32 gate columns, three shared-memory reads for 32 multiply-adds. Threads of the cell: row = tid / 16, unit = tid % 16.
constexpr int kSeqRedLd = 36;
__global__ void __launch_bounds__(kSeqThreads) lstm_seq_bwd_kernel(const LstmSeqBwdParams p) {
  extern __shared__ __align__(16) float seq_smem[];
  __shared__ int failed;
  const LstmSeqBwdDir& D = p.d[blockIdx.z];
  const int H = p.h, B = p.b, T = p.t, H4 = 4 * p.h, hq = p.h / 4;
  const int j0 = blockIdx.x * kSeqUnits, tid = threadIdx.x;
  const int group_rows = p.passes * kSeqRows, row_base = blockIdx.y * group_rows;
  const int slices = gridDim.x, all_rows = gridDim.y * group_rows;
  float* ws = seq_smem;
  float* ds = ws + (size_t)64 * H;
  float* red = ds + 64 * kSeqRows;
  float* dh_s = red + 128 * kSeqRedLd;
  float* dc_s = dh_s + (size_t)group_rows * kSeqUnits;
  for (int idx = tid; idx < 64 * hq; idx += kSeqThreads) {
    const int row = idx / hq, k4 = idx % hq, q = row / kSeqUnits, j = row % kSeqUnits;
    *reinterpret_cast<float4*>(ws + (size_t)row * H + 4 * k4) = __ldg(reinterpret_cast<const float4*>(D.w_hh + (size_t)(q * H + j0 + j) * H) + k4);
  }
  for (int e = tid; e < group_rows * kSeqUnits; e += kSeqThreads) {
    const int b = row_base + e / kSeqUnits;
    const size_t idx = (size_t)b * H + j0 + e % kSeqUnits;
    dh_s[e] = (b < B && D.ghn) ? D.ghn[idx] : 0.f;
    dc_s[e] = (b < B && D.gcn) ? D.gcn[idx] : 0.f;
  }
  if (tid == 0) failed = 0;
  __syncthreads();
  const int khalf = tid >> 7, rhalf = (tid >> 6) & 1, cq0 = tid & 63;
  const int cr = tid >> 4, cj = tid & 15;            // the cell's (row, unit) of this thread
  const size_t bh = (size_t)B * H, slice_floats = (size_t)all_rows * H;
  float* part_dir = p.part + (size_t)blockIdx.z * 2 * slices * slice_floats;
  unsigned* counter = D.counter + blockIdx.y;
  float pre[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int s = 0; s < T; s++) {
    const int tt = D.reverse ? s : T - 1 - s;
    const int pt = D.reverse ? tt + 1 : tt - 1;
    const bool first = D.reverse ? tt == T - 1 : tt == 0;
    const float* cp = first ? D.c0 : D.c + (size_t)pt * bh;
    const float* gates_t = D.gates + (size_t)tt * B * H4;
    float* dg_t = D.dG + (size_t)tt * B * H4;
    float* part_s = part_dir + (size_t)(s & 1) * slices * slice_floats;
    const bool last = s == T - 1 && D.dh0 == nullptr;
    for (int pass = 0; pass < p.passes; pass++) {
      if (row_base + pass * kSeqRows >= B) break;
      // Gate gradients of this CTA's units (BackwardRecurrent.cs:37-57 of the reference, the same operation order). With one
      // pass per CTA the step's saved values were fetched ahead (they do not depend on dh).
      const int b = row_base + pass * kSeqRows + cr;
      float dg[4] = {0.f, 0.f, 0.f, 0.f};
      if (b < B) {
        const int e = (pass * kSeqRows + cr) * kSeqUnits + cj, jg = j0 + cj;
        const size_t idx = (size_t)b * H + jg;
        float* d = dg_t + (size_t)b * H4;
        float gi, gf, gg, go, tc, gyv, cpv;
        if (p.passes == 1 && s > 0) {
          gi = pre[0]; gf = pre[1]; gg = pre[2]; go = pre[3]; tc = pre[4]; gyv = pre[5]; cpv = pre[6];
        } else {
          const float* g = gates_t + (size_t)b * H4;
          gi = g[jg]; gf = g[H + jg]; gg = g[2 * H + jg]; go = g[3 * H + jg];
          tc = D.tanh_c[(size_t)tt * bh + idx];
          gyv = D.gy[(size_t)tt * bh + idx];
          cpv = cp ? cp[idx] : 0.f;
        }
        const float dH = gyv + dh_s[e];
        const float dO = dH * tc;
        const float dC = dc_s[e] + ((dH * go) * (1.f - (tc * tc)));
        const float dI = dC * gg, dF = dC * cpv, dGg = dC * gi;
        dc_s[e] = dC * gf;
        dg[0] = (dI * gi) * (1.f - gi);
        dg[1] = (dF * gf) * (1.f - gf);
        dg[2] = dGg * (1.f - (gg * gg));
        dg[3] = (dO * go) * (1.f - go);
#pragma unroll
        for (int q = 0; q < 4; q++) d[q * H + jg] = dg[q];
      }
      if (last) continue;
#pragma unroll
      for (int q = 0; q < 4; q++) ds[(q * kSeqUnits + cj) * kSeqRows + cr] = dg[q];
      __syncthreads();
      // this slice's share of dh, all units: rows of the pass x H
      for (int q0 = 0; q0 < hq; q0 += 64) {
        const int cq = q0 + cq0;
        float acc[8][4];
#pragma unroll
        for (int r = 0; r < 8; r++)
#pragma unroll
          for (int j = 0; j < 4; j++) acc[r][j] = 0.f;
        if (cq < hq) {
#pragma unroll 4
          for (int k = khalf * 32; k < khalf * 32 + 32; k++) {
            const float4 w = *reinterpret_cast<const float4*>(ws + (size_t)k * H + 4 * cq);
            const float4 d0 = *reinterpret_cast<const float4*>(ds + k * kSeqRows + rhalf * 8);
            const float4 d1 = *reinterpret_cast<const float4*>(ds + k * kSeqRows + rhalf * 8 + 4);
            const float dv[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
            for (int r = 0; r < 8; r++) {
              acc[r][0] = fmaf(dv[r], w.x, acc[r][0]);
              acc[r][1] = fmaf(dv[r], w.y, acc[r][1]);
              acc[r][2] = fmaf(dv[r], w.z, acc[r][2]);
              acc[r][3] = fmaf(dv[r], w.w, acc[r][3]);
            }
          }
        }
        float* mine = red + (size_t)(tid & 127) * kSeqRedLd;
        if (khalf == 1) {
#pragma unroll
          for (int r = 0; r < 8; r++) *reinterpret_cast<float4*>(mine + 4 * r) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        }
        __syncthreads();
        if (khalf == 0 && cq < hq) {
          float* out = part_s + (size_t)blockIdx.x * slice_floats + (size_t)(row_base + pass * kSeqRows + rhalf * 8) * H + 4 * cq;
#pragma unroll
          for (int r = 0; r < 8; r++) {
            const float4 o = *reinterpret_cast<const float4*>(mine + 4 * r);
            *reinterpret_cast<float4*>(out + (size_t)r * H) = make_float4(acc[r][0] + o.x, acc[r][1] + o.y, acc[r][2] + o.z, acc[r][3] + o.w);
          }
        }
        __syncthreads();   // red and ds are used again
      }
    }
    if (last) break;
    if (p.passes == 1 && s + 1 < T) {
      // the next step's saved values: on their way during the barrier
      const int b = row_base + cr;
      if (b < B) {
        const int tn = D.reverse ? s + 1 : T - 2 - s;
        const int pn = D.reverse ? tn + 1 : tn - 1;
        const bool first_n = D.reverse ? tn == T - 1 : tn == 0;
        const size_t idx = (size_t)b * H + j0 + cj;
        const float* g = D.gates + ((size_t)tn * B + b) * H4;
        pre[0] = g[j0 + cj]; pre[1] = g[H + j0 + cj]; pre[2] = g[2 * H + j0 + cj]; pre[3] = g[3 * H + j0 + cj];
        pre[4] = D.tanh_c[(size_t)tn * bh + idx];
        pre[5] = D.gy[(size_t)tn * bh + idx];
        const float* cpn = first_n ? D.c0 : D.c + (size_t)pn * bh;
        pre[6] = cpn ? cpn[idx] : 0.f;
      }
    }
    if (!seq_barrier(counter, (unsigned)(s + 1) * gridDim.x, p.status, &failed, 9200 + (int)blockIdx.z)) return;
    for (int pass = 0; pass < p.passes; pass++) {
      if (row_base + pass * kSeqRows >= B) break;
      // written by other CTAs of this launch: past L1
      const float* src = part_s + (size_t)(row_base + pass * kSeqRows + cr) * H + j0 + cj;
      float t = 0.f;
#pragma unroll 8
      for (int k = 0; k < slices; k++) t += __ldcg(src + (size_t)k * slice_floats);
      dh_s[(pass * kSeqRows + cr) * kSeqUnits + cj] = t;     // read by this thread alone
    }
  }
  __syncthreads();
  for (int e = tid; e < group_rows * kSeqUnits; e += kSeqThreads) {
    const int b = row_base + e / kSeqUnits;
    if (b >= B) continue;
    const size_t idx = (size_t)b * H + j0 + e % kSeqUnits;
    if (D.dh0) D.dh0[idx] = dh_s[e];
    if (D.dc0) D.dc0[idx] = dc_s[e];
  }
}

static_assert(kSeqThreads == kSeqRows * kSeqUnits, "the cell phases map one thread to one (row, unit)");

static size_t seq_fwd_smem(int h) { return sizeof(float) * ((size_t)(64 + kSeqRows) * (h + kSeqPad)); }
static size_t seq_bwd_smem(int h, int passes) {
  return sizeof(float) * ((size_t)64 * h + 64 * kSeqRows + 128 * kSeqRedLd + 2 * (size_t)passes * kSeqRows * kSeqUnits);
}

// The launch shape: row groups of `passes` x 16 rows, as few passes as lets all CTAs of `dirs` directions be resident at
// once. Returns false when the shape does not fit the kernels.
static bool seq_plan(om_ctx* ctx, int dirs, int b, int h, bool backward, int* passes_out, int* groups_out) {
  if (h < 16 || h % 16 != 0 || b < 1) return false;
  const void* fn = backward ? (const void*)lstm_seq_bwd_kernel : (const void*)lstm_seq_fwd_kernel;
  const int tiles = (int)ceil_div(b, kSeqRows);
  for (int passes = 1;; passes *= 2) {
    const int groups = (int)ceil_div(tiles, passes);
    if (groups <= kSeqMaxGroups) {
      const size_t smem = backward ? seq_bwd_smem(h, passes) : seq_fwd_smem(h);
      if (smem > 200 * 1024) return false;
      if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      int per_sm = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kSeqThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      if ((long long)per_sm * ctx->sm_count >= (long long)dirs * groups * (h / kSeqUnits)) {
        *passes_out = passes;
        *groups_out = groups;
        return true;
      }
    }
    if (passes >= tiles) return false;
  }
}

bool lstm_seq_supported(om_ctx* ctx, int dirs, int t, int b, int h, bool backward) {
  if (!(ctx->flags & OM_SEQ_KERNELS) || t < 2) return false;
  int passes = 0, groups = 0;
  return seq_plan(ctx, dirs, b, h, backward, &passes, &groups);
}

int32_t lstm_seq_fwd(om_ctx* ctx, int dirs, int t, int b, int h, const LstmSeqFwdDir* d) {
  LstmSeqFwdParams p;
  if (!seq_plan(ctx, dirs, b, h, false, &p.passes, &p.groups)) return fail(ctx, OM_ERR_UNSUPPORTED, "lstm_seq_fwd: B %d H %d", b, h);
  unsigned* counters = nullptr;
  OM_TRY(pool_alloc(ctx, 2 * kSeqMaxGroups * sizeof(unsigned), true, (void**)&counters));
  for (int k = 0; k < 2; k++) {
    p.d[k] = d[k < dirs ? k : 0];
    p.d[k].counter = counters + k * kSeqMaxGroups;
  }
  p.t = t;
  p.b = b;
  p.h = h;
  p.status = ctx->status_dev;
  void* args[] = {&p};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)lstm_seq_fwd_kernel, dim3((unsigned)(h / kSeqUnits), (unsigned)p.groups, (unsigned)dirs),
                                              dim3(kSeqThreads), args, seq_fwd_smem(h), ctx->stream);
  pool_free(ctx, counters);
  if (e != cudaSuccess) return check_cuda(ctx, e, "lstm_seq_fwd");
  return OM_OK;
}

int32_t lstm_seq_bwd(om_ctx* ctx, int dirs, int t, int b, int h, const LstmSeqBwdDir* d) {
  LstmSeqBwdParams p;
  if (!seq_plan(ctx, dirs, b, h, true, &p.passes, &p.groups)) return fail(ctx, OM_ERR_UNSUPPORTED, "lstm_seq_bwd: B %d H %d", b, h);
  unsigned* counters = nullptr;
  OM_TRY(pool_alloc(ctx, 2 * kSeqMaxGroups * sizeof(unsigned), true, (void**)&counters));
  // the slices' shares of dh: two steps x (H / 16) slices x rows x H a direction (4 MB at 64 rows, H 256)
  const int32_t st = pool_alloc(ctx, sizeof(float) * (size_t)dirs * 2 * (h / kSeqUnits) * ((size_t)p.groups * p.passes * kSeqRows) * h, false, (void**)&p.part);
  if (st != OM_OK) {
    pool_free(ctx, counters);
    return st;
  }
  for (int k = 0; k < 2; k++) {
    p.d[k] = d[k < dirs ? k : 0];
    p.d[k].counter = counters + k * kSeqMaxGroups;
  }
  p.t = t;
  p.b = b;
  p.h = h;
  p.status = ctx->status_dev;
  void* args[] = {&p};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)lstm_seq_bwd_kernel, dim3((unsigned)(h / kSeqUnits), (unsigned)p.groups, (unsigned)dirs),
                                              dim3(kSeqThreads), args, seq_bwd_smem(h, p.passes), ctx->stream);
  pool_free(ctx, counters);
  pool_free(ctx, p.part);
  if (e != cudaSuccess) return check_cuda(ctx, e, "lstm_seq_bwd");
  return OM_OK;
}

}  // namespace om
