// Bandwidth-bound kernels: RMSNorm (+residual gradient), RoPE, SwiGLU, embedding gather,
// cross-entropy over a logits chunk, column sums (bias gradient), gradient accumulation,
// sum of squares and the fused AdamW update. All use 128-bit accesses, fp32 math and bf16 storage.
//
// These replace what the reference gets from Liger's Triton kernels (rms_norm, rope, swiglu,
// cross_entropy) and ATen foreach ops (clip, AdamW).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "entries.h"
#include "ptx.cuh"

namespace mtb {

constexpr int EW_THREADS = 256;

struct bf16x8 {
  uint4 u;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void store(__nv_bfloat16* p) const { *reinterpret_cast<uint4*>(p) = u; }
  __device__ __forceinline__ void to_float(float (&f)[8]) const {
    float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
  }
  __device__ __forceinline__ void from_float(const float (&f)[8]) {
    u.x = pack_bf16(f[0], f[1]); u.y = pack_bf16(f[2], f[3]); u.z = pack_bf16(f[4], f[5]); u.w = pack_bf16(f[6], f[7]);
  }
};

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.f;
  if (w == 0) t = warp_sum(t);
  if (threadIdx.x == 0) red[0] = t;
  __syncthreads();
  return red[0];
}
__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : -INFINITY;
  if (w == 0) t = warp_max(t);
  if (threadIdx.x == 0) red[0] = t;
  __syncthreads();
  return red[0];
}

// ------------------------------------------------------------------------------ RMSNorm / LayerNorm fwd
// RMSNorm    y = bf16(x * rstd) * w ; rstd saved
// LayerNorm  y = ((x - mean) * rstd) * w + b ; statistics in two passes over the row in registers (the mean first, then the
//            centred sum of squares), mean and rstd saved
// A group of LANES threads (one to eight warps) holds a row in registers, VPT 8-wide vectors per thread, and a 256-thread block
// works on 256 / LANES consecutive rows at a time. Bound by reading x and writing y.
// BULK: blocks are persistent and rows arrive in shared memory by bulk copies NORM_STAGES row sets ahead: the bytes in flight cost no
// registers and do not stop for a row's barriers and stores, which is what held the register form back (RMSNorm, 16384 x 4096:
// 53 -> 47 us; 6000 x 3072: 16 -> 14 us; LayerNorm, 16384 x 3072: 51 -> 43 us). Otherwise (RMSNorm) a block is one row set, loaded straight
// into registers: with a set or two per block nothing runs ahead, and the stages only cost residency (6000 x 1024: 8.3 us by bulk
// copies, 6.9 straight; 500 x 12288: 10.4 and 8.3).
constexpr int NORM_STAGES = 3;

__device__ __forceinline__ float group_sum(float v, float (&red)[EW_THREADS / 32], int lanes, int sub) {
  v = warp_sum(v);
  if (lanes > 32) {   // uniform over the block
    const int wpr = lanes >> 5;
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.f;
    for (int k = 0; k < wpr; ++k) v += red[sub * wpr + k];
  }
  return v;
}

template <bool LN, int VPT, bool BULK>
__global__ void __launch_bounds__(EW_THREADS) norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                             const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y,
                                                             float* __restrict__ mean_out, float* __restrict__ rstd_out, float eps, int T,
                                                             int H, int lanes, int* status) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(128) uint8_t norm_smem[];
  __shared__ uint64_t full[NORM_STAGES];
  __shared__ float red[2][2][EW_THREADS / 32];   // [parity of the row set][mean, square]
  __shared__ int abort_word;
  constexpr bool HOLD = BULK;   // weight and bias: once per persistent block, or behind the row's own loads
  volatile int* abort_flag = &abort_word;
  const int rows_per_block = EW_THREADS / lanes;
  const int sub = threadIdx.x / lanes, l = threadIdx.x % lanes;
  const uint32_t set_bytes = static_cast<uint32_t>(rows_per_block) * H * 2;
  const long long step = static_cast<long long>(gridDim.x) * rows_per_block;
  const long long first0 = static_cast<long long>(blockIdx.x) * rows_per_block;
  auto request = [&](long long first, int s) {   // one thread
    if (first >= T) return;
    const uint32_t bytes = static_cast<uint32_t>(T - first < rows_per_block ? T - first : rows_per_block) * H * 2;
    mbar_arrive_expect_tx(&full[s], bytes);
    bulk_load(norm_smem + s * set_bytes, x + first * H, bytes, &full[s]);
  };
  if (BULK && threadIdx.x == 0) {
    for (int s = 0; s < NORM_STAGES; ++s) mbar_init(&full[s], 1);
    abort_word = 0;
    fence_mbar_init();
    for (int s = 0; s < NORM_STAGES; ++s) request(first0 + s * step, s);
  }
  bf16x8 wv[HOLD ? VPT : 1], bv[LN && HOLD ? VPT : 1];
  if constexpr (HOLD) {
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int c = (l + k * lanes) * 8;
      wv[k].u = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (LN) bv[k].u = wv[k].u;
      if (c < H) { wv[k].load(w + c); if constexpr (LN) bv[k].load(b + c); }
    }
  }
  if (BULK) __syncthreads();
  int it = 0;
  for (long long first = first0; first < T; first += step, ++it) {
    const int s = it % NORM_STAGES, par = it & 1;
    const long long row = first + sub;
    const bool row_ok = row < T;
    if (BULK && !mbar_wait(&full[s], (it / NORM_STAGES) & 1, abort_flag)) { atomicExch(status, 70); break; }
    const __nv_bfloat16* src = BULK ? reinterpret_cast<const __nv_bfloat16*>(norm_smem + s * set_bytes) + sub * H : x + row * H;
    float f[VPT][8];
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int c = (l + k * lanes) * 8;
      bf16x8 v; v.u = make_uint4(0u, 0u, 0u, 0u);
      if (row_ok && c < H) v.load(src + c);
      v.to_float(f[k]);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc += LN ? f[k][i] : f[k][i] * f[k][i];
    }
    float mean = 0.f;
    if (LN) {
      mean = group_sum(acc, red[par][0], lanes, sub) / H;
      acc = 0.f;
#pragma unroll
      for (int k = 0; k < VPT; ++k) {
        if ((l + k * lanes) * 8 < H) {
#pragma unroll
          for (int i = 0; i < 8; ++i) { f[k][i] -= mean; acc += f[k][i] * f[k][i]; }
        }
      }
    }
    const float ss = group_sum(acc, red[par][1], lanes, sub);
    if (BULK) {
      if (lanes <= 32) __syncthreads();
      // every thread has its part of the rows in registers: the stage may be refilled
      if (threadIdx.x == 0) request(first + NORM_STAGES * step, s);
    }
    if (!row_ok) continue;
    const float rstd = rsqrtf(ss / H + eps);
    if (l == 0) { rstd_out[row] = rstd; if (LN) mean_out[row] = mean; }
    __nv_bfloat16* yr = y + row * H;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int c = (l + k * lanes) * 8;
      if (c < H) {
        float g[8], h[8];
        if constexpr (!HOLD) { wv[0].load(w + c); bv[0].load(b + c); }
        wv[HOLD ? k : 0].to_float(g);
        if constexpr (LN) bv[HOLD ? k : 0].to_float(h);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[k][i] = LN ? f[k][i] * rstd * g[i] + h[i] : __bfloat162float(__float2bfloat16(f[k][i] * rstd)) * g[i];
        bf16x8 o; o.from_float(f[k]); o.store(yr + c);
      }
    }
  }
}

// LayerNorm forward with one 256-thread block per row, VPT 8-wide vectors per thread, for short batches and for widths at which the
// form above leaves a quarter of its threads idle with registers for two blocks per SM (norm_fwd): 500 x 4096 5.1 us here and 6.3 there,
// 2000 x 2048 6.8 and 8.2, 16384 x 5120 69 and 78.
template <int VPT>
__global__ void __launch_bounds__(EW_THREADS) layernorm_row_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                  const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y,
                                                                  float* __restrict__ mean_out, float* __restrict__ rstd_out, float eps, int H) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * H;
  float f[VPT][8];
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int c = (threadIdx.x + k * EW_THREADS) * 8;
    if (c < H) {
      bf16x8 v; v.load(xr + c); v.to_float(f[k]);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += f[k][i];
    }
  }
  const float mean = block_sum(s, red) / H;
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int c = (threadIdx.x + k * EW_THREADS) * 8;
    if (c < H) {
#pragma unroll
      for (int i = 0; i < 8; ++i) { f[k][i] -= mean; ss += f[k][i] * f[k][i]; }
    }
  }
  const float rstd = rsqrtf(block_sum(ss, red) / H + eps);
  if (threadIdx.x == 0) { mean_out[row] = mean; rstd_out[row] = rstd; }
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int c = (threadIdx.x + k * EW_THREADS) * 8;
    if (c < H) {
      bf16x8 wv, bv; wv.load(w + c); bv.load(b + c);
      float fw[8], fb[8], o[8]; wv.to_float(fw); bv.to_float(fb);
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = f[k][i] * rstd * fw[i] + fb[i];
      bf16x8 ov; ov.from_float(o); ov.store(y + row * H + c);
    }
  }
}

// ------------------------------------------------------------------------------ RMSNorm / LayerNorm bwd
// RMSNorm    dx = rstd * (g - xhat * mean(g * xhat)) (+ add_to), g = dy * w, xhat = x * rstd;
//            dw partial per block in fp32: dwp[block, H] += dy * bf16(xhat)
// LayerNorm  dx = rstd * (g - mean(g) - xhat * mean(g * xhat)) (+ add_to), xhat = (x - mean) * rstd;
//            partials dwp[block, 0, :] += dy * xhat, dwp[block, 1, :] += dy (the bias gradient)
// Partials are summed over blocks by reduce_rows_kernel: no atomics. Bound by reading dy, x (and add_to) and writing dx.
// Persistent blocks loop over rows, one row per block, VPT 8-wide vectors per thread. Rows arrive in shared memory by bulk
// copies, `stages` ahead, and the row's statistics one row ahead; the reduction takes one barrier (every thread adds the
// warps' sums itself, two buffers). Before, a row was load, three barriers, store, and little was in flight meanwhile
// (RMSNorm with add_to, 16384 x 4096: 149 -> 98 us, 5987 x 1536: 58 -> 31 us; LayerNorm, 16384 x 4096: 222 -> 145 us, 7001 x 3072:
// 106 -> 52 us; all with the sum over blocks).
template <bool LN, int VPT>
__global__ void __launch_bounds__(512) norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                      const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                                                      const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ add_to,
                                                      __nv_bfloat16* __restrict__ dx, float* __restrict__ dwp, int T, int H, int stages,
                                                      int* status) {
  pdl_trigger();
  pdl_wait();
  constexpr bool KEEP = VPT <= 2;   // wider rows form xhat and g again after the reduction instead of holding them
  extern __shared__ __align__(128) uint8_t norm_smem[];
  __shared__ uint64_t full[8];
  __shared__ float2 red[2][16];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int nt = blockDim.x, wid = threadIdx.x >> 5;
  const uint32_t row_bytes = static_cast<uint32_t>(H) * 2;
  const uint32_t stage_bytes = row_bytes * (add_to != nullptr ? 3 : 2);
  auto request = [&](long long row, int s) {   // one thread
    if (row >= T) return;
    mbar_arrive_expect_tx(&full[s], stage_bytes);
    uint8_t* d = norm_smem + s * stage_bytes;
    bulk_load(d, dy + row * H, row_bytes, &full[s]);
    bulk_load(d + row_bytes, x + row * H, row_bytes, &full[s]);
    if (add_to != nullptr) bulk_load(d + 2 * row_bytes, add_to + row * H, row_bytes, &full[s]);
  };
  if (threadIdx.x < 32) red[threadIdx.x >> 4][threadIdx.x & 15] = make_float2(0.f, 0.f);   // warps that do not exist add zeros
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&full[s], 1);
    abort_word = 0;
    fence_mbar_init();
    for (int s = 0; s < stages; ++s) request(blockIdx.x + static_cast<long long>(s) * gridDim.x, s);
  }
  float2 dwacc[VPT][4], dbacc[LN ? VPT : 1][4];
  bf16x8 wv[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * nt) * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) { dwacc[v][i] = make_float2(0.f, 0.f); if (LN) dbacc[v][i] = make_float2(0.f, 0.f); }
    wv[v].u = make_uint4(0u, 0u, 0u, 0u);
    if (c < H) wv[v].load(w + c);
  }
  float mean = 0.f, rstd = 0.f;
  if (blockIdx.x < T) { rstd = rstd_in[blockIdx.x]; if (LN) mean = mean_in[blockIdx.x]; }
  __syncthreads();
  int it = 0, s = 0;
  uint32_t ph = 0;
  for (long long row = blockIdx.x; row < T; row += gridDim.x, ++it) {
    const long long next = row + gridDim.x;
    float nmean = 0.f, nrstd = 0.f;
    if (next < T) { nrstd = rstd_in[next]; if (LN) nmean = mean_in[next]; }
    if (!mbar_wait(&full[s], ph, abort_flag)) { atomicExch(status, 71); break; }
    const __nv_bfloat16* sdy = reinterpret_cast<const __nv_bfloat16*>(norm_smem + s * stage_bytes);
    const float2 rs2 = make_float2(rstd, rstd), mm2 = make_float2(-mean, -mean);
    auto load2 = [&](const __nv_bfloat16* p, int c, float2 (&f)[4]) {
      uint4 u = make_uint4(0u, 0u, 0u, 0u);
      if (c < H) u = *reinterpret_cast<const uint4*>(p + c);
      f[0] = unpack_bf16(u.x); f[1] = unpack_bf16(u.y); f[2] = unpack_bf16(u.z); f[3] = unpack_bf16(u.w);
    };
    auto w2 = [&](int v, int i) { return unpack_bf16(i == 0 ? wv[v].u.x : i == 1 ? wv[v].u.y : i == 2 ? wv[v].u.z : wv[v].u.w); };
    auto xhat = [&](float2 b) { return LN ? fmul2(fadd2(b, mm2), rs2) : fmul2(b, rs2); };
    float2 g[KEEP ? VPT : 1][4], xh[KEEP ? VPT : 1][4];
    float2 d1 = make_float2(0.f, 0.f), d2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (threadIdx.x + v * nt) * 8;
      float2 a[4], b[4];
      load2(sdy, c, a); load2(sdy + H, c, b);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 xv = xhat(b[i]), gv = fmul2(a[i], w2(v, i));
        if (LN) d1 = fadd2(d1, gv);
        d2 = ffma2(gv, xv, d2);
        dwacc[v][i] = ffma2(a[i], LN ? xv : unpack_bf16(pack_bf16(xv.x, xv.y)), dwacc[v][i]);
        if (LN) dbacc[v][i] = fadd2(dbacc[v][i], a[i]);
        if (KEEP) { g[v][i] = gv; xh[v][i] = xv; }
      }
    }
    float2 (&rd)[16] = red[it & 1];
    const float s1 = LN ? warp_sum(d1.x + d1.y) : 0.f, s2 = warp_sum(d2.x + d2.y);
    if ((threadIdx.x & 31) == 0) rd[wid] = make_float2(s1, s2);
    __syncthreads();
    // all threads are past the previous row's last reads: its stage may be refilled
    if (threadIdx.x == 0 && it > 0) request(row + static_cast<long long>(stages - 1) * gridDim.x, s == 0 ? stages - 1 : s - 1);
    d1 = d2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 16; k += 2) {
      const float2 t = rd[k], u = rd[k + 1];
      if (LN) d1 = fadd2(d1, make_float2(t.x, u.x));
      d2 = fadd2(d2, make_float2(t.y, u.y));
    }
    const float m1 = LN ? (d1.x + d1.y) / H : 0.f, m2 = (d2.x + d2.y) / H;
    const float2 nm1 = make_float2(-m1, -m1), nm2 = make_float2(-m2, -m2);
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (threadIdx.x + v * nt) * 8;
      if (c < H) {
        float2 a[4], b[4], r[4], o[4];
        if (!KEEP) { load2(sdy, c, a); load2(sdy + H, c, b); }
        if (add_to != nullptr) load2(sdy + 2 * H, c, r);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float2 gv, xv;
          if constexpr (KEEP) { gv = g[v][i]; xv = xh[v][i]; } else { gv = fmul2(a[i], w2(v, i)); xv = xhat(b[i]); }
          if (LN) gv = fadd2(gv, nm1);
          o[i] = fmul2(ffma2(xv, nm2, gv), rs2);
          if (add_to != nullptr) o[i] = fadd2(o[i], r[i]);
        }
        *reinterpret_cast<uint4*>(dx + row * H + c) = make_uint4(pack_bf16(o[0].x, o[0].y), pack_bf16(o[1].x, o[1].y),
                                                                 pack_bf16(o[2].x, o[2].y), pack_bf16(o[3].x, o[3].y));
      }
    }
    mean = nmean; rstd = nrstd;
    if (++s == stages) { s = 0; ph ^= 1; }
  }
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * nt) * 8;
    if (c < H) {
      float* dst = dwp + static_cast<long long>(blockIdx.x) * (LN ? 2 : 1) * H + c;
      *reinterpret_cast<float4*>(dst) = make_float4(dwacc[v][0].x, dwacc[v][0].y, dwacc[v][1].x, dwacc[v][1].y);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(dwacc[v][2].x, dwacc[v][2].y, dwacc[v][3].x, dwacc[v][3].y);
      if (LN) {
        *reinterpret_cast<float4*>(dst + H) = make_float4(dbacc[v][0].x, dbacc[v][0].y, dbacc[v][1].x, dbacc[v][1].y);
        *reinterpret_cast<float4*>(dst + H + 4) = make_float4(dbacc[v][2].x, dbacc[v][2].y, dbacc[v][3].x, dbacc[v][3].y);
      }
    }
  }
}

// Sums of R partial rows of C columns; columns [0, D) go to out_a, the rest to out_b (a row may hold the partials of two
// vectors; D = C when it holds one). 32 columns per block, 16 warps share the rows: a chain of R / 16 loads instead of R
// (296 rows of 4096: 15 -> 5 us). Few rows are one thread's work per column (reduce_few_rows_kernel): with a batch of eight tokens the
// barrier and the many blocks took longer than the sum (colsum of 8 x 896: 6.3 us, 4.7 like this; below 512 columns there are few blocks).
__global__ void __launch_bounds__(512) reduce_rows_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ out_a, __nv_bfloat16* __restrict__ out_b,
                                                         int R, int C, int D) {
  pdl_trigger();
  pdl_wait();
  __shared__ float sm[16][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < C) {
#pragma unroll 8
    for (int r = wid; r < R; r += 16) s += part[static_cast<long long>(r) * C + c];
  }
  sm[wid][lane] = s;
  __syncthreads();
  if (wid == 0 && c < C) {
#pragma unroll
    for (int k = 1; k < 16; ++k) s += sm[k][lane];
    if (c < D) out_a[c] = __float2bfloat16(s); else out_b[c - D] = __float2bfloat16(s);
  }
}
__global__ void __launch_bounds__(256) reduce_few_rows_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ out_a, __nv_bfloat16* __restrict__ out_b,
                                                             int R, int C, int D) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= C) return;
  float s = 0.f;
  for (int r = 0; r < R; ++r) s += part[static_cast<long long>(r) * C + c];
  if (c < D) out_a[c] = __float2bfloat16(s); else out_b[c - D] = __float2bfloat16(s);
}

// ------------------------------------------------------------------------------ RoPE
// In place on the first n_heads (q then k) heads of each row of qkv[T, ld]. Rotate-half
// convention: (x1, x2) -> (x1 cos - x2 sin, x2 cos + x1 sin), angle = fp32(pos) * inv_freq[i]
// (the fp32 product and fp32 sine / cosine that the Hugging Face rotary embedding computes).
// A thread owns 8 frequencies of one token for ROPE_HPT consecutive heads (grid.y = head groups):
// all of its loads are issued before the first store, so a thread keeps 2 * ROPE_HPT 16-byte loads in flight.
constexpr int ROPE_HPT = 4;
__global__ void __launch_bounds__(EW_THREADS) rope_kernel(__nv_bfloat16* __restrict__ qkv, const int* __restrict__ pos,
                                                         const float* __restrict__ inv_freq, int T, long long ld,
                                                         int n_heads, int D, float sign) {
  pdl_trigger();
  pdl_wait();
  const int half = D >> 1;
  const int vec_per_tok = half >> 3;  // 8 frequencies per thread
  const long long gid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (gid >= static_cast<long long>(T) * vec_per_tok) return;
  const int t = static_cast<int>(gid / vec_per_tok);
  const int i0 = static_cast<int>(gid % vec_per_tok) * 8;
  const int h0 = blockIdx.y * ROPE_HPT;
  __nv_bfloat16* row = qkv + static_cast<long long>(t) * ld;
  bf16x8 a[ROPE_HPT], b[ROPE_HPT];
#pragma unroll
  for (int j = 0; j < ROPE_HPT; ++j) {
    if (h0 + j < n_heads) { a[j].load(row + (h0 + j) * D + i0); b[j].load(row + (h0 + j) * D + i0 + half); }
  }
  const float p = static_cast<float>(pos[t]);
  float cs[8], sn[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    sincosf(p * inv_freq[i0 + i], &sn[i], &cs[i]);
    sn[i] *= sign;
  }
#pragma unroll
  for (int j = 0; j < ROPE_HPT; ++j) {
    if (h0 + j < n_heads) {
      float x1[8], x2[8], o1[8], o2[8]; a[j].to_float(x1); b[j].to_float(x2);
#pragma unroll
      for (int i = 0; i < 8; ++i) { o1[i] = x1[i] * cs[i] - x2[i] * sn[i]; o2[i] = x2[i] * cs[i] + x1[i] * sn[i]; }
      a[j].from_float(o1); b[j].from_float(o2);
      a[j].store(row + (h0 + j) * D + i0); b[j].store(row + (h0 + j) * D + i0 + half);
    }
  }
}

// ------------------------------------------------------------------------------ per-head RMSNorm (q_norm / k_norm)
// Qwen3 normalises every q and k head over head_dim before the rotary embedding, with one weight vector for all q
// heads and one for all k heads. In place on the first n_heads (q then k) heads of each row of qkv[T, ld]: a warp takes
// HEADS_PER_WARP heads of one token, a lane holds EPL = head_dim / 32 consecutive elements, the sum of squares is a shuffle
// reduction. y = bf16(x * rstd) * w, rstd[token * n_heads + head] saved.
// ROPE: the rotary embedding of the normalised heads in the same pass. Element i pairs with i + head_dim / 2, which the lane 16
// further holds; sine and cosine are shared by the warp's heads. `pre` (optional) receives the heads before the norm, which
// backward reads. Bound by reading and writing the heads once: with the copy, the norm and the rotation as passes of their
// own they were read three times and written three times (4099 tokens x 24 heads of 128: forward 54 -> 17 us, backward 36 -> 26 us).
// Forward: HPW heads of a token per warp; four, so that they share the angles and several loads are in flight, or one where that
// leaves fewer than two blocks per SM (33 tokens x 24 heads of 128, without the rotation, cold: 8.2 and 6.1 us; backward, whose blocks also
// add up partials, is the faster with four at any height).
constexpr int HEADS_PER_WARP = 4;
template <int EPL>
struct HeadVec {
  uint32_t raw[EPL / 2];
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    if constexpr (EPL == 8) { const uint4 v = *reinterpret_cast<const uint4*>(p); raw[0] = v.x; raw[1] = v.y; raw[2] = v.z; raw[3] = v.w; }
    else if constexpr (EPL == 4) { const uint2 v = *reinterpret_cast<const uint2*>(p); raw[0] = v.x; raw[1] = v.y; }
    else { raw[0] = *reinterpret_cast<const uint32_t*>(p); }
  }
  __device__ __forceinline__ void store(__nv_bfloat16* p) const {
    if constexpr (EPL == 8) *reinterpret_cast<uint4*>(p) = make_uint4(raw[0], raw[1], raw[2], raw[3]);
    else if constexpr (EPL == 4) *reinterpret_cast<uint2*>(p) = make_uint2(raw[0], raw[1]);
    else *reinterpret_cast<uint32_t*>(p) = raw[0];
  }
  __device__ __forceinline__ void to_float(float (&f)[EPL]) const {
#pragma unroll
    for (int i = 0; i < EPL / 2; ++i) { const float2 a = unpack_bf16(raw[i]); f[2 * i] = a.x; f[2 * i + 1] = a.y; }
  }
  __device__ __forceinline__ void from_float(const float (&f)[EPL]) {
#pragma unroll
    for (int i = 0; i < EPL / 2; ++i) raw[i] = pack_bf16(f[2 * i], f[2 * i + 1]);
  }
};

// Sines and cosines of a token for the EPL frequencies of this lane (lanes l and l + 16 share them: each evaluates half).
template <int EPL>
__device__ __forceinline__ void head_angles(float pos, const float* __restrict__ inv_freq, int lane, float (&cs)[EPL], float (&sn)[EPL]) {
  const bool hi = lane >= 16;
  float c0[EPL / 2], s0[EPL / 2];
#pragma unroll
  for (int j = 0; j < EPL / 2; ++j) sincosf(pos * inv_freq[(lane & 15) * EPL + (hi ? EPL / 2 : 0) + j], &s0[j], &c0[j]);
#pragma unroll
  for (int j = 0; j < EPL / 2; ++j) {
    const float co = __shfl_xor_sync(0xffffffffu, c0[j], 16), so = __shfl_xor_sync(0xffffffffu, s0[j], 16);
    cs[j] = hi ? co : c0[j]; sn[j] = hi ? so : s0[j];
    cs[EPL / 2 + j] = hi ? c0[j] : co; sn[EPL / 2 + j] = hi ? s0[j] : so;
  }
}
// Rotation of a head spread over the warp (sign -1: the inverse).
template <int EPL>
__device__ __forceinline__ void head_rotate(float (&f)[EPL], const float (&cs)[EPL], const float (&sn)[EPL], int lane, float sign) {
  const float sg = lane < 16 ? -sign : sign;   // x1 cos - x2 sin | x2 cos + x1 sin
#pragma unroll
  for (int i = 0; i < EPL; ++i) f[i] = f[i] * cs[i] + sg * __shfl_xor_sync(0xffffffffu, f[i], 16) * sn[i];
}

template <int EPL, bool ROPE, int HPW>
__global__ void __launch_bounds__(EW_THREADS) head_rmsnorm_fwd_kernel(__nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
                                                                     const __nv_bfloat16* __restrict__ wk, __nv_bfloat16* __restrict__ pre,
                                                                     float* __restrict__ rstd_out, const int* __restrict__ pos,
                                                                     const float* __restrict__ inv_freq, float eps, long long n_items, int groups,
                                                                     long long ld, int n_q, int n_heads) {
  pdl_trigger();
  pdl_wait();
  constexpr int D = EPL * 32;
  const long long r = static_cast<long long>(blockIdx.x) * (EW_THREADS / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= n_items) return;   // whole warps leave together
  const long long t = r / groups;
  const int h0 = static_cast<int>(r - t * groups) * HPW;
  __nv_bfloat16* p = qkv + t * ld + static_cast<long long>(h0) * D + lane * EPL;
  HeadVec<EPL> xv[HPW];
#pragma unroll
  for (int k = 0; k < HPW; ++k) if (h0 + k < n_heads) xv[k].load(p + k * D);
  float cs[EPL], sn[EPL];
  if (ROPE) head_angles<EPL>(static_cast<float>(pos[t]), inv_freq, lane, cs, sn);
#pragma unroll
  for (int k = 0; k < HPW; ++k) {
    const int h = h0 + k;
    if (h >= n_heads) break;
    if (pre != nullptr) xv[k].store(pre + t * (static_cast<long long>(n_heads) * D) + static_cast<long long>(h) * D + lane * EPL);
    HeadVec<EPL> wv;
    wv.load((h < n_q ? wq : wk) + lane * EPL);
    float f[EPL], g[EPL];
    xv[k].to_float(f); wv.to_float(g);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < EPL; ++i) ss += f[i] * f[i];
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / D + eps);
    if (lane == 0) rstd_out[t * n_heads + h] = rstd;
#pragma unroll
    for (int i = 0; i < EPL; ++i) f[i] = __bfloat162float(__float2bfloat16(f[i] * rstd)) * g[i];
    xv[k].from_float(f);
    if (ROPE) {   // of the normalised heads as bf16, as if they had been stored in between
      xv[k].to_float(f);
      head_rotate<EPL>(f, cs, sn, lane, 1.f);
      xv[k].from_float(f);
    }
    xv[k].store(p + k * D);
  }
}

// Backward, in place on dqkv (gradient of the normalised, and with ROPE rotated, heads in, gradient of the projection output
// out): dx = rstd * (g - xhat * mean(g * xhat)), g = dy * w, xhat = x * rstd with x the heads BEFORE the norm (pre[T, ld_pre],
// q then k heads). Weight gradients: dwp[block, 2, D] += dy * bf16(xhat) per block in fp32 (q heads in row 0, k heads in
// row 1), summed over blocks by reduce_rows_kernel: no atomics. Persistent warps loop over groups of heads of a token; a lane
// keeps the same columns throughout, so its partial sums stay in registers.
template <int EPL, bool ROPE>
__global__ void __launch_bounds__(EW_THREADS) head_rmsnorm_bwd_kernel(__nv_bfloat16* __restrict__ dqkv, const __nv_bfloat16* __restrict__ pre,
                                                                     const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ wq,
                                                                     const __nv_bfloat16* __restrict__ wk, float* __restrict__ dwp,
                                                                     const int* __restrict__ pos, const float* __restrict__ inv_freq,
                                                                     long long n_items, int groups, long long ld, long long ld_pre, int n_q,
                                                                     int n_heads) {
  pdl_trigger();
  pdl_wait();
  constexpr int D = EPL * 32;
  constexpr int WARPS = EW_THREADS / 32;
  __shared__ float sm[WARPS][2][D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float wqf[EPL], wkf[EPL], accq[EPL], acck[EPL];
  {
    HeadVec<EPL> a, b;
    a.load(wq + lane * EPL); b.load(wk + lane * EPL);
    a.to_float(wqf); b.to_float(wkf);
  }
#pragma unroll
  for (int i = 0; i < EPL; ++i) { accq[i] = 0.f; acck[i] = 0.f; }
  const long long stride = static_cast<long long>(gridDim.x) * WARPS;
  for (long long r = static_cast<long long>(blockIdx.x) * WARPS + warp; r < n_items; r += stride) {
    const long long t = r / groups;
    const int h0 = static_cast<int>(r - t * groups) * HEADS_PER_WARP;
    __nv_bfloat16* gp = dqkv + t * ld + static_cast<long long>(h0) * D + lane * EPL;
    const __nv_bfloat16* xp = pre + t * ld_pre + static_cast<long long>(h0) * D + lane * EPL;
    HeadVec<EPL> gv[HEADS_PER_WARP], xv[HEADS_PER_WARP];
    float rs[HEADS_PER_WARP];
#pragma unroll
    for (int k = 0; k < HEADS_PER_WARP; ++k) {
      if (h0 + k < n_heads) { gv[k].load(gp + k * D); xv[k].load(xp + k * D); rs[k] = rstd_in[t * n_heads + h0 + k]; }
    }
    float cs[EPL], sn[EPL];
    if (ROPE) head_angles<EPL>(static_cast<float>(pos[t]), inv_freq, lane, cs, sn);
#pragma unroll
    for (int k = 0; k < HEADS_PER_WARP; ++k) {
      if (h0 + k >= n_heads) break;
      const bool is_q = h0 + k < n_q;
      float dy[EPL], x[EPL], g[EPL], xh[EPL];
      gv[k].to_float(dy); xv[k].to_float(x);
      if (ROPE) {   // rounded to bf16, as if it had been stored in between
        head_rotate<EPL>(dy, cs, sn, lane, -1.f);
        gv[k].from_float(dy);
        gv[k].to_float(dy);
      }
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < EPL; ++i) {
        xh[i] = x[i] * rs[k];
        g[i] = dy[i] * (is_q ? wqf[i] : wkf[i]);
        dot += g[i] * xh[i];
        const float c = dy[i] * __bfloat162float(__float2bfloat16(xh[i]));
        if (is_q) accq[i] += c; else acck[i] += c;
      }
      dot = warp_sum(dot) / D;
#pragma unroll
      for (int i = 0; i < EPL; ++i) g[i] = rs[k] * (g[i] - xh[i] * dot);
      gv[k].from_float(g);
      gv[k].store(gp + k * D);
    }
  }
#pragma unroll
  for (int i = 0; i < EPL; ++i) { sm[warp][0][lane * EPL + i] = accq[i]; sm[warp][1][lane * EPL + i] = acck[i]; }
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * D; c += EW_THREADS) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) s += sm[w][c / D][c % D];
    dwp[static_cast<long long>(blockIdx.x) * 2 * D + c] = s;
  }
}

// ------------------------------------------------------------------------------ gated MLP activations
// act(gate) * up over gu = [gate | up]. ACT 0: SiLU (SwiGLU: Llama, Qwen, Mistral, Granite, Mixtral, Phi-3);
// ACT 1: tanh-approximated GELU (GeGLU: Gemma's gelu_pytorch_tanh).
// glu_act and gelu_gate are in ptx.cuh: 0.5 * (1 + tanh(u)) = sigmoid(2 u), which costs what SiLU costs (with tanhf the GELU kernels were bound
// by instructions: 7001 x 12288 forward 92 -> 69 us).
template <int ACT>
__global__ void __launch_bounds__(EW_THREADS) swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act,
                                                               long long T, int F) {
  pdl_trigger();
  pdl_wait();
  // grid = (tokens, column blocks): no 64-bit division per thread
  const long long t = blockIdx.x;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= F) return;
  bf16x8 g, u; g.load(gu + t * 2 * F + c); u.load(gu + t * 2 * F + F + c);
  float fg[8], fu[8], o[8]; g.to_float(fg); u.to_float(fu);
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = glu_act<ACT>(fg[i]) * fu[i];
  g.from_float(o); g.store(act + t * F + c);
}

// WITH_ACT: the forward output act(gate) * up is also produced, written over dact (each thread reads its
// dact vector before it stores there), for a backward that did not keep it: one pass over gate/up
// instead of a forward kernel plus this one.
template <bool WITH_ACT, int ACT>
__global__ void __launch_bounds__(EW_THREADS) swiglu_bwd_kernel(__nv_bfloat16* dact, const __nv_bfloat16* __restrict__ gu,
                                                               __nv_bfloat16* __restrict__ dgu, long long T, int F) {
  pdl_trigger();
  pdl_wait();
  // grid = (tokens, column blocks): no 64-bit division per thread
  const long long t = blockIdx.x;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= F) return;
  bf16x8 g, u, d; g.load(gu + t * 2 * F + c); u.load(gu + t * 2 * F + F + c); d.load(dact + t * F + c);
  float fg[8], fu[8], fd[8], og[8], ou[8]; g.to_float(fg); u.to_float(fu); d.to_float(fd);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if constexpr (ACT == 0) {
      const float sig = __fdividef(1.f, 1.f + exp_ftz(-fg[i]));
      og[i] = fd[i] * fu[i] * sig * (1.f + fg[i] * (1.f - sig));
      ou[i] = fd[i] * fg[i] * sig;
    } else {
      og[i] = fd[i] * fu[i] * glu_act_grad<ACT>(fg[i]);
      ou[i] = fd[i] * glu_act<ACT>(fg[i]);
    }
  }
  if (WITH_ACT) {
    float o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = glu_act<ACT>(fg[i]) * fu[i];   // same expression as the forward kernel
    d.from_float(o); d.store(dact + t * F + c);
  }
  g.from_float(og); u.from_float(ou);
  g.store(dgu + t * 2 * F + c); u.store(dgu + t * 2 * F + F + c);
}

// Plain (not gated) activation over n elements, forward and backward: Starcoder2's MLP is c_proj(gelu(c_fc(x))).
// WITH_ACT: the forward output is also produced, written over dy, for a backward that did not keep it.
template <int ACT>
__global__ void __launch_bounds__(EW_THREADS) act_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, long long n) {
  pdl_trigger();
  pdl_wait();
  const long long i0 = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
  if (i0 >= n) return;
  bf16x8 v; v.load(x + i0);
  float f[8]; v.to_float(f);
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = glu_act<ACT>(f[i]);
  v.from_float(f); v.store(y + i0);
}
template <bool WITH_ACT, int ACT>
__global__ void __launch_bounds__(EW_THREADS) act_bwd_kernel(__nv_bfloat16* dy, const __nv_bfloat16* __restrict__ x, __nv_bfloat16* dx, long long n) {
  pdl_trigger();
  pdl_wait();
  const long long i0 = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
  if (i0 >= n) return;
  bf16x8 v, d; v.load(x + i0); d.load(dy + i0);
  float f[8], g[8]; v.to_float(f); d.to_float(g);
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] *= glu_act_grad<ACT>(f[i]);
  d.from_float(g); d.store(dx + i0);
  if (WITH_ACT) {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = glu_act<ACT>(f[i]);   // same expression as the forward kernel
    v.from_float(f); v.store(dy + i0);
  }
}

// ------------------------------------------------------------------------------ embedding
// An id outside [0, V) (a tokenizer larger than the embedding table) is not dereferenced: the row is zero-filled
// and code 60 is recorded in the status word, which the host turns into an exception.
__global__ void __launch_bounds__(128) embedding_fwd_kernel(const __nv_bfloat16* __restrict__ w, const long long* __restrict__ ids,
                                                           __nv_bfloat16* __restrict__ out, int H, int V, int* status) {
  pdl_trigger();
  pdl_wait();
  const long long t = blockIdx.x;
  const long long id = ids[t];
  __nv_bfloat16* dst = out + t * H;
  if (id < 0 || id >= V) {
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 60);
    for (int c = threadIdx.x * 8; c < H; c += 128 * 8) *reinterpret_cast<uint4*>(dst + c) = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const __nv_bfloat16* src = w + id * H;
  for (int c = threadIdx.x * 8; c < H; c += 128 * 8) *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(src + c);
}

// dW[id, :] += sum over the tokens t with ids[t] == id of dx[t, :], deterministic: the token ids arrive
// sorted (stable, so equal ids keep their token order) with the permutation that sorted them. The block
// at the first position of each run of equal ids sums the run's rows in fp32, in that fixed order, adds
// what dW already holds (the LM-head gradient when the embeddings are tied) and rounds once. The other
// blocks of the run exit at once. No atomics, so the result does not depend on scheduling.
__global__ void __launch_bounds__(128) embedding_bwd_kernel(__nv_bfloat16* __restrict__ dw, const long long* __restrict__ sorted_ids,
                                                           const long long* __restrict__ order, const __nv_bfloat16* __restrict__ dx,
                                                           int T, int H, int V, int* status) {
  pdl_trigger();
  pdl_wait();
  const int j = blockIdx.x;
  const long long id = sorted_ids[j];
  if (j > 0 && sorted_ids[j - 1] == id) return;
  if (id < 0 || id >= V) {   // skipped and reported, never dereferenced
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 60);
    return;
  }
  __nv_bfloat16* dst = dw + id * H;
  for (int c = threadIdx.x * 8; c < H; c += 128 * 8) {
    float acc[8];
    {
      const uint4 v = *reinterpret_cast<const uint4*>(dst + c);
      const float2 a0 = unpack_bf16(v.x), a1 = unpack_bf16(v.y), a2 = unpack_bf16(v.z), a3 = unpack_bf16(v.w);
      acc[0] = a0.x; acc[1] = a0.y; acc[2] = a1.x; acc[3] = a1.y; acc[4] = a2.x; acc[5] = a2.y; acc[6] = a3.x; acc[7] = a3.y;
    }
    for (int k = j; k < T && sorted_ids[k] == id; ++k) {
      const uint4 v = *reinterpret_cast<const uint4*>(dx + order[k] * H + c);
      const float2 a0 = unpack_bf16(v.x), a1 = unpack_bf16(v.y), a2 = unpack_bf16(v.z), a3 = unpack_bf16(v.w);
      acc[0] += a0.x; acc[1] += a0.y; acc[2] += a1.x; acc[3] += a1.y; acc[4] += a2.x; acc[5] += a2.y; acc[6] += a3.x; acc[7] += a3.y;
    }
    *reinterpret_cast<uint4*>(dst + c) = make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
  }
}

// The same without the sort, for up to EMB_SCAN tokens: the block of a token looks through all the others. One that finds its id earlier ends,
// the first of an id lists the later ones in token order (each thread a stretch of them) and sums as above, bit for bit. The comparisons
// grow with the square of the tokens; sorting is five launches, which take the host longer still
// (640 tokens x 512 46 -> 6.5 us, 4096 x 256 50 -> 17, 6000 x 1536 107 -> 33, 8192 x 1024 110 -> 55).
constexpr int EMB_SCAN = 8192;
__global__ void __launch_bounds__(EW_THREADS) embedding_bwd_scan_kernel(__nv_bfloat16* __restrict__ dw, const long long* __restrict__ ids,
                                                                       const __nv_bfloat16* __restrict__ dx, int T, int H, int V, int* status) {
  pdl_trigger();
  pdl_wait();
  __shared__ unsigned short later[EMB_SCAN];
  __shared__ int wsum[EW_THREADS / 32];
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long id = ids[t];
  bool seen = false;
#pragma unroll 8
  for (int j = threadIdx.x; j < t; j += EW_THREADS) seen |= ids[j] == id;
  if (__syncthreads_or(seen)) return;
  if (id < 0 || id >= V) {   // skipped and reported, never dereferenced
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 60);
    return;
  }
  const int per = (T - t - 1 + EW_THREADS - 1) / EW_THREADS;
  const int j0 = t + 1 + threadIdx.x * per, j1 = min(T, j0 + per);
  int mine = 0;
#pragma unroll 4
  for (int j = j0; j < j1; ++j) mine += ids[j] == id;
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  int at = incl - mine, n = 0;
#pragma unroll
  for (int k = 0; k < EW_THREADS / 32; ++k) { if (k < warp) at += wsum[k]; n += wsum[k]; }
  if (mine > 0)
    for (int j = j0; j < j1; ++j) if (ids[j] == id) later[at++] = static_cast<unsigned short>(j);
  __syncthreads();
  __nv_bfloat16* dst = dw + id * H;
  for (int c = threadIdx.x * 8; c < H; c += EW_THREADS * 8) {
    float acc[8], f[8];
    bf16x8 v; v.load(dst + c); v.to_float(acc);
    for (int k = -1; k < n; ++k) {
      v.load(dx + static_cast<long long>(k < 0 ? t : later[k]) * H + c); v.to_float(f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += f[i];
    }
    v.from_float(acc); v.store(dst + c);
  }
}

// Zeros into n 16-byte pieces and m fp32, one launch that starts under its predecessor's tail. Zeros and rows together, two
// memsets before: 480 rows into 640 x 512 9.1 -> 3.1 us, 3069 into 4096 x 256 9.2 -> 5.5, 3720 into 6000 x 1536 14.4 -> 8.3, 12000 into 16384 x 4096 56 -> 51.
__global__ void __launch_bounds__(EW_THREADS) zero_rows_kernel(uint4* out, long long n, float* vout, int m) {
  pdl_trigger();
  pdl_wait();
  const long long first = static_cast<long long>(blockIdx.x) * EW_THREADS + threadIdx.x, step = static_cast<long long>(gridDim.x) * EW_THREADS;
  for (long long i = first; i < n; i += step) out[i] = make_uint4(0u, 0u, 0u, 0u);
  for (long long i = first; i < m; i += step) vout[i] = 0.f;
}

// out[rows[r]] = src[r] for rows of H columns, and the same for a vector of fp32.
__global__ void __launch_bounds__(128) scatter_rows_kernel(const long long* __restrict__ rows, const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ out,
                                                          const float* __restrict__ vsrc, float* __restrict__ vout, int H, int T, int* status) {
  pdl_trigger();
  pdl_wait();
  const long long r = blockIdx.x, t = rows[r];
  if (t < 0 || t >= T) {   // skipped and reported, never dereferenced
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 60);
    return;
  }
  if (threadIdx.x == 0) vout[t] = vsrc[r];
  for (int c = threadIdx.x * 8; c < H; c += 128 * 8)
    *reinterpret_cast<uint4*>(out + t * H + c) = *reinterpret_cast<const uint4*>(src + r * H + c);
}

// ------------------------------------------------------------------------------ cross-entropy
// One block per row of a logits chunk ([R, V] fp32 or bf16, leading dimension ld). Pass 1: online
// max / sum-exp; or, when the GEMM that made the logits left the statistics of every 256 columns (`stats`,
// [R, ceil(V / 256)]), only their combination. Pass 2: dlogits = (softmax - onehot) * scale in bf16. Rows whose target is
// ignore_index get zero loss and zero gradient. With bf16 logits the gradient may be written over
// the logits (dlogits == logits): a thread reads a vector of the row before it overwrites the same
// vector, and pass 2 starts after the block-wide reductions that end pass 1. Bound by the row's traffic: a row of a large
// vocabulary (300 KB) does not stay on the SM between the passes, so pass 1 costs a third read (3720 x 151936: 578 -> 375 us with statistics).
template <typename LogitT>
__device__ __forceinline__ void load8(const LogitT* p, float (&f)[8]) {
  if constexpr (sizeof(LogitT) == 2) { bf16x8 v; v.load(reinterpret_cast<const __nv_bfloat16*>(p)); v.to_float(f); }
  else {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
}

template <typename LogitT, bool STATS>
__global__ void __launch_bounds__(1024) ce_fwd_bwd_kernel(const LogitT* logits, long long ld, const float2* __restrict__ stats,
                                                         const long long* __restrict__ targets, float* __restrict__ loss,
                                                         __nv_bfloat16* dlogits, long long ldd, int V, float grad_scale,
                                                         long long ignore_index) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const LogitT* lr = logits + row * ld;
  __nv_bfloat16* dr = dlogits + row * ldd;
  const long long tgt = targets[row];
  if (tgt == ignore_index) {
    for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) *reinterpret_cast<uint4*>(dr + c) = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) loss[row] = 0.f;
    return;
  }
  float m = -INFINITY, s = 0.f;
  if constexpr (STATS) {
    const int tiles = (V + 255) / 256;
    for (int c = threadIdx.x; c < tiles; c += blockDim.x) {
      const float2 t = stats[row * tiles + c];
      if (t.x > m) { s *= exp_ftz(m - t.x); m = t.x; }
      s += t.y * exp_ftz(t.x - (m == -INFINITY ? 0.f : m));
    }
  }
  else for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
    float v[8];
    load8(lr + c, v);
    float mx = v[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) mx = fmaxf(mx, v[i]);
    if (mx > m) { s *= exp_ftz(m - mx); m = mx; }
    const float base = m == -INFINITY ? 0.f : m;   // nothing but masked columns so far
#pragma unroll
    for (int i = 0; i < 8; ++i) s += exp_ftz(v[i] - base);
  }
  const float gm = block_max(m, red);
  s *= exp_ftz(m - gm);
  const float gs = block_sum(s, red);
  const float lse = gm + logf(gs);
  if (threadIdx.x == 0) {
    float t = NAN;   // of a target that is no column
    if (tgt >= 0 && tgt < V) {
      if constexpr (sizeof(LogitT) == 2) t = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(lr)[tgt]); else t = lr[tgt];
    }
    loss[row] = lse - t;
  }
  __syncthreads();   // the target logit has been read before any thread overwrites the row
  const float inv = grad_scale / gs;
  // two vectors per thread are loaded before the first is overwritten (the buffers may be the same, so the compiler cannot)
  const int step = blockDim.x * 8;
  for (int c0 = threadIdx.x * 8; c0 < V; c0 += 2 * step) {
    float o[2][8];
    load8(lr + c0, o[0]);
    const bool two = c0 + step < V;
    if (two) load8(lr + c0 + step, o[1]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k == 1 && !two) break;
      const int c = c0 + k * step;
#pragma unroll
      for (int i = 0; i < 8; ++i) o[k][i] = exp_ftz(o[k][i] - gm) * inv;
      if (tgt >= c && tgt < c + 8) {
#pragma unroll
        for (int i = 0; i < 8; ++i) if (tgt - c == i) o[k][i] -= grad_scale;   // no dynamic index: the array stays in registers
      }
      bf16x8 ov; ov.from_float(o[k]); ov.store(dr + c);
    }
  }
}

// The same for bf16 rows of up to 32768 columns without statistics: persistent blocks hold a row in registers, four 8-wide vectors per thread, and
// read the next one while they work on this one. The exponentials are formed once, against the thread's own maximum, and scaled by
// the difference to the row's when they are written. Bound by reading and writing the row, and beyond 16384 columns, where one block fills
// the SM, by the wait at each row's reduction: 4000 x 4096 41 -> 12 us, 3000 x 16384 62 -> 35, 3069 x 32000 106 -> 76 (0.79 of the measured copy
// rate); 64 x 32000 9.4 -> 6.0. The form above reads the row twice and forms two exponentials per element, with up to 1024 threads on
// rows that have work for a few.
constexpr int CE_ROW_VECS = 4;
__global__ void __launch_bounds__(1024, 1) ce_row_kernel(const __nv_bfloat16* logits, long long ld, const long long* __restrict__ targets, float* __restrict__ loss,
                                                        __nv_bfloat16* dlogits, long long ldd, int R, int V, float grad_scale, long long ignore_index) {
  pdl_wait();
  __shared__ float2 red[2][32];
  const int c0 = threadIdx.x * 8, step = blockDim.x * 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 64; i += blockDim.x) red[i >> 5][i & 31] = make_float2(-INFINITY, 0.f);   // of warps that are not there
  __syncthreads();
  uint4 next[CE_ROW_VECS];
  auto fetch = [&](int row) {
#pragma unroll
    for (int k = 0; k < CE_ROW_VECS; ++k) {
      next[k] = make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // -infinity
      if (c0 + k * step < V) next[k] = *reinterpret_cast<const uint4*>(logits + row * ld + c0 + k * step);
    }
  };
  fetch(blockIdx.x);
  int par = 0;
  for (int row = blockIdx.x; row < R; row += gridDim.x, par ^= 1) {
    const long long tgt = targets[row];
    const bool ignored = tgt == ignore_index;
    float t = NAN;   // of a target that is no column
    if (threadIdx.x == 0 && tgt >= 0 && tgt < V) t = __bfloat162float(logits[row * ld + tgt]);
    float e[CE_ROW_VECS][8];
    float m = -INFINITY, s = 0.f;
#pragma unroll
    for (int k = 0; k < CE_ROW_VECS; ++k) {
      bf16x8 v; v.u = next[k];
      v.to_float(e[k]);
      m = fmax3(m, fmax3(e[k][0], e[k][1], e[k][2]), fmax3(e[k][3], e[k][4], e[k][5]));
      m = fmax3(m, e[k][6], e[k][7]);
    }
    if (row + gridDim.x < R) fetch(row + gridDim.x);
    const float base = m == -INFINITY ? 0.f : m;
#pragma unroll
    for (int k = 0; k < CE_ROW_VECS; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        e[k][i] = exp_ftz(e[k][i] - base);
        s += e[k][i];
      }
    // maximum and sum of the row from the threads' own; a sum beside a maximum of -infinity is zero, or NaN where a logit is
    float gm = warp_max(m);
    float gs = warp_sum(m == -INFINITY ? s : s * exp_ftz(m - gm));
    if (lane == 0) red[par][warp] = make_float2(gm, gs);
    __syncthreads();   // and the target's logit has been read before any thread overwrites the row
    const float2 w = red[par][lane];
    gm = warp_max(w.x);
    gs = warp_sum(w.x == -INFINITY ? w.y : w.y * exp_ftz(w.x - gm));
    if (threadIdx.x == 0) loss[row] = ignored ? 0.f : gm + logf(gs) - t;
    const float scale = exp_ftz(m - gm) * (grad_scale / gs);   // zero for a thread that has nothing but -infinity, whatever the row's maximum
    __nv_bfloat16* dr = dlogits + row * ldd;
#pragma unroll
    for (int k = 0; k < CE_ROW_VECS; ++k) {
      const int c = c0 + k * step;
      if (c >= V) break;
      bf16x8 ov; ov.u = make_uint4(0, 0, 0, 0);
      if (!ignored) {
#pragma unroll
        for (int i = 0; i < 8; ++i) e[k][i] *= scale;
        if (tgt >= c && tgt < c + 8) {
#pragma unroll
          for (int i = 0; i < 8; ++i) if (tgt - c == i) e[k][i] -= grad_scale;
        }
        ov.from_float(e[k]);
      }
      ov.store(dr + c);
    }
  }
  pdl_trigger();
}

// ------------------------------------------------------------------------------ column sums (bias grad)
// part[split, c] = sum over this split's rows of x[r, c]; then reduce_rows_kernel. A lane adds V neighbouring columns of every
// eighth row: V = 8 (16-byte loads) where rows are 16-byte aligned, V = 2 for any even width, and for few columns and rows, where more
// blocks count. Bound by reading x (7001 rows of 3072 to 12288 columns, four calls: 96 -> 73 us). UNROLL rows are in flight per
// warp: eight where few blocks read many rows (64000 x 1024: 82 -> 64 us, V = 2 70), four otherwise (16384 x 6144: 48 us with eight, 38).
template <int V, int UNROLL>
__global__ void __launch_bounds__(256) colsum_partial_kernel(const __nv_bfloat16* __restrict__ x, long long ld, float* __restrict__ part,
                                                            int T, int N) {
  pdl_trigger();
  pdl_wait();
  __shared__ float sm[8][32 * V];
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + lane) * V;
  const int rows_per = (T + gridDim.y - 1) / gridDim.y;
  const int r0 = blockIdx.y * rows_per, r1 = min(T, r0 + rows_per);
  float a[V];
#pragma unroll
  for (int i = 0; i < V; ++i) a[i] = 0.f;
  if (c < N) {
#pragma unroll UNROLL
    for (int r = r0 + wy; r < r1; r += 8) {
      const __nv_bfloat16* p = x + static_cast<long long>(r) * ld + c;
      if constexpr (V == 8) {
        bf16x8 v; v.load(p);
        float f[8]; v.to_float(f);
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] += f[i];
      } else {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
        a[0] += v.x; a[1] += v.y;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < V; ++i) sm[wy][lane * V + i] = a[i];
  __syncthreads();
  if (threadIdx.x < 32 * V) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += sm[i][threadIdx.x];
    const int cc = blockIdx.x * 32 * V + threadIdx.x;
    if (cc < N) part[static_cast<long long>(blockIdx.y) * N + cc] = s;
  }
}

// ------------------------------------------------------------------------------ optimizer-side
// acc = (accumulate ? acc : 0) + src   (fp32 accumulator, bf16 or fp32 source)
template <typename SrcT>
__global__ void __launch_bounds__(EW_THREADS) accumulate_kernel(float* __restrict__ acc, const SrcT* __restrict__ src, long long n, int accumulate) {
  pdl_trigger();
  pdl_wait();
  const long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  float f[8];
  if constexpr (sizeof(SrcT) == 2) { bf16x8 v; v.load(reinterpret_cast<const __nv_bfloat16*>(src) + i); v.to_float(f); }
  else {
    const float4 a = *reinterpret_cast<const float4*>(src + i), b = *reinterpret_cast<const float4*>(src + i + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
  float4* d = reinterpret_cast<float4*>(acc + i);
  if (accumulate) {
    const float4 a = d[0], b = d[1];
    f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w; f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
  }
  d[0] = make_float4(f[0], f[1], f[2], f[3]);
  d[1] = make_float4(f[4], f[5], f[6], f[7]);
}

// dst(bf16) = (accumulate ? dst : 0) + src(fp32)
__global__ void __launch_bounds__(EW_THREADS) f32_to_bf16_kernel(__nv_bfloat16* __restrict__ dst, const float* __restrict__ src, long long n, int accumulate) {
  pdl_trigger();
  pdl_wait();
  const long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  const float4 a = *reinterpret_cast<const float4*>(src + i), b = *reinterpret_cast<const float4*>(src + i + 4);
  float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  if (accumulate) {
    bf16x8 v; v.load(dst + i); float g[8]; v.to_float(g);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] += g[k];
  }
  bf16x8 o; o.from_float(f); o.store(dst + i);
}

// out[0] += sum(x^2): per-block partial sums combined with one atomic per block.
__global__ void __launch_bounds__(EW_THREADS) sumsq_kernel(const float* __restrict__ x, long long n, float* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  float s = 0.f;
  for (long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 4; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x * 4) {
    const float4 v = *reinterpret_cast<const float4*>(x + i);
    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

// Fused AdamW on a shard: g = grad * coef; moments in fp32 or bf16; master fp32; bf16 working copy refreshed. Four elements from `i` on.
struct AdamwParams {
  float lr, beta1, beta2, eps, wd, inv_bc1, inv_sqrt_bc2;
};
template <typename StateT>
__device__ __forceinline__ void adamw4(float* __restrict__ master, StateT* __restrict__ m, StateT* __restrict__ v, const float* __restrict__ grad,
                                       __nv_bfloat16* __restrict__ param, long long i, float c, const AdamwParams& p) {
  const float4 g4 = *reinterpret_cast<const float4*>(grad + i);
  float4 w4 = *reinterpret_cast<float4*>(master + i);
  float g[4] = {g4.x * c, g4.y * c, g4.z * c, g4.w * c};
  float w[4] = {w4.x, w4.y, w4.z, w4.w};
  float mm[4], vv[4];
  if constexpr (sizeof(StateT) == 4) {
    const float4 a = *reinterpret_cast<const float4*>(m + i), b = *reinterpret_cast<const float4*>(v + i);
    mm[0] = a.x; mm[1] = a.y; mm[2] = a.z; mm[3] = a.w; vv[0] = b.x; vv[1] = b.y; vv[2] = b.z; vv[3] = b.w;
  } else {
    const uint2 a = *reinterpret_cast<const uint2*>(m + i), b = *reinterpret_cast<const uint2*>(v + i);
    float2 t;
    t = unpack_bf16(a.x); mm[0] = t.x; mm[1] = t.y; t = unpack_bf16(a.y); mm[2] = t.x; mm[3] = t.y;
    t = unpack_bf16(b.x); vv[0] = t.x; vv[1] = t.y; t = unpack_bf16(b.y); vv[2] = t.x; vv[3] = t.y;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    w[k] *= (1.f - p.lr * p.wd);
    mm[k] = p.beta1 * mm[k] + (1.f - p.beta1) * g[k];
    vv[k] = p.beta2 * vv[k] + (1.f - p.beta2) * g[k] * g[k];
    const float denom = sqrtf(vv[k]) * p.inv_sqrt_bc2 + p.eps;
    w[k] -= p.lr * p.inv_bc1 * mm[k] / denom;
  }
  *reinterpret_cast<float4*>(master + i) = make_float4(w[0], w[1], w[2], w[3]);
  if constexpr (sizeof(StateT) == 4) {
    *reinterpret_cast<float4*>(m + i) = make_float4(mm[0], mm[1], mm[2], mm[3]);
    *reinterpret_cast<float4*>(v + i) = make_float4(vv[0], vv[1], vv[2], vv[3]);
  } else {
    *reinterpret_cast<uint2*>(m + i) = make_uint2(pack_bf16(mm[0], mm[1]), pack_bf16(mm[2], mm[3]));
    *reinterpret_cast<uint2*>(v + i) = make_uint2(pack_bf16(vv[0], vv[1]), pack_bf16(vv[2], vv[3]));
  }
  *reinterpret_cast<uint2*>(param + i) = make_uint2(pack_bf16(w[0], w[1]), pack_bf16(w[2], w[3]));
}

template <typename StateT>
__global__ void __launch_bounds__(EW_THREADS) adamw_kernel(float* __restrict__ master, StateT* __restrict__ m, StateT* __restrict__ v,
                                                          const float* __restrict__ grad, __nv_bfloat16* __restrict__ param,
                                                          long long n, AdamwParams p, const float* __restrict__ coef) {
  pdl_trigger();
  pdl_wait();
  const long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  if (i < n) adamw4(master, m, v, grad, param, i, coef[0], p);
}

// The same over up to OPT_GROUPS groups in one launch, with the clip coefficient min(1, max_norm / (norm + 1e-6)) formed here from the sum
// of squares; the first block also leaves the norm. A small model's step was five launches for the coefficient and two per group, each
// taking the host 5 to 10 us: 13 launches became 2 for 4 groups, a step of 640 tokens through 2 layers 1055 -> 978 us, of 4096 tokens 1168 -> 1086.
constexpr int OPT_GROUPS = 48;   // 56 bytes each: the parameters of a launch stay below 4 KB
struct OptGroup {
  float* master;
  void *m, *v;
  const float* grad;
  __nv_bfloat16* param;
  long long n;
  int first_block;   // of this group in the launch
};
struct OptTable {
  OptGroup g[OPT_GROUPS];
  int groups;
};
__device__ __forceinline__ int opt_group(const OptTable& t) {   // of this block (uniform): the last group that starts at or before it
  int lo = 0, hi = t.groups - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.g[mid].first_block <= static_cast<int>(blockIdx.x)) lo = mid; else hi = mid - 1;
  }
  return lo;
}
template <typename StateT>
__global__ void __launch_bounds__(EW_THREADS) adamw_groups_kernel(const __grid_constant__ OptTable t, AdamwParams p, const float* __restrict__ sumsq,
                                                                 float max_norm, float* __restrict__ norm_out) {
  pdl_trigger();
  pdl_wait();
  const float norm = sqrtf(sumsq[0]);
  float c = 1.f;
  if (max_norm > 0.f) {
    c = max_norm / (norm + 1e-6f);
    c = c > 1.f ? 1.f : c;   // a norm that is not a number stays one
  }
  if (norm_out != nullptr && blockIdx.x == 0 && threadIdx.x == 0) norm_out[0] = norm;
  if (t.groups == 0) return;   // one block, for the norm
  const OptGroup& g = t.g[opt_group(t)];
  const long long i = (static_cast<long long>(blockIdx.x - g.first_block) * blockDim.x + threadIdx.x) * 4;
  if (i < g.n) adamw4(g.master, static_cast<StateT*>(g.m), static_cast<StateT*>(g.v), g.grad, g.param, i, c, p);
}

// out[0] += sum of squares over all groups.
__global__ void __launch_bounds__(EW_THREADS) sumsq_groups_kernel(const __grid_constant__ OptTable t, float* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  const int k = opt_group(t);
  const OptGroup& g = t.g[k];
  const int blocks = (k + 1 < t.groups ? t.g[k + 1].first_block : static_cast<int>(gridDim.x)) - g.first_block;
  float s = 0.f;
  for (long long i = (static_cast<long long>(blockIdx.x - g.first_block) * blockDim.x + threadIdx.x) * 4; i < g.n;
       i += static_cast<long long>(blocks) * blockDim.x * 4) {
    const float4 v = *reinterpret_cast<const float4*>(g.grad + i);
    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

static inline int cdiv(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }
static void reduce_rows(const float* part, void* out_a, void* out_b, int R, int C, int D, cudaStream_t st) {
  if (R <= 16 && C >= 512) launch_pdl(reduce_few_rows_kernel, cdiv(C, 256), 256, 0, st, part, (__nv_bfloat16*)out_a, (__nv_bfloat16*)out_b, R, C, D);
  else launch_pdl(reduce_rows_kernel, cdiv(C, 32), 512, 0, st, part, (__nv_bfloat16*)out_a, (__nv_bfloat16*)out_b, R, C, D);
}
static inline int launch_ok() { return cudaGetLastError() == cudaSuccess ? 0 : -5; }
static int num_sms() {
  static int n = 0;
  if (n == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev); }
  return n;
}

}  // namespace mtb

using namespace mtb;
typedef __nv_bfloat16 bf16;

template <bool LN, int VPT, bool BULK>
static int launch_norm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, float eps, int T, int H, int lanes,
                           int* status, cudaStream_t st) {
  auto kern = norm_fwd_kernel<LN, VPT, BULK>;
  const int rows = EW_THREADS / lanes;
  const int smem = BULK ? NORM_STAGES * rows * H * 2 : 0;
  int grid = cdiv(T, rows);
  if constexpr (BULK) {
    static bool configured = false;
    if (!configured) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, NORM_STAGES * 8 * 8 * EW_THREADS * 2) != cudaSuccess) return -4;
      configured = true;
    }
    static thread_local int for_smem = -1, resident = 0;   // the occupancy of the last shape this thread launched
    if (for_smem != smem) {
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, EW_THREADS, smem) != cudaSuccess || resident < 1) return -4;
      for_smem = smem;
    }
    const int most = num_sms() * resident;
    if (grid > most) grid = most;
  }
  launch_pdl(kern, grid, EW_THREADS, smem, st, (const bf16*)x, (const bf16*)w, (const bf16*)b, (bf16*)y, mean, rstd, eps, T, H, lanes, status);
  return launch_ok();
}

template <bool LN>
static int norm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, float eps, int T, int H, int* status, cudaStream_t st) {
  if (T <= 0) return 0;
  if (H <= 0 || H % 8 || H > (LN ? 4 : 8) * 8 * EW_THREADS) return -10;
  if ((reinterpret_cast<uintptr_t>(x) & 15)) return -11;
  // about four vectors per thread; a row is held by 32 .. 256 threads (a power of two)
  const int vecs = H / 8;
  int lanes = 32;
  while (lanes < EW_THREADS && lanes * 4 < vecs) lanes *= 2;
  const int vpt = cdiv(vecs, lanes);
  if constexpr (LN) {
    // Rows of up to 1024 elements: eight and more per block pay from 1024 rows on (16384 x 1024: 14.5 us, 27 with a block per row; cold,
    // 8 x 1024: 8.2 and 6.4). Wider ones want a batch that lasts: equal at 4000 x 2048 and 6000 x 4096. Three vectors of 256 threads
    // (4104 .. 6144) never win.
    const long long n = static_cast<long long>(T) * H;
    const bool bulk = H <= 1024 ? T >= 1024 : (H <= 2048 ? n >= 6000000 : n >= 24000000 && !(lanes == EW_THREADS && vpt == 3));
    if (!bulk) {
#define LF(V) launch_pdl(layernorm_row_kernel<V>, T, EW_THREADS, 0, st, (const bf16*)x, (const bf16*)w, (const bf16*)b, (bf16*)y, mean, rstd, eps, H)
      const int v = cdiv(H, 8 * EW_THREADS);
      if (v <= 1) LF(1); else if (v == 2) LF(2); else if (v == 3) LF(3); else LF(4);
#undef LF
      return launch_ok();
    }
#define NF(V) return launch_norm_fwd<true, V, true>(x, w, b, y, mean, rstd, eps, T, H, lanes, status, st)
    if (vpt <= 1) NF(1);
    if (vpt <= 2) NF(2);
    if (vpt <= 3) NF(3);
    NF(4);
#undef NF
  } else {
    // By bulk copies when a block gets more than two and a half row sets: blocks that fit on an SM with the stages, eight at most.
    const int rows = EW_THREADS / lanes, stages = NORM_STAGES * rows * H * 2 + 1280;
    const int fit = 227 * 1024 / stages < 8 ? 227 * 1024 / stages : 8;
    const bool bulk = 2 * cdiv(T, rows) > 5 * fit * num_sms();
#define NF(V) return bulk ? launch_norm_fwd<false, V, true>(x, w, b, y, mean, rstd, eps, T, H, lanes, status, st) \
                          : launch_norm_fwd<false, V, false>(x, w, b, y, mean, rstd, eps, T, H, lanes, status, st)
    if (vpt <= 1) NF(1);
    if (vpt <= 2) NF(2);
    if (vpt <= 3) NF(3);
    if (vpt <= 4) NF(4);
    NF(8);
#undef NF
  }
}


// Threads of a norm backward block: the row's vectors over as few vectors per thread as 512 threads allow.
static int norm_bwd_vpt(int H) { return cdiv(H, 8 * 512); }
static int norm_bwd_threads(int H) { return cdiv(cdiv(H / 8, norm_bwd_vpt(H)), 32) * 32; }

// Number of row-partials the backward of either norm writes (rows of the dw_partial scratch, fp32: [blocks, H], LayerNorm [blocks, 2, H]).
// Two blocks per SM at 512 threads, more of the smaller ones: every row in flight hides another's reduction.
extern "C" int mtb200_norm_bwd_blocks(int T, int H) {
  const int per_sm = 1024 / norm_bwd_threads(H);
  const int b = num_sms() * (per_sm < 2 ? 2 : (per_sm > 6 ? 6 : per_sm));
  return T < b ? (T > 0 ? T : 1) : b;
}

template <bool LN, int VPT>
static int launch_norm_bwd(const void* dy, const void* x, const float* mean, const float* rstd, const void* w, const void* add_to, void* dx,
                           float* dwp, int T, int H, int blocks, int threads, int* status, cudaStream_t st) {
  auto kern = norm_bwd_kernel<LN, VPT>;
  constexpr int most = 200 * 1024;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return -4;
    configured = true;
  }
  // up to four rows ahead in the block's share of the SM (blocks / SMs of them are resident), two at least
  const int stage = H * 2 * (add_to != nullptr ? 3 : 2), per_sm = cdiv(blocks, num_sms());
  int stages = most / (per_sm * stage);
  stages = stages > 4 ? 4 : (stages < 2 ? 2 : stages);
  launch_pdl(kern, blocks, threads, stages * stage, st, (const bf16*)dy, (const bf16*)x, mean, rstd, (const bf16*)w, (const bf16*)add_to, (bf16*)dx, dwp, T, H,
                                                stages, status);
  return launch_ok();
}

static bool aligned16(const void* a, const void* b, const void* c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

extern "C" {

int mtb200_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, float eps, int T, int H, int* status, cudaStream_t st) {
  return norm_fwd<false>(x, w, nullptr, y, nullptr, rstd, eps, T, H, status, st);
}

// LayerNorm with bias over rows of H <= 8192 elements; mean / rstd: [T] fp32 each.
int mtb200_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, float eps, int T, int H, int* status,
                         cudaStream_t st) {
  return norm_fwd<true>(x, w, b, y, mean, rstd, eps, T, H, status, st);
}

int mtb200_rmsnorm_bwd(const void* dy, const void* x, const float* rstd, const void* w, const void* add_to, void* dx,
                       float* dw_partial, void* dw_out, int T, int H, int* status, cudaStream_t st) {
  if (T <= 0) return 0;
  if (H <= 0 || H % 8 || H > 4 * 8 * 512) return -10;
  if (!aligned16(dy, x, add_to)) return -11;
  const int blocks = mtb200_norm_bwd_blocks(T, H), vpt = norm_bwd_vpt(H), threads = norm_bwd_threads(H);
  int rc;
#define RB(V) launch_norm_bwd<false, V>(dy, x, nullptr, rstd, w, add_to, dx, dw_partial, T, H, blocks, threads, status, st)
  if (vpt <= 1) rc = RB(1); else if (vpt == 2) rc = RB(2); else if (vpt == 3) rc = RB(3); else rc = RB(4);
#undef RB
  if (rc) return rc;
  reduce_rows(dw_partial, dw_out, nullptr, blocks, H, H, st);
  return launch_ok();
}

// dw_partial: [mtb200_norm_bwd_blocks(T, H), 2, H] fp32 scratch; dw_out / db_out: [H] bf16 each.
int mtb200_layernorm_bwd(const void* dy, const void* x, const float* mean, const float* rstd, const void* w, const void* add_to, void* dx,
                         float* dw_partial, void* dw_out, void* db_out, int T, int H, int* status, cudaStream_t st) {
  if (T <= 0) return 0;
  if (H <= 0 || H % 8 || H > 4 * 8 * EW_THREADS) return -10;
  if (!aligned16(dy, x, add_to)) return -11;
  const int blocks = mtb200_norm_bwd_blocks(T, H), threads = norm_bwd_threads(H);
  int rc;
#define LB(V) launch_norm_bwd<true, V>(dy, x, mean, rstd, w, add_to, dx, dw_partial, T, H, blocks, threads, status, st)
  if (norm_bwd_vpt(H) <= 1) rc = LB(1); else rc = LB(2);
#undef LB
  if (rc) return rc;
  reduce_rows(dw_partial, dw_out, db_out, blocks, 2 * H, H, st);
  return launch_ok();
}

int mtb200_rope(void* qkv, const int* pos, const float* inv_freq, int T, long long ld, int n_heads, int D, int inverse, cudaStream_t st) {
  if (T <= 0) return 0;
  if (D % 16 || ld % 8) return -10;
  const long long n = static_cast<long long>(T) * (D / 16);
  launch_pdl(rope_kernel, dim3(cdiv(n, EW_THREADS), cdiv(n_heads, ROPE_HPT)), EW_THREADS, 0, st, (bf16*)qkv, pos, inv_freq, T, ld, n_heads, D,
                                                                                        inverse ? -1.f : 1.f);
  return launch_ok();
}

static int heads_per_warp(int T, int n_heads) {
  return static_cast<long long>(T) * cdiv(n_heads, HEADS_PER_WARP) < 2LL * num_sms() * (EW_THREADS / 32) ? 1 : HEADS_PER_WARP;
}

// Per-head RMSNorm of the q and k heads (n_q then n_heads - n_q) of qkv[T, ld], in place; rstd: [T * n_heads] fp32. With
// inv_freq [D / 2] (and pos [T]) the heads are also rotated; pre (optional): [T, n_heads * D], the heads as they came.
int mtb200_head_rmsnorm_fwd(void* qkv, const void* wq, const void* wk, void* pre, float* rstd, const int* pos, const float* inv_freq, float eps,
                            int T, long long ld, int n_q, int n_heads, int D, cudaStream_t st) {
  if (T <= 0 || n_heads <= 0) return 0;
  if ((D != 64 && D != 128 && D != 256) || ld % 8 || n_q < 0 || n_q > n_heads || (inv_freq && !pos)) return -10;
  const int hpw = heads_per_warp(T, n_heads), groups = cdiv(n_heads, hpw);
  const long long n_items = static_cast<long long>(T) * groups;
  const unsigned blocks = static_cast<unsigned>(cdiv(n_items, EW_THREADS / 32));
#define HF(E, R) if (hpw == 1) HFW(E, R, 1); else HFW(E, R, HEADS_PER_WARP)
#define HFW(E, R, W) launch_pdl(head_rmsnorm_fwd_kernel<E, R, W>, blocks, EW_THREADS, 0, st, (bf16*)qkv, (const bf16*)wq, (const bf16*)wk, (bf16*)pre, rstd, pos, inv_freq, eps, n_items, groups, ld, n_q, n_heads)
  if (inv_freq) { if (D == 64) { HF(2, true); } else if (D == 128) { HF(4, true); } else { HF(8, true); } }
  else { if (D == 64) { HF(2, false); } else if (D == 128) { HF(4, false); } else { HF(8, false); } }
#undef HF
#undef HFW
  return launch_ok();
}

// Rows of the dw_partial scratch ([blocks, 2, D] fp32) the backward writes.
int mtb200_head_rmsnorm_bwd_blocks(int T, int n_heads) {
  const long long items = static_cast<long long>(T) * cdiv(n_heads, HEADS_PER_WARP);
  const long long want = cdiv(items, EW_THREADS / 32);
  const long long cap = num_sms() * 4;
  return static_cast<int>(want < cap ? (want > 0 ? want : 1) : cap);
}

// dqkv (q and k heads) in place; pre: the heads before the norm, [T, ld_pre]; dwq_out / dwk_out: [D] bf16 each. With inv_freq the
// rotation is undone first.
int mtb200_head_rmsnorm_bwd(void* dqkv, const void* pre, const float* rstd, const void* wq, const void* wk, float* dw_partial,
                            void* dwq_out, void* dwk_out, const int* pos, const float* inv_freq, int T, long long ld, long long ld_pre, int n_q,
                            int n_heads, int D, cudaStream_t st) {
  if (T <= 0 || n_heads <= 0) return 0;
  if ((D != 64 && D != 128 && D != 256) || ld % 8 || ld_pre % 8 || n_q < 0 || n_q > n_heads || (inv_freq && !pos)) return -10;
  const int groups = cdiv(n_heads, HEADS_PER_WARP);
  const long long n_items = static_cast<long long>(T) * groups;
  const int blocks = mtb200_head_rmsnorm_bwd_blocks(T, n_heads);
#define HB(E, R) launch_pdl(head_rmsnorm_bwd_kernel<E, R>, blocks, EW_THREADS, 0, st, (bf16*)dqkv, (const bf16*)pre, rstd, (const bf16*)wq, (const bf16*)wk, dw_partial, pos, inv_freq, n_items, groups, ld, ld_pre, n_q, n_heads)
  if (inv_freq) { if (D == 64) HB(2, true); else if (D == 128) HB(4, true); else HB(8, true); }
  else { if (D == 64) HB(2, false); else if (D == 128) HB(4, false); else HB(8, false); }
#undef HB
  // partial rows are [2, D]: columns 0..D-1 belong to the q weight, D..2D-1 to the k weight
  reduce_rows(dw_partial, dwq_out, dwk_out, blocks, 2 * D, D, st);
  return launch_ok();
}

int mtb200_swiglu_fwd(const void* gu, void* act, long long T, int F, cudaStream_t st) {
  if (T <= 0) return 0;
  if (F % 8) return -10;
  launch_pdl(swiglu_fwd_kernel<0>, dim3(static_cast<unsigned>(T), cdiv(F / 8, EW_THREADS)), EW_THREADS, 0, st, (const bf16*)gu, (bf16*)act, T, F);
  return launch_ok();
}

int mtb200_swiglu_bwd(const void* dact, const void* gu, void* dgu, long long T, int F, cudaStream_t st) {
  if (T <= 0) return 0;
  if (F % 8) return -10;
  launch_pdl(swiglu_bwd_kernel<false, 0>, dim3(static_cast<unsigned>(T), cdiv(F / 8, EW_THREADS)), EW_THREADS, 0, st, (bf16*)const_cast<void*>(dact), (const bf16*)gu, (bf16*)dgu, T, F);
  return launch_ok();
}

// Same, and dact_inout is overwritten with the forward output silu(gate) * up.
int mtb200_swiglu_bwd_act(void* dact_inout, const void* gu, void* dgu, long long T, int F, cudaStream_t st) {
  if (T <= 0) return 0;
  if (F % 8) return -10;
  launch_pdl(swiglu_bwd_kernel<true, 0>, dim3(static_cast<unsigned>(T), cdiv(F / 8, EW_THREADS)), EW_THREADS, 0, st, (bf16*)dact_inout, (const bf16*)gu, (bf16*)dgu, T, F);
  return launch_ok();
}

// GeGLU (tanh-approximated GELU on the gate): same three entry points as SwiGLU.
int mtb200_geglu_fwd(const void* gu, void* act, long long T, int F, cudaStream_t st) {
  if (T <= 0) return 0;
  if (F % 8) return -10;
  launch_pdl(swiglu_fwd_kernel<1>, dim3(static_cast<unsigned>(T), cdiv(F / 8, EW_THREADS)), EW_THREADS, 0, st, (const bf16*)gu, (bf16*)act, T, F);
  return launch_ok();
}
int mtb200_geglu_bwd(const void* dact, const void* gu, void* dgu, long long T, int F, cudaStream_t st) {
  if (T <= 0) return 0;
  if (F % 8) return -10;
  launch_pdl(swiglu_bwd_kernel<false, 1>, dim3(static_cast<unsigned>(T), cdiv(F / 8, EW_THREADS)), EW_THREADS, 0, st, (bf16*)const_cast<void*>(dact), (const bf16*)gu, (bf16*)dgu, T, F);
  return launch_ok();
}
int mtb200_geglu_bwd_act(void* dact_inout, const void* gu, void* dgu, long long T, int F, cudaStream_t st) {
  if (T <= 0) return 0;
  if (F % 8) return -10;
  launch_pdl(swiglu_bwd_kernel<true, 1>, dim3(static_cast<unsigned>(T), cdiv(F / 8, EW_THREADS)), EW_THREADS, 0, st, (bf16*)dact_inout, (const bf16*)gu, (bf16*)dgu, T, F);
  return launch_ok();
}

// y = gelu_tanh(x) over n elements; dx = dy * gelu_tanh'(x) (dx may be dy).
int mtb200_gelu_fwd(const void* x, void* y, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8) return -10;
  launch_pdl(act_fwd_kernel<1>, static_cast<unsigned>(cdiv(n / 8, EW_THREADS)), EW_THREADS, 0, st, (const bf16*)x, (bf16*)y, n);
  return launch_ok();
}
int mtb200_gelu_bwd(const void* dy, const void* x, void* dx, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8) return -10;
  launch_pdl(act_bwd_kernel<false, 1>, static_cast<unsigned>(cdiv(n / 8, EW_THREADS)), EW_THREADS, 0, st, (bf16*)const_cast<void*>(dy), (const bf16*)x, (bf16*)dx, n);
  return launch_ok();
}
// Same, and dy_inout is overwritten with gelu_tanh(x); dx is another buffer.
int mtb200_gelu_bwd_act(void* dy_inout, const void* x, void* dx, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8 || dx == dy_inout) return -10;
  launch_pdl(act_bwd_kernel<true, 1>, static_cast<unsigned>(cdiv(n / 8, EW_THREADS)), EW_THREADS, 0, st, (bf16*)dy_inout, (const bf16*)x, (bf16*)dx, n);
  return launch_ok();
}

int mtb200_embedding_fwd(const void* w, const long long* ids, void* out, int T, int H, int V, int* status, cudaStream_t st) {
  if (T <= 0) return 0;
  if (H % 8) return -10;
  launch_pdl(embedding_fwd_kernel, T, 128, 0, st, (const bf16*)w, ids, (bf16*)out, H, V, status);
  return launch_ok();
}

int mtb200_embedding_bwd(void* dw, const long long* sorted_ids, const long long* order, const void* dx, int T, int H, int V,
                         int* status, cudaStream_t st) {
  if (T <= 0) return 0;
  if (H % 8) return -10;
  launch_pdl(embedding_bwd_kernel, T, 128, 0, st, (bf16*)dw, sorted_ids, order, (const bf16*)dx, T, H, V, status);
  return launch_ok();
}

// The same from the ids as they come, for at most EMB_SCAN tokens.
int mtb200_embedding_bwd_scan(void* dw, const long long* ids, const void* dx, int T, int H, int V, int* status, cudaStream_t st) {
  if (T <= 0) return 0;
  if (H % 8 || T > EMB_SCAN) return -10;
  launch_pdl(embedding_bwd_scan_kernel, T, EW_THREADS, 0, st, (bf16*)dw, ids, (const bf16*)dx, T, H, V, status);
  return launch_ok();
}

// out [T, H] and vout [T] are zero but in `rows` [R], where they are src [R, H] and vsrc [R].
int mtb200_scatter_rows(const long long* rows, const void* src, void* out, const float* vsrc, float* vout, int R, int H, int T, int* status, cudaStream_t st) {
  if (T <= 0 || R < 0) return 0;
  if (H % 8) return -10;
  const long long pieces = static_cast<long long>(T) * H / 8, blocks = (pieces + 4 * EW_THREADS - 1) / (4 * EW_THREADS);
  if (pieces > (8 << 20)) {   // above 128 MB the memsets are the faster ones: 64000 x 4096 179 us, 187 by the kernel
    if (cudaMemsetAsync(out, 0, pieces * 16, st) != cudaSuccess || cudaMemsetAsync(vout, 0, static_cast<size_t>(T) * 4, st) != cudaSuccess) return -5;
  } else launch_pdl(zero_rows_kernel, static_cast<int>(blocks < num_sms() * 8 ? (blocks > 0 ? blocks : 1) : num_sms() * 8), EW_THREADS, 0, st, (uint4*)out, pieces, vout, T);
  if (R > 0) launch_pdl(scatter_rows_kernel, R, 128, 0, st, rows, (const bf16*)src, (bf16*)out, vsrc, vout, H, T, status);
  return launch_ok();
}

// logits: [R, V] fp32, or bf16 when logits_bf16 (dlogits may then be the same buffer). stats: optional, bf16 logits only.
int mtb200_ce_fwd_bwd(const void* logits, long long ld, int logits_bf16, const float2* stats, const long long* targets, float* loss,
                      void* dlogits, long long ldd, int R, int V, float grad_scale, long long ignore_index, cudaStream_t st) {
  if (R <= 0) return 0;
  if (V % 8 || ld % 8 || ldd % 8 || (stats && !logits_bf16)) return -10;
  // Four rows at a time on an SM hide each other's reductions better than two, when there are rows enough to go round: with statistics 8000 x 17008
  // 151 -> 108 us, x 32000 194 -> 167, 3720 x 49152 127 -> 119, x 151936 level; without 4000 x 40000 152 -> 133, x 57344 200 -> 187, but 2048 x 65536
  // 114 -> 117 and x 128256 222 -> 262, where the rows at work on no longer stay in L2. 900 x 32000 25 -> 23, 600 level, 200 6.4 -> 9.3.
  const int per_row = logits_bf16 && V <= 57344 && R >= 6 * num_sms() ? 512 : 1024;
#define CE(T, S) launch_pdl(ce_fwd_bwd_kernel<T, S>, R, per_row, 0, st, (const T*)logits, ld, stats, targets, loss, (bf16*)dlogits, ldd, V, grad_scale, ignore_index)
  const int threads = cdiv(V, CE_ROW_VECS * 8 * 32) * 32;
  if (logits_bf16 && !stats && threads <= 1024) {
    const int most = num_sms() * (1024 / threads);   // what 64 registers a thread let an SM hold
    launch_pdl(ce_row_kernel, R < most ? R : most, threads, 0, st, (const bf16*)logits, ld, targets, loss, (bf16*)dlogits, ldd, R, V, grad_scale, ignore_index);
    return launch_ok();
  }
  if (stats) CE(bf16, true); else if (logits_bf16) CE(bf16, false); else CE(float, false);
#undef CE
  return launch_ok();
}

static void launch_colsum(const void* x, long long ld, void* out, float* scratch, int T, int N, cudaStream_t st) {
  const int splits = T < 32 ? 1 : 32;
  const bool many = T >= 8192;   // at least four times eight rows per warp
  const bool wide = N % 8 == 0 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (many || N > 1024);
  const dim3 grid(cdiv(N, wide ? 256 : 64), splits);
  if (wide && many && N <= 5120) launch_pdl(colsum_partial_kernel<8, 8>, grid, 256, 0, st, (const bf16*)x, ld, scratch, T, N);
  else if (wide) launch_pdl(colsum_partial_kernel<8, 4>, grid, 256, 0, st, (const bf16*)x, ld, scratch, T, N);
  else launch_pdl(colsum_partial_kernel<2, 4>, grid, 256, 0, st, (const bf16*)x, ld, scratch, T, N);
  reduce_rows(scratch, out, nullptr, splits, N, N, st);
}

// out[N] (bf16) = column sums of x[T, N]. scratch: fp32 [32, N].
int mtb200_colsum(const void* x, long long ld, void* out, float* scratch, int T, int N, cudaStream_t st) {
  if (T <= 0 || N <= 0) return 0;
  if (N % 2) return -10;
  launch_colsum(x, ld, out, scratch, T, N, st);
  return launch_ok();
}

int mtb200_accumulate(float* acc, const void* src, long long n, int src_is_f32, int accumulate, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8) return -10;
  if (src_is_f32) launch_pdl(accumulate_kernel<float>, cdiv(n / 8, EW_THREADS), EW_THREADS, 0, st, acc, (const float*)src, n, accumulate);
  else launch_pdl(accumulate_kernel<bf16>, cdiv(n / 8, EW_THREADS), EW_THREADS, 0, st, acc, (const bf16*)src, n, accumulate);
  return launch_ok();
}

int mtb200_f32_to_bf16(void* dst, const float* src, long long n, int accumulate, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8) return -10;
  launch_pdl(f32_to_bf16_kernel, cdiv(n / 8, EW_THREADS), EW_THREADS, 0, st, (bf16*)dst, src, n, accumulate);
  return launch_ok();
}

int mtb200_sumsq(const float* x, long long n, float* out, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 4) return -10;
  const int blocks = static_cast<int>(min(static_cast<long long>(num_sms() * 8), (n / 4 + EW_THREADS - 1) / EW_THREADS));
  launch_pdl(sumsq_kernel, blocks, EW_THREADS, 0, st, x, n, out);
  return launch_ok();
}

int mtb200_adamw(float* master, void* m, void* v, int state_is_f32, const float* grad, void* param, long long n, float lr,
                 float beta1, float beta2, float eps, float wd, int step, const float* coef, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 4) return -10;
  const float inv_bc1 = 1.f / (1.f - powf(beta1, static_cast<float>(step)));
  const float inv_sqrt_bc2 = 1.f / sqrtf(1.f - powf(beta2, static_cast<float>(step)));
  const AdamwParams p{lr, beta1, beta2, eps, wd, inv_bc1, inv_sqrt_bc2};
  const int blocks = cdiv(n / 4, EW_THREADS);
  if (state_is_f32) launch_pdl(adamw_kernel<float>, blocks, EW_THREADS, 0, st, master, (float*)m, (float*)v, grad, (bf16*)param, n, p, coef);
  else launch_pdl(adamw_kernel<bf16>, blocks, EW_THREADS, 0, st, master, (bf16*)m, (bf16*)v, grad, (bf16*)param, n, p, coef);
  return launch_ok();
}

// table: [groups][6] = master, m, v, gradient (fp32), working copy, elements. One launch per OPT_GROUPS groups.
// most_blocks: of a group (0: as many as give every thread four elements).
static int fill_table(OptTable& t, const long long* table, int groups, int most_blocks, long long* blocks) {
  long long at = 0;
  t.groups = 0;
  for (int k = 0; k < groups; ++k) {
    const long long* r = table + k * 6;
    if (r[5] <= 0) continue;
    if (r[5] % 4) return -10;
    OptGroup& g = t.g[t.groups++];
    g.master = reinterpret_cast<float*>(r[0]); g.m = reinterpret_cast<void*>(r[1]); g.v = reinterpret_cast<void*>(r[2]);
    g.grad = reinterpret_cast<const float*>(r[3]); g.param = reinterpret_cast<bf16*>(r[4]); g.n = r[5];
    g.first_block = static_cast<int>(at);
    const long long want = (r[5] / 4 + EW_THREADS - 1) / EW_THREADS;
    at += most_blocks > 0 && want > most_blocks ? most_blocks : want;
    if (at > 0x7fffffffLL) return -10;
  }
  *blocks = at;
  return 0;
}

// out[0] += sum of squares of the groups' gradients.
int mtb200_sumsq_groups(const long long* table, int groups, float* out, cudaStream_t st) {
  for (int first = 0; first < groups; first += OPT_GROUPS) {
    OptTable t;
    long long blocks = 0;
    const int k = groups - first < OPT_GROUPS ? groups - first : OPT_GROUPS;
    const int rc = fill_table(t, table + first * 6, k, num_sms() * 8, &blocks);
    if (rc) return rc;
    if (blocks > 0) launch_pdl(sumsq_groups_kernel, static_cast<unsigned>(blocks), EW_THREADS, 0, st, t, out);
  }
  return launch_ok();
}

// AdamW on all groups with the gradients scaled by min(1, max_norm / (sqrt(sumsq) + 1e-6)) (max_norm 0: by one); norm_out[0] = sqrt(sumsq).
int mtb200_adamw_groups(const long long* table, int groups, int state_is_f32, const float* sumsq, float max_norm, float* norm_out, float lr, float beta1,
                        float beta2, float eps, float wd, int step, cudaStream_t st) {
  const float inv_bc1 = 1.f / (1.f - powf(beta1, static_cast<float>(step)));
  const float inv_sqrt_bc2 = 1.f / sqrtf(1.f - powf(beta2, static_cast<float>(step)));
  const AdamwParams p{lr, beta1, beta2, eps, wd, inv_bc1, inv_sqrt_bc2};
  for (int first = 0; first == 0 || first < groups; first += OPT_GROUPS) {
    OptTable t;
    long long blocks = 0;
    const int k = groups - first < OPT_GROUPS ? groups - first : OPT_GROUPS;
    const int rc = fill_table(t, table + first * 6, k, 0, &blocks);
    if (rc) return rc;
    if (blocks == 0 && first > 0) continue;
    if (blocks == 0) blocks = 1;   // the first launch leaves the norm, whatever its groups hold
    float* out = first == 0 ? norm_out : nullptr;
    if (state_is_f32) launch_pdl(adamw_groups_kernel<float>, static_cast<unsigned>(blocks), EW_THREADS, 0, st, t, p, sumsq, max_norm, out);
    else launch_pdl(adamw_groups_kernel<bf16>, static_cast<unsigned>(blocks), EW_THREADS, 0, st, t, p, sumsq, max_norm, out);
  }
  return launch_ok();
}

}  // extern "C"

// ------------------------------------------------------------------------------------------
// Allocation-free variant of mtb200_colsum (declared in mtb200_noalloc.h).
//
// For callers that cannot allocate device memory when they need the kernel: the fp32 partial-sum
// workspace lives in a file-scope device array. In host code the array's name is only a handle,
// never a pointer a kernel could dereference, so its device address is looked up once per device
// with cudaGetSymbolAddress and that address is what the kernels receive.
// ------------------------------------------------------------------------------------------
#include "mtb200_noalloc.h"

static __device__ __align__(256) float g_colsum_noalloc_ws[32 * MTB200_COLSUM_NOALLOC_MAX_N];

namespace {
constexpr int kMaxDevices = 64;
float* g_colsum_ws_addr[kMaxDevices] = {nullptr};

// Device address of the workspace on the current device (looked up on first use per device).
float* colsum_noalloc_workspace() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  if (g_colsum_ws_addr[dev] == nullptr) {
    float* ptr = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_colsum_noalloc_ws) != cudaSuccess) return nullptr;
    g_colsum_ws_addr[dev] = ptr;
  }
  return g_colsum_ws_addr[dev];
}
}  // namespace

extern "C" int mtb200_colsum_noalloc(const void* x, long long ld, void* out, int T, int N, cudaStream_t st) {
  if (T <= 0 || N <= 0) return 0;
  if (N % 2 || ld < N) return -10;
  if (N > MTB200_COLSUM_NOALLOC_MAX_N) return -11;   // beyond the built-in workspace
  float* ws = colsum_noalloc_workspace();
  if (ws == nullptr) return -12;
  // Every element of ws[0 : splits * N] that the second kernel reads is written by the first one,
  // so nothing left over from an earlier call can reach the result and no clearing pass is needed.
  launch_colsum(x, ld, out, ws, T, N, st);
  return launch_ok();
}

