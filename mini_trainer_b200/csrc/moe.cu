// Mixture-of-experts support kernels: grouping of (token, slot) pairs by expert, row gather, SwiGLU gradient with the
// expert weights, combination of a token's experts, router gradient. The expert projections themselves are the grouped
// GEMMs of gemm_tcgen05.cu.
//
// Row buffers hold one slab of rows per expert, slabs start at multiples of 128 rows (GROUP_ALIGN) and the rows between a
// slab's end and the next start are zero. Row counts stay on the device: nothing here needs a host read.
//   pair  = token * k + slot (as chosen by the router);  pair_of[row] = pair or -1 in padding;  row_of[pair] = row
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "gemm_epilogue.cuh"
#include "ptx.cuh"

namespace mtb {

typedef __nv_bfloat16 bf16;
constexpr int MOE_THREADS = 256;
constexpr int PLAN_THREADS = 1024;   // 32 warps: one lane per warp total

struct Vec8 {
  uint4 u;
  __device__ __forceinline__ void load(const bf16* p) { u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void store(bf16* p) const { *reinterpret_cast<uint4*>(p) = u; }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
  }
  __device__ __forceinline__ void set(const float (&f)[8]) {
    u = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
  }
};

// Router of a layer, one warp per token: fp32 softmax of the logits, the k largest (the lower index of equal ones, the largest first) and their
// weights, renormalised over the chosen ones when `renorm`. A lane holds experts lane, lane + 32, ... As tensor operations these were
// six launches of 2 to 11 us and the gaps between them (2051 tokens, 64 experts, 8 chosen: 28 us and 10 of
// gaps, now 6.6; the layer's forward and backward 1053 -> 1019).
__global__ void __launch_bounds__(MOE_THREADS) moe_route_kernel(const bf16* __restrict__ logits, int T, int E, int k, int renorm, float* __restrict__ probs,
                                                               long long* __restrict__ topi, float* __restrict__ w) {
  pdl_trigger();
  pdl_wait();
  const long long t = (static_cast<long long>(blockIdx.x) * MOE_THREADS + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  constexpr int PER = GROUP_MAX / 32;
  float x[PER];
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + i * 32;
    x[i] = e < E ? __bfloat162float(logits[t * E + e]) : -INFINITY;
    m = fmaxf(m, x[i]);
  }
  m = warp_max(m);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) { x[i] = lane + i * 32 < E ? expf(x[i] - m) : 0.f; s += x[i]; }
  s = warp_sum(s);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + i * 32;
    x[i] /= s;
    if (e < E) probs[t * E + e] = x[i];
    x[i] = e >= E ? -1.f : (x[i] != x[i] ? INFINITY : x[i]);   // what is not a number counts as the largest, as in a sort
  }
  float mine = 0.f, sum = 0.f;   // lane s holds the s-th weight
  for (int c = 0; c < k; ++c) {
    float best = -2.f;
    int at = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) if (x[i] > best) { best = x[i]; at = lane + i * 32; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) if (at == lane + i * 32) x[i] = -1.f;   // taken
    const float v = best == INFINITY ? NAN : best;
    if (lane == c) { mine = v; topi[t * k + c] = at; }
    sum += v;
  }
  if (lane < k) w[t * k + lane] = renorm ? mine / sum : mine;
}

// One block per expert. Every block counts all experts (the chosen indices are a few hundred KB at most and stay in L2), so
// the slab starts need no second launch; it then walks the pairs once more and numbers its own, in pair order: the row order
// inside a slab, and with it every sum over a slab, does not depend on scheduling.
__global__ void __launch_bounds__(PLAN_THREADS) moe_plan_kernel(const long long* __restrict__ topi, int n, int E, int cap,
                                                               int* __restrict__ starts, int* __restrict__ counts,
                                                               int* __restrict__ pair_of, int* __restrict__ row_of, int* status) {
  pdl_trigger();
  pdl_wait();
  __shared__ int hist[GROUP_MAX];
  __shared__ int wsum[2][PLAN_THREADS / 32];
  __shared__ int start_sh;
  const int me = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < E; i += PLAN_THREADS) hist[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += PLAN_THREADS) {
    const long long e = topi[i];
    if (e >= 0 && e < E) atomicAdd(&hist[e], 1);
    else if (status != nullptr) atomicExch(status, 62);   // an index that is no expert: its pair gets no row
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0;
    for (int e = 0; e < E; ++e) {
      if (e == me) start_sh = at;
      if (me == 0) { starts[e] = at; counts[e] = hist[e]; }
      at += (hist[e] + GROUP_ALIGN - 1) / GROUP_ALIGN * GROUP_ALIGN;
    }
    if (me == 0) starts[E] = at;
  }
  __syncthreads();
  const int start = start_sh;
  int next = start;
  // (all threads run the same number of rounds; two buffers of warp totals, so one barrier per round)
  for (int i0 = 0, it = 0; i0 < n; i0 += PLAN_THREADS, ++it) {
    const int i = i0 + threadIdx.x;
    const long long e = i < n ? topi[i] : -1;
    const bool hit = e == me;
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) wsum[it & 1][warp] = __popc(m);
    __syncthreads();
    const int mine = wsum[it & 1][lane];   // every warp scans the warps' totals for itself
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
    const int before = __shfl_sync(0xffffffffu, incl - mine, warp), total = __shfl_sync(0xffffffffu, incl, 31);
    if (hit) {
      const int row = next + before + __popc(m & ((1u << lane) - 1));
      pair_of[row] = i;
      row_of[i] = row;
    }
    if (me == 0 && i < n && (e < 0 || e >= E)) row_of[i] = -1;
    next += total;
  }
  const int end = start + (hist[me] + GROUP_ALIGN - 1) / GROUP_ALIGN * GROUP_ALIGN;
  for (int r = start + hist[me] + threadIdx.x; r < end; r += PLAN_THREADS) pair_of[r] = -1;
  if (me == E - 1) for (int r = end + threadIdx.x; r < cap; r += PLAN_THREADS) pair_of[r] = -1;
}

// out[row] = scale * src[pair_of[row] / k], zeros in padding. Rows past the last slab are left alone. A warp per row, eight vectors of it
// in flight per lane (a block of 128 threads per row had two; layer of 64 experts, three gathers of 20 500 rows of 2048: 1047 -> 1019 us; eight experts level:
// bound by writing the rows).
constexpr int GATHER_WARPS = 4;
__global__ void __launch_bounds__(32 * GATHER_WARPS) moe_gather_kernel(const bf16* __restrict__ src, const int* __restrict__ pair_of, const int* __restrict__ starts,
                                                                      int E, int k, int cap, int H, float scale, bf16* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const long long row = static_cast<long long>(blockIdx.x) * GATHER_WARPS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= cap || row >= starts[E]) return;
  const int pair = pair_of[row];
  bf16* dst = out + row * H;
  const bf16* s = pair < 0 ? nullptr : src + static_cast<long long>(pair / k) * H;
  for (int c0 = lane * 8; c0 < H; c0 += 8 * 256) {
    Vec8 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j].u = make_uint4(0u, 0u, 0u, 0u);
      if (s != nullptr && c0 + j * 256 < H) v[j].load(s + c0 + j * 256);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (c0 + j * 256 >= H) break;
      if (scale != 1.f) {
        float f[8]; v[j].get(f);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] *= scale;
        v[j].set(f);
      }
      v[j].store(dst + c0 + j * 256);
    }
  }
}

template <int ACT>
__device__ __forceinline__ void act_and_grad(float g, float& a, float& da) {
  if constexpr (ACT == 0) {   // SiLU
    const float sig = __fdividef(1.f, 1.f + exp_ftz(-g));
    a = g * sig;
    da = sig * (1.f + g * (1.f - sig));
  } else {                    // tanh-approximated GELU
    const float s = gelu_gate(g);
    a = g * s;
    da = s + g * s * (1.f - s) * 1.5957691216057308f * (1.f + 0.134145f * g * g);
  }
}

// Per routed row, with du the gradient of the activation before the expert weight w:
//   dgu = d(act(g) * u) for the incoming gradient w * du,  du <- w * act(g) * u (the row the down projection's weight
//   gradient needs),  dw[pair] = du . (act(g) * u)
// One pass over gate/up and du instead of the forward activation, two scalings, a dot product and the activation gradient as passes of their
// own. TPR threads per row: a warp for narrow rows, whose reduction then needs no barrier (20 500 rows of 1024: 60 us with a block per row,
// 40 with a warp; the layer of 64 experts 1042 -> 1019), up to the whole block for wide ones (14 336: 221 us either way, the copy bandwidth).
template <int ACT, int TPR>
__global__ void __launch_bounds__(MOE_THREADS) moe_glu_bwd_kernel(bf16* __restrict__ du, const bf16* __restrict__ gu, const float* __restrict__ w,
                                                                 const int* __restrict__ pair_of, const int* __restrict__ starts, int E, int cap, int F,
                                                                 bf16* __restrict__ dgu, float* __restrict__ dw) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[MOE_THREADS / 32];
  const int l = threadIdx.x % TPR;
  const long long row = static_cast<long long>(blockIdx.x) * (MOE_THREADS / TPR) + threadIdx.x / TPR;
  const bool here = row < cap && row < starts[E];
  const int pair = here ? pair_of[row] : -1;
  const float wr = pair < 0 ? 0.f : w[pair];
  float dot = 0.f;
#pragma unroll 2
  for (int c = l * 8; here && c < F; c += TPR * 8) {
    Vec8 g, u, d;
    g.load(gu + row * 2 * F + c); u.load(gu + row * 2 * F + F + c); d.load(du + row * F + c);
    float fg[8], fu[8], fd[8], oa[8];
    g.get(fg); u.get(fu); d.get(fd);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float a, da;
      act_and_grad<ACT>(fg[i], a, da);
      const float y = a * fu[i], dd = fd[i] * wr;
      dot += fd[i] * y;
      oa[i] = y * wr;
      fg[i] = dd * fu[i] * da;
      fu[i] = dd * a;
    }
    d.set(oa); g.set(fg); u.set(fu);
    d.store(du + row * F + c);
    g.store(dgu + row * 2 * F + c);
    u.store(dgu + row * 2 * F + F + c);
  }
  dot = warp_sum(dot);
  if constexpr (TPR > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dot;
    __syncthreads();
    dot = 0.f;
#pragma unroll
    for (int i = 0; i < TPR / 32; ++i) dot += red[threadIdx.x / TPR * (TPR / 32) + i];
  }
  if (l == 0 && pair >= 0) dw[pair] = dot;
}

// out[t] = base[t] + scale * (sum over slots of w[t, slot] * rows[row_of[t, slot]] + add[t]), summed in fp32 in slot order.
// w, add (fp32) may be null.
__global__ void __launch_bounds__(MOE_THREADS) moe_combine_kernel(const bf16* __restrict__ rows, const int* __restrict__ row_of,
                                                                 const float* __restrict__ w, const float* __restrict__ add,
                                                                 const bf16* __restrict__ base, float scale, int k, int H, bf16* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const long long t = blockIdx.x;
  const int* ro = row_of + t * k;
  for (int c = threadIdx.x * 8; c < H; c += MOE_THREADS * 8) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll 4
    for (int s = 0; s < k; ++s) {
      const int r = ro[s];
      if (r < 0) continue;
      const float ws = w == nullptr ? 1.f : w[t * k + s];
      Vec8 v; v.load(rows + static_cast<long long>(r) * H + c);
      float f[8]; v.get(f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += ws * f[i];
    }
    if (add != nullptr) {
      const float4 a = *reinterpret_cast<const float4*>(add + t * H + c), b = *reinterpret_cast<const float4*>(add + t * H + c + 4);
      acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w; acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
    }
    Vec8 v; v.load(base + t * H + c);
    float f[8]; v.get(f);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] += scale * acc[i];
    v.set(f);
    v.store(out + t * H + c);
  }
}

// Gradient of the router logits, one warp per token: chosen weights -> renormalisation over the chosen experts (when
// `renorm`) -> selection -> softmax. probs, w: fp32 [T, E], [T, k]; dw: fp32 [T, k]; dlogits: bf16 [T, E].
__global__ void __launch_bounds__(MOE_THREADS) moe_route_bwd_kernel(const float* __restrict__ probs, const long long* __restrict__ topi,
                                                                   const float* __restrict__ w, const float* __restrict__ dw, int renorm,
                                                                   int T, int E, int k, bf16* __restrict__ dlogits) {
  pdl_trigger();
  pdl_wait();
  const long long t = (static_cast<long long>(blockIdx.x) * MOE_THREADS + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  const float* pr = probs + t * E;
  float dot = 0.f, sum = 0.f;      // sum_s dw_s w_s and sum of the chosen probabilities
  for (int s = lane; s < k; s += 32) { dot += dw[t * k + s] * w[t * k + s]; sum += pr[topi[t * k + s]]; }
  dot = warp_sum(dot); sum = warp_sum(sum);
  auto dtop = [&](int s) { return renorm ? (dw[t * k + s] - dot) / sum : dw[t * k + s]; };
  float inner = 0.f;               // sum_e dprobs_e probs_e: only chosen experts have a dprobs
  for (int s = lane; s < k; s += 32) inner += dtop(s) * pr[topi[t * k + s]];
  inner = warp_sum(inner);
  for (int e = lane; e < E; e += 32) {
    float dp = 0.f;
    for (int s = 0; s < k; ++s) if (topi[t * k + s] == e) dp = dtop(s);
    dlogits[t * E + e] = __float2bfloat16(pr[e] * (dp - inner));
  }
}

static inline int ok() { return cudaGetLastError() == cudaSuccess ? 0 : -5; }

}  // namespace mtb

extern "C" {
using namespace mtb;

// topi: [n] int64 chosen experts of n = T * k pairs; pair_of: [cap], cap a multiple of GROUP_ALIGN and at least
// n + E * (GROUP_ALIGN - 1); row_of: [n]; starts: [E + 1]; counts: [E]. All int32.
int mtb200_moe_plan(const long long* topi, int n, int E, int cap, int* starts, int* counts, int* pair_of, int* row_of, int* status,
                    cudaStream_t st) {
  if (n <= 0) return 0;
  if (E <= 0 || E > GROUP_MAX || cap % GROUP_ALIGN || cap < static_cast<long long>(n) + static_cast<long long>(E) * (GROUP_ALIGN - 1)) return -10;
  launch_pdl(moe_plan_kernel, E, PLAN_THREADS, 0, st, topi, n, E, cap, starts, counts, pair_of, row_of, status);
  return ok();
}

// probs [T, E], w [T, k]: fp32; topi [T, k]: int64.
int mtb200_moe_route(const void* logits, int T, int E, int k, int renorm, float* probs, long long* topi, float* w, cudaStream_t st) {
  if (T <= 0) return 0;
  if (E <= 0 || E > GROUP_MAX || k <= 0 || k > 32 || k > E) return -10;
  launch_pdl(moe_route_kernel, (T + MOE_THREADS / 32 - 1) / (MOE_THREADS / 32), MOE_THREADS, 0, st, (const bf16*)logits, T, E, k, renorm, probs, topi, w);
  return ok();
}

int mtb200_moe_gather(const void* src, const int* pair_of, const int* starts, int E, int k, int cap, int H, float scale, void* out,
                      cudaStream_t st) {
  if (cap <= 0) return 0;
  if (H % 8 || k <= 0) return -10;
  launch_pdl(moe_gather_kernel, (cap + GATHER_WARPS - 1) / GATHER_WARPS, 32 * GATHER_WARPS, 0, st, (const bf16*)src, pair_of, starts, E, k, cap, H, scale, (bf16*)out);
  return ok();
}

// act: 0 SiLU, 1 tanh-approximated GELU
int mtb200_moe_glu_bwd(void* du, const void* gu, const float* w, const int* pair_of, const int* starts, int E, int cap, int F, int act,
                       void* dgu, float* dw, cudaStream_t st) {
  if (cap <= 0) return 0;
  if (F % 8) return -10;
  // a row of at most 2048 elements (eight vectors a lane) is a warp's, which needs no barrier; a thread of a wider one gets at least two vectors
#define GB(ACT, TPR) launch_pdl(moe_glu_bwd_kernel<ACT, TPR>, (cap + MOE_THREADS / TPR - 1) / (MOE_THREADS / TPR), MOE_THREADS, 0, st, (bf16*)du, (const bf16*)gu, w, pair_of, starts, E, cap, F, (bf16*)dgu, dw)
#define GBT(ACT) if (F <= 2048) GB(ACT, 32); else if (F <= 4096) GB(ACT, 128); else GB(ACT, 256)
  if (act == 0) { GBT(0); } else { GBT(1); }
#undef GBT
#undef GB
  return ok();
}

int mtb200_moe_combine(const void* rows, const int* row_of, const float* w, const float* add, const void* base, float scale, int T, int k,
                       int H, void* out, cudaStream_t st) {
  if (T <= 0) return 0;
  if (H % 8 || k <= 0) return -10;
  launch_pdl(moe_combine_kernel, T, MOE_THREADS, 0, st, (const bf16*)rows, row_of, w, add, (const bf16*)base, scale, k, H, (bf16*)out);
  return ok();
}

int mtb200_moe_route_bwd(const float* probs, const long long* topi, const float* w, const float* dw, int renorm, int T, int E, int k,
                         void* dlogits, cudaStream_t st) {
  if (T <= 0) return 0;
  if (E <= 0 || k <= 0) return -10;
  launch_pdl(moe_route_bwd_kernel, (T + MOE_THREADS / 32 - 1) / (MOE_THREADS / 32), MOE_THREADS, 0, st, probs, topi, w, dw, renorm, T, E, k, (bf16*)dlogits);
  return ok();
}

}  // extern "C"
