// Epilogue shared by the tcgen05 GEMM kernels: a warp turns its 32 rows x 256 columns of an fp32 accumulator in tensor
// memory into output rows (alpha, bias, residual, conversion), and the split-K form of it.
//
// Split-K: a tile's k-blocks are divided over `splits` work items when whole tiles would leave SMs idle (a weight gradient
// with few tiles and a long reduction, the tail of a two-wave grid). Every item leaves its fp32 partial in a workspace; the
// warp that arrives last at the counter of a (tile, 32-row quarter) adds the partials in split order and runs the ordinary
// epilogue. Nobody waits for anybody (the items may run in any order, on any number of SMs), the sum has one fixed order
// whoever arrives last, and the counters are back at zero when the launch ends.
#pragma once
#include "ptx.cuh"

namespace mtb {

struct EpiParams {
  int M, N;
  void* D;
  long long ldd;
  const void* R;          // optional residual / accumulate source, same dtype as D
  long long ldr;
  const __nv_bfloat16* bias;  // optional, [N]
  float alpha;            // the product is multiplied by alpha before bias and residual are added
  int splits;             // work items per tile
  float* ws;              // splits > 1: partials, SPLIT_UNIT floats per (128-row unit, split)
  unsigned* counters;     // splits > 1: one arrival counter per (128-row unit, quarter); zero between launches
};

constexpr int SPLIT_COUNTER_BYTES = 16384;
constexpr int SPLIT_UNIT = 128 * 256;   // floats of one partial: 128 rows x 256 columns

// 32 accumulator columns of one row -> D. `col0` < N; columns past N are not stored.
template <bool OUT_F32>
__device__ __forceinline__ void epilogue_row32(const EpiParams& p, float (&f)[32], int row, int col0) {
#pragma unroll
  for (int j = 0; j < 32; ++j) f[j] *= p.alpha;
  if (p.bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      if (col0 + j < p.N) {
        const uint4 b = *reinterpret_cast<const uint4*>(p.bias + col0 + j);
        const float2 b0 = unpack_bf16(b.x), b1 = unpack_bf16(b.y), b2 = unpack_bf16(b.z), b3 = unpack_bf16(b.w);
        f[j] += b0.x; f[j + 1] += b0.y; f[j + 2] += b1.x; f[j + 3] += b1.y;
        f[j + 4] += b2.x; f[j + 5] += b2.y; f[j + 6] += b3.x; f[j + 7] += b3.y;
      }
    }
  }
  if constexpr (OUT_F32) {
    float* dptr = reinterpret_cast<float*>(p.D) + static_cast<long long>(row) * p.ldd + col0;
    const float* rptr = p.R ? reinterpret_cast<const float*>(p.R) + static_cast<long long>(row) * p.ldr + col0 : nullptr;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      if (col0 + j < p.N) {
        float4 o = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
        if (rptr) { const float4 r = *reinterpret_cast<const float4*>(rptr + j); o.x += r.x; o.y += r.y; o.z += r.z; o.w += r.w; }
        *reinterpret_cast<float4*>(dptr + j) = o;
      }
    }
  } else {
    __nv_bfloat16* dptr = reinterpret_cast<__nv_bfloat16*>(p.D) + static_cast<long long>(row) * p.ldd + col0;
    const __nv_bfloat16* rptr = p.R ? reinterpret_cast<const __nv_bfloat16*>(p.R) + static_cast<long long>(row) * p.ldr + col0 : nullptr;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      if (col0 + j < p.N) {
        if (rptr) {
          const uint4 r = *reinterpret_cast<const uint4*>(rptr + j);
          const float2 r0 = unpack_bf16(r.x), r1 = unpack_bf16(r.y), r2 = unpack_bf16(r.z), r3 = unpack_bf16(r.w);
          f[j] += r0.x; f[j + 1] += r0.y; f[j + 2] += r1.x; f[j + 3] += r1.y;
          f[j + 4] += r2.x; f[j + 5] += r2.y; f[j + 6] += r3.x; f[j + 7] += r3.y;
        }
        uint4 o;
        o.x = pack_bf16(f[j], f[j + 1]); o.y = pack_bf16(f[j + 2], f[j + 3]);
        o.z = pack_bf16(f[j + 4], f[j + 5]); o.w = pack_bf16(f[j + 6], f[j + 7]);
        *reinterpret_cast<uint4*>(dptr + j) = o;
      }
    }
  }
}

// One warp's part of a work item: quarter `q` of the 128-row unit that starts at row `row0`, columns [tn0, tn0 + 256).
// `taddr`: tensor-memory address of the quarter. `unit`: index of the 128-row unit among all tiles' units.
// SPLIT = false (the gathering kernels, which never split) leaves the split-K part out.
template <bool OUT_F32, bool SPLIT>
__device__ __forceinline__ void epilogue_quarter(const EpiParams& p, uint32_t taddr, int row0, int tn0, int q, int lane,
                                                 int unit, int split) {
  const int row = row0 + q * 32 + lane;
  const bool row_ok = row < p.M;
  if (!SPLIT || p.splits == 1) {
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
      const int col0 = tn0 + c * 32;
      if (col0 >= p.N) break;  // uniform across the warp
      uint32_t v[32];
      tmem_ld_32x32(taddr + c * 32, v);
      tmem_ld_wait();
      if (row_ok) {
        float f[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
        epilogue_row32<OUT_F32>(p, f, row, col0);
      }
    }
    return;
  }
  // partial to the workspace: lane-interleaved 16-byte pieces, so every store and load is one contiguous 512 bytes
  float* mine = p.ws + (static_cast<long long>(unit) * p.splits + split) * SPLIT_UNIT + q * 8192 + lane * 4;
#pragma unroll 1
  for (int c = 0; c < 8; ++c) {
    if (tn0 + c * 32 >= p.N) break;
    uint32_t v[32];
    tmem_ld_32x32(taddr + c * 32, v);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j)
      __stcg(reinterpret_cast<float4*>(mine + c * 1024 + j * 128),
             make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])));
  }
  __threadfence();
  __syncwarp();
  unsigned old = 0;
  if (lane == 0) old = atomicAdd(p.counters + unit * 4 + q, 1u);
  old = __shfl_sync(0xffffffffu, old, 0);
  if (old != static_cast<unsigned>(p.splits) - 1) return;
  __threadfence();
  const float* base = p.ws + static_cast<long long>(unit) * p.splits * SPLIT_UNIT + q * 8192 + lane * 4;
#pragma unroll 1
  for (int c = 0; c < 8; ++c) {
    const int col0 = tn0 + c * 32;
    if (col0 >= p.N) break;
    float f[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = 0.f;
#pragma unroll 2
    for (int s = 0; s < p.splits; ++s) {
      const float* src = base + static_cast<long long>(s) * SPLIT_UNIT + c * 1024;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(src + j * 128));
        f[4 * j] += v.x; f[4 * j + 1] += v.y; f[4 * j + 2] += v.z; f[4 * j + 3] += v.w;
      }
    }
    if (row_ok) epilogue_row32<OUT_F32>(p, f, row, col0);
  }
  if (lane == 0) p.counters[unit * 4 + q] = 0;
}

// The same part of an output tile without a product.
template <bool OUT_F32>
__device__ __forceinline__ void epilogue_zero(const EpiParams& p, int row0, int tn0, int q, int lane) {
  const int row = row0 + q * 32 + lane;
  if (row >= p.M) return;
#pragma unroll 1
  for (int c = 0; c < 8 && tn0 + c * 32 < p.N; ++c) {
    float f[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = 0.f;
    epilogue_row32<OUT_F32>(p, f, row, tn0 + c * 32);
  }
}

// Grouped GEMM: one launch over the slabs of all experts of a mixture-of-experts layer. The rows of expert e are
// [starts[e], starts[e] + counts[e]) of the gathered row buffers, starts are multiples of GROUP_ALIGN and the rows between the
// slabs are zero, so a row tile never mixes experts and a reduction over a slab may run into its padding. The row counts are
// only known on the device: the host launches for the most tiles there can be.
//   ROWS    D[rows, N] = A[rows, K] * W_e: A and D hold the slabs, the weights are one 3-D tensor [E, ., .]
//   REDUCE  D_e = A[rows_e, M]^T * B[rows_e, N]: one output matrix per expert, zeros for an expert without rows
// One launch per product instead of one per expert: forward + backward of 4096 tokens through 8 experts of 4096 x 14336
// (2 chosen) 12.2 -> 7.6 ms, of 2051 tokens through 64 experts of 2048 x 1024 (8 chosen) 12.3 -> 1.2 ms, where the loop was bound by
// its 1200 launches and a grid of a few tiles per expert.
enum { GROUP_NONE = 0, GROUP_ROWS = 1, GROUP_REDUCE = 2 };
constexpr int GROUP_ALIGN = 128;
constexpr int GROUP_MAX = 256;   // experts

struct GroupParams {
  const int* starts;     // [E + 1]
  const int* counts;     // [E]
  int E;
  long long d_stride;    // REDUCE: elements between two experts' outputs
};

// Work items of a grouped launch in shared memory: tile_start[e] is the first tile of expert e.
struct GroupTable {
  int tile_start[GROUP_MAX + 1];
  int row[GROUP_MAX], rows[GROUP_MAX];
};

// Filled by one warp; the caller synchronises the block.
template <int GROUP>
__device__ __forceinline__ void fill_group_table(GroupTable& tab, const GroupParams& g, int tile_rows, int tiles_n, int tiles_per_matrix, int lane) {
  int base = 0;
  for (int e0 = 0; e0 < g.E; e0 += 32) {
    const int e = e0 + lane;
    const int rows = e < g.E ? g.counts[e] : 0;
    int n = e < g.E ? (GROUP == GROUP_ROWS ? (rows + tile_rows - 1) / tile_rows * tiles_n : tiles_per_matrix) : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
    if (e < g.E) { tab.tile_start[e] = base + incl - n; tab.row[e] = g.starts[e]; tab.rows[e] = rows; }
    base += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) tab.tile_start[g.E] = base;
}

// Number of work items per tile (of 0.4 us k-blocks on one SM): 1 when whole tiles fill the `workers` (SMs or CTA pairs) well, else the smallest cost in
// units of one k-block of a tile: full waves of items, plus what the extra partials cost (write, one counter, ordered sum).
// `max_items`: what the workspace holds.
inline int choose_splits(long long tiles, int kblocks, int workers, long long max_items) {
  if (tiles <= 0 || workers <= 0) return 1;
  auto waves = [&](long long items) { return (items + workers - 1) / workers; };
  const double whole = static_cast<double>(waves(tiles)) * kblocks + 8.0;
  int best = 1;
  double best_cost = whole * 0.95;   // a split has to win by more than the model's error
  for (int s = 2; s <= 16; ++s) {
    if (tiles * s > max_items || kblocks / s < 6) break;
    const double cost = static_cast<double>(waves(tiles * s)) * ((kblocks + s - 1) / s + 10.0) + 14.0 + 3.0 * s;
    if (cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

}  // namespace mtb
