// Epilogue shared by the tcgen05 GEMM kernels: a warp turns its 32 rows x 256 columns of an fp32 accumulator in tensor
// memory into output rows (alpha, bias, residual, conversion), and the split-K form of it.
//
// Split-K: a tile's k-blocks are divided over `splits` work items when whole tiles would leave SMs idle (a weight gradient
// with few tiles and a long reduction, the tail of a two-wave grid). Every item leaves its fp32 partial in a workspace; the
// warp that arrives last at the counter of a (tile, 32-row quarter) adds the partials in split order and runs the ordinary
// epilogue. Nobody waits for anybody (the items may run in any order, on any number of SMs), the sum has one fixed order
// whoever arrives last. A counter counts the arrivals of one launch, named by its epoch: whatever an earlier launch that gave up has
// left there does not count. 1536 x 1536 x 5987 (72 tiles on 148 SMs): 40 -> 33 us,
// 3720 x 1536 x 151936 (180 tiles): 1791 -> 1231 us.
#pragma once
#include "ptx.cuh"

namespace mtb {

struct EpiParams {
  int M, N;
  const void* R;          // optional residual / accumulate source, same dtype as D
  long long ldr;
  const __nv_bfloat16* bias;  // optional, [N]
  float alpha;            // the product is multiplied by alpha before bias and residual are added
  int splits;             // work items per tile
  float* ws;              // splits > 1: partials, SPLIT_UNIT floats per (128-row unit, split)
  float2* stats;          // optional (bf16 output): per row and column tile, maximum and sum of exp(x - maximum) of the stored
                          // values, [M, ceil(N / 256)]; saves the cross-entropy its first pass over the logits
  unsigned long long* counters;   // splits > 1: one arrival counter per (128-row unit, quarter)
  unsigned long long epoch;       // splits > 1: number of this launch, larger than that of any launch before it on these counters
};

constexpr int SPLIT_COUNTERS = 4096;
constexpr int SPLIT_UNIT = 128 * 256;   // floats of one partial: 128 rows x 256 columns

// Arrival at a counter (one thread); true for the last of the launch's `splits` arrivals. The two operations of a thread on one
// address are performed in order, so the count starts from this launch's epoch whatever was there. The caller sets the counter
// to zero once the partials are added, which makes the order of the epochs matter only after a launch that gave up.
__device__ __forceinline__ bool last_arrival(unsigned long long* counter, unsigned long long epoch, int splits) {
  atomicMax(counter, epoch << 16);
  return atomicAdd(counter, 1ull) == (epoch << 16) + static_cast<unsigned long long>(splits - 1);
}

// Running maximum and sum of exponentials of a row.
struct RowStats {
  float m = -INFINITY, s = 0.f;
};

// Eight bf16 values. Exponentials in two instructions (exp_ftz): of 3 us per tile that the statistics take where nothing hides them, a third
// (logits and gradient of 8000 x 32000 x 1536: 848 -> 792 us).
template <typename Stats>
__device__ __forceinline__ void row_stats8(Stats& st, uint4 o) {
  const float2 r0 = unpack_bf16(o.x), r1 = unpack_bf16(o.y), r2 = unpack_bf16(o.z), r3 = unpack_bf16(o.w);
  const float mx = fmaxf(fmax3(fmaxf(r0.x, r0.y), r1.x, r1.y), fmax3(fmaxf(r2.x, r2.y), r3.x, r3.y));
  if (mx > st.m) { st.s *= exp_ftz(st.m - mx); st.m = mx; }
  const auto base = st.m == -INFINITY ? 0.f : st.m;   // nothing but -infinity so far
  st.s += exp_ftz(r0.x - base) + exp_ftz(r0.y - base) + exp_ftz(r1.x - base) + exp_ftz(r1.y - base) + exp_ftz(r2.x - base) +
          exp_ftz(r2.y - base) + exp_ftz(r3.x - base) + exp_ftz(r3.y - base);
}

// Output staging. A row of a tile belongs to one thread, so storing it directly sends 32 half-sectors to 32 rows with every
// instruction: a 128 x 256 tile cost about 4000 clocks of the load/store unit, more than its MMAs when the reduction is short.
// A warp stages 128 bytes of each of its 32 rows in shared memory (128B-swizzled, conflict-free) and one TMA store writes the
// box, clipped to the matrix, while the next columns are read (5987 x 1536 x 1536: 28.6 -> 24.6 us, 5987 x 17920 x 1536: 270 -> 250 us;
// long reductions hide either form).
constexpr int STORE_BOX = 32 * 128;                  // bytes of one staged box: 32 rows x 128 bytes
constexpr int EPI_SMEM = 4 * 2 * STORE_BOX;          // four epilogue warps, two boxes each

struct EpiOut {
  const void* map;      // tensor map of D, box 32 rows x 128 bytes
  uint8_t* stage;       // this warp's two boxes
  int z;                // matrix of a 3-D map, or -1
  uint32_t n;           // boxes so far
};

// Buffer for the next box, of a warp's BOXES: free once at most the other buffer's store is still reading. Every box that is taken here is
// stored and committed, or the count of pending groups would no longer name the buffer.
template <int BOXES = 2>
__device__ __forceinline__ uint8_t* next_box(EpiOut& o, int lane) {
  if (lane == 0) bulk_wait_read<BOXES - 1>();
  __syncwarp();
  return o.stage + (BOXES == 2 ? (o.n & 1) * STORE_BOX : 0);
}
__device__ __forceinline__ void store_box(EpiOut& o, const uint8_t* box, int x, int y, int lane) {
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    if (o.z < 0) tma_store_2d(o.map, box, x, y);
    else tma_store_3d(o.map, box, x, y, o.z);
    bulk_commit();
  }
  ++o.n;
}
// Before the CTA's shared memory goes away.
__device__ __forceinline__ void drain_boxes() { bulk_wait_read<0>(); }

// 32 accumulator columns of one row through alpha, bias and residual, into the staged row `srow` (`part`: which 64 bytes of a
// bf16 box; an fp32 box holds 32 columns). Columns past N and rows past M are computed from nothing and clipped by the store.
template <bool OUT_F32, bool STATS, bool EXTRA>
__device__ __forceinline__ void epilogue_row32(const EpiParams& p, float (&f)[32], int row, bool row_ok, int col0, uint8_t* srow, int part, int lane,
                                               RowStats& st) {
#pragma unroll
  for (int j = 0; j < 32; ++j) f[j] *= p.alpha;
  if (EXTRA && p.bias != nullptr) {
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
  const bool res = EXTRA && p.R != nullptr && row_ok;
  if constexpr (OUT_F32) {
    const float* rptr = reinterpret_cast<const float*>(p.R) + static_cast<long long>(row) * p.ldr + col0;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      float4 o = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
      if (res && col0 + j < p.N) { const float4 r = *reinterpret_cast<const float4*>(rptr + j); o.x += r.x; o.y += r.y; o.z += r.z; o.w += r.w; }
      *reinterpret_cast<float4*>(srow + (((j >> 2) ^ (lane & 7)) << 4)) = o;
    }
  } else {
    const __nv_bfloat16* rptr = reinterpret_cast<const __nv_bfloat16*>(p.R) + static_cast<long long>(row) * p.ldr + col0;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      if (res && col0 + j < p.N) {
        const uint4 r = *reinterpret_cast<const uint4*>(rptr + j);
        const float2 r0 = unpack_bf16(r.x), r1 = unpack_bf16(r.y), r2 = unpack_bf16(r.z), r3 = unpack_bf16(r.w);
        f[j] += r0.x; f[j + 1] += r0.y; f[j + 2] += r1.x; f[j + 3] += r1.y;
        f[j + 4] += r2.x; f[j + 5] += r2.y; f[j + 6] += r3.x; f[j + 7] += r3.y;
      }
      uint4 o;
      o.x = pack_bf16(f[j], f[j + 1]); o.y = pack_bf16(f[j + 2], f[j + 3]);
      o.z = pack_bf16(f[j + 4], f[j + 5]); o.w = pack_bf16(f[j + 6], f[j + 7]);
      *reinterpret_cast<uint4*>(srow + (((part * 4 + (j >> 3)) ^ (lane & 7)) << 4)) = o;
      if constexpr (STATS) {
        if (col0 + j < p.N) row_stats8(st, o);   // of the values as stored
      }
    }
  }
}

// Split-K: this warp's 32 x COLS fp32 partial to the workspace, as lane-interleaved 16-byte pieces, so that every store and load is one contiguous
// 512 bytes; pieces past N are left out. `drained` is called when the accumulator has been read. True for the warp that arrives last.
template <int COLS = 256, typename Drained>
__device__ __forceinline__ bool leave_partial(const EpiParams& p, uint32_t taddr, int tn0, int q, int lane, int unit, int split, Drained drained) {
  float* mine = p.ws + (static_cast<long long>(unit) * p.splits + split) * (128 * COLS) + q * 32 * COLS + lane * 4;
#pragma unroll 1
  for (int c = 0; c < COLS / 32; ++c) {
    if (tn0 + c * 32 >= p.N) break;
    uint32_t v[32];
    tmem_ld_32x32(taddr + c * 32, v);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j)
      __stcg(reinterpret_cast<float4*>(mine + c * 1024 + j * 128),
             make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])));
  }
  drained();
  __threadfence();
  __syncwarp();
  unsigned last = 0;
  if (lane == 0) last = last_arrival(p.counters + unit * 4 + q, p.epoch, p.splits);
  last = __shfl_sync(0xffffffffu, last, 0);
  if (last) __threadfence();
  return last != 0;
}
// 32 columns (piece `c`) of the sum of a unit's partials, in split order.
template <int COLS = 256>
__device__ __forceinline__ void sum_partials(const EpiParams& p, float (&f)[32], int tn0, int c, int q, int lane, int unit) {
#pragma unroll
  for (int j = 0; j < 32; ++j) f[j] = 0.f;
  if (tn0 + c * 32 >= p.N) return;   // never written
  const float* base = p.ws + static_cast<long long>(unit) * p.splits * (128 * COLS) + q * 32 * COLS + lane * 4 + c * 1024;
#pragma unroll 2
  for (int s = 0; s < p.splits; ++s) {
    const float* src = base + static_cast<long long>(s) * (128 * COLS);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 v = __ldcg(reinterpret_cast<const float4*>(src + j * 128));
      f[4 * j] += v.x; f[4 * j + 1] += v.y; f[4 * j + 2] += v.z; f[4 * j + 3] += v.w;
    }
  }
}

// One warp's part of a work item: quarter `q` of the 128-row unit that starts at row `row0`, columns [tn0, tn0 + COLS).
// `taddr`: tensor-memory address of the quarter. `unit`: index of the 128-row unit among all tiles' units. `zero`: the item
// had nothing to multiply, the accumulator holds an older tile. SPLIT = false leaves the split-K part out, STATS = false the
// statistics, EXTRA = false bias and residual: a worker walks this code once per tile, and what it does not need has to be fetched
// and branched around all the same. With the statistics as a run-time branch in every product a launch of one wave took 2 us
// more (384 x 2048 x 2048: 18.6 and 16.5 us, 4736 x 1024 x 512: 11.3 and 10.4), with bias and residual another step for some
// (824 x 80 x 824: 12.3 and 10.6 us; on pairs 40000 x 768 x 768: 45.2 and 43.2).
template <bool OUT_F32, bool SPLIT, bool STATS, bool EXTRA, int COLS = 256>
__device__ __forceinline__ void epilogue_quarter(const EpiParams& p, EpiOut& out, uint32_t taddr, int row0, int tn0, int q, int lane,
                                                 int unit, int split, bool zero) {
  constexpr int PARTS = OUT_F32 ? 1 : 2;      // 32-column pieces per box
  if (row0 + q * 32 >= p.M) return;           // none of this warp's rows exist: nothing to stage, store or count
  const int row = row0 + q * 32 + lane;
  const bool row_ok = row < p.M;
  RowStats st;
  auto finish = [&]() {
    if (STATS && row_ok && tn0 < p.N)
      p.stats[static_cast<long long>(row) * ((p.N + 255) / 256) + tn0 / 256] = make_float2(st.m, st.s);
  };
  if (!SPLIT || p.splits == 1) {
#pragma unroll 1
    for (int c = 0; c < COLS / 32; c += PARTS) {
      const int col0 = tn0 + c * 32;
      if (col0 >= p.N) break;  // uniform across the warp
      uint32_t v[PARTS][32];
#pragma unroll
      for (int k = 0; k < PARTS; ++k) tmem_ld_32x32(taddr + (c + k) * 32, v[k]);
      uint8_t* box = next_box(out, lane);
      tmem_ld_wait();
#pragma unroll
      for (int k = 0; k < PARTS; ++k) {
        float f[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = zero ? 0.f : __uint_as_float(v[k][j]);
        epilogue_row32<OUT_F32, STATS, EXTRA>(p, f, row, row_ok, col0 + k * 32, box + lane * 128, k, lane, st);
      }
      store_box(out, box, col0, row0 + q * 32, lane);
    }
    finish();
    return;
  }
  if (!leave_partial<COLS>(p, taddr, tn0, q, lane, unit, split, [] {})) return;
#pragma unroll 1
  for (int c = 0; c < COLS / 32; c += PARTS) {
    const int col0 = tn0 + c * 32;
    if (col0 >= p.N) break;
    uint8_t* box = next_box(out, lane);
#pragma unroll 1
    for (int k = 0; k < PARTS; ++k) {
      float f[32];
      sum_partials<COLS>(p, f, tn0, c + k, q, lane, unit);
      epilogue_row32<OUT_F32, STATS, EXTRA>(p, f, row, row_ok, col0 + k * 32, box + lane * 128, k, lane, st);
    }
    store_box(out, box, col0, row0 + q * 32, lane);
  }
  finish();
  if (lane == 0) p.counters[unit * 4 + q] = 0;
}

// Wide tiles (gemm2_tcgen05.cu): the same part of an item for the eight epilogue warps of a CTA, one box each. The accumulator is wanted back at
// once, and reading it is the short part of an epilogue: `drained` is called when the 256 columns are in registers, rounded (`row_end`: the first row
// that is not the item's; `zero`: it had nothing to multiply; bias and residual come before the rounding, so with them the columns are stored as they
// are read; fp32 columns would not fit). 16384 x 28672 x 4096 in a loop at the power cap: 1320 TFLOP/s storing as it reads, 1413 this way. One box with rows
// of 128 bytes per warp is better than two with rows of 64, which cost the copy engine as many requests each: 75776 x 4096 x 512 269 -> 249 us, x 64 133 -> 125.
//
// Formed here: the compiler would move the rounding to where the value is stored, past `drained`, and hold the fp32 values until then.
__device__ __forceinline__ uint32_t formed(uint32_t x) {
  asm volatile("" : "+r"(x));
  return x;
}
// A loop over pieces that are held in registers works on the first of them and moves the others up: unrolled, the arithmetic of several pieces is
// started together and the registers spill.
template <int N, int BY>
__device__ __forceinline__ void next_pieces(uint32_t (*d)[16]) {
#pragma unroll
  for (int c = 0; c + BY < N; ++c)
#pragma unroll
    for (int j = 0; j < 16; ++j) d[c][j] = d[c + BY][j];
}
// 64 columns of this thread's row, in two pieces.
__device__ __forceinline__ void send_columns64(EpiOut& out, const uint32_t (*d)[16], int col0, int y0, int lane) {
  uint8_t* box = next_box<1>(out, lane);
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<uint4*>(box + lane * 128 + (((k * 4 + i) ^ (lane & 7)) << 4)) = make_uint4(d[k][4 * i], d[k][4 * i + 1], d[k][4 * i + 2], d[k][4 * i + 3]);
  store_box(out, box, col0, y0, lane);
}
template <bool OUT_F32, bool SPLIT, bool STATS, bool EXTRA, typename Drained>
__device__ __forceinline__ void epilogue_wide(const EpiParams& p, EpiOut& out, uint32_t taddr, int row0, int row_end, int tn0, int q, int lane, int unit,
                                              int split, bool zero, Drained drained) {
  constexpr int PARTS = OUT_F32 ? 1 : 2;
  const int y0 = row0 + q * 32, row = y0 + lane;
  if (y0 >= row_end) { drained(); return; }
  const bool row_ok = row < row_end;
  RowStats st;
  auto finish = [&]() {
    if (STATS && row_ok && tn0 < p.N) p.stats[static_cast<long long>(row) * ((p.N + 255) / 256) + tn0 / 256] = make_float2(st.m, st.s);
  };
  const bool partial = SPLIT && p.splits > 1;
  if (partial && !leave_partial(p, taddr, tn0, q, lane, unit, split, drained)) return;
  if (partial || EXTRA || OUT_F32) {
#pragma unroll 1
    for (int c = 0; c < 8 && tn0 + c * 32 < p.N; c += PARTS) {
      uint8_t* box = next_box<1>(out, lane);
#pragma unroll
      for (int k = 0; k < PARTS; ++k) {
        float f[32];
        if (partial) {
          sum_partials(p, f, tn0, c + k, q, lane, unit);
        } else {
          uint32_t v[32];
          tmem_ld_32x32(taddr + (c + k) * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
        }
        epilogue_row32<OUT_F32, STATS, EXTRA>(p, f, row, row_ok, tn0 + (c + k) * 32, box + lane * 128, k, lane, st);
      }
      store_box(out, box, tn0 + c * 32, y0, lane);
    }
    if (partial) { if (lane == 0) p.counters[unit * 4 + q] = 0; }
    else drained();
  } else {
    uint32_t d[8][16];
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      uint32_t v[2][32];
      tmem_ld_32x32(taddr + c * 32, v[0]);
      tmem_ld_32x32(taddr + c * 32 + 32, v[1]);
      tmem_ld_wait();
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 16; ++j) d[c + k][j] = zero ? 0u : formed(pack_bf16(__uint_as_float(v[k][2 * j]) * p.alpha, __uint_as_float(v[k][2 * j + 1]) * p.alpha));
    }
    drained();
    if constexpr (STATS) {
#pragma unroll 1
      for (int c = 0; c < 8 && tn0 + c * 32 < p.N; c += 2) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (tn0 + c * 32 + i * 8 < p.N) row_stats8(st, make_uint4(d[i / 4][i % 4 * 4], d[i / 4][i % 4 * 4 + 1], d[i / 4][i % 4 * 4 + 2], d[i / 4][i % 4 * 4 + 3]));
        send_columns64(out, d, tn0 + c * 32, y0, lane);
        next_pieces<8, 2>(d);
      }
    } else {
#pragma unroll
      for (int c = 0; c < 8; c += 2)
        if (tn0 + c * 32 < p.N) send_columns64(out, d + c, tn0 + c * 32, y0, lane);
    }
  }
  finish();
}

// Products of at most this many operations start under their predecessor's tail (launch_pdl). It saves about 2 us per launch whatever the
// size; on the other hand CTAs that are placed as SMs fall free, instead of in order, take neighbouring tiles to distant SMs, and
// long launches lose what that saves (this rule and every product early, in one process: 1.5B, q/k-norm and LayerNorm blocks within 1 %, which is
// their spread; 8B block 19.92 and 20.08 ms, LM head 4.66 and 4.73, eight-expert layer 7.88 and 8.13, sixty-four experts 1019 and 1040 us).
constexpr double PDL_MAX_FLOPS = 1e12;
// Grouped products, counted over the whole row buffers: 477 tokens through 4 experts of 2760 (0.01 TFLOP) 311 -> 301 us, 878 through 32 of 1080 (0.05) 350 -> 342;
// 2051 through 64 of 1024 (0.2) is the slower early.
constexpr float PDL_MAX_GROUPED_FLOPS = 1e11f;

// Grouped GEMM: one launch over the slabs of all experts of a mixture-of-experts layer. The rows of expert e are
// [starts[e], starts[e] + counts[e]) of the gathered row buffers, starts are multiples of GROUP_ALIGN and the rows between the
// slabs are zero, so a row tile never mixes experts and a reduction over a slab may run into its padding. The row counts are
// only known on the device: the host launches for the most tiles there can be.
//   ROWS    D[rows, N] = A[rows, K] * W_e: A and D hold the slabs, the weights are one 3-D tensor [E, ., .]
//   REDUCE  D_e = A[rows_e, M]^T * B[rows_e, N]: one output matrix per expert, zeros for an expert without rows
// One launch per product instead of one per expert: forward + backward of 4096 tokens through 8 experts of 4096 x 14336
// (2 chosen) 12.4 -> 8.2 ms, of 2051 tokens through 64 experts of 2048 x 1024 (8 chosen) 12.7 -> 1.1 ms, where the loop was bound by
// its 1200 launches and a grid of a few tiles per expert.
enum { GROUP_NONE = 0, GROUP_ROWS = 1, GROUP_REDUCE = 2 };
constexpr int GROUP_ALIGN = 128;
constexpr int GROUP_MAX = 256;   // experts

struct GroupParams {
  const int* starts;     // [E + 1]
  const int* counts;     // [E]
  int E;
  float flops;           // of the launch, at most: on all of the row buffers
};

// Work items of a grouped launch in shared memory: tile_start[e] is the first tile of expert e. (Slab starts and counts are read
// from global memory where they are needed, once per tile: shared memory is full.)
struct GroupTable {
  int tile_start[GROUP_MAX + 1];
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
    if (e < g.E) tab.tile_start[e] = base + incl - n;
    base += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) tab.tile_start[g.E] = base;
}

// Whether a split launch over `units` 128-row units fits its scratch and leaves every item a k-block.
inline bool split_fits(const EpiParams& e, long long units, int kblocks, long long part_bytes, int unit_floats = SPLIT_UNIT) {
  return e.ws != nullptr && e.counters != nullptr && e.splits <= kblocks && units * 4 <= SPLIT_COUNTERS &&
         units * e.splits * unit_floats * 4 <= part_bytes;
}

}  // namespace mtb
