// Persistent, warp-specialised bf16 GEMM for sm_100a: TMA -> 128B-swizzled shared memory ->
// tcgen05.mma with the fp32 accumulator in tensor memory -> tcgen05.ld epilogue.
//
//   D[M, N] = A * B (+ bias[N]) (+ R[M, N])        bf16 inputs, fp32 accumulate, bf16 or fp32 out
//
// A is an "M x K" operand and B an "N x K" operand; each may be stored K-major (row-major
// [rows, K]) or MN-major (row-major [K, rows]), which covers the three products of a linear layer
// without any transposed copies:
//   forward  Y[T,N]  = X[T,K]  * W[N,K]^T   A K-major,  B K-major
//   dgrad    dX[T,K] = dY[T,N] * W[N,K]     A K-major,  B MN-major (W read as [red=N, out=K])
//   wgrad    dW[N,K] = dY[T,N]^T * X[T,K]   A MN-major, B MN-major (both read as [red=T, .])
//
// CTA layout (192 threads, one CTA per SM, grid = min(work items, SMs); an item is a tile, or one
// split of its reduction):
//   warp 0     TMA producer: fills a STAGES-deep ring of {A 128x64, B 256x64} tiles
//   warp 1     allocates 512 TMEM columns (two 128x256 fp32 accumulators) and issues the MMAs
//   warps 2-5  epilogue: each reads its 32-lane quarter of the accumulator, adds bias / residual,
//              converts and stores; runs concurrently with the next tile's MMAs (double buffer)
// Tiles are visited in bands of GROUP_M row-tiles so the A band stays in L2 while B streams.
//
// Out-of-range rows/columns/K are zero-filled by TMA and masked in the epilogue, so M, N and K
// need no padding (N and the leading dimensions must be multiples of 8 elements: TMA strides
// are multiples of 16 bytes).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include "entries.h"
#include "gather.cuh"
#include "gemm_act.cuh"
#include "gemm_epilogue.cuh"
#include "ptx.cuh"

namespace mtb {

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int A_TILE_BYTES = BM * BK * 2;   // 16 KB
constexpr int RING_BYTES = 4 * (A_TILE_BYTES + BN * BK * 2);   // the ring of operand stages: 4 of 128 x 256 tiles, 8 of 128 x 64
// Tiles of 128 x 64 and 128 x 128 are for products that have fewer of them than there are SMs. Such a product is a row of latencies (fill, reduction,
// epilogue, and the partial sums, which the last arrival adds alone), and narrow tiles shorten all of them: the epilogue of a tile is a quarter or
// half as long, and a long reduction is divided into few splits. 640 x 512 x 3072 20.0 -> 10.9 us (in 256 x 256 tiles adding the partials took
// 12 of them), 256 x 688 x 4096 20.0 -> 10.6, 640 x 512 x 512 6.7 -> 5.4, 1200 x 1024 x 768 8.9 -> 7.0.
constexpr int GEMM_THREADS = 192;
constexpr int gemm_threads(int act) { return act == ACT_NONE ? GEMM_THREADS : 64 + 32 * ACT_WARPS; }
constexpr int GROUP_M = 16;
constexpr int GATHER_GROUP_N = 4;   // column-tiles per band in the all-gather variant
constexpr int GEMM_SMEM = RING_BYTES + EPI_SMEM + 1024 /*alignment slack*/ + 256 /*barriers*/;

struct GemmParams {
  int M, N, K;
  int* status;            // device word; set non-zero when a bounded wait expired
  int group_m;            // row-tiles per band of the tile order
  unsigned wait_hint_ns;  // suspend-time hint of the epilogue's and the MMA thread's long waits (0: plain polling)
  unsigned wait_limit_us; // > 0: every pipeline wait is bounded by this time instead of a poll count (fused reduce + GEMM)
  EpiParams e;            // output, epilogue operands, split-K
  ActParams act;          // ACT instances
};

// The fused all-gather variant (GATHER = true) adds the gather warps and the flag checker of gather.cuh;
// its tiles are visited in bands of GATHER_GROUP_N column-tiles.
// REDUCE (with GATHER): the gathered operand is A, and it is the SUM over ranks of a region of their gradient
// buffers (reduce_chunks in gather.cuh): the gradient reduce-scatter with ownership by tensor, fused into the GEMM
// that consumes the reduced gradient (OSFT factor gradients).
// GROUP: one launch over the expert slabs of a mixture-of-experts layer (gemm_epilogue.cuh).
// STATS: softmax statistics of the output rows (EpiParams). EXTRA: bias or residual. ACT: an activation in the epilogue (gemm_act.cuh).
template <bool A_MN, bool B_MN, bool OUT_F32, bool GATHER = false, bool REDUCE = false, int GROUP = GROUP_NONE, bool STATS = false, bool EXTRA = true,
          int ACT = ACT_NONE, int NT = BN>
__global__ void __launch_bounds__(GATHER ? GEMM_THREADS + GATHER_EXTRA_THREADS : gemm_threads(ACT), 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
            const __grid_constant__ CUtensorMap tmap_d, const __grid_constant__ ActMaps<ACT> maps, GemmParams p,
            const __grid_constant__ GatherParams g, GroupParams gr) {
  constexpr int B_TILE_BYTES = NT * BK * 2, STAGE_BYTES = A_TILE_BYTES + B_TILE_BYTES, STAGES = RING_BYTES / STAGE_BYTES;
  static_assert(NT == BN || (!GATHER && !GROUP && !STATS && !ACT), "the other forms have tiles of 128 x 256");
  __shared__ GroupTable gtab;   // unused (and not allocated) outside the grouped forms
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + RING_BYTES + EPI_SMEM);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;   // [2] accumulator ready for the epilogue
  uint64_t* tempty_bar = tfull_bar + 2;       // [2] accumulator drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* verified = tmem_slot + 2;   // gather variant: tiles of this CTA whose weight chunks have all arrived
  uint32_t* ticket_slot = tmem_slot + 3;   // gather variant: broadcast of the chunk ticket among the gather warps

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (p.M + BM - 1) / BM, tiles_n = (p.N + NT - 1) / NT;
  const int num_tiles = tiles_m * tiles_n;
  const int kblocks = (p.K + BK - 1) / BK;
  const int splits = (GATHER || GROUP) ? 1 : p.e.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull_bar[a], 1); mbar_init(&tempty_bar[a], ACT ? ACT_WARPS : 4); }
    *abort_flag = 0;
    *verified = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_d);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  pdl_wait();   // nothing so far has touched global memory
  if (GROUP && warp == 2) fill_group_table<GROUP>(gtab, gr, BM, tiles_n, num_tiles, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // item = split * num_tiles + tile: neighbours share operand tiles
  const int num_items = GROUP ? gtab.tile_start[gr.E] : num_tiles * splits;
  // The grouped forms walk the experts with the items: `e` only moves forward.
  auto group_coords = [&](int w, int& e, int& tm, int& tn) {
    while (w >= gtab.tile_start[e + 1]) ++e;
    const int rows_m = GROUP == GROUP_ROWS ? (gr.counts[e] + BM - 1) / BM : tiles_m;
    const int t = w - gtab.tile_start[e];
    const int band = t / (p.group_m * tiles_n);
    const int first_m = band * p.group_m;
    const int rows = min(p.group_m, rows_m - first_m);
    const int local = t - band * p.group_m * tiles_n;
    tm = first_m + local % rows;
    tn = local / rows;
  };
  auto k_range = [&](int split, int& kb0, int& kb1) {
    kb0 = static_cast<int>(static_cast<long long>(kblocks) * split / splits);
    kb1 = static_cast<int>(static_cast<long long>(kblocks) * (split + 1) / splits);
  };
  auto tile_coords = [&](int t, int& tm, int& tn) {
    if constexpr (GATHER && !REDUCE) {
      // Bands of GROUP_N column-tiles, all row-tiles inside a band: the weight is consumed front to
      // back at an even rate over the whole launch (a band of row-tiles would need the ENTIRE weight
      // within its first band, i.e. within the first few waves, faster than the links deliver it).
      const int band = t / (GATHER_GROUP_N * tiles_m);
      const int first_n = band * GATHER_GROUP_N;
      const int cols = min(GATHER_GROUP_N, tiles_n - first_n);
      const int local = t - band * GATHER_GROUP_N * tiles_m;
      tn = first_n + local % cols;
      tm = local / cols;
      return;
    }
    const int band = t / (p.group_m * tiles_n);
    const int first_m = band * p.group_m;
    const int rows = min(p.group_m, tiles_m - first_m);
    const int local = t - band * p.group_m * tiles_n;
    tm = first_m + local % rows;
    tn = local / rows;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t it = 0, tl = 0;
      unsigned long long waited_ns = 0;
      int e = 0;
      for (int w = blockIdx.x; w < num_items; w += gridDim.x) {
        int tm, tn, kb0, kb1;
        if constexpr (GROUP != GROUP_NONE) {
          group_coords(w, e, tm, tn);
          kb0 = 0;
          kb1 = GROUP == GROUP_REDUCE ? (gr.counts[e] + BK - 1) / BK : kblocks;
        } else {
          tile_coords(w % num_tiles, tm, tn);
          k_range(w / num_tiles, kb0, kb1);
        }
        const int a_row = GROUP == GROUP_ROWS ? gr.starts[e] + tm * BM : tm * BM;   // first row of the A tile
        const int k_row = GROUP == GROUP_REDUCE ? gr.starts[e] : 0;                 // first row of the reduction
        if (GATHER) {
          // the checker warp has seen the flags of every chunk under this tile's B rows
          if (!wait_verified(verified, tl, abort_flag, waited_ns, p.wait_limit_us)) { *abort_flag = 1; atomicExch(p.status, 5); goto done; }
          asm volatile("fence.proxy.async;" ::: "memory");   // peer data was written with ordinary stores, TMA reads it
          ++tl;
        }
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&empty_bar[s], ph ^ 1, abort_flag, 0, p.wait_limit_us)) { atomicExch(p.status, 1); goto done; }
          uint8_t* sa = smem + s * STAGE_BYTES;
          uint8_t* sb = sa + A_TILE_BYTES;
          mbar_arrive_expect_tx(&full_bar[s], STAGE_BYTES);
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * 8192, &tmap_a, &full_bar[s], a_row + j * 64, k_row + kb * BK);
          } else {
            tma_load_2d(sa, &tmap_a, &full_bar[s], kb * BK, a_row);
          }
          if (B_MN) {
#pragma unroll
            for (int j = 0; j < NT / 64; ++j) {
              if constexpr (GROUP == GROUP_ROWS) tma_load_3d(sb + j * 8192, &tmap_b, &full_bar[s], tn * NT + j * 64, kb * BK, e);
              else tma_load_2d(sb + j * 8192, &tmap_b, &full_bar[s], tn * NT + j * 64, k_row + kb * BK);
            }
          } else {
            if constexpr (ACT == ACT_GLU) {   // 128 rows of the gate's weight and the same of up's
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const int row = (j ? p.act.F : 0) + tn * (NT / 2);
                if constexpr (GROUP == GROUP_ROWS) tma_load_3d(sb + j * (B_TILE_BYTES / 2), &tmap_b, &full_bar[s], kb * BK, row, e);
                else tma_load_2d(sb + j * (B_TILE_BYTES / 2), &tmap_b, &full_bar[s], kb * BK, row);
              }
            } else if constexpr (GROUP == GROUP_ROWS) tma_load_3d(sb, &tmap_b, &full_bar[s], kb * BK, tn * NT, e);
            else tma_load_2d(sb, &tmap_b, &full_bar[s], kb * BK, tn * NT);
          }
        }
      }
      if (!GATHER && (!GROUP || gr.flops <= PDL_MAX_GROUPED_FLOPS)) pdl_trigger();   // what is left is a few products and the last epilogue
      if (GATHER && g.wait_ns != nullptr) {   // exposed-communication accounting: how long this producer starved
        atomicAdd(g.wait_ns, waited_ns);
        atomicAdd(g.wait_ns + 1, 1ull);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(BM, NT, A_MN, B_MN);
      uint32_t it = 0, tl = 0;
      int e = 0;
      for (int w = blockIdx.x; w < num_items; w += gridDim.x, ++tl) {
        int kb0, kb1;
        if constexpr (GROUP != GROUP_NONE) {
          while (w >= gtab.tile_start[e + 1]) ++e;
          kb0 = 0;
          kb1 = GROUP == GROUP_REDUCE ? (gr.counts[e] + BK - 1) / BK : kblocks;
        } else {
          k_range(w / num_tiles, kb0, kb1);
        }
        const int acc = tl & 1;
        const uint32_t aph = (tl >> 1) & 1;
        if (!mbar_wait(&tempty_bar[acc], aph ^ 1, abort_flag, p.wait_hint_ns, p.wait_limit_us)) { atomicExch(p.status, 2); goto done; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * NT;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&full_bar[s], ph, abort_flag, 0, p.wait_limit_us)) { atomicExch(p.status, 3); goto done; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES);
          const uint32_t sb = sa + A_TILE_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = A_MN ? make_smem_desc(sa + k * 2048, 8192, 1024) : make_smem_desc(sa + k * 32, 16, 1024);
            const uint64_t db = B_MN ? make_smem_desc(sb + k * 2048, 8192, 1024) : make_smem_desc(sb + k * 32, 16, 1024);
            umma_bf16(d_tmem, da, db, idesc, kb != kb0 || k != 0);
          }
          umma_commit(&empty_bar[s]);   // frees the stage when these MMAs have read it
        }
        umma_commit(&tfull_bar[acc]);   // accumulator complete
      }
    }
  } else if (GATHER && warp == 6 + GATHER_THREADS / 32) {
    // ------------------------------------------------------------------ flag checker (warp 14)
    // Runs ahead of the TMA producer, so the producer thread never waits on a chain of dependent global loads.
    uint32_t tl = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++tl) {
      int tm, tn;
      tile_coords(t, tm, tn);
      // rows [tn*NT, tn*NT+NT) of the K-major weight (reduce mode: rows [tm*BM, tm*BM+BM) of the K-major A operand)
      // are one contiguous byte range of the gathered buffer
      const unsigned long long lo = g.b_byte_off + static_cast<unsigned long long>(REDUCE ? tm * BM : tn * NT) * p.K * 2;
      const int rows = REDUCE ? min(BM, p.M - tm * BM) : min(NT, p.N - tn * NT);
      const unsigned long long hi = lo + static_cast<unsigned long long>(rows) * p.K * 2 - 1;
      const bool ok = wait_chunks(g, lo, hi, lane, abort_flag, p.wait_limit_us);
      __syncwarp();
      if (!ok) {
        if (lane == 0) { *abort_flag = 1; atomicExch(p.status, 5); }
        break;
      }
      if (lane == 0) st_release_cta_shared(verified, tl + 1);
    }
  } else if (GATHER && warp >= 6) {
    // ------------------------------------------------------------------ gather warps (6..13)
    if constexpr (REDUCE) reduce_chunks<8>(g, threadIdx.x - GEMM_THREADS, ticket_slot);
    else gather_chunks(g, threadIdx.x - GEMM_THREADS, ticket_slot);
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5; with an activation 2..9)
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    uint32_t tl = 0;
    int e = 0;
    EpiOut out{&tmap_d, smem + RING_BYTES + (ACT ? (warp - 2) * 2 * ACT_BOX : q * 2 * STORE_BOX), -1, 0};
    for (int w = blockIdx.x; w < num_items; w += gridDim.x, ++tl) {
      const int t = w % num_tiles;
      int tm, tn, row0;
      if constexpr (GROUP != GROUP_NONE) group_coords(w, e, tm, tn); else tile_coords(t, tm, tn);
      row0 = tm * BM;
      if constexpr (GROUP == GROUP_ROWS) row0 += gr.starts[e];   // slabs are padded to whole tiles: every row may be stored
      if constexpr (GROUP == GROUP_REDUCE) out.z = e;
      const int acc = tl & 1;
      const uint32_t aph = (tl >> 1) & 1;
      if (!mbar_wait(&tfull_bar[acc], aph, abort_flag, p.wait_hint_ns, p.wait_limit_us)) { atomicExch(p.status, 4); goto done; }
      tc_fence_after();
      if constexpr (ACT != ACT_NONE)
        epilogue_act<ACT>(p.e, p.act, maps, out, tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * NT, row0, tn, q, (warp - 2) >> 2, lane);
      else epilogue_quarter<OUT_F32, !GATHER && !GROUP, STATS, EXTRA && !GROUP, NT>(p.e, out, tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * NT, row0, tn * NT, q, lane, t,
                                                   w / num_tiles, GROUP == GROUP_REDUCE && gr.counts[e] == 0);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[acc]);
    }
  }
done:
  if (warp >= 2 && (ACT || warp < 6) && lane == 0) drain_boxes();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
int make_tmap_2d_f32(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                     uint32_t box_inner, uint32_t box_outer);
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// 2-D bf16 tensor map over a row-major [outer, inner] matrix with leading dimension `ld`.
int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 2) % 16) return -2;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// Same for an fp32 matrix (box_inner * 4 bytes must not exceed the 128-byte swizzle span).
int make_tmap_2d_f32(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                     uint32_t box_inner, uint32_t box_outer) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 4) % 16 || box_inner * 4 > 128) return -2;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * 4};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// 3-D bf16 tensor map over `n` row-major [outer, inner] matrices, `stride` elements from one to the next.
int make_tmap_3d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t n, uint64_t stride,
                      uint32_t box_inner, uint32_t box_outer) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || inner % 8 || stride % 8) return -2;
  cuuint64_t dims[3] = {inner, outer, n};
  cuuint64_t strides[2] = {inner * 2, stride * 2};
  cuuint32_t box[3] = {box_inner, box_outer, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// bf16 map for the boxes of the activation epilogues: 32 rows x 32 columns, 64B-swizzled; with wide tiles 32 rows x 64 columns, 128B-swizzled.
int make_tmap_act(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld, bool wide) {
  if (wide) return make_tmap_2d_bf16(out, base, inner, outer, ld, 64, 32);
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 2) % 16) return -2;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// Tensor map the epilogue stores D through: boxes of 32 rows x 128 bytes.
int make_tmap_out(CUtensorMap* out, const void* D, int M, int N, long long ldd, int out_f32) {
  return out_f32 ? make_tmap_2d_f32(out, D, N, M, ldd, 32, 32) : make_tmap_2d_bf16(out, D, N, M, ldd, 64, 32);
}

static int g_num_sms = 0;

// Tuning knobs read once from the environment (experiments; the defaults are what ships).
static int tune_group_m() {
  static int v = -1;
  if (v < 0) { const char* e = getenv("MTB200_GEMM_GROUP_M"); v = e ? atoi(e) : GROUP_M; if (v < 1) v = GROUP_M; }
  return v;
}
static unsigned tune_wait_hint() {
  static int v = -1;
  if (v < 0) { const char* e = getenv("MTB200_GEMM_WAIT_HINT_NS"); v = e ? atoi(e) : 0; if (v < 0) v = 0; }
  return static_cast<unsigned>(v);
}

namespace g2 {
int launch_act(int mode, bool wide, const CUtensorMap& ta, const CUtensorMap& tb, const ActMaps<ACT_GLU>& m, const EpiParams& e, const ActParams& a, int K,
               int* status, cudaStream_t stream);
int launch_grouped(int mode, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const ActMaps<ACT_GLU>& m, const EpiParams& e, const ActParams& a,
                   int K, const GroupParams& g, int* status, cudaStream_t stream);
int launch_gather(const void* A, long long lda, void* D, long long ldd, const void* bias, int M, int N, int K,
                  const void* w, int* status, const GatherParams& g, cudaStream_t stream);
}

template <bool A_MN, bool B_MN, bool OUT_F32, bool GATHER = false, bool REDUCE = false, int GROUP = GROUP_NONE, bool STATS = false, bool EXTRA = true,
          int ACT = ACT_NONE, int NT = BN>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, GemmParams p, cudaStream_t stream,
                  const GatherParams* gp = nullptr, long long part_bytes = 0, const GroupParams* grp = nullptr, const ActMaps<ACT>& maps = ActMaps<ACT>{}) {
  static bool configured = false;
  auto kern = gemm_kernel<A_MN, B_MN, OUT_F32, GATHER, REDUCE, GROUP, STATS, EXTRA, ACT, NT>;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM) != cudaSuccess) return -4;
    configured = true;
  }
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  int tiles = ((p.M + BM - 1) / BM) * ((p.N + NT - 1) / NT);
  if (GROUP == GROUP_REDUCE) tiles *= grp->E;
  if (p.e.splits > 1 && !split_fits(p.e, tiles, (p.K + BK - 1) / BK, part_bytes, 128 * NT)) return -11;
  // the gathering variant always uses every SM: its extra warps carry the transfer
  const int items = tiles * p.e.splits;
  const int grid = (GATHER || items >= g_num_sms) ? g_num_sms : items;
  static const GatherParams none{};
  // A gathering launch neither overlaps its predecessor nor lets a successor in: its CTAs are counted on to be resident. A long
  // launch (PDL_MAX_FLOPS) starts behind its predecessor too.
  if constexpr (GATHER) kern<<<grid, GEMM_THREADS + GATHER_EXTRA_THREADS, GEMM_SMEM, stream>>>(ta, tb, td, maps, p, *gp, GroupParams{});
  else if (GROUP ? grp->flops > PDL_MAX_GROUPED_FLOPS : 2.0 * p.M * p.N * p.K > PDL_MAX_FLOPS) kern<<<grid, gemm_threads(ACT), GEMM_SMEM, stream>>>(ta, tb, td, maps, p, none, grp ? *grp : GroupParams{});
  else launch_pdl(kern, grid, gemm_threads(ACT), GEMM_SMEM, stream, ta, tb, td, maps, p, none, grp ? *grp : GroupParams{});
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template <bool A_MN, bool B_MN, bool OUT_F32, int NT>
static int launch_narrow(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const GemmParams& p, long long part_bytes, cudaStream_t stream) {
  if (p.e.R != nullptr || p.e.bias != nullptr) return launch<A_MN, B_MN, OUT_F32, false, false, GROUP_NONE, false, true, ACT_NONE, NT>(ta, tb, td, p, stream, nullptr, part_bytes);
  return launch<A_MN, B_MN, OUT_F32, false, false, GROUP_NONE, false, false, ACT_NONE, NT>(ta, tb, td, p, stream, nullptr, part_bytes);
}

// `nt`: columns of a tile.
static int gemm(int nt, const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* D,
                long long ldd, int out_f32, const void* R, long long ldr, const void* bias, int M, int N, int K,
                float alpha, int splits, unsigned long long* counters, unsigned long long epoch, float* part, long long part_bytes, float2* stats, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (N % 8 || ldd % 8 || (R && ldr % 8) || (stats && (out_f32 || nt != BN)) || splits < 1) return -10;
  CUtensorMap ta, tb, td;
  int rc;
  if (a_mn) rc = make_tmap_2d_bf16(&ta, A, M, K, lda, 64, 64);
  else rc = make_tmap_2d_bf16(&ta, A, K, M, lda, BK, BM);
  if (rc) return rc;
  if (b_mn) rc = make_tmap_2d_bf16(&tb, B, N, K, ldb, 64, 64);
  else rc = make_tmap_2d_bf16(&tb, B, K, N, ldb, BK, nt);
  if (rc) return rc - 10;
  rc = make_tmap_out(&td, D, M, N, ldd, out_f32);
  if (rc) return rc - 20;
  GemmParams p{M, N, K, status, tune_group_m(), tune_wait_hint(), 0u,
               EpiParams{M, N, R, ldr, reinterpret_cast<const __nv_bfloat16*>(bias), alpha, splits, part, stats, counters, epoch}};
  if (stats != nullptr) {
    switch ((a_mn ? 2 : 0) | (b_mn ? 1 : 0)) {
      case 0: return launch<false, false, false, false, false, GROUP_NONE, true>(ta, tb, td, p, stream, nullptr, part_bytes);
      case 1: return launch<false, true, false, false, false, GROUP_NONE, true>(ta, tb, td, p, stream, nullptr, part_bytes);
      case 2: return launch<true, false, false, false, false, GROUP_NONE, true>(ta, tb, td, p, stream, nullptr, part_bytes);
      default: return launch<true, true, false, false, false, GROUP_NONE, true>(ta, tb, td, p, stream, nullptr, part_bytes);
    }
  }
#define GEMM(X, Y, Z) if (nt == 64) return launch_narrow<X, Y, Z, 64>(ta, tb, td, p, part_bytes, stream); \
                      if (nt == 128) return launch_narrow<X, Y, Z, 128>(ta, tb, td, p, part_bytes, stream); \
                      return R != nullptr || bias != nullptr ? launch<X, Y, Z>(ta, tb, td, p, stream, nullptr, part_bytes) \
                                                             : launch<X, Y, Z, false, false, GROUP_NONE, false, false>(ta, tb, td, p, stream, nullptr, part_bytes)
  const int sel = (a_mn ? 4 : 0) | (b_mn ? 2 : 0) | (out_f32 ? 1 : 0);
  switch (sel) {
    case 0: GEMM(false, false, false);
    case 1: GEMM(false, false, true);
    case 2: GEMM(false, true, false);
    case 3: GEMM(false, true, true);
    case 4: GEMM(true, false, false);
    case 5: GEMM(true, false, true);
    case 6: GEMM(true, true, false);
    default: GEMM(true, true, true);
  }
#undef GEMM
}

}  // namespace mtb

extern "C" {

// D[M,N] = alpha * op(A) * op(B) (+bias) (+R).
//   a_mn = 0: A is row-major [M, K] (lda >= K);  a_mn = 1: A is row-major [K, M] (lda >= M)
//   b_mn = 0: B is row-major [N, K] (ldb >= K);  b_mn = 1: B is row-major [K, N] (ldb >= N)
//   out_f32: D and R are fp32, else bf16. R may alias D (accumulate). bias is bf16 [N] or null.
//   splits: work items per output tile (ops/gemm_plan.py); more than one needs counters (SPLIT_COUNTERS words, zero before the first
//   call; launches that may overlap have their own), an epoch that grows with every launch on them, and part, fp32 scratch of part_bytes
//   stats: optional softmax statistics of the output rows (EpiParams), bf16 output only
// Returns 0 on success, a negative code on invalid arguments or launch failure.
int mtb200_gemm_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* D,
                     long long ldd, int out_f32, const void* R, long long ldr, const void* bias, int M, int N, int K,
                     float alpha, int splits, unsigned long long* counters, unsigned long long epoch, float* part, long long part_bytes, float2* stats, int* status, cudaStream_t stream) {
  return mtb::gemm(mtb::BN, A, lda, a_mn, B, ldb, b_mn, D, ldd, out_f32, R, ldr, bias, M, N, K, alpha, splits, counters, epoch, part, part_bytes, stats, status, stream);
}

// The same in tiles of 128 x 64 and of 128 x 128, without statistics.
int mtb200_gemm_n64_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* D,
                         long long ldd, int out_f32, const void* R, long long ldr, const void* bias, int M, int N, int K,
                         float alpha, int splits, unsigned long long* counters, unsigned long long epoch, float* part, long long part_bytes, float2* stats, int* status, cudaStream_t stream) {
  return mtb::gemm(64, A, lda, a_mn, B, ldb, b_mn, D, ldd, out_f32, R, ldr, bias, M, N, K, alpha, splits, counters, epoch, part, part_bytes, stats, status, stream);
}
int mtb200_gemm_n128_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* D,
                          long long ldd, int out_f32, const void* R, long long ldr, const void* bias, int M, int N, int K,
                          float alpha, int splits, unsigned long long* counters, unsigned long long epoch, float* part, long long part_bytes, float2* stats, int* status, cudaStream_t stream) {
  return mtb::gemm(128, A, lda, a_mn, B, ldb, b_mn, D, ldd, out_f32, R, ldr, bias, M, N, K, alpha, splits, counters, epoch, part, part_bytes, stats, status, stream);
}

// A product with an MLP's activation in its epilogue (gemm_act.cuh). `form`: FORM_ONE, FORM_PAIR or FORM_WIDE; narrow tiles have no such epilogue.
//   mode 1  out[M, 2F] = A[M, K] * W[2F, K]^T, act[M, F] = f(out[:, :F]) * out[:, F:]
//   mode 2  out[M, F] = A[M, K] * W[F, K]^T (+ bias), act[M, F] = f(out)
// All row-major, without padding between rows but in A. f: SiLU, or (gelu) the tanh-approximated GELU.
int mtb200_gemm_act(const void* A, long long lda, const void* W, void* out, void* act, const void* bias, int mode, int gelu, int M, int F, int K,
                    int form, int* status, cudaStream_t stream) {
  using namespace mtb;
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if ((mode != ACT_GLU && mode != ACT_PLAIN) || form < FORM_ONE || form > FORM_WIDE || F % 8 || K % 8 || (bias != nullptr && mode != ACT_PLAIN)) return -10;
  if (reinterpret_cast<uintptr_t>(bias) & 15) return -11;
  const int N = mode == ACT_GLU ? 2 * F : F;
  const bool wide = form == FORM_WIDE;
  CUtensorMap ta, tb;
  ActMaps<ACT_GLU> m;
  int rc = make_tmap_2d_bf16(&ta, A, K, M, lda, 64, 128);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tb, W, K, N, K, 64, mode == ACT_GLU || form != FORM_ONE ? 128 : 256);
  if (rc) return rc - 10;
  __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(out);
  rc = make_tmap_act(&m.gate, o, F, M, N, wide);
  if (!rc) rc = make_tmap_act(&m.up, mode == ACT_GLU ? o + F : o, F, M, N, wide);
  if (!rc) rc = make_tmap_act(&m.act, act, F, M, F, wide);
  if (rc) return rc - 20;
  const EpiParams e{M, N, nullptr, 0, reinterpret_cast<const __nv_bfloat16*>(bias), 1.0f, 1, nullptr, nullptr, nullptr, 0};
  const ActParams a{F, gelu};
  if (form != FORM_ONE) return g2::launch_act(mode, wide, ta, tb, m, e, a, K, status, stream);
  const GemmParams p{M, N, K, status, tune_group_m(), tune_wait_hint(), 0u, e, a};
  if (mode == ACT_GLU)
    return launch<false, false, false, false, false, GROUP_NONE, false, false, ACT_GLU>(ta, tb, m.gate, p, stream, nullptr, 0, nullptr, m);
  return launch<false, false, false, false, false, GROUP_NONE, false, false, ACT_PLAIN>(ta, tb, m.gate, p, stream, nullptr, 0, nullptr,
                                                                                     ActMaps<ACT_PLAIN>{m.gate, m.up, m.act});
}

enum { GROUPED_WIDE = 4 };
// Grouped GEMM over expert slabs (see gemm_epilogue.cuh); mode + GROUPED_WIDE: on CTA pairs with wide tiles (gemm2_tcgen05.cu). starts [E + 1] and counts [E] are device arrays, `rows` is the
// height of the row buffers.
//   mode 0  D[rows, N] = A[rows, K] * W_e[N, K]^T        W: E matrices [N, K], w_stride elements apart
//   mode 1  D[rows, N] = A[rows, K] * W_e[K, N]          W: E matrices [K, N], w_stride elements apart
//   mode 2  W_e[M, N] = A[rows_e, M]^T * B[rows_e, N]    D is W here: E outputs, w_stride elements apart, ldd = N; K is ignored
//   mode 3  as mode 0, and act[rows, N / 2] = f(gate) * up of D = [gate | up] (gemm_act.cuh); f: SiLU, or (gelu) the tanh-approximated GELU
int mtb200_gemm_grouped(const void* A, long long lda, const void* B, long long ldb, void* D, long long ldd, void* act, int gelu, int mode, int rows,
                        int M, int N, int K, const int* starts, const int* counts, int E, long long w_stride, int* status,
                        cudaStream_t stream) {
  using namespace mtb;
  const bool wide = mode >= GROUPED_WIDE;
  if (wide) mode -= GROUPED_WIDE;
  if (E <= 0 || rows <= 0 || N <= 0 || (mode == 2 ? M : K) <= 0) return 0;
  if (E > GROUP_MAX || N % 8 || ldd % 8 || rows % GROUP_ALIGN || w_stride % 8 || mode < 0 || mode > 3 || (mode == 3 && (act == nullptr || N % 16))) return -10;
  CUtensorMap ta, tb, td;
  int rc = mode == 2 ? make_tmap_2d_bf16(&ta, A, M, rows, lda, 64, 64) : make_tmap_2d_bf16(&ta, A, K, rows, lda, BK, BM);
  if (rc) return rc;
  if (mode == 0 || mode == 3) rc = make_tmap_3d_bf16(&tb, B, K, N, E, w_stride, BK, mode == 3 || wide ? BN / 2 : BN);
  else if (mode == 1) rc = make_tmap_3d_bf16(&tb, B, N, K, E, w_stride, 64, 64);
  else rc = make_tmap_2d_bf16(&tb, B, N, rows, ldb, 64, 64);
  if (rc) return rc - 10;
  const int out_rows = mode == 2 ? M : rows;
  if (mode == 2) rc = ldd == N ? make_tmap_3d_bf16(&td, D, N, M, E, w_stride, 64, 32) : -10;
  else rc = make_tmap_out(&td, D, rows, N, ldd, 0);
  if (rc) return rc - 20;
  const EpiParams ep{out_rows, N, nullptr, 0, nullptr, 1.0f, 1, nullptr, nullptr, nullptr, 0};
  const ActParams ap{N / 2, gelu};
  GroupParams g{starts, counts, E, static_cast<float>(2.0 * rows * N * (mode == 2 ? M : K))};
  ActMaps<ACT_GLU> m{};
  if (mode == 3) {
    rc = make_tmap_act(&m.gate, D, N / 2, rows, ldd, wide);
    if (!rc) rc = make_tmap_act(&m.up, reinterpret_cast<__nv_bfloat16*>(D) + N / 2, N / 2, rows, ldd, wide);
    if (!rc) rc = make_tmap_act(&m.act, act, N / 2, rows, N / 2, wide);
    if (rc) return rc - 20;
  }
  if (wide) return g2::launch_grouped(mode, ta, tb, td, m, ep, ap, K, g, status, stream);
  GemmParams p{out_rows, N, K, status, tune_group_m(), tune_wait_hint(), 0u, ep, ap};
  if (mode == 3) return launch<false, false, false, false, false, GROUP_ROWS, false, false, ACT_GLU>(ta, tb, td, p, stream, nullptr, 0, &g, m);
  if (mode == 0) return launch<false, false, false, false, false, GROUP_ROWS>(ta, tb, td, p, stream, nullptr, 0, &g);
  if (mode == 1) return launch<false, true, false, false, false, GROUP_ROWS>(ta, tb, td, p, stream, nullptr, 0, &g);
  return launch<true, true, false, false, false, GROUP_REDUCE>(ta, tb, td, p, stream, nullptr, 0, &g);
}

// Fused all-gather + GEMM:  D[M,N] = A[M,K] * W[N,K]^T (+bias) with W living in `full`, the local
// full parameter buffer of a sharded group that this same launch fills from the peers' shards.
//   bases/world       arena address of every rank; shard_off/shard_bytes locate the group's shard
//   full              local destination (world * shard_bytes); w_byte_off = offset of W inside it
//   flags/epoch       per-chunk (128 KB) completion words; a chunk is ready when its word == epoch
//   chunk_lo/chunk_hi chunks gathered by this launch (others must already carry `epoch`)
//   ticket            device word used to hand chunks out to whichever CTAs are resident (zeroed here)
//   wait_ns           optional device [2] counters: producer wait time summed over CTAs, CTA count
//   two_cta           run on CTA pairs (cta_group::2, 256 x 256 tiles) when the device can schedule them
// bias, if given, must lie in an already gathered part of `full` (or elsewhere).
int mtb200_gemm_bf16_allgather(const void* A, long long lda, void* D, long long ldd, const void* bias, int M, int N, int K,
                               const unsigned long long* bases, int world, unsigned long long shard_off,
                               unsigned long long shard_bytes, void* full, unsigned long long w_byte_off, unsigned int* flags,
                               unsigned int epoch, int chunk_lo, int chunk_hi, unsigned int* ticket, unsigned long long* wait_ns,
                               int two_cta, int* status, cudaStream_t stream) {
  using namespace mtb;
  if (M <= 0 || N <= 0 || K <= 0) return -10;
  if (N % 8 || ldd % 8 || K % 8 || world < 1 || world > GATHER_MAX_RANKS || shard_bytes % 16 || w_byte_off % 16) return -10;
  if (world > 1 && shard_bytes < static_cast<unsigned long long>(GATHER_CHUNK_BYTES)) return -11;   // a chunk may straddle one shard boundary at most
  CUtensorMap ta, tb, td;
  int rc = make_tmap_2d_bf16(&ta, A, K, M, lda, BK, BM);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tb, reinterpret_cast<const unsigned char*>(full) + w_byte_off, K, N, K, BK, BN);
  if (rc) return rc - 10;
  rc = make_tmap_out(&td, D, M, N, ldd, 0);
  if (rc) return rc - 20;
  GemmParams p{M, N, K, status, tune_group_m(), tune_wait_hint(), 0u,
               EpiParams{M, N, nullptr, 0, reinterpret_cast<const __nv_bfloat16*>(bias), 1.0f, 1, nullptr, nullptr, nullptr, 0}};
  GatherParams g{};
  for (int i = 0; i < world; ++i) g.peer_base[i] = bases[i];
  g.shard_off = shard_off; g.shard_bytes = shard_bytes; g.dst = reinterpret_cast<unsigned char*>(full);
  g.flags = flags; g.epoch = epoch; g.world = world; g.chunk_lo = chunk_lo; g.chunk_hi = chunk_hi;
  g.ticket = ticket; g.wait_ns = wait_ns;
  g.b_byte_off = w_byte_off;
  int first = static_cast<int>(w_byte_off / GATHER_CHUNK_BYTES);
  g.chunk_first = first < chunk_lo ? chunk_lo : (first >= chunk_hi ? chunk_lo : first);
  if (ticket == nullptr) return -10;
  if (cudaMemsetAsync(ticket, 0, sizeof(unsigned int), stream) != cudaSuccess) return -5;   // chunk tickets start at 0 in every launch
  if (two_cta) {
    rc = g2::launch_gather(A, lda, D, ldd, bias, M, N, K, reinterpret_cast<const unsigned char*>(full) + w_byte_off, status, g, stream);
    if (rc != -6) return rc;   // -6: CTA pairs cannot be scheduled here; fall through to the one-CTA kernel
  }
  return launch<false, false, false, true>(ta, tb, td, p, stream, &g);
}

// Fused gradient reduce + GEMM:  D[M,N] (fp32) = (sum over ranks of G_r)[M,K] * B[N,K]^T (+ R), where G_r is the region
// [src_off, src_off + M*K*2) of rank r's arena (a tensor of its block gradient buffer). Gather warps pull the region from
// every rank, sum in fp32 and write bf16 into `dst` (local, M*K elements), which the TMA producer reads as the A operand as
// its chunks complete. Handshake of the reduce-scatter: waits for every rank's ready epoch, signals consumed when done.
//   flags/epoch   per-chunk completion words of dst;  ticket, done: device words, zeroed here
//   ready_flags   local row of ready epochs;  consumed_off: byte offset of the consumed row in every arena
int mtb200_gemm_bf16_reduce_a(void* dst, const void* B, long long ldb, float* D, long long ldd, const float* R, long long ldr,
                              int M, int N, int K, const unsigned long long* bases, int world, int rank,
                              unsigned long long src_off, unsigned int* flags, unsigned int epoch, unsigned int* ticket,
                              unsigned int* done, const void* ready_flags, unsigned long long consumed_off, unsigned int rs_epoch,
                              unsigned int limit_us, int* status, cudaStream_t stream) {
  using namespace mtb;
  if (M <= 0 || N <= 0 || K <= 0) return -10;
  if (N % 8 || ldd % 8 || K % 8 || (R && ldr % 8) || world < 1 || world > 8 || src_off % 16 || ticket == nullptr || done == nullptr) return -10;
  CUtensorMap ta, tb, td;
  int rc = make_tmap_2d_bf16(&ta, dst, K, M, K, BK, BM);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tb, B, K, N, ldb, BK, BN);
  if (rc) return rc - 10;
  // every pipeline wait sits out the peers' skew: a little longer than the bound of the ready-flag wait itself
  const unsigned lim = limit_us ? limit_us : FLAG_SPIN_LIMIT;
  rc = make_tmap_out(&td, D, M, N, ldd, 1);
  if (rc) return rc - 20;
  GemmParams p{M, N, K, status, tune_group_m(), tune_wait_hint(), lim + lim / 2 + 10000000u,
               EpiParams{M, N, R, ldr, nullptr, 1.0f, 1, nullptr, nullptr, nullptr, 0}};
  GatherParams g{};
  for (int i = 0; i < world; ++i) g.peer_base[i] = bases[i];
  g.dst = reinterpret_cast<unsigned char*>(dst);
  g.total_bytes = static_cast<unsigned long long>(M) * K * 2;
  g.flags = flags; g.epoch = epoch; g.world = world; g.rank = rank;
  g.chunk_lo = 0; g.chunk_hi = static_cast<int>((g.total_bytes + GATHER_CHUNK_BYTES - 1) / GATHER_CHUNK_BYTES);
  g.chunk_first = 0; g.b_byte_off = 0;
  g.ticket = ticket; g.done = done; g.wait_ns = nullptr;
  g.src_off = src_off; g.ready_flags = reinterpret_cast<const unsigned int*>(ready_flags); g.consumed_off = consumed_off;
  g.rs_epoch = rs_epoch; g.limit_us = limit_us ? limit_us : FLAG_SPIN_LIMIT; g.status = status;
  if (cudaMemsetAsync(ticket, 0, sizeof(unsigned int), stream) != cudaSuccess) return -5;
  if (cudaMemsetAsync(done, 0, sizeof(unsigned int), stream) != cudaSuccess) return -5;
  return launch<false, false, true, true, true>(ta, tb, td, p, stream, &g);
}

}  // extern "C"
