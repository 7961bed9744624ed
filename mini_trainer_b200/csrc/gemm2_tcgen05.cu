// Two-CTA variant of the persistent bf16 GEMM: a cluster of two CTAs (two SMs) computes one
// 256 x 256 output tile with tcgen05.mma.cta_group::2. Each CTA stages its own 128 rows of A and
// HALF of the B tile (128 of the 256 N rows/columns), so per multiply the tensor core of each SM
// reads 8 KB of operands from shared memory instead of 12 KB, and the L2 -> SM traffic of B halves.
// That operand path, not the MMA itself, is what limits the one-CTA 128 x 256 kernel.
//
// Protocol (barriers live at the same shared-memory offsets in both CTAs):
//   full[s]    CTA 0 only. CTA 0's producer arms it with the bytes of BOTH CTAs; both producers'
//              TMA loads (cp.async.bulk.tensor ... .cta_group::2, no multicast) complete on it.
//   empty[s]   both CTAs; arrived by the leader's tcgen05.commit, multicast to the pair.
//   tfull[a]   both CTAs; accumulator `a` (128 lanes x 256 columns per CTA) is complete.
//   tempty[a]  CTA 0 only; the 8 epilogue warps of the pair arrive (CTA 1 remotely).
// Only CTA 0's MMA thread issues tcgen05.mma; every wait is bounded as in the one-CTA kernel.
// The two CTAs synchronise with barrier.cluster once after set-up and once before teardown.
//
// WIDE = true computes 256 x 512 tiles: a stage holds a pair's A once and two halves of B, and both 256-column accumulators belong to one tile, so
// that a product of 256 x 512 x 64 moves 48 KB per SM where two 256 x 256 tiles move 64. What bounds a long product is the 1000 W cap, and operands that
// travel from L2 (and, where the tiles in flight span more rows than L2 holds, from HBM again) cost as much of it as the multiplications' own smem
// reads: 28672 x 4096 x 16384 as a weight gradient reads 7.4 GB of HBM in 256 x 256 tiles and 4.2 in wide ones, and in a loop at the cap gives
// 1261 and 1360 TFLOP/s (single CTAs 1257, the library 1332); 16384 x 4096 x 28672 1239 and 1390 (1280, 1417), 16384 x 28672 x 4096 1376 and 1413 (1325, 1407).
// With no second pair of accumulators the epilogue would stand between tiles. So the second half runs WIDE_LAG k-blocks behind the first at either end,
// a warpgroup per half empties its accumulator into registers before it stores anything (epilogue_wide), and the first half's next tile starts
// while the second's is emptied. What is left of the gap is about 2500 clocks, which short reductions show (5987 x 17920 x 1536: 263 us in 256 x 256 tiles, 281 wide).
//
// GROUP is the grouped form over expert slabs (gemm_epilogue.cuh) in wide tiles: 4096 tokens through 2 of 8 experts of 4096 x 14336, forward and backward,
// 8.20 -> 7.78 ms.
//
// GATHER = true is the fused all-gather variant (see gather.cuh): both CTAs of a pair carry eight
// gather warps and a flag checker; each CTA's checker watches the chunks under ITS half of the B
// tile (128 weight rows, one contiguous byte range) and only that CTA's producer waits for them.
// No load in this file is multicast: every CTA issues its own TMA loads from local memory.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "entries.h"
#include "gather.cuh"
#include "gemm_act.cuh"
#include "gemm_epilogue.cuh"
#include "ptx.cuh"

namespace mtb {

int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);
int make_tmap_out(CUtensorMap* out, const void* D, int M, int N, long long ldd, int out_f32);

namespace g2 {

constexpr int BM = 128;            // rows of A / D per CTA (256 per pair)
constexpr int BN = 256;            // columns per pair; each CTA stages BN/2 of them
constexpr int BNH = BN / 2;
constexpr int BK = 64;
constexpr int STAGES = 6;
constexpr int A_BYTES = BM * BK * 2;     // 16 KB
constexpr int B_BYTES = BNH * BK * 2;    // 16 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int WIDE_STAGES = 4;                        // wide tiles: a second half of B in every stage
constexpr int WIDE_STAGE_BYTES = A_BYTES + 2 * B_BYTES;
constexpr int WIDE_LAG = 2;                           // k-blocks by which the second half of a wide tile runs behind the first at its ends
constexpr int WIDE_GROUP_M = 14;                      // row-tiles per band, about: the 74 tiles in flight then read 3600 rows of A and 2700 of B
// Three warpgroups: {TMA, MMA}, and the epilogue of either half, whose threads hold 256 columns as 128 registers and the piece at work on. In the grouped forms and
// those with an activation 5 to 16 words a thread are spilled all the same, and read back 17 to 42 times per item; the other splits
// of the registers (24 / 240, 56 / 224, 72 / 216) spill more, also in the plain forms.
constexpr int WIDE_THREADS = 384;
constexpr int WIDE_REGS = 168, WIDE_REGS_IO = 40, WIDE_REGS_EPI = 232;   // per thread at launch, and after the split
static_assert(WIDE_REGS_IO + 2 * WIDE_REGS_EPI == 3 * WIDE_REGS && 3 * 128 * WIDE_REGS <= 65536, "register split");
static_assert(2 * 4 * STORE_BOX == EPI_SMEM, "a box per warp");
static_assert(WIDE_STAGES * WIDE_STAGE_BYTES == STAGES * STAGE_BYTES, "one shared-memory size");
constexpr int THREADS = 192;
constexpr int GROUP_M = 8;               // band of 8 pair-tiles = 2048 rows
constexpr int GATHER_GROUP_N = 4;        // column-tiles per band in the all-gather variant
constexpr int SMEM = STAGES * STAGE_BYTES + EPI_SMEM + 1024 + 256;
constexpr uint32_t PEER_MASK = 0xFEFFFFFFu;   // clears the CTA-rank bit of a shared::cluster address -> CTA 0

// How many of a launch's wide tiles are given out whole: a last round that half of the pairs have a tile for goes as half tiles.
__host__ __device__ inline int whole_tiles(int tiles, int pairs) {
  const int rest = tiles % pairs;
  return 2 * rest <= pairs ? tiles - rest : tiles;
}
inline int wide_group_m(int tiles_m) {
  const int bands = (tiles_m + WIDE_GROUP_M / 2) / WIDE_GROUP_M;
  return bands > 1 ? (tiles_m + bands - 1) / bands : tiles_m;
}

struct Params {
  int M, N, K;
  int* status;
  int num_pairs;
  int group_m;      // wide tiles: row-tiles per band
  int whole;        // wide tiles: items that are whole tiles, the rest of the tiles go as two halves each
  EpiParams e;
  ActParams act;   // ACT instances
};

constexpr int threads_of(int act, bool wide) { return wide ? WIDE_THREADS : act == ACT_NONE ? THREADS : 64 + 32 * ACT_WARPS; }

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t bar_addr_cta0, int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_addr_cta0), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const void* tmap, uint32_t bar_addr_cta0, int32_t c0, int32_t c1, int32_t c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_addr_cta0), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void umma2_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this shared-memory offset in BOTH CTAs once the leader's MMAs are done.
__device__ __forceinline__ void umma2_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cta0(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & PEER_MASK) : "memory");
}

template <bool A_MN, bool B_MN, bool OUT_F32, bool GATHER = false, bool STATS = false, bool EXTRA = true, int ACT = ACT_NONE, bool WIDE = false,
          int GROUP = GROUP_NONE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GATHER ? THREADS + GATHER_EXTRA_THREADS : threads_of(ACT, WIDE), 1)
gemm2_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
             const __grid_constant__ CUtensorMap tmap_d, const __grid_constant__ ActMaps<ACT> maps, Params p,
             const __grid_constant__ GatherParams g, GroupParams gr) {
  static_assert(GROUP == GROUP_NONE || WIDE, "the grouped forms are wide");
  __shared__ GroupTable gtab;   // unused (and not allocated) outside the grouped forms
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES + EPI_SMEM);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* verified = tmem_slot + 2;      // gather variant: tiles whose chunks under this CTA's B half have arrived
  uint32_t* ticket_slot = tmem_slot + 3;   // gather variant: broadcast of the chunk ticket among the gather warps

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1;
  const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM), tiles_n = (p.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int kblocks = (p.K + BK - 1) / BK;
  const int splits = GATHER || GROUP ? 1 : p.e.splits;
  const int wide_n = (p.N + 2 * BN - 1) / (2 * BN);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull_bar[a], 1); mbar_init(&tempty_bar[a], ACT && !WIDE ? 2 * ACT_WARPS : 8); }
    *abort_flag = 0;
    *verified = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_d);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_wait();   // nothing so far has touched global memory
  if (GROUP && warp == 2) fill_group_table<GROUP>(gtab, gr, 2 * BM, wide_n, tiles_m * wide_n, lane);
  tc_fence_before();
  __syncthreads();
  cluster_sync();          // the partner's barriers are initialised before anything is sent to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // item = split * num_tiles + tile: neighbours share operand tiles. Wide tiles: the first `whole` items are whole tiles, then come half tiles.
  const int wide_tiles = GROUP ? gtab.tile_start[gr.E] : tiles_m * wide_n;
  const int whole = GROUP ? whole_tiles(wide_tiles, p.num_pairs) : p.whole;
  const int num_items = WIDE ? wide_tiles * splits + (wide_tiles - whole) : num_tiles * splits;
  auto k_range = [&](int split, int& kb0, int& kb1) {
    kb0 = static_cast<int>(static_cast<long long>(kblocks) * split / splits);
    kb1 = static_cast<int>(static_cast<long long>(kblocks) * (split + 1) / splits);
  };
  auto tile_coords = [&](int t, int& tm, int& tn) {
    if constexpr (GATHER) {   // bands of column-tiles: the weight is consumed front to back at an even rate
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

  // Wide tiles: row-tile, first column and number of 256-column halves (0: a half tile past the last column) of an item. The grouped forms walk
  // the experts with the items: `e` only moves forward.
  auto wide_coords = [&](int w, int& e, int& tm, int& col0, int& halves, int& kb0, int& kb1) {
    k_range(splits > 1 ? w / wide_tiles : 0, kb0, kb1);
    if (splits > 1) w %= wide_tiles;
    int t = w < whole ? w : whole + (w - whole) / 2;
    int rows_m = tiles_m;
    if constexpr (GROUP != GROUP_NONE) {
      while (t >= gtab.tile_start[e + 1]) ++e;
      t -= gtab.tile_start[e];
      if (GROUP == GROUP_ROWS) rows_m = (gr.counts[e] + 2 * BM - 1) / (2 * BM);
      else { kb0 = 0; kb1 = (gr.counts[e] + BK - 1) / BK; }
    }
    const int band = t / (p.group_m * wide_n);
    const int first_m = band * p.group_m;
    const int rows = min(p.group_m, rows_m - first_m);
    const int local = t - band * p.group_m * wide_n;
    tm = first_m + local % rows;
    col0 = local / rows * 2 * BN;
    if (w < whole) {
      halves = col0 + BN < p.N ? 2 : 1;
    } else {
      col0 += ((w - whole) & 1) * BN;
      halves = col0 < p.N ? 1 : 0;
    }
  };

  if (WIDE && warp < 4) setmaxnreg_dec<WIDE_REGS_IO>();
  if (WIDE && warp == 0) {
    // ------------------------------------------------------------------ wide tiles: TMA producer (both CTAs)
    if (elect_one()) {
      uint32_t it = 0;
      int e = 0;
      for (int w = pair; w < num_items; w += p.num_pairs) {
        int tm, col0, halves, kb0, kb1;
        wide_coords(w, e, tm, col0, halves, kb0, kb1);
        if (halves == 0) continue;
        int row0 = tm * 2 * BM + rank * BM;
        if (GROUP == GROUP_ROWS) {   // a slab may end with CTA 0's rows: CTA 1 multiplies zeros then (from past the matrix), and stores nothing
          row0 += gr.starts[e];
          if (row0 >= gr.starts[e + 1]) row0 = p.M;
        }
        const int k_row = GROUP == GROUP_REDUCE ? gr.starts[e] : 0;   // first row of the reduction
        // this CTA's part of each half of B: 128 of its columns; with a gated activation CTA 0 has the gate's weight and CTA 1 up's
        const int b0 = ACT == ACT_GLU ? col0 / 2 + static_cast<int>(rank) * p.act.F : col0 + rank * BNH;
        constexpr int b_step = ACT == ACT_GLU ? BNH : BN;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % WIDE_STAGES;
          const uint32_t ph = (it / WIDE_STAGES) & 1;
          if (!mbar_wait(&empty_bar[s], ph ^ 1, abort_flag)) { atomicExch(p.status, 51); goto done; }
          uint8_t* sa = smem + s * WIDE_STAGE_BYTES;
          const uint32_t fb = smem_u32(&full_bar[s]) & PEER_MASK;   // CTA 0's barrier
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * (A_BYTES + halves * B_BYTES));
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * 8192, &tmap_a, fb, row0 + j * 64, k_row + kb * BK);
          } else {
            tma_load_2d_pair(sa, &tmap_a, fb, kb * BK, row0);
          }
          for (int h = 0; h < halves; ++h) {
            uint8_t* sb = sa + A_BYTES + h * B_BYTES;
            if (B_MN) {
#pragma unroll
              for (int j = 0; j < BNH / 64; ++j) {
                if constexpr (GROUP == GROUP_ROWS) tma_load_3d_pair(sb + j * 8192, &tmap_b, fb, b0 + h * b_step + j * 64, kb * BK, e);
                else tma_load_2d_pair(sb + j * 8192, &tmap_b, fb, b0 + h * b_step + j * 64, k_row + kb * BK);
              }
            } else {
              if constexpr (GROUP == GROUP_ROWS) tma_load_3d_pair(sb, &tmap_b, fb, kb * BK, b0 + h * b_step, e);
              else tma_load_2d_pair(sb, &tmap_b, fb, kb * BK, b0 + h * b_step);
            }
          }
        }
      }
      if (!GROUP || gr.flops <= PDL_MAX_GROUPED_FLOPS) pdl_trigger();
    }
  } else if (WIDE && warp == 1) {
    // ------------------------------------------------------------------ wide tiles: MMA issuer (leader CTA only)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      uint32_t it = 0, used0 = 0, used1 = 0;   // stages so far; tiles that used each accumulator
      int e = 0;
      for (int w = pair; w < num_items; w += p.num_pairs) {
        int tm, col0, halves, kb0, kb1;
        wide_coords(w, e, tm, col0, halves, kb0, kb1);
        if (halves == 0) continue;
        auto filled = [&](int j) { return mbar_wait(&full_bar[(it + j) % WIDE_STAGES], ((it + j) / WIDE_STAGES) & 1, abort_flag); };
        auto multiply = [&](int j, int h) {
          const uint32_t sa = smem_u32(smem + (it + j) % WIDE_STAGES * WIDE_STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES + h * B_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = A_MN ? make_smem_desc(sa + k * 2048, 8192, 1024) : make_smem_desc(sa + k * 32, 16, 1024);
            const uint64_t db = B_MN ? make_smem_desc(sb + k * 2048, 8192, 1024) : make_smem_desc(sb + k * 32, 16, 1024);
            umma2_bf16(tmem_base + h * BN, da, db, idesc, j != 0 || k != 0);
          }
        };
        auto release = [&](int j) { umma2_commit_pair(&empty_bar[(it + j) % WIDE_STAGES]); };
        if (!mbar_wait(&tempty_bar[0], (used0 & 1) ^ 1, abort_flag)) { atomicExch(p.status, 52); goto done; }
        ++used0;
        tc_fence_after();
        const int n = kb1 - kb0;
        const int lag = halves == 2 ? min(WIDE_LAG, n / 2) : 0;
        for (int j = 0; j < lag; ++j) {
          if (!filled(j)) { atomicExch(p.status, 53); goto done; }
          tc_fence_after();
          multiply(j, 0);
        }
        if (halves == 2) {
          if (!mbar_wait(&tempty_bar[1], (used1 & 1) ^ 1, abort_flag)) { atomicExch(p.status, 52); goto done; }
          ++used1;
          tc_fence_after();
          for (int j = 0; j < lag; ++j) { multiply(j, 1); release(j); }
        }
        for (int j = lag; j < n - lag; ++j) {
          if (!filled(j)) { atomicExch(p.status, 53); goto done; }
          tc_fence_after();
          multiply(j, 0);
          if (halves == 2) multiply(j, 1);
          release(j);
        }
        for (int j = n - lag; j < n; ++j) {
          if (!filled(j)) { atomicExch(p.status, 53); goto done; }
          tc_fence_after();
          multiply(j, 0);
        }
        umma2_commit_pair(&tfull_bar[0]);
        for (int j = n - lag; j < n; ++j) { multiply(j, 1); release(j); }
        if (halves == 2) umma2_commit_pair(&tfull_bar[1]);
        it += n;
      }
    }
  } else if (WIDE && warp >= 4) {
    // ------------------------------------------------------------------ wide tiles: epilogue (both CTAs; warps 4..7 half 0, 8..11 half 1)
    setmaxnreg_inc<WIDE_REGS_EPI>();
    const int q = warp & 3, h = (warp - 4) >> 2;
    EpiOut out{&tmap_d, smem + WIDE_STAGES * WIDE_STAGE_BYTES + (warp - 4) * STORE_BOX, -1, 0};
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + h * BN;
    uint32_t used = 0;
    int e = 0;
    for (int w = pair; w < num_items; w += p.num_pairs) {
      int tm, col0, halves, kb0, kb1;
      wide_coords(w, e, tm, col0, halves, kb0, kb1);
      if (h >= halves) continue;
      if (!mbar_wait(&tfull_bar[h], used & 1, abort_flag)) { atomicExch(p.status, 54); goto done; }
      ++used;
      tc_fence_after();
      int row0 = tm * 2 * BM + rank * BM, row_end = p.M;
      if constexpr (GROUP == GROUP_ROWS) { row0 += gr.starts[e]; row_end = gr.starts[e + 1]; }   // slabs are padded to 128 rows, all of which may be stored
      if constexpr (GROUP == GROUP_REDUCE) out.z = e;
      auto drained = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cta0(&tempty_bar[h]);
      };
      if constexpr (ACT != ACT_NONE) epilogue_act_wide<ACT>(p.e, p.act, maps, out, taddr, row0, row_end, col0 / BN + h, q, lane, drained);
      else epilogue_wide<OUT_F32, !GROUP, STATS, EXTRA>(p.e, out, taddr, row0, row_end, col0 + h * BN, q, lane, 2 * (tm * tiles_n + col0 / BN + h) + static_cast<int>(rank),
                                                splits > 1 ? w / wide_tiles : 0, GROUP == GROUP_REDUCE && kb1 == 0, drained);
    }
  } else if (WIDE) {
    // warps 2 and 3 have no part
  } else if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      uint32_t it = 0, tl = 0;
      unsigned long long waited_ns = 0;
      for (int w = pair; w < num_items; w += p.num_pairs) {
        int tm, tn, kb0, kb1;
        tile_coords(w % num_tiles, tm, tn);
        k_range(w / num_tiles, kb0, kb1);
        const int row0 = tm * 2 * BM + rank * BM;        // this CTA's rows of A
        // this CTA's half of the B tile; with a gated activation CTA 0 has the gate's weight and CTA 1 up's
        const int col0 = ACT == ACT_GLU ? tn * BNH + static_cast<int>(rank) * p.act.F : tn * BN + rank * BNH;
        if (GATHER) {
          if (!wait_verified(verified, tl, abort_flag, waited_ns)) { *abort_flag = 1; atomicExch(p.status, 55); goto done; }
          asm volatile("fence.proxy.async;" ::: "memory");   // peer data was written with ordinary stores, TMA reads it
          ++tl;
        }
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&empty_bar[s], ph ^ 1, abort_flag)) { atomicExch(p.status, 51); goto done; }
          uint8_t* sa = smem + s * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          const uint32_t fb = smem_u32(&full_bar[s]) & PEER_MASK;   // CTA 0's barrier
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * 8192, &tmap_a, fb, row0 + j * 64, kb * BK);
          } else {
            tma_load_2d_pair(sa, &tmap_a, fb, kb * BK, row0);
          }
          if (B_MN) {
#pragma unroll
            for (int j = 0; j < BNH / 64; ++j) tma_load_2d_pair(sb + j * 8192, &tmap_b, fb, col0 + j * 64, kb * BK);
          } else {
            tma_load_2d_pair(sb, &tmap_b, fb, kb * BK, col0);
          }
        }
      }
      if (!GATHER) pdl_trigger();   // what is left is a few products and the last epilogue
      if (GATHER && g.wait_ns != nullptr) {
        atomicAdd(g.wait_ns, waited_ns);
        atomicAdd(g.wait_ns + 1, 1ull);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      uint32_t it = 0, tl = 0;
      for (int w = pair; w < num_items; w += p.num_pairs, ++tl) {
        int kb0, kb1;
        k_range(w / num_tiles, kb0, kb1);
        const int acc = tl & 1;
        const uint32_t aph = (tl >> 1) & 1;
        if (!mbar_wait(&tempty_bar[acc], aph ^ 1, abort_flag)) { atomicExch(p.status, 52); goto done; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&full_bar[s], ph, abort_flag)) { atomicExch(p.status, 53); goto done; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = A_MN ? make_smem_desc(sa + k * 2048, 8192, 1024) : make_smem_desc(sa + k * 32, 16, 1024);
            const uint64_t db = B_MN ? make_smem_desc(sb + k * 2048, 8192, 1024) : make_smem_desc(sb + k * 32, 16, 1024);
            umma2_bf16(d_tmem, da, db, idesc, kb != kb0 || k != 0);
          }
          umma2_commit_pair(&empty_bar[s]);
        }
        umma2_commit_pair(&tfull_bar[acc]);
      }
    }
  } else if (GATHER && warp == 6 + GATHER_THREADS / 32) {
    // ------------------------------------------------------------------ flag checker (warp 14, both CTAs)
    uint32_t tl = 0;
    for (int t = pair; t < num_tiles; t += p.num_pairs, ++tl) {
      int tm, tn;
      tile_coords(t, tm, tn);
      const int col0 = tn * BN + rank * BNH;
      bool ok = true;
      if (col0 < p.N) {   // rows [col0, col0 + BNH) of the K-major weight: one contiguous byte range
        const unsigned long long lo = g.b_byte_off + static_cast<unsigned long long>(col0) * p.K * 2;
        const int rows = min(BNH, p.N - col0);
        ok = wait_chunks(g, lo, lo + static_cast<unsigned long long>(rows) * p.K * 2 - 1, lane, abort_flag);
      }
      __syncwarp();
      if (!ok) {
        if (lane == 0) { *abort_flag = 1; atomicExch(p.status, 55); }
        break;
      }
      if (lane == 0) st_release_cta_shared(verified, tl + 1);
    }
  } else if (GATHER && warp >= 6) {
    // ------------------------------------------------------------------ gather warps (6..13, both CTAs)
    gather_chunks(g, threadIdx.x - THREADS, ticket_slot);
  } else {
    // ------------------------------------------------------------------ epilogue (both CTAs; warps 2..5, with an activation 2..9)
    const int q = warp & 3;
    EpiOut out{&tmap_d, smem + STAGES * STAGE_BYTES + (ACT ? (warp - 2) * 2 * ACT_BOX : q * 2 * STORE_BOX), -1, 0};
    uint32_t tl = 0;
    for (int w = pair; w < num_items; w += p.num_pairs, ++tl) {
      const int t = w % num_tiles;
      int tm, tn;
      tile_coords(t, tm, tn);
      const int acc = tl & 1;
      const uint32_t aph = (tl >> 1) & 1;
      if (!mbar_wait(&tfull_bar[acc], aph, abort_flag)) { atomicExch(p.status, 54); goto done; }
      tc_fence_after();
      if constexpr (ACT != ACT_NONE)
        epilogue_act<ACT>(p.e, p.act, maps, out, tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN, tm * 2 * BM + rank * BM, tn, q,
                              (warp - 2) >> 2, lane);
      else epilogue_quarter<OUT_F32, !GATHER, STATS, EXTRA>(p.e, out, tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN, tm * 2 * BM + rank * BM, tn * BN, q, lane,
                                2 * t + static_cast<int>(rank), w / num_tiles, false);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cta0(&tempty_bar[acc]);
    }
  }
done:
  if (warp >= 2 && (ACT || WIDE || warp < 6) && lane == 0) drain_boxes();
  tc_fence_before();
  __syncthreads();
  cluster_sync();          // nobody tears down while the partner may still signal or read
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

// Clusters of two that can be co-resident (0: unsupported), plain / gather variant. Instances differ in threads and registers (wide tiles: 384 of 168)
// and in static shared memory (the grouped forms' table), but with tensor memory taken whole and more than half of an SM's shared memory every one
// of them fits an SM exactly once, so one is asked, once.
static_assert(SMEM + sizeof(GroupTable) <= 227 * 1024 && 2 * SMEM > 228 * 1024, "one CTA to an SM, in every instance");
template <bool GATHER>
static int co_resident_pairs() {
  static int pairs = -1;
  if (pairs < 0) {
    auto kern = gemm2_kernel<false, false, false, GATHER>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(GATHER ? THREADS + GATHER_EXTRA_THREADS : THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
    pairs = n;
  }
  return pairs;
}

template <bool A_MN, bool B_MN, bool OUT_F32, bool GATHER = false, bool STATS = false, bool EXTRA = true, int ACT = ACT_NONE, bool WIDE = false,
          int GROUP = GROUP_NONE>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, Params p, cudaStream_t stream, const GatherParams* gp = nullptr,
                  long long part_bytes = 0, const ActMaps<ACT>& maps = ActMaps<ACT>{}, const GroupParams* grp = nullptr) {
  auto kern = gemm2_kernel<A_MN, B_MN, OUT_F32, GATHER, STATS, EXTRA, ACT, WIDE, GROUP>;
  constexpr int threads = GATHER ? THREADS + GATHER_EXTRA_THREADS : threads_of(ACT, WIDE);
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) return -4;
    configured = true;
  }
  const int pairs = co_resident_pairs<GATHER>();
  if (pairs <= 0) return -6;
  const int tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + BN - 1) / BN);
  if (p.e.splits > 1 && !split_fits(p.e, 2 * tiles, (p.K + BK - 1) / BK, part_bytes)) return -11;
  // the gathering variant always uses every pair: its extra warps carry the transfer
  int items = tiles * p.e.splits;
  p.group_m = GROUP_M;
  if constexpr (WIDE) {
    const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM), wide = tiles_m * ((p.N + 2 * BN - 1) / (2 * BN));
    p.group_m = wide_group_m(tiles_m);
    p.whole = p.e.splits == 1 ? whole_tiles(wide, pairs) : wide;
    items = wide * p.e.splits + (wide - p.whole);
    if (GROUP == GROUP_REDUCE) items *= grp->E;   // at most, both forms
  }
  p.num_pairs = (GATHER || items >= pairs) ? pairs : items;
  static const GatherParams none{};
  if constexpr (GATHER) kern<<<2 * p.num_pairs, threads, SMEM, stream>>>(ta, tb, td, maps, p, *gp, GroupParams{});
  else if (GROUP ? grp->flops > PDL_MAX_GROUPED_FLOPS : 2.0 * p.M * p.N * p.K > PDL_MAX_FLOPS) kern<<<2 * p.num_pairs, threads, SMEM, stream>>>(ta, tb, td, maps, p, none, grp ? *grp : GroupParams{});
  else launch_pdl(kern, 2 * p.num_pairs, threads, SMEM, stream, ta, tb, td, maps, p, none, grp ? *grp : GroupParams{});
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// Fused all-gather + GEMM on CTA pairs; called by mtb200_gemm_bf16_allgather.
int launch_gather(const void* A, long long lda, void* D, long long ldd, const void* bias, int M, int N, int K,
                  const void* w, int* status, const GatherParams& g, cudaStream_t stream) {
  CUtensorMap ta, tb, td;
  int rc = make_tmap_2d_bf16(&ta, A, K, M, lda, BK, BM);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tb, w, K, N, K, BK, BNH);
  if (rc) return rc - 10;
  rc = make_tmap_out(&td, D, M, N, ldd, 0);
  if (rc) return rc - 20;
  Params p{M, N, K, status, 0, 0, 0, EpiParams{M, N, nullptr, 0, reinterpret_cast<const __nv_bfloat16*>(bias), 1.0f, 1, nullptr, nullptr, nullptr, 0}};
  return launch<false, false, false, true>(ta, tb, td, p, stream, &g);
}

// Products with an activation in the epilogue; called by mtb200_gemm_act.
int launch_act(int mode, bool wide, const CUtensorMap& ta, const CUtensorMap& tb, const ActMaps<ACT_GLU>& m, const EpiParams& e, const ActParams& a, int K,
               int* status, cudaStream_t stream) {
  const Params p{e.M, e.N, K, status, 0, 0, 0, e, a};
  const ActMaps<ACT_PLAIN> plain{m.gate, m.up, m.act};
  if (wide) return mode == ACT_GLU ? launch<false, false, false, false, false, false, ACT_GLU, true>(ta, tb, m.gate, p, stream, nullptr, 0, m)
                                   : launch<false, false, false, false, false, false, ACT_PLAIN, true>(ta, tb, m.gate, p, stream, nullptr, 0, plain);
  if (mode == ACT_GLU) return launch<false, false, false, false, false, false, ACT_GLU>(ta, tb, m.gate, p, stream, nullptr, 0, m);
  return launch<false, false, false, false, false, false, ACT_PLAIN>(ta, tb, m.gate, p, stream, nullptr, 0, plain);
}

// Grouped products on wide tiles; called by mtb200_gemm_grouped. `td`, `m`: maps of boxes of 32 rows x 128 bytes.
int launch_grouped(int mode, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const ActMaps<ACT_GLU>& m, const EpiParams& e, const ActParams& a,
                   int K, const GroupParams& g, int* status, cudaStream_t stream) {
  const Params p{e.M, e.N, K, status, 0, 0, 0, e, a};
  if (mode == 3) return launch<false, false, false, false, false, false, ACT_GLU, true, GROUP_ROWS>(ta, tb, td, p, stream, nullptr, 0, m, &g);
  if (mode == 0) return launch<false, false, false, false, false, false, ACT_NONE, true, GROUP_ROWS>(ta, tb, td, p, stream, nullptr, 0, ActMaps<ACT_NONE>{}, &g);
  if (mode == 1) return launch<false, true, false, false, false, false, ACT_NONE, true, GROUP_ROWS>(ta, tb, td, p, stream, nullptr, 0, ActMaps<ACT_NONE>{}, &g);
  return launch<true, true, false, false, false, false, ACT_NONE, true, GROUP_REDUCE>(ta, tb, td, p, stream, nullptr, 0, ActMaps<ACT_NONE>{}, &g);
}

template <bool A_MN, bool B_MN>
static int launch_wide(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const Params& p, bool out_f32, long long part_bytes, cudaStream_t stream) {
  if (out_f32) return launch<A_MN, B_MN, true, false, false, true, ACT_NONE, true>(ta, tb, td, p, stream, nullptr, part_bytes);
  if (p.e.R != nullptr || p.e.bias != nullptr) return launch<A_MN, B_MN, false, false, false, true, ACT_NONE, true>(ta, tb, td, p, stream, nullptr, part_bytes);
  return launch<A_MN, B_MN, false, false, false, false, ACT_NONE, true>(ta, tb, td, p, stream, nullptr, part_bytes);
}

static int gemm2(bool wide, const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* D, long long ldd, int out_f32, const void* R,
                 long long ldr, const void* bias, int M, int N, int K, float alpha, int splits, unsigned long long* counters, unsigned long long epoch,
                 float* part, long long part_bytes, float2* stats, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (N % 8 || ldd % 8 || (R && ldr % 8) || (stats && out_f32) || splits < 1) return -10;
  if (stats != nullptr && (a_mn || b_mn || R || bias)) wide = false;   // of the products with statistics only the plain forward one has wide tiles
  CUtensorMap ta, tb, td;
  int rc;
  if (a_mn) rc = make_tmap_2d_bf16(&ta, A, M, K, lda, 64, 64);
  else rc = make_tmap_2d_bf16(&ta, A, K, M, lda, BK, BM);
  if (rc) return rc;
  if (b_mn) rc = make_tmap_2d_bf16(&tb, B, N, K, ldb, 64, 64);
  else rc = make_tmap_2d_bf16(&tb, B, K, N, ldb, BK, BNH);
  if (rc) return rc - 10;
  rc = make_tmap_out(&td, D, M, N, ldd, out_f32);
  if (rc) return rc - 20;
  Params p{M, N, K, status, 0, 0, 0, EpiParams{M, N, R, ldr, reinterpret_cast<const __nv_bfloat16*>(bias), alpha, splits, part, stats, counters, epoch}};
  if (wide) {
    if (stats != nullptr) return launch<false, false, false, false, true, false, ACT_NONE, true>(ta, tb, td, p, stream, nullptr, part_bytes);
    switch ((a_mn ? 2 : 0) | (b_mn ? 1 : 0)) {
      case 0: return launch_wide<false, false>(ta, tb, td, p, out_f32, part_bytes, stream);
      case 1: return launch_wide<false, true>(ta, tb, td, p, out_f32, part_bytes, stream);
      case 2: return launch_wide<true, false>(ta, tb, td, p, out_f32, part_bytes, stream);
      default: return launch_wide<true, true>(ta, tb, td, p, out_f32, part_bytes, stream);
    }
  }
  if (stats != nullptr) {
    switch ((a_mn ? 2 : 0) | (b_mn ? 1 : 0)) {
      case 0: return launch<false, false, false, false, true>(ta, tb, td, p, stream, nullptr, part_bytes);
      case 1: return launch<false, true, false, false, true>(ta, tb, td, p, stream, nullptr, part_bytes);
      case 2: return launch<true, false, false, false, true>(ta, tb, td, p, stream, nullptr, part_bytes);
      default: return launch<true, true, false, false, true>(ta, tb, td, p, stream, nullptr, part_bytes);
    }
  }
#define GEMM2(X, Y, Z) return R != nullptr || bias != nullptr ? launch<X, Y, Z>(ta, tb, td, p, stream, nullptr, part_bytes) \
                                                              : launch<X, Y, Z, false, false, false>(ta, tb, td, p, stream, nullptr, part_bytes)
  const int sel = (a_mn ? 4 : 0) | (b_mn ? 2 : 0) | (out_f32 ? 1 : 0);
  switch (sel) {
    case 0: GEMM2(false, false, false);
    case 1: GEMM2(false, false, true);
    case 2: GEMM2(false, true, false);
    case 3: GEMM2(false, true, true);
    case 4: GEMM2(true, false, false);
    case 5: GEMM2(true, false, true);
    case 6: GEMM2(true, true, false);
    default: GEMM2(true, true, true);
  }
#undef GEMM2
}

}  // namespace g2
}  // namespace mtb

extern "C" {

// Same contract as mtb200_gemm_bf16, computed by CTA pairs (256 x 256 tiles). Returns -6 when
// clusters of two cannot be scheduled on this device (mtb200_gemm2_pairs() is 0); callers then use the one-CTA kernel.
int mtb200_gemm2_pairs() { return mtb::g2::co_resident_pairs<false>(); }

int mtb200_gemm2_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* D,
                      long long ldd, int out_f32, const void* R, long long ldr, const void* bias, int M, int N, int K,
                      float alpha, int splits, unsigned long long* counters, unsigned long long epoch, float* part, long long part_bytes, float2* stats, int* status, cudaStream_t stream) {
  return mtb::g2::gemm2(false, A, lda, a_mn, B, ldb, b_mn, D, ldd, out_f32, R, ldr, bias, M, N, K, alpha, splits, counters, epoch, part, part_bytes, stats, status, stream);
}

// The same with wide tiles (256 x 512).
int mtb200_gemm2_wide_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* D,
                           long long ldd, int out_f32, const void* R, long long ldr, const void* bias, int M, int N, int K,
                           float alpha, int splits, unsigned long long* counters, unsigned long long epoch, float* part, long long part_bytes, float2* stats, int* status, cudaStream_t stream) {
  return mtb::g2::gemm2(true, A, lda, a_mn, B, ldb, b_mn, D, ldd, out_f32, R, ldr, bias, M, N, K, alpha, splits, counters, epoch, part, part_bytes, stats, status, stream);
}

}  // extern "C"
