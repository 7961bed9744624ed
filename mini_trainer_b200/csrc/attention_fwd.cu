// Varlen causal GQA attention forward for sm_100a.
//
// A work item is a PAIR of 128-row query tiles A and B that read the same keys: two query heads of one kv head (even GQA
// ratio), or two consecutive query blocks of one head (odd ratio). Q, K and V are read straight out of the fused qkv
// activation [T, (Hq + 2 Hkv) * D] through ONE tensor map (128B swizzle):
//   S = Q K^T      tcgen05.mma, M=128 queries, N=128 keys, K=D      (one accumulator per tile in TMEM)
//   P = softmax    one warpgroup per tile, one thread per query row: S from TMEM, bf16 P written back over S
//   O += P V       tcgen05.mma with P as the tensor-memory A operand  (one accumulator per tile)
// Roles: warp 0 = TMA (K and V double-buffered), warp 1 = MMA issue, warps 4-7 = softmax + epilogue of A, 8-11 of B.
//
// Why pairs: a tile's chain is S -> softmax -> P V, and with one tile per CTA the tensor core idles under the softmax and the
// softmax under the products, or (with two S buffers of one tile) all softmax warps do the same phase at the same time and
// queue on the special-function unit. Two independent tiles take turns: while A is in its softmax the tensor core runs
// P V and the next S of B. K and V are loaded once per pair. A row belongs to one thread, so nothing is exchanged between
// threads (two threads per row with their maxima exchanged through shared memory measured 1.92 ms below). P is handed over in
// two halves of 64 keys, so the first half's products run under the second half's exponentials.
// 1 x 16384 tokens, 32/8 heads, D = 128: 1.65 ms; 41 samples, 12 345 tokens, 16/4 heads, D = 64: 53 us (one tile per CTA, two
// threads per row: 1.94 ms and 94 us). Launches with few pairs are faster in that other form (attention_fwd_one.cu);
// a long sequence at D = 64 is level (1 x 16384, 32/8 heads: 1.54 ms there, 1.50 here).
//
// CTAs are persistent (one per SM): barriers and tensor memory are set up once, K and V of the next item are prefetched
// under the current one's tail, and the epilogue of an item runs under the next item's first product. Items come most work
// first and are dealt in alternating direction, so the CTAs' totals differ by about one item.
//
// A row's reference maximum only moves (and its accumulator is only rescaled) when the running maximum grew by more than
// 2^8, which is exact: the same reference is used throughout. Only the last key tile of a query tile touches the causal
// diagonal: its code is its own, a warp leaves out the pieces of 32 keys that none of its rows see, and masks one.
//
// What a unit costs beside its key tiles is what short samples are bound by: 3.7 us at D = 64, where a key tile of the pair takes 0.8. Of that, the
// unit's row of the table and the divisions that find it took 0.7, masking 0.6, storing the output 0.7 (1.4 to 2.9 at D = 128). Without them
// (before, now): 148 samples of 128 tokens, 16/4 heads, 36.5 -> 30.4 us at D = 64 and 57.6 -> 42.6 at 128, 37 of 1024 163 -> 149 and 232 -> 188,
// 41 of 12 to 1489 tokens 55.9 -> 53; 1 x 16384 level.
//
// Masked scores are -inf. The exponentials that run on the special-function unit turn them into exact zeros;
// the quarter that runs on the FMA pipe (ex2_fma2) clamps its argument at -126 and returns about 1e-38 instead, so
// on the diagonal tile one masked key in four of the masked piece adds a term of that size to a row sum that is at least 1 (the row's
// maximum contributes exp2(0)) and to P: 38 orders of magnitude below either, no effect on out or lse.
//
// Outputs: out [T, Hq*D] bf16 and lse [Hq, T] fp32 (natural log, scaled scores), as needed by
// the backward. Sequence boundaries come from a host-built work table (seq_start, seq_len, q0),
// so there is no device-side search in cu_seqlens.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "entries.h"
#include "ptx.cuh"

namespace mtb {

int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);

constexpr int ATT_B = 128;         // query tile and key tile edge
constexpr int POLY = 4;            // every POLY-th exponential pair runs on the FMA pipe (2 and 8 measured the same within the spread)
constexpr int ATT_THREADS = 384;   // three warpgroups: TMA / MMA, softmax of A, softmax of B
// Registers per thread after the split; over the three warpgroups they add up to at most the 3 x 168 of the launch.
// A softmax thread holds the 128 scores of its row.
constexpr int ATT_REGS_IO = 88, ATT_REGS_SOFTMAX = 208;
static_assert(ATT_REGS_IO + 2 * ATT_REGS_SOFTMAX <= 3 * 168, "register split");

template <int D>
struct AttFwdSmem {
  static constexpr int TILE = ATT_B * D * 2;         // a [128, D] bf16 tile
  static constexpr int OFF_Q = 0;                    // A, B
  static constexpr int OFF_K = 2 * TILE;             // 2 stages
  static constexpr int OFF_V = 4 * TILE;             // 2 stages
  static constexpr int OFF_OUT = 6 * TILE;           // staged output: a box of 32 rows x 64 columns for each softmax warp
  static constexpr int OFF_BAR = OFF_OUT + 8 * 4096;
  static constexpr int TOTAL = OFF_BAR + 256 + 1024;
};

struct AttFwdParams {
  __nv_bfloat16* out;
  long long ldo;
  float* lse;
  const int* plan;   // [n_items, 3] = seq_start, seq_len, q0
  int n_items;
  int T, Hq, Hkv;
  int row_pairs;     // 0: item x two heads of a kv head; 1: item (256 rows) x one head
  float scale;
  int* status;
};

struct AttTrue { static constexpr bool value = true; };
struct AttFalse { static constexpr bool value = false; };

// One unit of work: the two query tiles of a pair. n = key tiles (0: no such tile).
struct AttWork {
  int seq_start, seq_len, hk, h[2], q0[2], n[2];
  __device__ __forceinline__ int tiles() const { return n[0] > n[1] ? n[0] : n[1]; }
};

// Where the next unit of this CTA is in the table. A unit's row is fetched while the unit before it is worked on: read when it is needed, it cost
// every role 1300 to 3000 clocks, a fifth of a unit of one key tile.
// x / d for 0 <= x < 2^31 and d > 0, with m = (2^32 - 1) / d: the product is at most one too small.
struct AttDiv {
  unsigned m;
  int d;
  __device__ __forceinline__ explicit AttDiv(int div) : m(0xffffffffu / static_cast<unsigned>(div)), d(div) {}
  __device__ __forceinline__ int operator()(int x) const {
    const int q = static_cast<int>(__umulhi(static_cast<unsigned>(x), m));
    return x - q * d >= d ? q + 1 : q;
  }
};
struct AttNext {
  int item, x;                      // item: -1 for none (the last round may be partial in either direction)
  int seq_start, seq_len, q0;
  bool more;                        // whether there is such a round at all
};
__device__ __forceinline__ void att_fetch(const AttFwdParams& p, const AttDiv& per_item, int round, AttNext& f) {
  const int total = p.n_items * per_item.d, grid = static_cast<int>(gridDim.x);
  f.more = round * grid < total;
  const int u = round * grid + ((round & 1) ? grid - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x));
  f.item = -1;
  if (!f.more || u >= total) return;
  f.item = per_item(u);
  f.x = u - f.item * per_item.d;
  f.seq_start = p.plan[f.item * 3 + 0]; f.seq_len = p.plan[f.item * 3 + 1]; f.q0 = p.plan[f.item * 3 + 2];
}
// The unit that was fetched. A row of the table that does not lie inside the packed batch yields a unit without tiles, which every role skips.
__device__ __forceinline__ void att_unit(const AttFwdParams& p, const AttDiv& group, const AttNext& f, AttWork& w) {
  w.n[0] = w.n[1] = 0;
  if (f.item < 0) return;
  w.seq_start = f.seq_start; w.seq_len = f.seq_len;
  const int q0 = f.q0;
  if (w.seq_start < 0 || w.seq_len <= 0 || q0 < 0 || q0 >= w.seq_len || static_cast<long long>(w.seq_start) + w.seq_len > p.T) {
    atomicExch(p.status, 61);   // reported, not dereferenced
    return;
  }
  w.h[0] = p.row_pairs ? f.x : 2 * f.x;
  w.h[1] = p.row_pairs ? f.x : 2 * f.x + 1;
  w.hk = group(w.h[0]);
  w.q0[0] = q0;
  w.q0[1] = p.row_pairs ? q0 + ATT_B : q0;
  w.n[0] = q0 / ATT_B + 1;
  w.n[1] = w.q0[1] < w.seq_len ? w.q0[1] / ATT_B + 1 : 0;
}

template <int D>
__global__ void __launch_bounds__(ATT_THREADS, 1) attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tmap_out, AttFwdParams p) {
  using L = AttFwdSmem<D>;
  constexpr int KB = D / 64;  // 64-element (128 B) column blocks of a D-wide row
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* q_full = bars;            // both Q tiles of a unit landed
  uint64_t* q_free = bars + 1;        // every S of the unit has completed
  uint64_t* k_full = bars + 2;        // [2]
  uint64_t* k_empty = bars + 4;       // [2] S of both tiles against this K has completed
  uint64_t* v_full = bars + 6;        // [2]
  uint64_t* v_empty = bars + 8;       // [2] P V of both tiles has completed
  uint64_t* s_full = bars + 10;       // [A, B]
  uint64_t* p_ready = bars + 12;      // [A, B][keys 0-63, keys 64-127] P in tensor memory, O rescaled (4 arrivals)
  uint64_t* pv_done = bars + 16;      // [A, B] P V complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1); mbar_init(q_free, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&v_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_ready[2 * i], 4); mbar_init(&p_ready[2 * i + 1], 4); mbar_init(&pv_done[i], 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap);
    tma_prefetch_desc(&tmap_out);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  pdl_wait();   // nothing so far has touched global memory
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const AttDiv per_item(p.row_pairs ? p.Hq : p.Hq / 2), group(p.Hq / p.Hkv);
  const uint32_t tmem_base = *tmem_slot;   // S of A and B at columns 0 and 128, O at 256 and 256 + D

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ATT_REGS_IO));
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (elect_one()) {
        AttWork w;
        AttNext f;
        uint32_t units = 0, kt = 0;   // units with tiles so far; key tiles so far
        att_fetch(p, per_item, 0, f);
        for (int round = 1; f.more; ++round) {
          att_unit(p, group, f, w);
          att_fetch(p, per_item, round, f);
          const int n = w.tiles();
          if (n == 0) continue;
          if (units > 0 && !mbar_wait(q_free, (units - 1) & 1, abort_flag)) { atomicExch(p.status, 11); goto done; }
          mbar_arrive_expect_tx(q_full, w.n[1] > 0 ? 2 * L::TILE : L::TILE);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (w.n[g] == 0) continue;
#pragma unroll
            for (int kb = 0; kb < KB; ++kb)
              tma_load_2d(smem + L::OFF_Q + g * L::TILE + kb * 16384, &tmap, q_full, w.h[g] * D + kb * 64, w.seq_start + w.q0[g]);
          }
          for (int j = 0; j < n; ++j, ++kt) {
            const int s = kt & 1;
            const uint32_t ph = ((kt >> 1) & 1) ^ 1;
            const int row = w.seq_start + j * ATT_B;
            if (!mbar_wait(&k_empty[s], ph, abort_flag)) { atomicExch(p.status, 11); goto done; }
            mbar_arrive_expect_tx(&k_full[s], L::TILE);
#pragma unroll
            for (int kb = 0; kb < KB; ++kb)
              tma_load_2d(smem + L::OFF_K + s * L::TILE + kb * 16384, &tmap, &k_full[s], (p.Hq + w.hk) * D + kb * 64, row);
            if (!mbar_wait(&v_empty[s], ph, abort_flag)) { atomicExch(p.status, 11); goto done; }
            mbar_arrive_expect_tx(&v_full[s], L::TILE);
#pragma unroll
            for (int kb = 0; kb < KB; ++kb)
              tma_load_2d(smem + L::OFF_V + s * L::TILE + kb * 16384, &tmap, &v_full[s], (p.Hq + p.Hkv + w.hk) * D + kb * 64, row);
          }
          ++units;
        }
        pdl_trigger();   // what is left is the last key tiles' softmax and products
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      if (elect_one()) {
        constexpr uint32_t idesc_qk = make_idesc_bf16(ATT_B, ATT_B, false, false);
        constexpr uint32_t idesc_pv = make_idesc_bf16(ATT_B, D, false, true);
        // descriptors of tiles at fixed addresses are built once; a k-step is one add
        const uint32_t dQ = smem_desc_lo(smem_u32(smem + L::OFF_Q), 16);
        const uint32_t dK = smem_desc_lo(smem_u32(smem + L::OFF_K), 16);
        const uint32_t dV = smem_desc_lo(smem_u32(smem + L::OFF_V), 16384);
        auto kstep = [](int k) { return static_cast<uint32_t>((k >> 2) * 1024 + (k & 3) * 2); };
        auto stage = [](uint32_t t) { return (t & 1) * static_cast<uint32_t>(L::TILE >> 4); };
        auto issue_s = [&](int g, uint32_t t) {
#pragma unroll
          for (int k = 0; k < D / 16; ++k)
            umma_bf16_lo(tmem_base + g * ATT_B, dQ + g * (L::TILE >> 4) + kstep(k), dK + stage(t) + kstep(k), idesc_qk, k != 0);
          umma_commit(&s_full[g]);
        };
        auto issue_pv = [&](int g, uint32_t t, bool first, int half) {   // the products with 64 keys; both halves make a P V
#pragma unroll
          for (int k = 0; k < ATT_B / 32; ++k) {   // 16 keys = 8 packed columns of P
            const int kk = half * (ATT_B / 32) + k;
            umma_bf16_ts_lo(tmem_base + 2 * ATT_B + g * D, tmem_base + g * ATT_B + kk * 8, dV + stage(t) + kk * 128, idesc_pv, !first || kk != 0);
          }
        };
        AttWork w;
        AttNext f;
        uint32_t units = 0, kt = 0;
        uint32_t cnt[2] = {0, 0};   // tiles of each group so far
        att_fetch(p, per_item, 0, f);
        for (int round = 1; f.more; ++round) {
          att_unit(p, group, f, w);
          att_fetch(p, per_item, round, f);
          const int n = w.tiles();
          if (n == 0) continue;
          if (!mbar_wait(q_full, units & 1, abort_flag)) { atomicExch(p.status, 12); goto done; }
          if (!mbar_wait(&k_full[kt & 1], (kt >> 1) & 1, abort_flag)) { atomicExch(p.status, 13); goto done; }
          tc_fence_after();
          issue_s(0, kt);
          if (w.n[1] > 0) issue_s(1, kt);
          umma_commit(&k_empty[kt & 1]);
          if (n == 1) umma_commit(q_free);
          for (int j = 0; j < n; ++j) {
            const uint32_t t = kt + j;
            if (!mbar_wait(&v_full[t & 1], (t >> 1) & 1, abort_flag)) { atomicExch(p.status, 16); goto done; }
            bool k_next = false;
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              if (j >= w.n[g]) continue;
#pragma unroll
              for (int half = 0; half < 2; ++half) {
                if (!mbar_wait(&p_ready[2 * g + half], cnt[g] & 1, abort_flag)) { atomicExch(p.status, 15); goto done; }
                tc_fence_after();
                issue_pv(g, t, j == 0, half);
              }
              umma_commit(&pv_done[g]);
              ++cnt[g];
              if (j + 1 < w.n[g]) {   // P was the last reader of these columns: the next S of this tile follows at once
                if (!k_next && !mbar_wait(&k_full[(t + 1) & 1], ((t + 1) >> 1) & 1, abort_flag)) { atomicExch(p.status, 14); goto done; }
                k_next = true;
                tc_fence_after();
                issue_s(g, t + 1);
              }
            }
            umma_commit(&v_empty[t & 1]);
            if (j + 1 < n) {
              umma_commit(&k_empty[(t + 1) & 1]);
              if (j + 2 == n) umma_commit(q_free);
            }
          }
          kt += n;
          ++units;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax + epilogue, one thread per query row
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ATT_REGS_SOFTMAX));
    const int g = (warp >> 2) - 1;            // tile A or B
    const int r = (warp & 3) * 32 + lane;     // row inside the query tile
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t ts = tmem_base + g * ATT_B + lane_addr, to = tmem_base + 2 * ATT_B + g * D + lane_addr;
    const float sl2 = p.scale * 1.4426950408889634f;
    const int wq = warp & 3;
    uint8_t* box = smem + L::OFF_OUT + (warp - 4) * 4096;
    const float2 sl2v = make_float2(sl2, sl2);
    uint32_t cnt = 0;
    AttWork w;
    AttNext f;
    att_fetch(p, per_item, 0, f);
    for (int round = 1; f.more; ++round) {
      att_unit(p, group, f, w);
      const int n = g == 0 ? w.n[0] : w.n[1];
      if (n == 0) { att_fetch(p, per_item, round, f); continue; }
      const int qpos = (g == 0 ? w.q0[0] : w.q0[1]) + r;
      float m_ref = -INFINITY, l = 0.f;
      // One key tile. DIAG: the last one, on the causal diagonal. Of its keys, 32 at a time, the warp's rows see all before piece `wq`, the first
      // lane + 1 of that piece, and none behind it: nothing is computed for those.
      auto key_tile = [&](auto diag, int j) -> bool {
        constexpr bool DIAG = decltype(diag)::value;
        // the row of S is read from tensor memory once and stays in registers for the maximum and the exponentials
        uint32_t sv[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c)
          tmem_ld_32x32(ts + c * 32, sv[c]);
        tmem_ld_wait();
        float mc[4];   // four independent chains
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          mc[c] = -INFINITY;
          if (DIAG && c > wq) continue;
          if (DIAG && c == wq) {
#pragma unroll
            for (int i = 1; i < 32; ++i)
              if (i > lane) sv[c][i] = 0xff800000u;   // -inf
          }
          mc[c] = fmaxf(__uint_as_float(sv[c][0]), __uint_as_float(sv[c][1]));
#pragma unroll
          for (int i = 2; i < 32; i += 2) mc[c] = fmax3(mc[c], __uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1]));
        }
        const float mt = fmax3(fmaxf(mc[0], mc[1]), mc[2], mc[3]);
        float factor = 1.f;
        bool rescale = false;
        if (mt > m_ref && (mt - m_ref) * sl2 > 8.f) {   // includes the first tile (m_ref = -inf)
          factor = (m_ref == -INFINITY) ? 0.f : ex2_mufu((m_ref - mt) * sl2);
          rescale = j > 0;
          m_ref = mt;
          l *= factor;
        }
        if (j > 0 && __any_sync(0xffffffffu, rescale)) {   // O must be complete through tile j-1 before it is rescaled
          if (!mbar_wait(&pv_done[g], (cnt - 1) & 1, abort_flag)) return false;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t v[16];
            tmem_ld_32x16(to + c * 16, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * factor);
            tmem_st_32x16(to + c * 16, v);
          }
        }
        // probabilities -> bf16 P over the columns of S, row sum; exp2(-inf) = 0 masks
        const float mo = (m_ref == -INFINITY) ? 0.f : m_ref * sl2;
        const float2 nmo = make_float2(-mo, -mo);
        float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
          if (!DIAG || c <= wq) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              // scale and shift two scores with one packed FMA; of every POLY pairs one runs its exponentials on the FMA pipe
              const float2 x = ffma2(make_float2(__uint_as_float(sv[c][2 * i]), __uint_as_float(sv[c][2 * i + 1])), sl2v, nmo);
              const float2 e = (i % POLY == POLY - 1) ? ex2_fma2(x) : make_float2(ex2_mufu(x.x), ex2_mufu(x.y));
              l2[i & 1] = fadd2(l2[i & 1], e);
              pk[i] = pack_bf16(e.x, e.y);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[i] = 0u;
          }
          tmem_st_32x16(ts + c * 16, pk);
          if (c & 1) {   // half of the keys: their products start under the other half's exponentials
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[2 * g + (c >> 1)]);
          }
        }
        l += (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y);
        return true;
      };
      for (int j = 0; j < n; ++j, ++cnt) {
        if (!mbar_wait(&s_full[g], cnt & 1, abort_flag)) { atomicExch(p.status, 17); goto done; }
        tc_fence_after();
        bool ok;
        if (j == n - 1) {
          att_fetch(p, per_item, round, f);   // here, so that its registers are not held through the other tiles
          ok = key_tile(AttTrue{}, j);
        } else {
          ok = key_tile(AttFalse{}, j);
        }
        if (!ok) { atomicExch(p.status, 18); goto done; }
      }
      // epilogue: O / l -> out, lse. The next unit's first P V overwrites O only after this thread has handed over its P. A warp whose rows all exist
      // stages 64 columns at a time for a tensor store: the rows of a tile are far apart, and 16-byte stores of 32 of them at a time took 1300 clocks
      // per tile at D = 64 and 2700 to 5400 at 128.
      if (!mbar_wait(&pv_done[g], (cnt - 1) & 1, abort_flag)) { atomicExch(p.status, 19); goto done; }
      tc_fence_after();
      const bool ok = qpos < w.seq_len;
      const bool whole = qpos - lane + 31 < w.seq_len;   // uniform over the warp
      const float inv = 1.f / l;
      const int h = g == 0 ? w.h[0] : w.h[1];
      const long long tok = static_cast<long long>(w.seq_start) + qpos;
      __nv_bfloat16* orow = p.out + tok * p.ldo + h * D;
#pragma unroll 1
      for (int c = 0; c < D / 32; c += 2) {
        uint32_t v[2][32];
        tmem_ld_32x32(to + c * 32, v[0]);
        tmem_ld_32x32(to + c * 32 + 32, v[1]);
        if (whole) {   // the box is free once the last store has read it
          if (lane == 0) bulk_wait_read<0>();
          __syncwarp();
        }
        tmem_ld_wait();
        if (whole || ok) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            float o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = __uint_as_float(v[k >> 2][(k & 3) * 8 + i]) * inv;
            const uint4 d = make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
            if (whole) *reinterpret_cast<uint4*>(box + lane * 128 + ((k ^ (lane & 7)) << 4)) = d;
            else *reinterpret_cast<uint4*>(orow + c * 32 + k * 8) = d;
          }
        }
        if (whole) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmap_out, box, h * D + c * 32, w.seq_start + qpos);
            bulk_commit();
          }
        }
      }
      if (ok) p.lse[static_cast<long long>(h) * p.T + tok] = m_ref * p.scale + logf(l);
    }
  }
done:
  if (warp >= 4 && lane == 0) bulk_wait_read<0>();   // before the shared memory goes away
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int D>
static int launch_fwd(const CUtensorMap& tm, const CUtensorMap& to, const AttFwdParams& p, cudaStream_t st) {
  static bool configured = false;
  static int sms = 0;
  auto kern = attn_fwd_kernel<D>;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, AttFwdSmem<D>::TOTAL) != cudaSuccess) return -4;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    configured = true;
  }
  const long long units = static_cast<long long>(p.n_items) * (p.row_pairs ? p.Hq : p.Hq / 2);
  if (units > (1 << 30)) return -10;
  launch_pdl(kern, static_cast<int>(units < sms ? units : sms), ATT_THREADS, AttFwdSmem<D>::TOTAL, st, tm, to, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // namespace mtb

// plan: query-block work table [n_items, 3] = (seq_start, seq_len, q0), most work first: blocks of 128 rows when Hq / Hkv is
// even, of 256 rows (row_pairs) when it is odd.
extern "C" int mtb200_attn_fwd(const void* qkv, long long ld, void* out, long long ldo, float* lse, const int* plan, int n_items,
                               int T, int Hq, int Hkv, int D, int row_pairs, float scale, int* status, cudaStream_t st) {
  using namespace mtb;
  if (n_items <= 0 || T <= 0) return 0;
  if ((D != 64 && D != 128) || Hkv <= 0 || Hq % Hkv || ld % 8 || ldo % 8 || (!row_pairs && (Hq / Hkv) % 2)) return -10;
  CUtensorMap tm;
  CUtensorMap to;
  int rc = make_tmap_2d_bf16(&tm, qkv, static_cast<uint64_t>(ld), static_cast<uint64_t>(T), static_cast<uint64_t>(ld), 64, 128);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&to, out, static_cast<uint64_t>(Hq) * D, static_cast<uint64_t>(T), static_cast<uint64_t>(ldo), 64, 32);
  if (rc) return rc - 10;
  AttFwdParams p{reinterpret_cast<__nv_bfloat16*>(out), ldo, lse, plan, n_items, T, Hq, Hkv, row_pairs, scale, status};
  return D == 128 ? launch_fwd<128>(tm, to, p, st) : launch_fwd<64>(tm, to, p, st);
}
