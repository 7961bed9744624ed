// Varlen causal GQA attention backward for sm_100a.
//
// One CTA owns one (sequence, 128-key block, kv head): K and V of that block stay in shared memory
// and dK, dV accumulate in tensor memory over every query head of the GQA group and every query
// block at or below the causal diagonal, so they are written once, without atomics. Per
// (query head, query block) the CTA runs five tcgen05 GEMMs on TRANSPOSED scores (keys on the lanes):
//   S^T = K Q^T        dP^T = V dO^T                        (TMEM, 128 columns each)
//   P^T = exp(S^T*scale - lse), dS^T = P^T * (dP^T - delta) * scale   (8 warps)
//   dV += P^T dO       dK += dS^T Q       dQ = dS K
// With keys on the lanes, P^T and dS^T are the A operands of dV and dK as they stand: they are written back over the
// columns of tensor memory they were computed from and never become shared-memory tiles (a 128 x 128 product with both
// operands in shared memory already reads the 128 bytes per clock that shared memory has). Only dS has a shared-memory
// tile, for dQ, where it is read MN-major. The room that frees holds a second Q tile.
//
// The MMAs of neighbouring iterations interleave so that the softmax of one runs under the products of another. Issue order:
//   ... dK(i) dQ(i) | dP(i+1) dV(i+1) S(i+2) | dK(i+1) dQ(i+1) | ...            (D = 64: dQ in front of dK)
// P(i+1) is computed while dK(i), dQ(i) run and dQ(i) is drained, dS(i+1) while dV(i+1) and S(i+2) run. The chain that bounds
// an iteration is dS -> dK dQ -> drain -> dP -> dS, where the form with everything in one chain (S dP | softmax | dK dV dQ |
// drain) had five products, the whole softmax and the drain. At D = 128 an iteration takes about 4950 clocks for 2560 of MMA,
// the same for every order of the products tried: the chain's hand-offs and latencies, and dQ's tensor reduces of 64 KB.
// 1 x 16384 tokens, 32/8 heads: 6.5 -> 5.5 ms at D = 128 (main kernel),
// 5.3 -> 3.2 ms at D = 64 (all passes; 3.6 with dV in front of dP and the shared columns).
//
// dQ shares the columns of dP at D = 128 (it is read out before the next dP is issued) and has its own at D = 64. Its tiles
// (several key blocks contribute to one query block) go through a 32 KB staging buffer, 64 columns at a time, into an fp32
// [T, Hq*D] accumulator with TMA tensor reduces (cp.reduce.async.bulk.tensor .add, one 32-column x 128-row box each,
// 128B-swizzled so the staging stores are free of bank conflicts); a small kernel rounds the accumulator to bf16 afterwards.
// Four warps of their own drain, one more issues the reduces, so the softmax warps see nothing of dQ.
//
// Rows past the end of the sequence contribute nothing: a query's lse is staged as +infinity, a key's dS is zero.
//
// With short samples a CTA has few iterations, and its first loads and its stores count: the loads go out before tensor memory is allocated, and dK and dV
// leave by tensor stores. 148 samples of 128 tokens, 16/4 heads: 106 -> 102 us at D = 64, 193 -> 182 at 128 (all passes); 37 of 1024 492 -> 482, 879 -> 871.
// The rest of it is dQ's accumulator, which is written, added to and read in fp32: 78 MB of it in 101 us.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "entries.h"
#include "gemm_epilogue.cuh"
#include "ptx.cuh"

namespace mtb {

int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);
int make_tmap_2d_f32(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                     uint32_t box_inner, uint32_t box_outer);

constexpr int AB_B = 128;          // block edge (queries and keys)
// four warpgroups: {TMA, MMA, dQ reduce, row statistics}, 2 x softmax (two threads per key row), dQ drain
constexpr int AB_THREADS = 512;
// Registers per thread after the split; over the four warpgroups they add up to the 4 x 128 of the launch.
constexpr int AB_REGS_IO = 104, AB_REGS_SOFTMAX = 152, AB_REGS_DRAIN = 104;
static_assert(AB_REGS_IO + 2 * AB_REGS_SOFTMAX + AB_REGS_DRAIN == 4 * 128, "register split");

template <int D>
struct AttBwdSmem {
  static constexpr int TILE = AB_B * D * 2;         // a [128, D] bf16 tile
  static constexpr int OFF_K = 0, OFF_V = TILE, OFF_DO = 2 * TILE, OFF_Q = 3 * TILE;   // Q: 2 buffers
  static constexpr int OFF_DS = 5 * TILE;           // dS as [key, query], 128 x 128 bf16
  static constexpr int OFF_ST = OFF_DS + AB_B * AB_B * 2;    // dQ staging: 2 boxes of 128 rows x 32 fp32 columns
  static constexpr int OFF_STAT = OFF_ST + 2 * 16384;        // 2 buffers x {-lse * log2 e, -delta * scale} x 128 queries
  static constexpr int OFF_BAR = OFF_STAT + 2 * 2 * 128 * 4;
  // D = 128 fills the shared memory of an SM, so there is no slack to align with: the kernel checks that the window
  // starts on a 1024-byte boundary (swizzle atom).
  static constexpr int TOTAL = OFF_BAR + 256;
};

struct AttBwdParams {
  __nv_bfloat16* dqkv;
  long long ldq;
  const float* lse;
  const float* delta;
  float* dq_acc;        // [T, Hq*D] fp32, zeroed by attn_delta_kernel
  const int* plan;      // [n_items, 3] = seq_start, seq_len, k0
  int T, Hq, Hkv;
  int G;                // Hq / Hkv
  unsigned hkv_inv;     // (2^32 - 1) / Hkv
  int splits;           // CTAs that share a key block's query heads
  float* ws;            // splits > 1: fp32 partials of dK and dV
  unsigned long long* counters;   // splits > 1: one arrival counter per (key block, warp); last_arrival in gemm_epilogue.cuh
  unsigned long long epoch;
  float scale;
  int* status;
};


template <int D>
__global__ void __launch_bounds__(AB_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_dkv, AttBwdParams p) {
  using L = AttBwdSmem<D>;
  constexpr int KB = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {   // uniform over the CTA: nothing has been allocated or armed yet
    if (threadIdx.x == 0) atomicExch(p.status, 20);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* kv_full = bars;          // K and V resident
  uint64_t* q_full = bars + 1;       // [2] Q landed
  uint64_t* q_free = bars + 3;       // [2] dK has read Q
  uint64_t* do_full = bars + 5;      // dO landed
  uint64_t* do_free = bars + 6;      // dV and dP have read dO
  uint64_t* s_full = bars + 7;       // S^T complete
  uint64_t* dp_full = bars + 8;      // dP^T complete; every earlier MMA too, so the dS tile is writable
  uint64_t* p_ready = bars + 9;      // P^T in tensor memory (8 arrivals)
  uint64_t* ds_ready = bars + 10;    // dS^T in tensor memory and dS in shared memory (8 arrivals)
  uint64_t* dq_full = bars + 11;     // dQ complete
  uint64_t* dq_read = bars + 12;     // dQ read out of tensor memory (4 arrivals): dP columns reusable
  uint64_t* stage_full = bars + 13;  // 64 columns of dQ staged (4 arrivals)
  uint64_t* stage_free = bars + 14;  // the tensor reduces have read the staging buffer
  uint64_t* stat_full = bars + 15;   // [2] lse / delta of a query block staged
  uint64_t* stat_free = bars + 17;   // [2] consumed (8 arrivals)
  uint64_t* all_done = bars + 19;    // dK and dV complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  pdl_wait();   // the work table comes first
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = p.splits == 1 ? blockIdx.x : blockIdx.x / p.splits, sub = blockIdx.x - unit * p.splits;
  int item = static_cast<int>(__umulhi(static_cast<unsigned>(unit), p.hkv_inv));   // unit / Hkv, or one less
  if (unit - item * p.Hkv >= p.Hkv) ++item;
  const int hk = unit - item * p.Hkv;
  const int G = p.G;
  const int h_first = hk * G + (p.splits == 1 ? 0 : G * sub / p.splits), heads = p.splits == 1 ? G : G * (sub + 1) / p.splits - G * sub / p.splits;
  const int seq_start = p.plan[item * 3 + 0], seq_len = p.plan[item * 3 + 1], k0 = p.plan[item * 3 + 2];
  const int jblk = k0 / AB_B;
  const int nq = (seq_len + AB_B - 1) / AB_B;      // query blocks of the sequence
  const int per_head = nq - jblk;                  // query blocks at or below the diagonal
  const int n_iters = heads * per_head;
  // bounds check of the host-built work item (uniform over the CTA; nothing allocated or armed yet)
  if (seq_start < 0 || seq_len <= 0 || k0 < 0 || k0 >= seq_len || static_cast<long long>(seq_start) + seq_len > p.T) {
    if (threadIdx.x == 0) atomicExch(p.status, 61);
    return;
  }

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1); mbar_init(do_full, 1); mbar_init(do_free, 1); mbar_init(s_full, 1); mbar_init(dp_full, 1);
    mbar_init(p_ready, 8); mbar_init(ds_ready, 8); mbar_init(dq_full, 1); mbar_init(dq_read, 4);
    mbar_init(stage_full, 4); mbar_init(stage_free, 1); mbar_init(all_done, 1);
    for (int b = 0; b < 2; ++b) { mbar_init(&q_full[b], 1); mbar_init(&q_free[b], 1); mbar_init(&stat_full[b], 1); mbar_init(&stat_free[b], 8); }
    *abort_flag = 0;
    fence_mbar_init();
    // the first loads go out before anything else is set up
    mbar_arrive_expect_tx(kv_full, 2 * L::TILE);
    mbar_arrive_expect_tx(&q_full[0], L::TILE);
    mbar_arrive_expect_tx(do_full, L::TILE);
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) {
      tma_load_2d(smem + L::OFF_K + kb * 16384, &tm_qkv, kv_full, (p.Hq + hk) * D + kb * 64, seq_start + k0);
      tma_load_2d(smem + L::OFF_Q + kb * 16384, &tm_qkv, &q_full[0], h_first * D + kb * 64, seq_start + jblk * AB_B);
      tma_load_2d(smem + L::OFF_V + kb * 16384, &tm_qkv, kv_full, (p.Hq + p.Hkv + hk) * D + kb * 64, seq_start + k0);
      tma_load_2d(smem + L::OFF_DO + kb * 16384, &tm_do, do_full, h_first * D + kb * 64, seq_start + jblk * AB_B);
    }
    tma_prefetch_desc(&tm_dq);
    tma_prefetch_desc(&tm_dkv);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t t_s = tmem_base, t_dp = tmem_base + 128, t_dv = tmem_base + 256, t_dk = tmem_base + 256 + D;
  // dQ has columns of its own where they are left over (D = 64); at D = 128 it shares those of dP
  constexpr bool DQ_OWN = 2 * 128 + 3 * D <= 512;
  const uint32_t t_dq = DQ_OWN ? tmem_base + 256 + 2 * D : t_dp;

  if (warp < 4) {
    setmaxnreg_dec<AB_REGS_IO>();
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (elect_one()) {
        int h = h_first, i = jblk;
        if (++i == nq) { i = jblk; ++h; }
        for (int it = 1; it < n_iters; ++it) {   // the first iteration's tiles have been asked for above
          const int b = it & 1;
          if (it > 1 && !mbar_wait(&q_free[b], ((it - 2) >> 1) & 1, abort_flag)) { atomicExch(p.status, 21); goto done; }
          mbar_arrive_expect_tx(&q_full[b], L::TILE);
#pragma unroll
          for (int kb = 0; kb < KB; ++kb)
            tma_load_2d(smem + L::OFF_Q + b * L::TILE + kb * 16384, &tm_qkv, &q_full[b], h * D + kb * 64, seq_start + i * AB_B);
          if (it > 0 && !mbar_wait(do_free, (it - 1) & 1, abort_flag)) { atomicExch(p.status, 21); goto done; }
          mbar_arrive_expect_tx(do_full, L::TILE);
#pragma unroll
          for (int kb = 0; kb < KB; ++kb)
            tma_load_2d(smem + L::OFF_DO + kb * 16384, &tm_do, do_full, h * D + kb * 64, seq_start + i * AB_B);
          if (++i == nq) { i = jblk; ++h; }
        }
        pdl_trigger();   // what is left is the last iteration and the stores of dK and dV
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      if (elect_one()) {
        constexpr uint32_t id_nt = make_idesc_bf16(AB_B, AB_B, false, false);   // S^T, dP^T
        constexpr uint32_t id_ts = make_idesc_bf16(AB_B, D, false, true);       // dV, dK (A in tensor memory)
        constexpr uint32_t id_dq = make_idesc_bf16(AB_B, D, true, true);        // dQ = dS K
        // every tile lives at a fixed shared-memory address, so the descriptors are built once; inside
        // the loop a k-step is one add (start-address field, in 16-byte units)
        const uint32_t sk = smem_u32(smem + L::OFF_K), sq = smem_u32(smem + L::OFF_Q), sdo = smem_u32(smem + L::OFF_DO);
        const uint32_t dKk = smem_desc_lo(sk, 16), dVk = smem_desc_lo(smem_u32(smem + L::OFF_V), 16);
        const uint32_t dQk = smem_desc_lo(sq, 16), dDOk = smem_desc_lo(sdo, 16);
        const uint32_t dDSm = smem_desc_lo(smem_u32(smem + L::OFF_DS), 16384), dKm = smem_desc_lo(sk, 16384);
        const uint32_t dQm = smem_desc_lo(sq, 16384), dDOm = smem_desc_lo(sdo, 16384);
        auto kstep = [](int k) { return static_cast<uint32_t>((k >> 2) * 1024 + (k & 3) * 2); };   // K-major: 32 B per step, 16 KB per 64
        auto mstep = [](int k) { return static_cast<uint32_t>(k * 128); };                           // MN-major: 2048 B per step
        auto astep = [](int k) { return static_cast<uint32_t>(k < 4 ? k * 8 : 64 + (k - 4) * 8); };   // bf16 A operand in tensor memory
        auto qbuf = [&](int it) { return static_cast<uint32_t>((it & 1) * (L::TILE >> 4)); };
        auto issue_s = [&](int it) {
#pragma unroll
          for (int k = 0; k < D / 16; ++k) umma_bf16_lo(t_s, dKk + kstep(k), dQk + qbuf(it) + kstep(k), id_nt, k != 0);
          umma_commit(s_full);
        };
        auto issue_dp = [&]() {
#pragma unroll
          for (int k = 0; k < D / 16; ++k) umma_bf16_lo(t_dp, dVk + kstep(k), dDOk + kstep(k), id_nt, k != 0);
          umma_commit(dp_full);
        };
        auto issue_dv = [&](int it) {   // dP of the same iteration has been issued: dO is free when both are done
#pragma unroll
          for (int k = 0; k < AB_B / 16; ++k) umma_bf16_ts_lo(t_dv, t_s + astep(k), dDOm + mstep(k), id_ts, it != 0 || k != 0);
          umma_commit(do_free);
        };
        if (!mbar_wait(kv_full, 0, abort_flag)) { atomicExch(p.status, 22); goto done; }
        if (!mbar_wait(&q_full[0], 0, abort_flag)) { atomicExch(p.status, 23); goto done; }
        tc_fence_after();
        issue_s(0);
        if (!mbar_wait(do_full, 0, abort_flag)) { atomicExch(p.status, 23); goto done; }
        tc_fence_after();
        issue_dp();
        if (!mbar_wait(p_ready, 0, abort_flag)) { atomicExch(p.status, 25); goto done; }
        tc_fence_after();
        issue_dv(0);
        if (n_iters > 1) {
          if (!mbar_wait(&q_full[1], 0, abort_flag)) { atomicExch(p.status, 23); goto done; }
          tc_fence_after();
          issue_s(1);
        }
        auto issue_dk = [&](int it) {
#pragma unroll
          for (int k = 0; k < AB_B / 16; ++k) umma_bf16_ts_lo(t_dk, t_dp + astep(k), dQm + qbuf(it) + mstep(k), id_ts, it != 0 || k != 0);
          umma_commit(&q_free[it & 1]);
        };
        auto issue_dq = [&]() {
#pragma unroll
          for (int k = 0; k < AB_B / 16; ++k) umma_bf16_lo(t_dq, dDSm + mstep(k), dKm + mstep(k), id_dq, k != 0);
          umma_commit(dq_full);
        };
        for (int it = 0; it < n_iters; ++it) {
          if (!mbar_wait(ds_ready, it & 1, abort_flag)) { atomicExch(p.status, 25); goto done; }
          if (DQ_OWN && it > 0 && !mbar_wait(dq_read, (it - 1) & 1, abort_flag)) { atomicExch(p.status, 24); goto done; }
          tc_fence_after();
          if (DQ_OWN) { issue_dq(); issue_dk(it); }
          else { issue_dk(it); issue_dq(); }     // dK reads dS^T from the columns that dQ overwrites
          if (it + 1 < n_iters) {
            if (!mbar_wait(do_full, (it + 1) & 1, abort_flag)) { atomicExch(p.status, 23); goto done; }
            if (!DQ_OWN && !mbar_wait(dq_read, it & 1, abort_flag)) { atomicExch(p.status, 24); goto done; }
            tc_fence_after();
            issue_dp();
            if (!mbar_wait(p_ready, (it + 1) & 1, abort_flag)) { atomicExch(p.status, 25); goto done; }
            tc_fence_after();
            issue_dv(it + 1);
            if (it + 2 < n_iters) {
              if (!mbar_wait(&q_full[it & 1], ((it + 2) >> 1) & 1, abort_flag)) { atomicExch(p.status, 23); goto done; }
              tc_fence_after();
              issue_s(it + 2);
            }
          }
        }
        umma_commit(all_done);
      }
    } else if (warp == 2) {
      // ------------------------------------------------------------------ dQ reduce warp
      if (elect_one()) {
        const uint32_t stage = smem_u32(smem + L::OFF_ST);
        int h = h_first, i = jblk, n = 0;
        for (int it = 0; it < n_iters; ++it) {
          for (int part = 0; part < KB; ++part, ++n) {
            if (!mbar_wait(stage_full, n & 1, abort_flag)) { atomicExch(p.status, 30); goto done; }
#pragma unroll
            for (int c = 0; c < 2; ++c)
              asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
                           ::"l"(reinterpret_cast<uint64_t>(&tm_dq)), "r"(stage + c * 16384), "r"(h * D + part * 64 + c * 32),
                             "r"(seq_start + i * AB_B) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            mbar_arrive(stage_free);
          }
          if (++i == nq) { i = jblk; ++h; }
        }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // every add has been performed before the CTA exits
      }
    } else {
      // ------------------------------------------------------------------ row statistics of the query blocks
      float* stat = reinterpret_cast<float*>(smem + L::OFF_STAT);
      int h = h_first, i = jblk;
      for (int it = 0; it < n_iters; ++it) {
        const int b = it & 1;
        if (it > 1 && !mbar_wait(&stat_free[b], ((it - 2) >> 1) & 1, abort_flag)) { atomicExch(p.status, 32); goto done; }
        const long long base = static_cast<long long>(h) * p.T + seq_start;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int x = j * 32 + lane, qpos = i * AB_B + x;
          const bool ok = qpos < seq_len;
          stat[b * 256 + x] = ok ? p.lse[base + qpos] * -1.4426950408889634f : -INFINITY;
          stat[b * 256 + 128 + x] = ok ? p.delta[base + qpos] * -p.scale : 0.f;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&stat_full[b]);
        if (++i == nq) { i = jblk; ++h; }
      }
    }
  } else if (warp >= 12) {
    // ------------------------------------------------------------------ dQ drain (one thread per query row)
    setmaxnreg_dec<AB_REGS_DRAIN>();
    const int r = (warp & 3) * 32 + lane;
    const uint32_t src = t_dq + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    uint8_t* rowp = smem + L::OFF_ST + r * 128;
    int n = 0;
    for (int it = 0; it < n_iters; ++it) {
      if (!mbar_wait(dq_full, it & 1, abort_flag)) { atomicExch(p.status, 28); goto done; }
      tc_fence_after();
#pragma unroll 1
      for (int part = 0; part < KB; ++part, ++n) {
        uint32_t v[2][32];
        tmem_ld_32x32(src + part * 64, v[0]);
        tmem_ld_32x32(src + part * 64 + 32, v[1]);
        tmem_ld_wait();
        if (part == KB - 1) {   // the last columns are in registers: the next dP may overwrite them
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_read);
        }
        if (n > 0 && !mbar_wait(stage_free, (n - 1) & 1, abort_flag)) { atomicExch(p.status, 31); goto done; }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int g = 0; g < 8; ++g)
            *reinterpret_cast<uint4*>(rowp + c * 16384 + ((g ^ (r & 7)) << 4)) = make_uint4(v[c][g * 4], v[c][g * 4 + 1], v[c][g * 4 + 2], v[c][g * 4 + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(stage_full);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax (two threads per key row)
    setmaxnreg_inc<AB_REGS_SOFTMAX>();
    const int q = warp & 3;
    const int half = (warp >> 2) - 1;      // which 64 queries (softmax) / which half of the D columns (epilogue)
    const int r = q * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t ts = t_s + lane_addr + half * 64, tp = t_dp + lane_addr + half * 64;
    const float sl2 = p.scale * 1.4426950408889634f;
    const float2 sl2v = make_float2(sl2, sl2), scv = make_float2(p.scale, p.scale);
    uint8_t* ds_row = smem + L::OFF_DS + half * 16384 + r * 128;
    int i = jblk;
    for (int it = 0; it < n_iters; ++it) {
      const int b = it & 1;
      const float* stat = reinterpret_cast<const float*>(smem + L::OFF_STAT) + b * 256 + half * 64;
      if (!mbar_wait(&stat_full[b], (it >> 1) & 1, abort_flag)) { atomicExch(p.status, 26); goto done; }
      if (!mbar_wait(s_full, it & 1, abort_flag)) { atomicExch(p.status, 26); goto done; }
      tc_fence_after();
      float2 pr[32];      // probabilities of this thread's 64 (key, query) pairs
      {
        uint32_t sv[2][32];
        tmem_ld_32x32(ts, sv[0]);
        tmem_ld_32x32(ts + 32, sv[1]);
        tmem_ld_wait();
        if (i == jblk) {   // diagonal block: of the queries, 32 at a time, a warp's keys are seen by none before piece q, by those from the lane on in it
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            if (half * 2 + cc <= q) {
#pragma unroll
              for (int x = 0; x < 32; ++x)
                if (half * 2 + cc < q || lane > x) sv[cc][x] = 0xff800000u;   // exp2(-inf) = 0
            }
          }
        }
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t pk[16];
#pragma unroll
          for (int x = 0; x < 32; x += 4) {
            const float4 nl = *reinterpret_cast<const float4*>(stat + cc * 32 + x);
            // packed fp32 pairs: one FMA scales and shifts two scores
            const float2 a0 = ffma2(make_float2(__uint_as_float(sv[cc][x]), __uint_as_float(sv[cc][x + 1])), sl2v, make_float2(nl.x, nl.y));
            const float2 a1 = ffma2(make_float2(__uint_as_float(sv[cc][x + 2]), __uint_as_float(sv[cc][x + 3])), sl2v, make_float2(nl.z, nl.w));
            // a quarter of the exponentials runs on the FMA pipe: the special-function unit bounds this phase
            const float2 e0 = make_float2(ex2_mufu(a0.x), ex2_mufu(a0.y)), e1 = make_float2(ex2_mufu(a1.x), ex2_fma(a1.y));
            pr[cc * 16 + (x >> 1)] = e0;
            pr[cc * 16 + (x >> 1) + 1] = e1;
            pk[x >> 1] = pack_bf16(e0.x, e0.y);
            pk[(x >> 1) + 1] = pack_bf16(e1.x, e1.y);
          }
          tmem_st_32x16(ts + cc * 16, pk);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      if (!mbar_wait(dp_full, it & 1, abort_flag)) { atomicExch(p.status, 27); goto done; }
      tc_fence_after();
      uint32_t dv[2][32];
      tmem_ld_32x32(tp, dv[0]);
      tmem_ld_32x32(tp + 32, dv[1]);
      tmem_ld_wait();
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t dk[16];
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
          const float4 nd = *reinterpret_cast<const float4*>(stat + 128 + cc * 32 + x);
          // one FMA forms (dP - delta) * scale for two entries
          const float2 d0 = ffma2(make_float2(__uint_as_float(dv[cc][x]), __uint_as_float(dv[cc][x + 1])), scv, make_float2(nd.x, nd.y));
          const float2 d1 = ffma2(make_float2(__uint_as_float(dv[cc][x + 2]), __uint_as_float(dv[cc][x + 3])), scv, make_float2(nd.z, nd.w));
          const float2 s0 = fmul2(pr[cc * 16 + (x >> 1)], d0), s1 = fmul2(pr[cc * 16 + (x >> 1) + 1], d1);
          dk[x >> 1] = pack_bf16(s0.x, s0.y);
          dk[(x >> 1) + 1] = pack_bf16(s1.x, s1.y);
        }
        if (k0 + AB_B > seq_len) {   // last key block: keys past the sequence give nothing to dQ (their rows of dK and dV are not stored)
#pragma unroll
          for (int x = 0; x < 16; ++x) dk[x] = k0 + r < seq_len ? dk[x] : 0u;
        }
        tmem_st_32x16(tp + cc * 16, dk);
#pragma unroll
        for (int g = 0; g < 4; ++g)
          *reinterpret_cast<uint4*>(ds_row + (((cc * 4 + g) ^ (r & 7)) << 4)) = make_uint4(dk[g * 4], dk[g * 4 + 1], dk[g * 4 + 2], dk[g * 4 + 3]);
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(ds_ready); mbar_arrive(&stat_free[b]); }
      if (++i == nq) i = jblk;
    }
    // epilogue: dK, dV (rows = keys)
    if (!mbar_wait(all_done, 0, abort_flag)) { atomicExch(p.status, 29); goto done; }
    tc_fence_after();
    const int kpos = k0 + r;
    const bool ok = kpos < seq_len;
    const bool whole = kpos - lane + 31 < seq_len;   // uniform over the warp
    __nv_bfloat16* rowp = p.dqkv + (static_cast<long long>(seq_start) + kpos) * p.ldq;
    // A warp has 64 columns of one gradient (D = 64: dK or dV) or of both (D = 128), in pieces of 32; rows that all exist leave by tensor stores, staged
    // where Q was (stored 16 bytes at a time to rows that are far apart, they took 3500 clocks per CTA at D = 64 and 9000 at 128).
    constexpr int PIECES = D / 32, BOXES = D / 64;
    constexpr int PART = PIECES * 1024;   // floats of a warp's partial
    uint8_t* box = smem + L::OFF_Q + (warp - 4) * BOXES * 4096;
    auto gradient = [&](int x) { return D == 64 ? half : x >> 1; };                          // 0: dK, 1: dV
    auto column = [&](int x) { return D == 64 ? x * 32 : half * 64 + (x & 1) * 32; };
    auto store = [&](int x, const float (&f)[32]) {   // piece x of this thread's row
      const int col = (gradient(x) == 0 ? p.Hq + hk : p.Hq + p.Hkv + hk) * D + column(x);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const uint4 d = make_uint4(pack_bf16(f[g * 8], f[g * 8 + 1]), pack_bf16(f[g * 8 + 2], f[g * 8 + 3]),
                                   pack_bf16(f[g * 8 + 4], f[g * 8 + 5]), pack_bf16(f[g * 8 + 6], f[g * 8 + 7]));
        if (whole) *reinterpret_cast<uint4*>(box + (x >> 1) * 4096 + lane * 128 + ((((x & 1) * 4 + g) ^ (lane & 7)) << 4)) = d;
        else if (ok) *reinterpret_cast<uint4*>(rowp + col + g * 8) = d;
      }
      if (whole && (x & 1)) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tm_dkv, box + (x >> 1) * 4096, col - 32, seq_start + kpos);
          bulk_commit();
        }
      }
    };
    float* base = p.ws + (static_cast<long long>(unit) * p.splits * 8 + (warp - 4)) * PART + lane * 4;   // split s: + s * 8 * PART
#pragma unroll 1
    for (int x = 0; x < PIECES; ++x) {
      uint32_t v[32];
      tmem_ld_32x32((gradient(x) == 0 ? t_dk : t_dv) + lane_addr + column(x), v);
      tmem_ld_wait();
      float f[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
      if (p.splits == 1) store(x, f);
      else {   // lane-interleaved 16-byte pieces: every access is one contiguous 512 bytes
#pragma unroll
        for (int j = 0; j < 8; ++j)
          __stcg(reinterpret_cast<float4*>(base + static_cast<long long>(sub) * 8 * PART + x * 1024 + j * 128), make_float4(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]));
      }
    }
    if (p.splits > 1) {   // the warp that arrives last adds the partials, in split order whoever that is; nobody waits
      unsigned long long* counter = p.counters + unit * 8 + (warp - 4);
      __threadfence();
      __syncwarp();
      unsigned last = 0;
      if (lane == 0) last = last_arrival(counter, p.epoch, p.splits);
      last = __shfl_sync(0xffffffffu, last, 0);
      if (last) {
        __threadfence();
#pragma unroll 1
        for (int x = 0; x < PIECES; ++x) {
          float f[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = 0.f;
#pragma unroll 2
          for (int s = 0; s < p.splits; ++s) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 t = __ldcg(reinterpret_cast<const float4*>(base + static_cast<long long>(s) * 8 * PART + x * 1024 + j * 128));
              f[4 * j] += t.x; f[4 * j + 1] += t.y; f[4 * j + 2] += t.z; f[4 * j + 3] += t.w;
            }
          }
          store(x, f);
        }
        if (lane == 0) *counter = 0;
      }
    }
    if (lane == 0) bulk_wait_read<0>();   // before the shared memory goes away
  }
done:
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d], and zeros into the dQ accumulator; D / 8 lanes per (t, h), one 16-byte load of each operand per
// lane and row, two rows in flight. Bound by reading dO and O and writing the accumulator once (as a launch of its own the zeroing
// took 9 us next to 14 us for 12 345 tokens x 16 heads of 64, forward and backward together 177 us, now 168).
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o, long long ldo, const __nv_bfloat16* __restrict__ dout,
                                                        long long lddo, float* __restrict__ delta, float* __restrict__ dq_acc, int T, int Hq, int D) {
  pdl_trigger();
  pdl_wait();
  const int lanes = D >> 3;   // 8 or 16: a power of two that divides the warp
  const int per_block = 256 / lanes, sub = threadIdx.x / lanes, c = (threadIdx.x & (lanes - 1)) * 8;
  const long long rows = static_cast<long long>(T) * Hq, first = static_cast<long long>(blockIdx.x) * 2 * per_block + sub;
  uint4 a[2], b[2];
  int t[2], h[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const long long row = first + k * per_block;
    a[k] = b[k] = make_uint4(0u, 0u, 0u, 0u);
    t[k] = rows <= 0xffffffffLL ? static_cast<int>(static_cast<unsigned>(row) / static_cast<unsigned>(Hq)) : static_cast<int>(row / Hq);
    h[k] = static_cast<int>(row - static_cast<long long>(t[k]) * Hq);
    if (row < rows) {
      a[k] = *reinterpret_cast<const uint4*>(o + static_cast<long long>(t[k]) * ldo + h[k] * D + c);
      b[k] = *reinterpret_cast<const uint4*>(dout + static_cast<long long>(t[k]) * lddo + h[k] * D + c);
    }
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const long long row = first + k * per_block;
    const uint32_t av[4] = {a[k].x, a[k].y, a[k].z, a[k].w}, bv[4] = {b[k].x, b[k].y, b[k].z, b[k].w};
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 u = unpack_bf16(av[i]), v = unpack_bf16(bv[i]);
      s += u.x * v.x + u.y * v.y;
    }
    for (int m = lanes >> 1; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (row < rows) {
      if (c == 0) delta[static_cast<long long>(h[k]) * T + t[k]] = s;
      float4* z = reinterpret_cast<float4*>(dq_acc + row * D + c);
      z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// dqkv[t, 0:Hq*D] = bf16(dq_acc[t, :])
__global__ void __launch_bounds__(256) attn_dq_store_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dqkv, long long ldq,
                                                           long long T, int HqD) {
  pdl_trigger();
  pdl_wait();
  // grid = (tokens, column blocks): no 64-bit division per thread
  const long long t = blockIdx.x;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= HqD) return;
  const float4 a = *reinterpret_cast<const float4*>(acc + t * HqD + c), b = *reinterpret_cast<const float4*>(acc + t * HqD + c + 4);
  *reinterpret_cast<uint4*>(dqkv + t * ldq + c) =
      make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
}

template <int D>
static int launch_bwd(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& c, const CUtensorMap& d, const AttBwdParams& p, int n_items, bool in_order, cudaStream_t st) {
  static bool configured = false;
  auto kern = attn_bwd_kernel<D>;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, AttBwdSmem<D>::TOTAL) != cudaSuccess) return -4;
    configured = true;
  }
  // Blocks that come under their predecessor's tail stand on whatever SMs are free first; launched behind its end (in_order), consecutive ones (the kv heads of a
  // key block) go round the chip in order. Where a block has many iterations that decides more than the 3 us of an early launch: the kernel alone, D = 128, 4313 tokens,
  // 32/8 heads, 174 us in order and 195 early with 4 samples, 370 and 406 with one. The rule is attention_plan.backward_in_order.
  const unsigned grid = n_items * p.Hkv * p.splits;
  if (in_order) kern<<<grid, AB_THREADS, AttBwdSmem<D>::TOTAL, st>>>(a, b, c, d, p);
  else launch_pdl(kern, grid, AB_THREADS, AttBwdSmem<D>::TOTAL, st, a, b, c, d, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // namespace mtb

// plan: key-block work table [n_items, 3] = (seq_start, seq_len, k0), most work first.
// dq_acc: fp32 [T, Hq*D] scratch, 16-byte aligned; delta: fp32 [Hq, T] scratch.
// splits: CTAs that share the query heads of a key block; more than one needs counters, an epoch and scratch as the split-K GEMM does.
// in_order: the kernel is launched behind its predecessor's end (launch_bwd).
extern "C" int mtb200_attn_bwd(const void* qkv, long long ld, const void* out, long long ldo, const void* dout, long long lddo,
                               void* dqkv, long long ldq, const float* lse, float* delta, float* dq_acc, const int* plan,
                               int n_items, int T, int Hq, int Hkv, int D, int splits, unsigned long long* counters, unsigned long long epoch, float* part, long long part_bytes, float scale, int in_order, int* status, cudaStream_t st) {
  using namespace mtb;
  if (n_items <= 0 || T <= 0) return 0;
  if ((D != 64 && D != 128) || Hq % Hkv || ld % 8 || ldo % 8 || lddo % 8 || ldq % 8 || splits < 1 || splits > Hq / Hkv) return -10;
  const long long units = static_cast<long long>(n_items) * Hkv;
  if (splits > 1 && (part == nullptr || counters == nullptr || units * 8 > SPLIT_COUNTERS || splits * units * 2 * AB_B * D * 4 > part_bytes)) return -11;
  CUtensorMap tq, tdo, tdq, tdkv;
  int rc = make_tmap_2d_bf16(&tq, qkv, static_cast<uint64_t>(ld), static_cast<uint64_t>(T), static_cast<uint64_t>(ld), 64, 128);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tdo, dout, static_cast<uint64_t>(Hq) * D, static_cast<uint64_t>(T), static_cast<uint64_t>(lddo), 64, 128);
  if (rc) return rc - 10;
  rc = make_tmap_2d_f32(&tdq, dq_acc, static_cast<uint64_t>(Hq) * D, static_cast<uint64_t>(T), static_cast<uint64_t>(Hq) * D, 32, 128);
  if (rc) return rc - 20;
  rc = make_tmap_2d_bf16(&tdkv, dqkv, (static_cast<uint64_t>(Hq) + 2 * Hkv) * D, static_cast<uint64_t>(T), static_cast<uint64_t>(ldq), 64, 32);
  if (rc) return rc - 30;
  const int per_block = 2 * 256 / (D / 8);
  launch_pdl(attn_delta_kernel, static_cast<unsigned>((static_cast<long long>(T) * Hq + per_block - 1) / per_block), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(out), ldo, reinterpret_cast<const __nv_bfloat16*>(dout), lddo, delta, dq_acc, T, Hq, D);
  AttBwdParams p{reinterpret_cast<__nv_bfloat16*>(dqkv), ldq, lse, delta, dq_acc, plan, T, Hq, Hkv, Hq / Hkv, 0xffffffffu / static_cast<unsigned>(Hkv), splits,
                 part, counters, epoch, scale, status};
  rc = D == 128 ? launch_bwd<128>(tq, tdo, tdq, tdkv, p, n_items, in_order != 0, st) : launch_bwd<64>(tq, tdo, tdq, tdkv, p, n_items, in_order != 0, st);
  if (rc) return rc;
  launch_pdl(attn_dq_store_kernel, dim3(static_cast<unsigned>(T), (Hq * D / 8 + 255) / 256), 256, 0, st, dq_acc, reinterpret_cast<__nv_bfloat16*>(dqkv), ldq, T, Hq * D);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
