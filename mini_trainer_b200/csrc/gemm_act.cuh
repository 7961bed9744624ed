// Products that end at an MLP's activation take it into their epilogue, so that the pre-activations are not read back and passed over again by
// a bandwidth-bound kernel. They are rounded to bf16 before the activation reads them, as if they had been stored in between.
//   ACT_GLU    pre = A * [Wg; Wu]^T, act = f(g) * u. A tile's 256 columns are 128 of the gate and the same 128 of up, so that one thread has both.
//   ACT_PLAIN  pre = A * B (+ bias), act = f(pre): an MLP without a gate
// Eight warps, two per 32-row quarter: with four (one per scheduler) the arithmetic of a tile took longer than short reductions. They work on
// 32 columns at a time, staged as boxes of 32 rows x 64 bytes (64B-swizzled). Bound by the product. With its activation, in a loop of its own on a B200:
// 5987 x 17920 x 1536 272 -> 231 us (product alone 220), 4099 x 12288 x 2048 167 -> 153, 16384 x 28672 x 4096 3.16 -> 2.8 ms, 7001 x 12288 x 3072 without
// a gate 448 -> 375 us; over the slabs of 64 experts (20 500 rows x 2048 x 2048) 150 + 24 -> 153, of 8 (9200 x 28672 x 4096) 1378 + 117 -> 1434.
// Forward and backward of whole layers, without and with it in one process: 1.5B block 1830 -> 1796 us, q/k-norm block 1700 -> 1680, 64 experts 1042 -> 1024,
// 8 experts 7985 -> 7897; an 8B block (20.0 ms) and a LayerNorm block (4.2 ms) by less than their runs differ.
//
// The other direction, the activation's gradient in the epilogue of the product in front of it, was tried with the pre-activations loaded
// by TMA two boxes ahead and either form of stores. It gained up to a fifth alone (5987 x 8960 x 1536 243 -> 190 us) and nothing in a
// block: five tensors of a tile's width pass through its epilogue, which then takes longer than its products up to a reduction of 2000, and
// longer ones run at the power cap, where the time is given by what is computed and moved.
#pragma once
#include <cuda.h>

#include "gemm_epilogue.cuh"
#include "ptx.cuh"

namespace mtb {

enum { ACT_NONE = 0, ACT_GLU = 1, ACT_PLAIN = 2 };

struct ActParams {
  int F;          // width of the activation
  int gelu;       // 0: SiLU, 1: tanh-approximated GELU
};
// Tensor maps of gate (or x), up and act, boxes of 32 rows x 32 columns, 64B-swizzled; nothing in instances without an activation.
template <int ACT> struct ActMaps { CUtensorMap gate, up, act; };
template <> struct ActMaps<ACT_NONE> {};

constexpr int ACT_WARPS = 8;
constexpr int ACT_BOX = 32 * 64;                     // bytes of a box
static_assert(ACT_WARPS * 2 * ACT_BOX == EPI_SMEM, "two boxes per warp");

// A thread's row in a box: four 16-byte pieces.
__device__ __forceinline__ uint4* box_piece(uint8_t* box, int lane, int i) {
  return reinterpret_cast<uint4*>(box + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4));
}
__device__ __forceinline__ float2 sigmoid2(float2 x) {   // 1 / (1 + exp(-x))
  return make_float2(__fdividef(1.f, 1.f + exp_ftz(-x.x)), __fdividef(1.f, 1.f + exp_ftz(-x.y)));
}
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }
// The factor s of f(x) = x * s, for two x.
__device__ __forceinline__ float2 act_gate2(float2 x, bool gelu) {
  if (!gelu) return sigmoid2(x);
  const float2 q = ffma2(fmul2(x, x), f2(0.044715f), f2(1.f));            // gelu_gate on pairs
  return sigmoid2(fmul2(fmul2(x, q), f2(1.5957691216057308f)));
}
__device__ __forceinline__ uint32_t pack2(float2 v) { return pack_bf16(v.x, v.y); }

// Two columns: f(g) (GATED: times u) of the rounded pre-activations.
template <bool GATED>
__device__ __forceinline__ uint32_t act_pair(uint32_t g, uint32_t u, bool gelu) {
  const float2 x = unpack_bf16(g);
  float2 f = fmul2(x, act_gate2(x, gelu));
  if (GATED) f = fmul2(f, unpack_bf16(u));
  return pack2(f);
}
// One warp's part of a tile, `half` of its columns (gated: 64 of the gate and the same of up, else 128). `out`: this warp's two boxes.
template <int ACT>
__device__ __forceinline__ void epilogue_act(const EpiParams& p, const ActParams& ap, const ActMaps<ACT>& maps, EpiOut& out, uint32_t taddr, int row0,
                                                 int tn, int q, int half, int lane) {
  constexpr bool GLU = ACT == ACT_GLU;
  const int y0 = row0 + q * 32;
  if (y0 >= p.M) return;
  auto send = [&](const CUtensorMap& map, const uint32_t (&d)[16], int col) {
    if (lane == 0) bulk_wait_read<1>();
    __syncwarp();
    uint8_t* box = out.stage + (out.n & 1) * ACT_BOX;
#pragma unroll
    for (int i = 0; i < 4; ++i) *box_piece(box, lane, i) = make_uint4(d[4 * i], d[4 * i + 1], d[4 * i + 2], d[4 * i + 3]);
    out.map = &map;
    store_box(out, box, col, y0, lane);
  };
#pragma unroll 1
  for (int c = 0; c < (GLU ? 2 : 4); ++c) {
    const int at = half * (GLU ? 64 : 128) + c * 32, col = tn * (GLU ? 128 : 256) + at;
    if (col >= ap.F) break;
    uint32_t v[32], g[16], u[GLU ? 16 : 1];
    tmem_ld_32x32(taddr + at, v);
    tmem_ld_wait();
    if (ACT == ACT_PLAIN && p.bias != nullptr) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (col + i * 8 < ap.F) {
          const uint4 b = *reinterpret_cast<const uint4*>(p.bias + col + i * 8);
          const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 bb = unpack_bf16(bw[j]);
            v[i * 8 + 2 * j] = __float_as_uint(__uint_as_float(v[i * 8 + 2 * j]) + bb.x);
            v[i * 8 + 2 * j + 1] = __float_as_uint(__uint_as_float(v[i * 8 + 2 * j + 1]) + bb.y);
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) g[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
    if constexpr (GLU) tmem_ld_32x32(taddr + 128 + at, v);
    send(maps.gate, g, col);
    if constexpr (GLU) {
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) u[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
      send(maps.up, u, col);
    }
    if (ap.gelu) {
#pragma unroll
      for (int j = 0; j < 16; ++j) g[j] = act_pair<GLU>(g[j], u[GLU ? j : 0], true);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) g[j] = act_pair<GLU>(g[j], u[GLU ? j : 0], false);
    }
    send(maps.act, g, col);
  }
}

// The same for wide tiles: one warp has all 256 columns of its quarter and reads them before it works on any; boxes of 32 rows x 128 bytes, one per
// warp (epilogue_wide). The maps are of such boxes.
template <int ACT, typename Drained>
__device__ __forceinline__ void epilogue_act_wide(const EpiParams& p, const ActParams& ap, const ActMaps<ACT>& maps, EpiOut& out, uint32_t taddr,
                                                  int row0, int row_end, int tn, int q, int lane, Drained drained) {
  constexpr bool GLU = ACT == ACT_GLU;
  const int y0 = row0 + q * 32;
  if (y0 >= row_end) { drained(); return; }
  uint32_t d[8][16];   // gated: four pieces of the gate, then four of up
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    uint32_t v[32];
    tmem_ld_32x32(taddr + c * 32, v);
    tmem_ld_wait();
    if (ACT == ACT_PLAIN && p.bias != nullptr) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = tn * 256 + c * 32 + i * 8;
        if (col < ap.F) {
          const uint4 b = *reinterpret_cast<const uint4*>(p.bias + col);
          const float2 b0 = unpack_bf16(b.x), b1 = unpack_bf16(b.y), b2 = unpack_bf16(b.z), b3 = unpack_bf16(b.w);
          const float add[8] = {b0.x, b0.y, b1.x, b1.y, b2.x, b2.y, b3.x, b3.y};
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i * 8 + j] = __float_as_uint(__uint_as_float(v[i * 8 + j]) + add[j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) d[c][j] = formed(pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])));
  }
  drained();
#pragma unroll 1
  for (int c = 0; c < (GLU ? 4 : 8); c += 2) {
    const int col = tn * (GLU ? 128 : 256) + c * 32;
    if (col >= ap.F) break;
    out.map = &maps.gate;
    send_columns64(out, d, col, y0, lane);
    if constexpr (GLU) {
      out.map = &maps.up;
      send_columns64(out, d + 4, col, y0, lane);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (ap.gelu) {
#pragma unroll
        for (int j = 0; j < 16; ++j) d[k][j] = act_pair<GLU>(d[k][j], d[GLU ? 4 + k : k][j], true);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) d[k][j] = act_pair<GLU>(d[k][j], d[GLU ? 4 + k : k][j], false);
      }
    }
    out.map = &maps.act;
    send_columns64(out, d, col, y0, lane);
    next_pieces<GLU ? 4 : 8, 2>(d);
    if constexpr (GLU) next_pieces<4, 2>(d + 4);
  }
}

}  // namespace mtb
