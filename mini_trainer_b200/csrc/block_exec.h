// Structures and entry points of a decoder block that is queued by one call (block_exec.cu), for the file that queues several (step_exec.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

extern "C" {

typedef unsigned long long u64;

// Products of a block, in the order of the plan: forward qkv, o, gate/up, down; backward the input gradients and the weight gradients.
enum { G_QKV, G_O, G_GU, G_DOWN, D_DOWN, D_GU, D_O, D_QKV, W_DOWN, W_GU, W_O, W_QKV, GEMMS };

struct BlockSpec {
  int T, H, F, Hq, Hkv, D;
  int gated, gelu, layernorm, qk_norm;
  float eps, scale, alpha;
  int form[GEMMS], splits[GEMMS];   // kernel (FORM_ of entries.h) and splits of each product (ops/gemm_plan.py)
  int act_form;                     // kernel of the gate/up product where the activation is in it
  int need_out;                     // 0: the forward stops before the activation
  int attn_form;                    // 0: one query tile per CTA, 1: pairs of heads, 2: pairs of row blocks
  int fwd_items, bwd_items, bwd_splits, bwd_in_order;
};
// Parameters, or their gradients; null where the model has none.
struct BlockParams {
  void *ln1, *bln1, *wqkv, *bqkv, *qn, *kn, *wo, *bo, *ln2, *bln2, *wgu, *bgu, *wd, *bd;
};
struct BlockIO {
  const void* x;
  void *n1, *qkv, *attn, *h1, *n2, *gu, *act, *out, *qk_pre;   // n1, n2, act, out: null where they are not kept (out: not wanted)
  float *mean1, *rstd1, *lse, *mean2, *rstd2, *rstd_qk;
  const int *pos, *fwd_plan, *bwd_plan;
  const float* inv_freq;
  int have_attn;          // attn and lse are there already
  const void* dout;       // backward
  void* dx;
  void* ws;               // workspace
  u64* counters;          // split launches: arrival counters of the stream, growing epochs (used in launch order: GEMMS + 1 are enough), partial sums
  const u64* epochs;
  float* part;
  long long part_bytes;
  int* status;
};

long long mtb200_block_workspace(const BlockSpec* s, const BlockIO* io, int bwd);
int mtb200_block_forward(const BlockSpec* s, const BlockParams* p, const BlockIO* io, int* launches, cudaStream_t st);
int mtb200_block_backward(const BlockSpec* s, const BlockParams* p, const BlockParams* g, const BlockIO* io, int* launches, cudaStream_t st);
}

struct Carver {   // 256-byte aligned pieces of the workspace; with a null base only their sum
  uint8_t* base;
  long long at = 0;
  template <typename T = void> T* take(long long bytes) {
    T* p = base ? reinterpret_cast<T*>(base + at) : nullptr;
    at += (bytes + 255) / 256 * 256;
    return p;
  }
};
