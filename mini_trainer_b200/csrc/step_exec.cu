// Forward and backward of one minibatch through a whole small model, queued by one call: embedding, blocks (block_exec.cu), head with its loss, the
// blocks' backward, embedding gradient, and the accumulation of every group's gradient. It is the schedule of parallel/engine.py for one rank that
// keeps every block's activations, with the same kernels in the same order. What goes is the interpreter around the blocks, which is what a step of a
// small model is bound by: about 70 launches take the host 2 to 3 us each, and took 10 with what stood between them. Training step of 640 tokens
// through 2 layers 976 -> 553 us, of 4096 tokens 1072 -> 950 (where the device is the bound).
//
// Memory: one workspace from the caller, laid out here (mtb200_step_workspace says how large), which holds the activations of all blocks; nothing is
// kept between calls.
#include <cuda_runtime.h>
#include <stdint.h>

#include "block_exec.h"
#include "entries.h"

extern "C" {

constexpr int STEP_PARAMS = 14;   // of a block, in the order of BlockParams

struct StepSpec {
  BlockSpec block;                   // of every block
  int layers, V, R;                  // R: rows that the head runs on, T: all of them
  int tied;
  float logit_alpha, grad_scale;
  int form[3], splits[3];            // products of the head: logits, input gradient, weight gradient
  long long off[STEP_PARAMS];        // elements from the start of a block's buffers, -1: the model has no such tensor
  long long off_embed, off_norm, off_bnorm, off_lm;   // in the embedding's buffers; in the head's (tied: off_lm in the embedding's)
};
struct StepGroup {                   // flat buffers of a parameter group
  void *param, *grad;                // bf16
  float* acc;                        // fp32 accumulator
  long long n;
  int add;                           // 0: the accumulator holds nothing yet
};
struct StepIO {
  const StepGroup *embed, *blocks, *head;   // blocks: one per layer
  const float* const* inv_freq;             // per layer, null: no rotation
  const long long *ids, *targets, *rows;    // targets of the R rows; rows: null when R == T
  const int *pos, *fwd_plan, *bwd_plan;
  float* loss;                              // [T]
  void* ws;
  u64* counters;                            // as in BlockIO; 13 epochs per layer and 3 for the head
  const u64* epochs;
  float* part;
  long long part_bytes;
  int* status;
};
}

namespace {

// What a block keeps from its forward to its backward.
struct Kept {
  void *x, *qkv, *attn, *h1, *gu, *qk_pre;
  float *mean1, *rstd1, *lse, *mean2, *rstd2, *rstd_qk;
};

long long run(const StepSpec& s, const StepIO& io, bool measure, cudaStream_t st, int* launches) {
  const BlockSpec& b = s.block;
  const long long T = b.T, H = b.H, q = static_cast<long long>(b.Hq) * b.D, kv = static_cast<long long>(b.Hkv) * b.D, R = s.R, V = s.V;
  const bool ln = b.layernorm != 0;
  Carver ws{measure ? nullptr : static_cast<uint8_t*>(io.ws)};
  constexpr int MOST_LAYERS = 256;
  static_assert(sizeof(Kept) * MOST_LAYERS < 64 * 1024, "on the stack");
  if (s.layers < 1 || s.layers > MOST_LAYERS || R < 1 || R > T) return -10;
  Kept kept[MOST_LAYERS];
  for (int i = 0; i < s.layers; ++i) {
    Kept& k = kept[i];
    k.x = ws.take(T * H * 2);
    k.qkv = ws.take(T * (q + 2 * kv) * 2);
    k.attn = ws.take(T * q * 2);
    k.h1 = ws.take(T * H * 2);
    k.gu = ws.take(T * (b.gated ? 2LL * b.F : b.F) * 2);
    k.qk_pre = b.qk_norm ? ws.take(T * (q + kv) * 2) : nullptr;
    k.rstd_qk = b.qk_norm ? ws.take<float>(T * (b.Hq + b.Hkv) * 4) : nullptr;
    k.lse = ws.take<float>(T * b.Hq * 4);
    k.mean1 = ln ? ws.take<float>(T * 4) : nullptr;
    k.rstd1 = ws.take<float>(T * 4);
    k.mean2 = ln ? ws.take<float>(T * 4) : nullptr;
    k.rstd2 = ws.take<float>(T * 4);
  }
  void* last = ws.take(T * H * 2);                      // hidden state behind the last block
  void* grad[2] = {ws.take(T * H * 2), ws.take(T * H * 2)};   // gradient of the hidden states, in turn
  // The head and the blocks take their temporaries from the same place: the head runs between the blocks' two directions.
  const long long shared = ws.at;
  void* xs = io.rows ? ws.take(R * H * 2) : nullptr;
  void* normed = ws.take(R * H * 2);
  float* mean = ln ? ws.take<float>(R * 4) : nullptr;
  float* rstd = ws.take<float>(R * 4);
  void* logits = ws.take(R * V * 2);
  float* loss = io.rows ? ws.take<float>(R * 4) : io.loss;
  void* dnormed = ws.take(R * H * 2);
  void* dxs = io.rows ? ws.take(R * H * 2) : grad[0];
  float* norm_rows = ws.take<float>(static_cast<long long>(mtb200_norm_bwd_blocks(s.R, b.H)) * (ln ? 2 : 1) * H * 4);
  const long long after_head = ws.at;
  BlockIO bio{};
  const long long block_ws = [&] {
    const long long f = mtb200_block_workspace(&b, &bio, 0), g = mtb200_block_workspace(&b, &bio, 1);
    return f > g ? f : g;
  }();
  const long long size = after_head > shared + block_ws ? after_head : shared + block_ws;
  if (measure) return size;

  auto params = [&](const StepGroup& g, bool gradient) {
    BlockParams p;
    void** to = reinterpret_cast<void**>(&p);
    for (int i = 0; i < STEP_PARAMS; ++i) to[i] = s.off[i] < 0 ? nullptr : static_cast<uint8_t*>(gradient ? g.grad : g.param) + 2 * s.off[i];
    return p;
  };
  static_assert(sizeof(BlockParams) == STEP_PARAMS * sizeof(void*), "one pointer per tensor");
  auto block_io = [&](int i, void* out) {
    const Kept& k = kept[i];
    BlockIO x{};
    x.x = k.x; x.qkv = k.qkv; x.attn = k.attn; x.h1 = k.h1; x.gu = k.gu; x.out = out; x.qk_pre = k.qk_pre;
    x.mean1 = k.mean1; x.rstd1 = k.rstd1; x.lse = k.lse; x.mean2 = k.mean2; x.rstd2 = k.rstd2; x.rstd_qk = k.rstd_qk;
    x.pos = io.pos; x.fwd_plan = io.fwd_plan; x.bwd_plan = io.bwd_plan; x.inv_freq = io.inv_freq[i];
    x.ws = static_cast<uint8_t*>(io.ws) + shared;
    x.counters = io.counters; x.part = io.part; x.part_bytes = io.part_bytes; x.status = io.status;
    return x;
  };
  auto at = [](void* base, long long elements) -> void* { return elements < 0 ? nullptr : static_cast<uint8_t*>(base) + 2 * elements; };
#define RUN(call, n) do { const int rc_ = (call); if (rc_) return rc_; *launches += (n); } while (0)
  const u64* epoch = io.epochs;   // in launch order
  auto add = [&](const StepGroup& g) { return mtb200_accumulate(g.acc, g.grad, g.n, 0, g.add, st); };

  // forward
  RUN(mtb200_embedding_fwd(at(io.embed->param, s.off_embed), io.ids, kept[0].x, b.T, b.H, s.V, io.status, st), 1);
  for (int i = 0; i < s.layers; ++i) {
    const BlockParams p = params(io.blocks[i], false);
    BlockIO x = block_io(i, i + 1 < s.layers ? kept[i + 1].x : last);
    x.epochs = epoch;
    epoch += 4;
    RUN(mtb200_block_forward(&b, &p, &x, launches, st), 0);
  }

  // head
  const StepGroup& lm = s.tied ? *io.embed : *io.head;
  // A group whose gradients are all written below, gaps there are none, needs no zeros: the head's, and the embedding's when the head's product fills it
  // (32000 x 256: 10 us for zeroing 16 MB and adding them to the product).
  const long long table = static_cast<long long>(s.V) * b.H;
  const bool filled = s.tied && io.embed->n == table;
  if (io.head->n != (ln ? 2 : 1) * b.H + (s.tied ? 0 : table) && cudaMemsetAsync(io.head->grad, 0, io.head->n * 2, st) != cudaSuccess) return -5;
  if (!filled && cudaMemsetAsync(io.embed->grad, 0, io.embed->n * 2, st) != cudaSuccess) return -5;
  const void* hidden = last;
  if (io.rows) {
    RUN(mtb200_embedding_fwd(last, io.rows, xs, s.R, b.H, b.T, io.status, st), 1);
    hidden = xs;
  }
  void *w = at(io.head->param, s.off_norm), *wb = at(io.head->param, s.off_bnorm), *dw = at(io.head->grad, s.off_norm), *dwb = at(io.head->grad, s.off_bnorm);
  RUN(ln ? mtb200_layernorm_fwd(hidden, w, wb, normed, mean, rstd, b.eps, s.R, b.H, io.status, st)
         : mtb200_rmsnorm_fwd(hidden, w, normed, rstd, b.eps, s.R, b.H, io.status, st), 1);
  auto product = [&](int which, const void* a, long long lda, int a_mn, const void* w_, long long ldw, int w_mn, void* d, long long ldd, int M, int N, int K,
                     const void* r) {
    const int splits = io.part != nullptr ? s.splits[which] : 1;
    GemmEntry* f = gemm_entry(s.form[which]);
    if (f == nullptr) return -10;
    return f(a, lda, a_mn, w_, ldw, w_mn, d, ldd, 0, r, r ? ldd : 0, nullptr, M, N, K, s.logit_alpha, splits,
             splits > 1 ? io.counters : nullptr, splits > 1 ? *epoch++ : 0, splits > 1 ? io.part : nullptr, splits > 1 ? io.part_bytes : 0, nullptr, io.status, st);
  };
  const void* W = at(lm.param, s.off_lm);
  void* dW = at(lm.grad, s.off_lm);
  RUN(product(0, normed, H, 0, W, H, 0, logits, V, s.R, s.V, b.H, nullptr), 1);
  RUN(mtb200_ce_fwd_bwd(logits, V, 1, nullptr, io.targets, loss, logits, V, s.R, s.V, s.grad_scale, -100, st), 1);
  RUN(product(1, logits, V, 0, W, H, 1, dnormed, H, s.R, b.H, s.V, nullptr), 1);
  RUN(product(2, logits, V, 1, normed, H, 1, dW, H, s.V, b.H, s.R, s.tied && !filled ? dW : nullptr), 1);
  RUN(ln ? mtb200_layernorm_bwd(dnormed, hidden, mean, rstd, w, nullptr, dxs, norm_rows, dw, dwb, s.R, b.H, io.status, st)
         : mtb200_rmsnorm_bwd(dnormed, hidden, rstd, w, nullptr, dxs, norm_rows, dw, s.R, b.H, io.status, st), 2);
  if (io.rows) RUN(mtb200_scatter_rows(io.rows, dxs, grad[0], loss, io.loss, s.R, b.H, b.T, io.status, st), 2);
  RUN(add(*io.head), 1);

  // backward through the blocks
  for (int i = s.layers - 1, turn = 0; i >= 0; --i, turn ^= 1) {
    const BlockParams p = params(io.blocks[i], false), g = params(io.blocks[i], true);
    BlockIO x = block_io(i, nullptr);
    x.dout = grad[turn];
    x.dx = grad[turn ^ 1];
    x.epochs = epoch;
    epoch += 9;
    RUN(mtb200_block_backward(&b, &p, &g, &x, launches, st), 0);
    RUN(add(io.blocks[i]), 1);
  }
  RUN(mtb200_embedding_bwd_scan(at(io.embed->grad, s.off_embed), io.ids, grad[s.layers & 1], b.T, b.H, s.V, io.status, st), 1);
  RUN(add(*io.embed), 1);
  return 0;
}

}  // namespace

extern "C" {

void mtb200_step_sizes(int* out) {
  out[0] = sizeof(StepSpec); out[1] = sizeof(StepGroup); out[2] = sizeof(StepIO);
}
// Bytes of io->ws; negative: not a model that can be queued like this. Only io->rows is looked at.
long long mtb200_step_workspace(const StepSpec* s, const StepIO* io) { return run(*s, *io, true, nullptr, nullptr); }
int mtb200_step_forward_backward(const StepSpec* s, const StepIO* io, int* launches, cudaStream_t st) {
  return static_cast<int>(run(*s, *io, false, st, launches));
}

}  // extern "C"
