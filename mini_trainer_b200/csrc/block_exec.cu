// One decoder block, forward or backward, queued by one call: the host side of models/decoder.py's dense pre-norm block for a rank that
// holds its parameters whole. The kernels, their order and their results are those of the Python form; what goes is the interpreter
// between the launches (5 to 8 us per launch next to the 2 to 3 us of the launch itself), which is what a step of a small model and
// a block on a short minibatch are bound by. Training step of 640 tokens through 2 layers 1207 -> 978 us, of 4096 tokens 1355 -> 1088; a block of
// 5987 tokens x 1536, which the device bounds, 1798 either way.
//
// Memory comes from the caller: what outlives the call as tensors of their own, the rest as one workspace laid out here
// (mtb200_block_workspace says how large), so nothing is allocated and nothing is kept between calls.
#include <cuda_runtime.h>
#include <stdint.h>

#include "block_exec.h"
#include "entries.h"

namespace {

// `epoch`: the next one. Arrivals on these counters are told apart by epochs that grow from launch to launch.
int gemm(const BlockSpec& s, const BlockIO& io, const u64*& epoch, int which, const void* a, long long lda, int a_mn, const void* b, long long ldb, int b_mn, void* d, int M, int N,
         int K, const void* r, const void* bias, float alpha, cudaStream_t st) {
  const int splits = io.part != nullptr ? s.splits[which] : 1;
  GemmEntry* f = gemm_entry(s.form[which]);
  if (f == nullptr) return -10;
  return f(a, lda, a_mn, b, ldb, b_mn, d, N, 0, r, N, bias, M, N, K, alpha, splits, splits > 1 ? io.counters : nullptr, splits > 1 ? *epoch++ : 0,
           splits > 1 ? io.part : nullptr, splits > 1 ? io.part_bytes : 0, nullptr, io.status, st);
}

#define RUN(call, n) do { const int rc_ = (call); if (rc_) return rc_; *launches += (n); } while (0)

int norm(const BlockSpec& s, const BlockIO& io, const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, cudaStream_t st) {
  return s.layernorm ? mtb200_layernorm_fwd(x, w, b, y, mean, rstd, s.eps, s.T, s.H, io.status, st)
                     : mtb200_rmsnorm_fwd(x, w, y, rstd, s.eps, s.T, s.H, io.status, st);
}

long long forward(const BlockSpec& s, const BlockParams& p, const BlockIO& io, bool measure, cudaStream_t st, int* launches) {
  const long long T = s.T, q = static_cast<long long>(s.Hq) * s.D, nh = s.Hq + s.Hkv, Q = (nh + s.Hkv) * s.D, width = s.gated ? 2LL * s.F : s.F;
  Carver ws{measure ? nullptr : static_cast<uint8_t*>(io.ws)};
  void* n1 = io.n1 ? io.n1 : ws.take(T * s.H * 2);
  void* n2 = io.n2 ? io.n2 : ws.take(T * s.H * 2);
  void* act = io.act ? io.act : ws.take(T * s.F * 2);
  if (measure) return ws.at;
  const u64* epoch = io.epochs;
  RUN(norm(s, io, io.x, p.ln1, p.bln1, n1, io.mean1, io.rstd1, st), 1);
  RUN(gemm(s, io, epoch, G_QKV, n1, s.H, 0, p.wqkv, s.H, 0, io.qkv, s.T, Q, s.H, nullptr, p.bqkv, 1.f, st), 1);
  if (s.qk_norm) RUN(mtb200_head_rmsnorm_fwd(io.qkv, p.qn, p.kn, io.qk_pre, io.rstd_qk, io.inv_freq ? io.pos : nullptr, io.inv_freq, s.eps, s.T, Q, s.Hq, nh, s.D, st), 1);
  else if (io.inv_freq) RUN(mtb200_rope(io.qkv, io.pos, io.inv_freq, s.T, Q, nh, s.D, 0, st), 1);
  if (!io.have_attn) {
    if (s.attn_form == 0) RUN(mtb200_attn_fwd_one(io.qkv, Q, io.attn, q, io.lse, io.fwd_plan, s.fwd_items, s.T, s.Hq, s.Hkv, s.D, s.scale, io.status, st), 1);
    else RUN(mtb200_attn_fwd(io.qkv, Q, io.attn, q, io.lse, io.fwd_plan, s.fwd_items, s.T, s.Hq, s.Hkv, s.D, s.attn_form - 1, s.scale, io.status, st), 1);
  }
  RUN(gemm(s, io, epoch, G_O, io.attn, q, 0, p.wo, q, 0, io.h1, s.T, s.H, q, io.x, p.bo, s.alpha, st), 1);
  RUN(norm(s, io, io.h1, p.ln2, p.bln2, n2, io.mean2, io.rstd2, st), 1);
  if (!s.need_out) {
    RUN(gemm(s, io, epoch, G_GU, n2, s.H, 0, p.wgu, s.H, 0, io.gu, s.T, width, s.H, nullptr, p.bgu, 1.f, st), 1);
    return 0;
  }
  if (s.splits[G_GU] > 1) {   // a split product has no room for the activation (ops/native.py, linear_act)
    RUN(gemm(s, io, epoch, G_GU, n2, s.H, 0, p.wgu, s.H, 0, io.gu, s.T, width, s.H, nullptr, p.bgu, 1.f, st), 1);
    if (!s.gated) RUN(mtb200_gelu_fwd(io.gu, act, T * s.F, st), 1);
    else RUN(s.gelu ? mtb200_geglu_fwd(io.gu, act, T, s.F, st) : mtb200_swiglu_fwd(io.gu, act, T, s.F, st), 1);
  } else {
    RUN(mtb200_gemm_act(n2, s.H, p.wgu, io.gu, act, p.bgu, s.gated ? 1 : 2, s.gelu, s.T, s.F, s.H, s.act_form, io.status, st), 1);
  }
  RUN(gemm(s, io, epoch, G_DOWN, act, s.F, 0, p.wd, s.F, 0, io.out, s.T, s.H, s.F, io.h1, p.bd, s.alpha, st), 1);
  return 0;
}

long long backward(const BlockSpec& s, const BlockParams& p, const BlockParams& g, const BlockIO& io, bool measure, cudaStream_t st, int* launches) {
  const long long T = s.T, q = static_cast<long long>(s.Hq) * s.D, nh = s.Hq + s.Hkv, Q = (nh + s.Hkv) * s.D, width = s.gated ? 2LL * s.F : s.F;
  Carver ws{measure ? nullptr : static_cast<uint8_t*>(io.ws)};
  auto most = [](long long a, long long b) { return a > b ? a : b; };
  void* dgu = ws.take(T * most(width, Q) * 2);      // then dqkv
  void* dact = ws.take(T * s.F * 2);                // then, unless it was kept, the activation
  void* dn = ws.take(T * s.H * 2);                  // gradient of the normalised rows, of either norm
  void* n2 = io.n2 ? io.n2 : ws.take(T * s.H * 2);
  void* n1 = io.n1 ? io.n1 : io.n2 ? ws.take(T * s.H * 2) : n2;   // n2 is read for the last time before n1 is formed
  void* dh1 = ws.take(T * s.H * 2);
  void* dattn = ws.take(T * q * 2);
  float* delta = ws.take<float>(T * s.Hq * 4);
  float* dq = ws.take<float>(T * q * 4);
  const int norm_rows = mtb200_norm_bwd_blocks(s.T, s.H) * (s.layernorm ? 2 : 1);
  float* rows = ws.take<float>(most(static_cast<long long>(norm_rows) * s.H, s.qk_norm ? 2LL * mtb200_head_rmsnorm_bwd_blocks(s.T, nh) * s.D : 0) * 4);
  float* cols = ws.take<float>(32 * most(width, most(Q, s.H)) * 4);
  float* again = ws.take<float>(T * 2 * 4);         // statistics of a norm that is formed again
  void* dqkv = dgu;
  if (measure) return ws.at;
  const u64* epoch = io.epochs;
  auto wgrad = [&](int which, const void* dy, long long N, const void* x, long long K, void* dw, void* db) -> int {
    int rc = gemm(s, io, epoch, which, dy, N, 1, x, K, 1, dw, N, K, s.T, nullptr, nullptr, which == W_DOWN || which == W_O ? s.alpha : 1.f, st);
    if (!rc && db) { rc = mtb200_colsum(dy, N, db, cols, s.T, N, st); *launches += 2; }
    ++*launches;
    return rc;
  };
  auto norm_bwd = [&](const void* x, const float* mean, const float* rstd, const void* w, const void* add, void* dx, void* dw, void* db) {
    *launches += 2;
    return s.layernorm ? mtb200_layernorm_bwd(dn, x, mean, rstd, w, add, dx, rows, dw, db, s.T, s.H, io.status, st)
                       : mtb200_rmsnorm_bwd(dn, x, rstd, w, add, dx, rows, dw, s.T, s.H, io.status, st);
  };
  // MLP
  RUN(gemm(s, io, epoch, D_DOWN, io.dout, s.H, 0, p.wd, s.F, 1, dact, s.T, s.F, s.H, nullptr, nullptr, s.alpha, st), 1);
  if (io.act) {
    if (!s.gated) RUN(mtb200_gelu_bwd(dact, io.gu, dgu, T * s.F, st), 1);
    else RUN(s.gelu ? mtb200_geglu_bwd(dact, io.gu, dgu, T, s.F, st) : mtb200_swiglu_bwd(dact, io.gu, dgu, T, s.F, st), 1);
  } else {
    if (!s.gated) RUN(mtb200_gelu_bwd_act(dact, io.gu, dgu, T * s.F, st), 1);
    else RUN(s.gelu ? mtb200_geglu_bwd_act(dact, io.gu, dgu, T, s.F, st) : mtb200_swiglu_bwd_act(dact, io.gu, dgu, T, s.F, st), 1);
  }
  RUN(wgrad(W_DOWN, io.dout, s.H, io.act ? io.act : dact, s.F, g.wd, g.bd), 0);
  RUN(gemm(s, io, epoch, D_GU, dgu, width, 0, p.wgu, s.H, 1, dn, s.T, s.H, width, nullptr, nullptr, 1.f, st), 1);
  if (!io.n2) RUN(norm(s, io, io.h1, p.ln2, p.bln2, n2, again, again + T, st), 1);
  RUN(wgrad(W_GU, dgu, width, n2, s.H, g.wgu, g.bgu), 0);
  RUN(norm_bwd(io.h1, io.mean2, io.rstd2, p.ln2, io.dout, dh1, g.ln2, g.bln2), 0);
  // attention
  RUN(gemm(s, io, epoch, D_O, dh1, s.H, 0, p.wo, q, 1, dattn, s.T, q, s.H, nullptr, nullptr, s.alpha, st), 1);
  RUN(wgrad(W_O, dh1, s.H, io.attn, q, g.wo, g.bo), 0);
  const int splits = io.part != nullptr ? s.bwd_splits : 1;
  RUN(mtb200_attn_bwd(io.qkv, Q, io.attn, q, dattn, q, dqkv, Q, io.lse, delta, dq, io.bwd_plan, s.bwd_items, s.T, s.Hq, s.Hkv, s.D, splits,
                      splits > 1 ? io.counters : nullptr, splits > 1 ? *epoch++ : 0, splits > 1 ? io.part : nullptr, splits > 1 ? io.part_bytes : 0, s.scale,
                      s.bwd_in_order, io.status, st), 3);
  if (s.qk_norm) RUN(mtb200_head_rmsnorm_bwd(dqkv, io.qk_pre, io.rstd_qk, p.qn, p.kn, rows, g.qn, g.kn, io.inv_freq ? io.pos : nullptr, io.inv_freq, s.T, Q, nh * s.D,
                                             s.Hq, nh, s.D, st), 2);
  else if (io.inv_freq) RUN(mtb200_rope(dqkv, io.pos, io.inv_freq, s.T, Q, nh, s.D, 1, st), 1);
  RUN(gemm(s, io, epoch, D_QKV, dqkv, Q, 0, p.wqkv, s.H, 1, dn, s.T, s.H, Q, nullptr, nullptr, 1.f, st), 1);
  if (!io.n1) RUN(norm(s, io, io.x, p.ln1, p.bln1, n1, again, again + T, st), 1);
  RUN(wgrad(W_QKV, dqkv, Q, n1, s.H, g.wqkv, g.bqkv), 0);
  RUN(norm_bwd(io.x, io.mean1, io.rstd1, p.ln1, dh1, io.dx, g.ln1, g.bln1), 0);
  return 0;
}

}  // namespace

extern "C" {

// Sizes of the structures, for a caller that lays them out itself (ops/block_exec.py).
void mtb200_block_sizes(int* out) {
  out[0] = sizeof(BlockSpec); out[1] = sizeof(BlockParams); out[2] = sizeof(BlockIO);
}
// Entry point of a product's kernel by its number, null past the last, for a caller that numbers them itself.
const char* mtb200_gemm_form(int form) {
#define F(form, entry) case form: return #entry;
  switch (form) { GEMM_FORMS(F) default: return nullptr; }
#undef F
}
// Bytes of io->ws for a call with these arguments (backward: with gradients).
long long mtb200_block_workspace(const BlockSpec* s, const BlockIO* io, int bwd) {
  const BlockParams none{};
  int n = 0;
  return bwd ? backward(*s, none, none, *io, true, nullptr, &n) : forward(*s, none, *io, true, nullptr, &n);
}
// launches: kernels launched, added to. Returns what the first failing launch returned, or 0.
int mtb200_block_forward(const BlockSpec* s, const BlockParams* p, const BlockIO* io, int* launches, cudaStream_t st) {
  return static_cast<int>(forward(*s, *p, *io, false, st, launches));
}
int mtb200_block_backward(const BlockSpec* s, const BlockParams* p, const BlockParams* g, const BlockIO* io, int* launches, cudaStream_t st) {
  return static_cast<int>(backward(*s, *p, *g, *io, false, st, launches));
}

}  // extern "C"
