// Host-side driver objects behind the level-2 (Linear) and level-3 (Model) C ABI.
// They mirror the reference's Linear (src/linear.rs:38-122), Attention/Mlp/Block
// (src/attention.rs, src/model.rs:92-218) and Model (src/model.rs:292-687), with every
// tensor resident in HBM.
#pragma once
#include "ctx.h"
#include "graph_cache.h"
#include "ops.h"
#include <map>
#include <string>
#include <vector>

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  // grow-only; returns false on allocation failure
  bool reserve(size_t want, bool zero = false);
  void release();
  template <class T> T* as() const { return (T*)p; }
};

// Page-locked host memory, grow-only.
struct PinnedBuf {
  void* p = nullptr;
  size_t bytes = 0;
  bool reserve(size_t want);
  void release();
};

struct LoraDev {
  int rank = 0;
  float alpha = 0.f;
  float *a = nullptr, *b = nullptr, *ga = nullptr, *gb = nullptr;  // views into flat f32 buffers
  __half *a_s = nullptr, *a_h = nullptr, *bp = nullptr, *bt_s = nullptr;  // 16-bit operand copies
  DevBuf shadows;
  bool stale = true;  // operand copies need rebuilding from a, b
  uint64_t version = 1;  // bumped with every change of a, b: stacked copies elsewhere compare it
  float scale() const { return alpha / (float)rank; }
};

struct rt_linear {
  rt_ctx* ctx = nullptr;
  int device = 0;
  std::string name;
  rt_frozen* w = nullptr;
  bool owns_w = false;
  float* bias = nullptr;  // device [out] or null
  bool has_lora = false, lora_enabled = true;
  LoraDev lora;
  DevBuf own_params;  // standalone linears own their a|b|ga|gb; model linears point into the model's buffers
  int in_dim() const { return w->w.cols; }
  int out_dim() const { return w->w.rows; }
  bool lora_active() const { return has_lora && lora_enabled; }
};

// Scratch of the Linear calls of a model, or of those on a ctx outside any model (one call at a time per ctx).
struct LinearScratch {
  DevBuf hs, gs[rt::LORA_GRAD_JOBS], grad_ws;
  // Adapter gradients wait here for the other linears of their block (`defer`), to be computed by one
  // launch: what they read has to stay in place until lora_grads_flush.
  bool defer = false;
  int n_jobs = 0;
  rt::LoraGradJob jobs[rt::LORA_GRAD_JOBS];
  void release() {
    hs.release();
    for (DevBuf& g : gs) g.release();
    grad_ws.release();
  }
};

namespace rt {
// hs_keep: optional [M x 64] f16 buffer (zero beyond the rank) that receives Hs = X.(sA)^T so the
// backward can reuse it instead of recomputing it.
rt_status linear_forward_dev(rt_linear* l, LinearScratch& sc, const __half* x16, int M, void* y, int y_dtype,
                             int accumulate, __half* hs_keep = nullptr, bool hs_ready = false, const float* residual = nullptr);
// Hs alone (the forward of a linear whose output is not needed).
rt_status linear_lora_h(rt_linear* l, const __half* x16, int M, __half* hs_out);
// dy16 is row-normalised f16 with per-row scales `dscale` (null = all ones).  With
// unscaled_f16_out, dx receives f16 rows WITHOUT their factor dscale[row] (the consumer applies
// it): half the output bytes, no accumulate.  gs_ready: Gs lies in sc.gs[sc.n_jobs] already.
rt_status linear_backward_dev(rt_linear* l, LinearScratch& sc, const __half* x16, const __half* dy16,
                              const float* dscale, int M, void* dx, int accumulate,
                              const __half* hs_saved = nullptr, bool unscaled_f16_out = false, bool gs_ready = false);
// computes the adapter gradients that are waiting in `sc`
rt_status lora_grads_flush(rt_ctx* c, LinearScratch& sc, int M);
rt_status lora_refresh(rt_linear* l);
}  // namespace rt

// Linears that read the same input (q|k|v, gate|up) as ONE matmul: their packed weights lie
// stacked along the output rows in one buffer (the members' own handles point into it), so the
// forward is a single product with the stacked rows as output features and the backward a
// single product contracting over them, instead of one product per member plus accumulating
// passes.  The members' adapters become one stacked low-rank chunk: member i owns columns
// [rank_off[i], rank_off[i] + r_i) of Hs / Gs.
struct LinGroup {
  int n = 0;
  rt_linear* lin[3] = {nullptr, nullptr, nullptr};
  int row_off[3] = {0, 0, 0}, rank_off[3] = {0, 0, 0};
  int rows_total = 0, rank_total = 0;
  bool stacked = false;    // weights share one buffer
  bool lora_ok = false;    // the members' adapters fit one 64-wide chunk (or there are none)
  rt::QWeight w;
  DevBuf store, lora_copies;
  float* bias = nullptr;   // stacked biases (owned), null when no member has one
  __half *a_s = nullptr, *a_h = nullptr, *bp = nullptr, *bt_s = nullptr;
  uint64_t seen[3] = {0, 0, 0};
};

struct BlockDev {
  float *input_norm = nullptr, *post_norm = nullptr, *q_norm = nullptr, *k_norm = nullptr;
  rt_linear* lin[7] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};  // q k v o gate up down
  LinGroup qkv, gu;
};

struct rt_model {
  rt_ctx* ctx = nullptr;
  int device = 0;
  rt_model_config cfg;
  bool finalized = false;
  rt_frozen* embed = nullptr;
  rt_frozen* lm_head = nullptr;  // == embed when tied
  float* final_norm = nullptr;
  std::vector<float> rope_factors;  // host copy of rope_freqs.weight
  std::vector<BlockDev> blocks;
  std::vector<void*> owned;  // small device allocations (norms, biases)
  std::vector<rt_linear*> lora_order;  // adapted linears in parameter order

  // flat LoRA state: [A_0 | B_0 | A_1 | B_1 ...] in parameter order
  size_t n_params = 0;
  DevBuf P, G, Mo, Vo, opt_scalars;  // opt_scalars: 1024 f64 partials + 1 f64 sum
  uint64_t opt_t = 0;

  // RoPE tables
  DevBuf inv_freq, rope_cos, rope_sin;
  int rope_max_pos = 0;

  LinearScratch lsc;
  DevBuf hs_keep[7];  // Hs of a block's seven linears, kept from the forward (or its recompute) for the backward
  // What a block's backward needs from its forward is either kept for every layer (180 GB of HBM
  // holds it for the usual fine-tuning shapes) or rebuilt by running the block's forward again
  // just before its backward.  Decided when the token capacity grows; RT_B200_RECOMPUTE=1 forces
  // the second.
  bool store_acts = false;
  int recompute_policy = -1;  // -1: not read yet, 0: automatic, 1: always recompute, 2: always keep
  // activations, sized for `cap_tokens`
  int cap_tokens = 0, cap_targets = 0, cap_head_rows = 0;
  // q_raw holds q|k|v before RoPE (three regions, or one matrix with q, k, v as column slices when the
  // block runs them as a group); g16 holds gate|up the same way; dq16, dg16 likewise for the gradients
  DevBuf x, ckpt, h, n1, n2, q_raw, q16, k16, v16, o16, lse, delta, g16, hm16;
  DevBuf dx, dy16, sc_y, dhm, dg16, sc_g, sc_u, dn, dO16, dy16o, sc_yo, dq, dk, dv, dq16, sc_q, sc_k, sc_v;
  DevBuf xs, ns16, logits, dl16, sc_l, dns, dxs;
  DevBuf argmax;            // per target, the greedy token of the last pass that asked for it
  bool want_argmax = false;
  DevBuf refresh_tab;       // device copy of refresh_sent
  std::vector<rt::LoraRefreshJob> refresh_jobs, refresh_sent;
  // A batch travels as one block: laid out in pinned memory, one copy to `batch`, the pointers below into it
  // (they depend on the block's base, the token and target counts and whether there are gaps only).  Results come back as
  // one block too: hit count, then log-probabilities.
  DevBuf batch, results;
  PinnedBuf h_batch, h_results;
  cudaEvent_t batch_sent = nullptr;
  int *tokens = nullptr, *pos = nullptr, *seq_start = nullptr, *tpos = nullptr, *ttok = nullptr;
  int *tiles_q = nullptr, *tiles_k = nullptr;  // see AttnBatch
  rt::AttnBatch attn_batch(int M) const { return {seq_start, gap, tiles_q, tiles_k, M}; }
  int* gap = nullptr;       // per token (first, end) of the key range hidden from it: packed shared-prompt groups, or null
  float* tw = nullptr;
  int* hits() const { return results.as<int>(); }
  float* logp() const { return results.as<float>() + 4; }
  int staged_tokens = 0, staged_targets = 0;
  bool staged_has_weights = false;
  // CUDA graphs of the staged step, one per shape of batch once it has run eagerly.
  // A trainer meets several shapes in turn (accumulated batches, a preference update's three passes).
  struct Shape {
    int M, n_targets, backward;
    uint64_t sig;
    bool operator==(const Shape& o) const { return M == o.M && n_targets == o.n_targets && backward == o.backward && sig == o.sig; }
  };
  struct Graph { cudaGraphExec_t exec; unsigned long long kernels; };
  rt::GraphCache<Shape, Graph, 32> graphs;
  int use_graphs = -1;  // -1: decide from the environment on first use
};
