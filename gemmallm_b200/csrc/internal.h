// Entry points of libmoe_b200.so that the package's own host extension (host.cpp) calls besides the
// C ABI of include/moe_b200.h. C++ linkage, same conventions and return codes.
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <vector>

namespace moe {

// moe_b200_forward with the load-balancing loss written to `aux` (nullptr: the workspace's own word).
int forward_into(const void* x, const void* Wg, const void* bg, const void* plan, const void* residual,
                 const void* norm_weight, const void* norm_bias, float norm_eps, int64_t N, int d, int f,
                 int E, int k, int dtype, int flags, void* workspace, size_t workspace_bytes, void* out,
                 float* aux, void* stream);

// Where the gradients of a backward pass go; nullptr: not wanted, and its kernels are not launched.
struct TrainGrads {
  void* x;                   // [N, d]
  void *wg, *bg;             // router [E, d], [E]
  void *w1, *b1, *w2, *b2;   // experts [E, 2f, d], [E, 2f], [E, d, f], [E, d]
};

// LoRA gradients of both Linears (0: gate_and_up, 1: down); they are formed from w1, b1, w2 and b2 of TrainGrads: those
// that are not wanted are formed in the training workspace. A run: experts [first, first + count) of the same ranks and scale.
struct LoraRun {
  int first, count, rank[2];
  float scale;
  void *dA[2], *da[2], *dB[2], *db[2];   // [count, rank, in], [count, rank], [count, out, rank], [count, out]
};
// Given for every fine-tuning step, without runs where no LoRA tensor is wanted: such a step rounds dh, and what is wanted
// must not decide what the other gradients are.
struct LoraGrads {
  const void* const* tab;    // device [2][E][3]: A, a, B of every expert
  float* scratch;            // as many floats as the largest run asks for
  std::vector<LoraRun> runs;
};
// Linears with their LoRA branches folded in (moe_b200_lora_merge), in as few launches as can be.
struct LoraMerge {
  const void *W, *b, *A, *a_bias, *B, *b_lora;
  void *out_W, *out_b;
  float scale;
  int out_f, in_f, rank;
};
int lora_merges(const LoraMerge* merges, int n, int dtype, void* stream);
size_t lora_grads_scratch_floats(int d, int f, const LoraRun& run);

// moe_b200_forward_train with the load-balancing loss written to `aux` (nullptr: the workspace's word). lora: of a LoRA
// step, whose backward pass is given LoraGrads; it works on other saved values.
int forward_train_into(const void* x, const void* Wg, const void* bg, const void* plan, const void* residual,
                       int64_t N, int d, int f, int E, int k, int dtype, float dropout_p, uint64_t seed,
                       void* workspace, size_t workspace_bytes, void* train_ws, size_t train_ws_bytes, void* out,
                       float* aux, bool lora, void* stream);
// moe_b200_experts_train likewise.
int experts_train_into(const void* x_sorted, const int32_t* offsets, const void* plan, int64_t M, int d, int f, int E,
                       float dropout_p, uint64_t seed, void* train_ws, size_t train_ws_bytes, void* h, void* y, bool lora,
                       int32_t* status, void* stream);
// moe_b200_backward with the gradients written where the caller wants them and the loss's gradient read
// from device memory (grad_aux_dev, when not nullptr, instead of grad_aux).
int backward_into(const void* x, const void* Wg, const void* plan, const void* grad_out, float grad_aux,
                  const float* grad_aux_dev, int64_t N, int d, int f, int E, int k, int dtype, float dropout_p,
                  uint64_t seed, void* workspace, size_t workspace_bytes, void* train_ws, size_t train_ws_bytes,
                  const TrainGrads& grads, const LoraGrads* lora, void* stream);
// moe_b200_experts_backward likewise (grads.wg and grads.bg are not used).
int experts_backward_into(const void* x_sorted, const void* h, const int32_t* offsets, const void* plan,
                          const void* grad_y, int64_t M, int d, int f, int E, float dropout_p, uint64_t seed,
                          void* train_ws, size_t train_ws_bytes, const TrainGrads& grads, const LoraGrads* lora,
                          int32_t* status, void* stream);

// The attention of the decoder layer (bf16): QKV projection and head gate, on LayerNorm(x) where norm_weight is given, the core
// of moe_b200_attention, the output projection, plus skip where given. Three launches up to moe_b200_linear_rows_max() rows,
// beyond a fourth for the LayerNorm. Buffers: qkv [B S, (q + 2 kv) 64], gate [B S, q], core [B S, q 64]; x, out, skip and, where
// attention_normalises_apart() says so, xn [B S, hidden]; status: 16 words.
struct AttentionArgs {
  const void *x, *norm_weight, *norm_bias;
  float eps;
  const void *wqkv, *bqkv, *wgate, *bgate, *wo, *bo;
  const float *pos_emb, *mask;
  const void* skip;
  int64_t B;
  int S, hidden, q_heads, kv_heads, head_dim;
  float scaler;
  void *xn, *qkv, *gate, *core, *out;
  int32_t* status;
};
// Whether sizes and places are those that these launches take (and moe_b200_linear_rows) and the sizes are those where they are
// the faster ones (moe_b200_attention_linears).
bool attention_supported(const AttentionArgs& p);
bool attention_normalises_apart(const AttentionArgs& p);
int attention_layer(const AttentionArgs& p, void* stream);

}  // namespace moe
