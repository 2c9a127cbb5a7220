// extern "C" entry points of training mode (declared in include/moe_b200.h): the forward with
// dropout on h and the tensors the backward pass needs (reference model.py:164,183 under
// .train()), and the backward pass itself (what torch.autograd derives for model.py:200-276
// and 173-190 when the reference trains, train.py:140-141).
#include "common.cuh"
#include "internal.h"

namespace moe {
namespace {

size_t up1k(size_t v) { return (v + 1023) & ~(size_t)1023; }

int train_check(int64_t N, int d, int f, int E, int k, int dtype, float p) {
  if (dtype != MOE_B200_BF16)
    return set_error(MOE_B200_ERR_DTYPE, "training mode computes in bf16");
  if (N < 0 || d < 8 || (d & 7) || f < 8 || (f & 7) || E < 1 || E > kMaxExperts || k < 1 ||
      k > kMaxTopK || k > E || N * (int64_t)k >= (int64_t)1 << 31)
    return set_error(MOE_B200_ERR_SHAPE, "N, d, f, E or k out of range");
  if (!(p >= 0.f && p < 1.f)) return set_error(MOE_B200_ERR_SHAPE, "dropout probability must be in [0,1)");
  return 0;
}

void tws_layout(int64_t N, int d, int f, int E, int k, size_t* off, size_t* total) {
  const size_t M = (size_t)N * k;
  size_t sizes[MOE_B200_TWS_NUM] = {};
  sizes[MOE_B200_TWS_GU] = M * 2 * f * 2;
  sizes[MOE_B200_TWS_PAIR_OF] = M * sizeof(int32_t);
  sizes[MOE_B200_TWS_DY] = M * d * 2;
  sizes[MOE_B200_TWS_DXS] = M * d * 2;
  sizes[MOE_B200_TWS_DL] = (size_t)N * E * sizeof(float);
  sizes[MOE_B200_TWS_DW] = M * sizeof(float);
  sizes[MOE_B200_TWS_DWG_F32] = (size_t)router_bwd_scratch_floats(N, d, E) * sizeof(float);
  sizes[MOE_B200_TWS_G_WG] = (size_t)E * d * 2;
  sizes[MOE_B200_TWS_G_BG] = (size_t)E * 2;
  sizes[MOE_B200_TWS_G_W1] = (size_t)E * 2 * f * d * 2;
  sizes[MOE_B200_TWS_G_B1] = (size_t)E * 2 * f * 2;
  sizes[MOE_B200_TWS_G_W2] = (size_t)E * d * f * 2;
  sizes[MOE_B200_TWS_G_B2] = (size_t)E * d * 2;
  sizes[MOE_B200_TWS_MASK] = M * (f / 8);
  // one row per 128-row half of a 256-row tile for dg and du; the sums of dy take less
  const size_t tiles = (M + 255) / 256 + E;
  const size_t cols = (size_t)4 * f > (size_t)d ? (size_t)4 * f : (size_t)d;
  sizes[MOE_B200_TWS_COL_PART] = tiles * cols * sizeof(float);
  size_t pos = 0;
  for (int i = 0; i < MOE_B200_TWS_NUM; ++i) {
    off[i] = pos;
    pos += up1k(sizes[i] ? sizes[i] : 1);
  }
  *total = pos;
}

// lora: of a LoRA step, forward and backward alike
TrainArgs train_args(char* tws, const size_t* to, float p, uint64_t seed, bool lora) {
  TrainArgs tr;
  tr.gu = reinterpret_cast<__nv_bfloat16*>(tws + to[MOE_B200_TWS_GU]);
  tr.mask = reinterpret_cast<uint8_t*>(tws + to[MOE_B200_TWS_MASK]);
  tr.col_part = reinterpret_cast<float*>(tws + to[MOE_B200_TWS_COL_PART]);
  tr.pair_of = reinterpret_cast<const int32_t*>(tws + to[MOE_B200_TWS_PAIR_OF]);
  const double t = (double)p * 4294967296.0;
  tr.thresh = p <= 0.f ? 0u : (uint32_t)(t >= 4294967295.0 ? 4294967295.0 : t);
  tr.scale = 1.0f / (1.0f - p);
  tr.seed_lo = (uint32_t)seed;
  tr.seed_hi = (uint32_t)(seed >> 32);
  tr.keep_pre = lora;
  return tr;
}

// Backward of the grouped expert feed-forward (model.py:174-184) on sorted rows: given dy (gradient of y),
// h (the dropped h of the forward), what the forward kept in gu and mask (TrainArgs) and the sorted inputs, writes g.x (gradient of the
// sorted inputs) and the four parameter gradients.
int experts_backward(const void* perm, const void* h, const int32_t* offsets, const void* plan, const void* dy,
                     int64_t M, int d, int f, int E, const TrainArgs& tr, const TrainGrads& g, const LoraGrads* lora,
                     int32_t* status, cudaStream_t s) {
  const PlanView pv = plan_view(plan, E);
  int rc;
  // down Linear (model.py:184): db2 = column sums of dy, dW2 = dy^T h, dh = dy W2; the last one goes back
  // through dropout, product and GELU (model.py:180-183) in its epilogue: (g, u) -> (dg, du) in place
  if (g.b2 != nullptr) {
    rc = launch_colsum(dy, offsets, M, E, d, tr.col_part, g.b2, s);
    if (rc) return rc;
  }
  if (g.w2 != nullptr) {
    rc = launch_grouped_wgrad(dy, h, M, d, f, offsets, g.w2, E, status, s);
    if (rc) return rc;
  }
  if (g.x == nullptr && g.w1 == nullptr && g.b1 == nullptr) return 0;   // (LoRA gradients need w1)
  rc = launch_grouped_dx(dy, M, d, pv.tmap_W2_dec, offsets, E, f, nullptr, &tr, lora != nullptr, status, s);
  if (rc) return rc;
  // gate_and_up Linear (model.py:174): db1 = column sums of dgu, dx = dgu W1, dW1 = dgu^T x
  if (g.b1 != nullptr) {
    rc = launch_colsum_finish(tr.col_part, 2, offsets, E, 2 * f, g.b1, s);
    if (rc) return rc;
  }
  if (g.x != nullptr) {
    rc = launch_grouped_dx(tr.gu, M, 2 * f, pv.tmap_W1_dec, offsets, E, d, g.x, nullptr, false, status, s);
    if (rc) return rc;
  }
  if (g.w1 != nullptr) {
    rc = launch_grouped_wgrad(tr.gu, perm, M, 2 * f, d, offsets, g.w1, E, status, s);
    if (rc) return rc;
  }
  if (lora == nullptr) return 0;
  const void* const G[2] = {g.w1, g.w2};
  const void* const gb[2] = {g.b1, g.b2};
  for (const LoraRun& run : lora->runs) {
    rc = launch_lora_grads(lora->tab, d, f, E, run, lora->scratch, G, gb, s);
    if (rc) return rc;
  }
  return 0;
}

// the gradient regions of the training workspace
TrainGrads own_grads(char* tws, const size_t* to, void* grad_x) {
  return TrainGrads{grad_x, tws + to[MOE_B200_TWS_G_WG], tws + to[MOE_B200_TWS_G_BG], tws + to[MOE_B200_TWS_G_W1],
                    tws + to[MOE_B200_TWS_G_B1], tws + to[MOE_B200_TWS_G_W2], tws + to[MOE_B200_TWS_G_B2]};
}

// `g` with the workspace's own place for what LoRA gradients need besides
TrainGrads with_own(TrainGrads g, const LoraGrads* lora, char* tws, const size_t* to) {
  if (lora == nullptr || lora->runs.empty()) return g;
  const TrainGrads own = own_grads(tws, to, nullptr);
  if (g.w1 == nullptr) g.w1 = own.w1;
  if (g.b1 == nullptr) g.b1 = own.b1;
  if (g.w2 == nullptr) g.w2 = own.w2;
  if (g.b2 == nullptr) g.b2 = own.b2;
  return g;
}

}  // namespace
}  // namespace moe

using namespace moe;

extern "C" {

size_t moe_b200_train_workspace_bytes(int64_t N, int d, int f, int E, int k, int dtype) {
  if (train_check(N, d, f, E, k, dtype, 0.f)) return 0;
  size_t off[MOE_B200_TWS_NUM], total;
  tws_layout(N, d, f, E, k, off, &total);
  return total;
}

int moe_b200_train_workspace_layout(int64_t N, int d, int f, int E, int k, int dtype, size_t* h_offsets) {
  if (!h_offsets) return set_error(MOE_B200_ERR_NULL, "h_offsets is NULL");
  int rc = train_check(N, d, f, E, k, dtype, 0.f);
  if (rc) return rc;
  size_t total;
  tws_layout(N, d, f, E, k, h_offsets, &total);
  return 0;
}

int moe_b200_train_setup(int64_t N, int d, int f, int E, int k, int dtype, void* train_ws,
                         size_t train_ws_bytes, void* stream) {
  int rc = train_check(N, d, f, E, k, dtype, 0.f);
  if (rc) return rc;
  if (!train_ws) return set_error(MOE_B200_ERR_NULL, "train_ws is NULL");
  size_t to[MOE_B200_TWS_NUM], total;
  tws_layout(N, d, f, E, k, to, &total);
  if (train_ws_bytes < total) return set_error(MOE_B200_ERR_WORKSPACE, "training workspace too small");
  if ((uintptr_t)train_ws & 1023) return set_error(MOE_B200_ERR_ALIGN, "training workspace must be 1024-byte aligned");
  (void)stream;
  return 0;
}

int moe_b200_forward_train(const void* x, const void* Wg, const void* bg, const void* plan,
                           const void* residual, int64_t N, int d, int f, int E, int k, int dtype,
                           float dropout_p, uint64_t seed, void* workspace, size_t workspace_bytes,
                           void* train_ws, size_t train_ws_bytes, void* out, void* stream) {
  return forward_train_into(x, Wg, bg, plan, residual, N, d, f, E, k, dtype, dropout_p, seed, workspace,
                            workspace_bytes, train_ws, train_ws_bytes, out, nullptr, false, stream);
}

int moe_b200_backward(const void* x, const void* Wg, const void* plan, const void* grad_out,
                      float grad_aux, int64_t N, int d, int f, int E, int k, int dtype,
                      float dropout_p, uint64_t seed, void* workspace, size_t workspace_bytes,
                      void* train_ws, size_t train_ws_bytes, void* grad_x, void* stream) {
  int rc = train_check(N, d, f, E, k, dtype, dropout_p);
  if (rc) return rc;
  if (!train_ws) return set_error(MOE_B200_ERR_NULL, "workspace is NULL");
  if (N > 0 && !grad_x) return set_error(MOE_B200_ERR_NULL, "NULL argument");
  size_t to[MOE_B200_TWS_NUM], ttotal;
  tws_layout(N, d, f, E, k, to, &ttotal);
  return backward_into(x, Wg, plan, grad_out, grad_aux, nullptr, N, d, f, E, k, dtype, dropout_p, seed, workspace,
                       workspace_bytes, train_ws, train_ws_bytes,
                       own_grads(static_cast<char*>(train_ws), to, grad_x), nullptr, stream);
}

// ---- the expert feed-forward alone (the reference's dense FeedForward, model.py:154-190, is one
// group; any grouping by offsets works) ----

int moe_b200_experts_train(const void* x_sorted, const int32_t* offsets, const void* plan, int64_t M,
                           int d, int f, int E, float dropout_p, uint64_t seed, void* train_ws,
                           size_t train_ws_bytes, void* h, void* y, int32_t* status, void* stream) {
  return experts_train_into(x_sorted, offsets, plan, M, d, f, E, dropout_p, seed, train_ws, train_ws_bytes, h, y, false,
                            status, stream);
}

int moe_b200_experts_backward(const void* x_sorted, const void* h, const int32_t* offsets,
                              const void* plan, const void* grad_y, int64_t M, int d, int f, int E,
                              float dropout_p, uint64_t seed, void* train_ws, size_t train_ws_bytes,
                              void* grad_x, int32_t* status, void* stream) {
  int rc = train_check(M, d, f, E, 1, MOE_B200_BF16, dropout_p);
  if (rc) return rc;
  if (M == 0) return 0;
  if (!train_ws || !grad_x) return set_error(MOE_B200_ERR_NULL, "NULL argument");
  size_t to[MOE_B200_TWS_NUM], ttotal;
  tws_layout(M, d, f, E, 1, to, &ttotal);
  return experts_backward_into(x_sorted, h, offsets, plan, grad_y, M, d, f, E, dropout_p, seed, train_ws,
                               train_ws_bytes, own_grads(static_cast<char*>(train_ws), to, grad_x), nullptr, status,
                               stream);
}

}  // extern "C"

namespace moe {

int experts_train_into(const void* x_sorted, const int32_t* offsets, const void* plan, int64_t M, int d, int f, int E,
                       float dropout_p, uint64_t seed, void* train_ws, size_t train_ws_bytes, void* h, void* y, bool lora,
                       int32_t* status, void* stream) {
  int rc = train_check(M, d, f, E, 1, MOE_B200_BF16, dropout_p);
  if (rc) return rc;
  if (M == 0) return 0;
  if (!x_sorted || !offsets || !plan || !train_ws || !h || !y || !status)
    return set_error(MOE_B200_ERR_NULL, "NULL argument");
  size_t to[MOE_B200_TWS_NUM], ttotal;
  tws_layout(M, d, f, E, 1, to, &ttotal);
  if (train_ws_bytes < ttotal) return set_error(MOE_B200_ERR_WORKSPACE, "training workspace too small");
  if ((uintptr_t)train_ws & 1023) return set_error(MOE_B200_ERR_ALIGN, "training workspace must be 1024-byte aligned");
  char* tws = static_cast<char*>(train_ws);
  cudaStream_t s = (cudaStream_t)stream;
  TrainArgs tr = train_args(tws, to, dropout_p, seed, lora);
  tr.pair_of = nullptr;     // row r is pair r: the dropout mask of element (r, c) depends on the row's position only
  return launch_experts_tc2(x_sorted, offsets, plan, M, d, f, E, h, y, nullptr, status, s, &tr);
}

int forward_train_into(const void* x, const void* Wg, const void* bg, const void* plan, const void* residual,
                       int64_t N, int d, int f, int E, int k, int dtype, float dropout_p, uint64_t seed,
                       void* workspace, size_t workspace_bytes, void* train_ws, size_t train_ws_bytes, void* out,
                       float* aux, bool lora, void* stream) {
  int rc = train_check(N, d, f, E, k, dtype, dropout_p);
  if (rc) return rc;
  if (!workspace || !train_ws) return set_error(MOE_B200_ERR_NULL, "workspace is NULL");
  size_t off[MOE_B200_WS_NUM], to[MOE_B200_TWS_NUM], ttotal;
  rc = moe_b200_workspace_layout(N, d, f, E, k, dtype, off);
  if (rc) return rc;
  if (workspace_bytes < moe_b200_workspace_bytes(N, d, f, E, k, dtype))
    return set_error(MOE_B200_ERR_WORKSPACE, "workspace too small");
  tws_layout(N, d, f, E, k, to, &ttotal);
  if (train_ws_bytes < ttotal) return set_error(MOE_B200_ERR_WORKSPACE, "training workspace too small");
  if (((uintptr_t)workspace & 1023) || ((uintptr_t)train_ws & 1023))
    return set_error(MOE_B200_ERR_ALIGN, "workspaces must be 1024-byte aligned");
  if (N == 0) return 0;
  if (!x || !Wg || !bg || !plan || !out) return set_error(MOE_B200_ERR_NULL, "NULL argument");
  char* ws = static_cast<char*>(workspace);
  char* tws = static_cast<char*>(train_ws);
  int32_t* status = reinterpret_cast<int32_t*>(ws + off[MOE_B200_WS_STATUS]);
  float* logits = reinterpret_cast<float*>(ws + off[MOE_B200_WS_LOGITS]);
  int32_t* idx = reinterpret_cast<int32_t*>(ws + off[MOE_B200_WS_IDX]);
  float* w = reinterpret_cast<float*>(ws + off[MOE_B200_WS_W]);
  float* psum_part = reinterpret_cast<float*>(ws + off[MOE_B200_WS_PSUM_PART]);
  int32_t* row_of = reinterpret_cast<int32_t*>(ws + off[MOE_B200_WS_ROW_OF]);
  int32_t* offsets = reinterpret_cast<int32_t*>(ws + off[MOE_B200_WS_OFFSETS]);
  void* perm = ws + off[MOE_B200_WS_PERM];
  void* h = ws + off[MOE_B200_WS_H];
  void* y = ws + off[MOE_B200_WS_Y];
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t M = N * k;
  // training always takes the large-N kernels: the backward pass works on their sorted buffers
  int32_t* scratch = reinterpret_cast<int32_t*>(ws + off[MOE_B200_WS_SCRATCH]);
  int32_t* cnt_slot = reinterpret_cast<int32_t*>(ws + off[MOE_B200_WS_CNT_SLOT]);
  float* psum = reinterpret_cast<float*>(ws + off[MOE_B200_WS_PSUM]);
  int32_t* pair_of = reinterpret_cast<int32_t*>(tws + to[MOE_B200_TWS_PAIR_OF]);
  if (aux == nullptr) aux = reinterpret_cast<float*>(ws + off[MOE_B200_WS_AUX]);
  int many = 0;
  if (aligned16(x) && aligned16(Wg)) {
    rc = front_many_tokens(N, d, E, k, dtype, false, &many);
    if (rc) return rc;
  }
  if (many > 0) {
    rc = launch_front_many(x, nullptr, nullptr, nullptr, Wg, bg, N, d, E, k, logits, idx, w, cnt_slot, offsets, row_of, perm,
                           pair_of, psum, aux, scratch, status, many, true, s);
    if (rc) return rc;
  } else {
    MOE_CUDA_CHECK(cudaMemsetAsync(status, 0, (MOE_B200_READY_OFFSET + MOE_B200_READY_INTS) * sizeof(int32_t), s));
    rc = moe_b200_router(x, Wg, bg, N, d, E, k, dtype, logits, idx, w, psum_part, status, stream);
    if (rc) return rc;
    rc = moe_b200_dispatch(x, idx, N, d, E, k, dtype, scratch, cnt_slot, offsets, row_of, perm, psum_part, psum, aux, status,
                           stream);
    if (rc) return rc;
    rc = launch_pair_of(row_of, M, pair_of, s);
    if (rc) return rc;
  }
  const TrainArgs tr = train_args(tws, to, dropout_p, seed, lora);
  rc = launch_experts_tc2(perm, offsets, plan, M, d, f, E, h, y, nullptr, status, s, &tr);
  if (rc) return rc;
  return moe_b200_combine(y, row_of, w, residual, N, d, k, dtype, out, stream);
}

int backward_into(const void* x, const void* Wg, const void* plan, const void* grad_out, float grad_aux,
                  const float* grad_aux_dev, int64_t N, int d, int f, int E, int k, int dtype, float dropout_p,
                  uint64_t seed, void* workspace, size_t workspace_bytes, void* train_ws, size_t train_ws_bytes,
                  const TrainGrads& grads, const LoraGrads* lora, void* stream) {
  int rc = train_check(N, d, f, E, k, dtype, dropout_p);
  if (rc) return rc;
  if (!workspace || !train_ws) return set_error(MOE_B200_ERR_NULL, "workspace is NULL");
  size_t off[MOE_B200_WS_NUM], to[MOE_B200_TWS_NUM], ttotal;
  rc = moe_b200_workspace_layout(N, d, f, E, k, dtype, off);
  if (rc) return rc;
  if (workspace_bytes < moe_b200_workspace_bytes(N, d, f, E, k, dtype))
    return set_error(MOE_B200_ERR_WORKSPACE, "workspace too small");
  tws_layout(N, d, f, E, k, to, &ttotal);
  if (train_ws_bytes < ttotal) return set_error(MOE_B200_ERR_WORKSPACE, "training workspace too small");
  if (N == 0) return 0;
  if (!x || !Wg || !plan || !grad_out) return set_error(MOE_B200_ERR_NULL, "NULL argument");
  if (!aligned16(grad_out) || !aligned16(grads.x) || !aligned16(x))
    return set_error(MOE_B200_ERR_ALIGN, "buffers must be 16-byte aligned");
  char* ws = static_cast<char*>(workspace);
  char* tws = static_cast<char*>(train_ws);
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t M = N * k;
  int32_t* status = reinterpret_cast<int32_t*>(ws + off[MOE_B200_WS_STATUS]);
  const float* logits = reinterpret_cast<const float*>(ws + off[MOE_B200_WS_LOGITS]);
  const int32_t* idx = reinterpret_cast<const int32_t*>(ws + off[MOE_B200_WS_IDX]);
  const float* w = reinterpret_cast<const float*>(ws + off[MOE_B200_WS_W]);
  const int32_t* cnt_slot = reinterpret_cast<const int32_t*>(ws + off[MOE_B200_WS_CNT_SLOT]);
  const int32_t* offsets = reinterpret_cast<const int32_t*>(ws + off[MOE_B200_WS_OFFSETS]);
  const int32_t* row_of = reinterpret_cast<const int32_t*>(ws + off[MOE_B200_WS_ROW_OF]);
  const void* perm = ws + off[MOE_B200_WS_PERM];
  const void* h = ws + off[MOE_B200_WS_H];
  const void* y = ws + off[MOE_B200_WS_Y];
  void* dy = tws + to[MOE_B200_TWS_DY];
  void* dxs = tws + to[MOE_B200_TWS_DXS];
  float* dl = reinterpret_cast<float*>(tws + to[MOE_B200_TWS_DL]);
  float* dw = reinterpret_cast<float*>(tws + to[MOE_B200_TWS_DW]);
  float* dwg32 = reinterpret_cast<float*>(tws + to[MOE_B200_TWS_DWG_F32]);
  const TrainArgs tr = train_args(tws, to, dropout_p, seed, lora != nullptr);

  // combine (model.py:271) and router (model.py:206-223)
  rc = launch_combine_bwd(grad_out, y, tr.pair_of, offsets, E, w, M, d, k, dy, dw, s);
  if (rc) return rc;
  if (grads.x != nullptr || grads.wg != nullptr || grads.bg != nullptr) {
    rc = launch_router_bwd(logits, idx, w, dw, cnt_slot, grad_aux, grad_aux_dev, x, N, d, E, k, dl, dwg32, grads.wg,
                           grads.bg, s);
    if (rc) return rc;
  }
  // the experts (model.py:174-184)
  TrainGrads eg = with_own(grads, lora, tws, to);
  eg.x = grads.x != nullptr ? dxs : nullptr;
  rc = experts_backward(perm, h, offsets, plan, dy, M, d, f, E, tr, eg, lora, status, s);
  if (rc || grads.x == nullptr) return rc;
  // gather (model.py:248-253) and the router's share
  return launch_combine_dx(dxs, row_of, dl, Wg, N, d, E, k, grads.x, s);
}

int experts_backward_into(const void* x_sorted, const void* h, const int32_t* offsets, const void* plan,
                          const void* grad_y, int64_t M, int d, int f, int E, float dropout_p, uint64_t seed,
                          void* train_ws, size_t train_ws_bytes, const TrainGrads& grads, const LoraGrads* lora,
                          int32_t* status, void* stream) {
  int rc = train_check(M, d, f, E, 1, MOE_B200_BF16, dropout_p);
  if (rc) return rc;
  if (M == 0) return 0;
  if (!x_sorted || !h || !offsets || !plan || !grad_y || !train_ws || !status)
    return set_error(MOE_B200_ERR_NULL, "NULL argument");
  if (!aligned16(x_sorted) || !aligned16(h)) return set_error(MOE_B200_ERR_ALIGN, "x and h must be 16-byte aligned");
  size_t to[MOE_B200_TWS_NUM], ttotal;
  tws_layout(M, d, f, E, 1, to, &ttotal);
  if (train_ws_bytes < ttotal) return set_error(MOE_B200_ERR_WORKSPACE, "training workspace too small");
  char* tws = static_cast<char*>(train_ws);
  cudaStream_t s = (cudaStream_t)stream;
  const TrainArgs tr = train_args(tws, to, dropout_p, seed, lora != nullptr);
  // gradients come as they come (a slice of a concatenation starts anywhere): those that TMA and 16-byte accesses cannot
  // take go through the workspace
  const size_t bytes = (size_t)M * d * 2;
  const void* dy = grad_y;
  if (!aligned16(grad_y)) {
    MOE_CUDA_CHECK(cudaMemcpyAsync(tws + to[MOE_B200_TWS_DY], grad_y, bytes, cudaMemcpyDeviceToDevice, s));
    dy = tws + to[MOE_B200_TWS_DY];
  }
  TrainGrads eg = with_own(grads, lora, tws, to);
  if (!aligned16(grads.x)) eg.x = tws + to[MOE_B200_TWS_DXS];
  rc = experts_backward(x_sorted, h, offsets, plan, dy, M, d, f, E, tr, eg, lora, status, s);
  if (rc) return rc;
  if (eg.x != grads.x) MOE_CUDA_CHECK(cudaMemcpyAsync(grads.x, eg.x, bytes, cudaMemcpyDeviceToDevice, s));
  return 0;
}

}  // namespace moe
