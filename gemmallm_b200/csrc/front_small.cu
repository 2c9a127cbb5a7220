// Router and dispatch of a small call in ONE launch: the kernel around front_small_body
// (front_small.cuh), its launcher and the size limits.
#include "front_small.cuh"

namespace moe {

namespace {

constexpr int kThreads = kFrontThreads;
constexpr int kMaxTok = kFrontMaxTok;
constexpr int kMaxE = kFrontMaxE;
constexpr int kMaxPairs = kFrontMaxPairs;

// fp32 tokens of a block: as few as 128 blocks allow, but four (their rows' copies and parts are the longest step of a block of
// 16, which stores 160 KB at d 512: 512 tokens 81.8 -> 76.0 us, 51 tokens 58.5 -> 55.1, 1024 134 -> 130). Up to 16 are one block's, which need not meet any other.
int f32_tokens_per_block(int64_t N) {
  if (N <= 16) return 16;
  const int64_t per = (N + 127) / 128;
  return per < 4 ? 4 : (int)per;
}

template <int NT, bool SPLIT, typename T>
__global__ void __launch_bounds__(kThreads, 1)
front_small_kernel(const T* __restrict__ x, const T* Wg, const T* bg, int Ntotal, int d, int E, int k,
                   float* __restrict__ out_logits, int32_t* __restrict__ out_idx,
                   float* __restrict__ out_w, int32_t* __restrict__ cnt_slot,
                   int32_t* __restrict__ offsets, int32_t* __restrict__ row_of,
                   T* __restrict__ perm, __nv_bfloat16* __restrict__ planes, float* __restrict__ psum,
                   float* __restrict__ aux, int* __restrict__ xch, int* __restrict__ counter,
                   int32_t* __restrict__ status, int per) {
  extern __shared__ float smem[];
  pdl_wait();                 // x may come from the kernel before this one
  pdl_launch_dependents();
  front_small_body<NT, SPLIT, T>(smem, x, Wg, bg, Ntotal, d, E, k, out_logits, out_idx, out_w, cnt_slot, offsets,
                                 row_of, perm, planes, psum, aux, xch, counter, status, per);
}

template <int NT, typename T>
int launch(const void* x, const void* Wg, const void* bg, int N, int d, int E, int k,
           float* out_logits, int32_t* out_idx, float* out_w, int32_t* cnt_slot, int32_t* offsets,
           int32_t* row_of, void* perm, void* planes, float* psum, float* aux, int* xch, int* counter,
           int32_t* status, cudaStream_t s) {
  // beyond 128 tokens repeating the routing in every block costs more than one exchange
  constexpr bool F32 = sizeof(T) == 4;
  const bool split = F32 || (xch != nullptr && counter != nullptr && status != nullptr && N > 128);
  const int per = F32 ? f32_tokens_per_block(N) : 16;
  const size_t smem = front_small_smem_bytes(NT, split ? per : N, E, k) + (F32 ? front_f32_chunk_bytes(NT) : 0);
  static PerDeviceOnce once_whole, once_split;
  auto fn = front_small_kernel<NT, true, T>;
  int rc = ensure_dynamic_smem(once_split, fn, 160 * 1024);
  if (rc) return rc;
  if constexpr (!F32) {
    rc = ensure_dynamic_smem(once_whole, front_small_kernel<NT, false, T>, 160 * 1024);
    if (rc) return rc;
    if (!split) fn = front_small_kernel<NT, false, T>;
  }
  const int blocks = (N + per - 1) / per;
  MOE_CUDA_CHECK(launch_pdl_as(fn, dim3(blocks), dim3(kThreads), 0, F32 && blocks > 1, smem, s, static_cast<const T*>(x),
                               static_cast<const T*>(Wg), static_cast<const T*>(bg), N, d, E, k, out_logits, out_idx,
                               out_w, cnt_slot, offsets, row_of, static_cast<T*>(perm),
                               static_cast<__nv_bfloat16*>(planes), psum, aux, xch, counter, status, per));
  return 0;
}

}  // namespace

bool front_small_supported(int64_t N, int E, int k, int dtype) {
  return dtype == MOE_B200_BF16 && N >= 1 && N <= kMaxTok && N * k <= kMaxPairs && E <= kMaxE;
}

// With the exchange buffer and the counter (blocks share the work): as many tokens as give a grid
// whose blocks are all resident at once with room to spare.
bool front_split_supported(int64_t N, int E, int k, int dtype) {
  return dtype == MOE_B200_BF16 && N >= 1 && N <= 16 * 128 && E <= kMaxE && k <= kMaxTopK;
}

// xch: int32 scratch of at least front_small_exchange_ints(N, E, k) words and counter: one int32
// that is zero on entry (both only used beyond 128 tokens; without them every block repeats the
// whole routing at every size).
int64_t front_small_exchange_ints(int64_t N, int E, int k) {
  const int per = f32_tokens_per_block(N);      // no fewer blocks than bf16 has
  const int64_t nb = (N + per - 1) / per;
  return nb * k * E + nb * E;
}

// fp32 calls: the general kernels took 36 us at 512 tokens (d 512, 8 experts: router 22, dispatch 14, with a memset in front).
// One block an SM, 128 of them at most: up to 2048 tokens on a whole GPU, fewer where a part of one is at hand.
bool front_f32_supported(int64_t N, int E, int k) {
  return N >= 1 && N <= 16 * 128 && E <= kMaxE && k <= kMaxTopK && N * k <= kRowsPathMaxRows;
}

int front_f32_resident(int64_t N, bool* yes) {
  int sms = 0;
  int rc = N > 16 ? sm_count(&sms) : 0;
  const int per = f32_tokens_per_block(N);
  *yes = rc == 0 && (N <= 16 || (N + per - 1) / per <= sms);
  return rc;
}

namespace {
template <typename T, typename... Args>
int launch_by_experts(int E, Args... args) {
  if (E <= 8) return launch<1, T>(args...);
  if (E <= 16) return launch<2, T>(args...);
  return launch<4, T>(args...);
}
}  // namespace

int launch_front_small(const void* x, const void* Wg, const void* bg, int64_t N, int d, int E, int k,
                       float* out_logits, int32_t* out_idx, float* out_w, int32_t* cnt_slot,
                       int32_t* offsets, int32_t* row_of, void* perm, float* psum, float* aux,
                       cudaStream_t s, int* xch, int* counter, int32_t* status, int dtype, void* planes) {
  if (dtype == MOE_B200_F32)
    return launch_by_experts<float>(E, x, Wg, bg, (int)N, d, E, k, out_logits, out_idx, out_w, cnt_slot, offsets, row_of,
                                    perm, planes, psum, aux, xch, counter, status, s);
  return launch_by_experts<__nv_bfloat16>(E, x, Wg, bg, (int)N, d, E, k, out_logits, out_idx, out_w, cnt_slot, offsets,
                                          row_of, perm, nullptr, psum, aux, xch, counter, status, s);
}

}  // namespace moe
