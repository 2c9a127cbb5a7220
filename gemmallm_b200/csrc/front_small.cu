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

template <int NT, typename T>
__global__ void __launch_bounds__(kThreads, 1)
front_small_kernel(const T* __restrict__ x, const T* Wg, const T* bg, int Ntotal, int d, int E, int k,
                   float* __restrict__ out_logits, int32_t* __restrict__ out_idx,
                   float* __restrict__ out_w, int32_t* __restrict__ cnt_slot,
                   int32_t* __restrict__ offsets, int32_t* __restrict__ row_of,
                   T* __restrict__ perm, __nv_bfloat16* __restrict__ planes, float* __restrict__ psum,
                   float* __restrict__ aux, int* __restrict__ xch, int32_t* __restrict__ status, int per) {
  extern __shared__ float smem[];
  pdl_wait();                 // x may come from the kernel before this one
  pdl_launch_dependents();
  front_small_body<NT, T>(smem, x, Wg, bg, Ntotal, d, E, k, out_logits, out_idx, out_w, cnt_slot, offsets, row_of, perm, planes,
                          psum, aux, xch, status, per);
}

// bf16 calls of more than 128 tokens: blocks of 16 tokens that share the work, of 16 warps. What a warp does counts four
// times and not eight, its loads (both its chunks of the tokens and of the weights, its token's row for the copy) are in flight
// together without spills, a token's softmax and top-k are a warp's and not a few lanes', and no step divides. Blocks meet
// at a counter (up to 128 of them, one an SM, on an otherwise idle GPU); the wait is bounded and reports a time-out.
// (front_small_body did it with 32 warps: 9.4 us from the wait to the end at 300 tokens, where this kernel takes 7.2. Whole
// calls, d 1024, f 4096, 8 experts: 130 tokens 53.1 -> 51.6 us, 300 59.3 -> 57.9, 400 62.0 -> 60.9, 1173 88.0 -> 86.8.)
constexpr int kMidWarps = 16, kMidTok = 16;

template <int NT>      // 8 NT >= E
__global__ void __launch_bounds__(32 * kMidWarps, 1)
front_mid_kernel(const __nv_bfloat16* x, const __nv_bfloat16* Wg, const __nv_bfloat16* bg, int Ntotal, int d, int E, int k,
                 float* __restrict__ out_logits, int32_t* __restrict__ out_idx, float* __restrict__ out_w,
                 int32_t* __restrict__ cnt_slot, int32_t* __restrict__ offsets, int32_t* __restrict__ row_of,
                 __nv_bfloat16* __restrict__ perm, float* __restrict__ psum, float* __restrict__ aux, int* __restrict__ xch,
                 int* __restrict__ counter, int32_t* __restrict__ status) {
  constexpr int ET = 8 * NT, P = 32 / ET;
  constexpr int kInFlight = 4;
  __shared__ __align__(16) float s_part[kMidWarps][kMidTok][ET];    // then block 0's probability sums of all blocks
  __shared__ float s_prob[kMidTok][ET];
  __shared__ int s_idx[kMidTok * kMaxTopK], s_row[kMidTok * kMaxTopK], s_tot[kMaxTopK * kMaxE], s_base[kMaxE];
  static_assert(sizeof(s_part) >= 128 * ET * sizeof(float), "the sums of 128 blocks");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int b = (int)blockIdx.x, nb = (int)gridDim.x;
  const int N = min(kMidTok, Ntotal - b * kMidTok);
  const int pieces = d >> 3, nchunk = (d + 31) >> 5;
  x += (size_t)b * kMidTok * d;
  out_idx += (size_t)b * kMidTok * k;
  out_w += (size_t)b * kMidTok * k;
  row_of += (size_t)b * kMidTok * k;
  if (tid < kMaxE) s_base[tid] = 0;
  pdl_wait();                 // x may come from the kernel before this one
  pdl_launch_dependents();

  // ---- logits: a warp's chunks of 32 of K, as in the body above ----
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const uint4* row = reinterpret_cast<const uint4*>(x) + (size_t)min(warp, N - 1) * pieces;      // the one this warp copies
  uint4 pre[kInFlight];
#pragma unroll
  for (int u = 0; u < kInFlight; ++u) pre[u] = lane + 32 * u < pieces ? __ldcg(row + lane + 32 * u) : zero;
  const uint4* xa = reinterpret_cast<const uint4*>(x) + (size_t)min(g, N - 1) * pieces + t;
  const uint4* xb = reinterpret_cast<const uint4*>(x) + (size_t)min(g + 8, N - 1) * pieces + t;
  const uint4* wg = reinterpret_cast<const uint4*>(Wg) + t;
  const float bias = lane % ET < E ? to_f32(bg[lane % ET]) : 0.f;
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
  for (int c0 = warp; c0 < nchunk; c0 += 2 * kMidWarps) {
    uint4 A[2], B[2], W[2][NT];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int p = 4 * (c0 + u * kMidWarps);
      const bool ok = p + t < pieces;
      A[u] = ok ? __ldcg(xa + p) : zero;
      B[u] = ok ? __ldcg(xb + p) : zero;
#pragma unroll
      for (int j = 0; j < NT; ++j) W[u][j] = ok ? wg[(size_t)min(8 * j + g, E - 1) * pieces + p] : zero;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma_bf16_16816(acc[j], A[u].x, B[u].x, A[u].y, B[u].y, W[u][j].x, W[u][j].y);
        mma_bf16_16816(acc[j], A[u].z, B[u].z, A[u].w, B[u].w, W[u][j].z, W[u][j].w);
      }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    *reinterpret_cast<float2*>(&s_part[warp][g][8 * j + 2 * t]) = make_float2(acc[j][0], acc[j][1]);
    *reinterpret_cast<float2*>(&s_part[warp][g + 8][8 * j + 2 * t]) = make_float2(acc[j][2], acc[j][3]);
  }
  __syncthreads();

  // ---- softmax, top-k, renormalise: a warp per token; lane = expert, groups of lanes share the sum over the slices ----
  if (warp < N) {
    const int e = lane % ET;
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < kMidWarps / P; ++q) v += s_part[q * P + lane / ET][warp][e];
#pragma unroll
    for (int o = ET; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    v += bias;
    const bool live = e < E;
    if (out_logits != nullptr && lane < E) out_logits[((size_t)b * kMidTok + warp) * E + lane] = v;
    v = live ? v + 0.f : -INFINITY;      // + 0: no negative zero
    const unsigned u = __float_as_uint(v);
    unsigned key = (u & 0x80000000u) ? ~u : (u | 0x80000000u);      // order-preserving; NaN is the largest
    const unsigned kmax = __reduce_max_sync(0xffffffffu, key);
    const float m = __uint_as_float((kmax & 0x80000000u) ? (kmax & 0x7fffffffu) : ~kmax);
    const float p = live ? expf(v - m) : 0.f;
    float sum = p;
#pragma unroll
    for (int o = ET / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv_sum = __frcp_rn(sum);
    if (lane < ET) s_prob[warp][lane] = p * inv_sum;
    int my_sel = 0;
    float my_val = 0.f, total = 0.f;
#pragma unroll 1
    for (int j = 0; j < k; ++j) {
      const unsigned km = __reduce_max_sync(0xffffffffu, key);
      const int winner = __ffs(__ballot_sync(0xffffffffu, key == km)) - 1;      // in the first group
      const float bv = __uint_as_float((km & 0x80000000u) ? (km & 0x7fffffffu) : ~km);
      const float val = expf(bv - m) * inv_sum;
      total += val;
      if (lane == j) { my_sel = winner; my_val = val; }
      if (e == winner) key = 0u;     // below every real key
    }
    if (lane < k) {
      s_idx[warp * k + lane] = my_sel;
      out_idx[warp * k + lane] = my_sel;
      out_w[warp * k + lane] = my_val * __frcp_rn(total);
    }
  } else {      // (no token: below, nothing has to ask)
    if (lane < k) s_idx[warp * k + lane] = -1;
    if (lane < ET) s_prob[warp][lane] = 0.f;
  }
  __syncthreads();

  // ---- this block's counts per (slot, expert), a count's blocks side by side, and its probability sums ----
  float* xps = reinterpret_cast<float*>(xch + nb * k * E);    // [nb][E]
  if (tid < k * E) {
    int c = 0;
    const int j = tid / E, e = tid - j * E;
#pragma unroll
    for (int tok = 0; tok < kMidTok; ++tok) c += s_idx[tok * k + j] == e ? 1 : 0;
    xch[tid * nb + b] = c;
  } else if (tid >= 32 * kMidWarps - E) {
    const int e = tid - (32 * kMidWarps - E);
    float ps = 0.f;
#pragma unroll
    for (int tok = 0; tok < kMidTok; ++tok) ps += s_prob[tok][e];
    xps[b * E + e] = ps;
  }
  __syncthreads();
  int left = 0;
  if (tid == 0) {
    __threadfence();
    atomicAdd(counter, 1);
    unsigned long long t0 = 0;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (uint32_t it = 0; ld_acquire_gpu_i32(counter) < nb; ++it) {
      if ((it & 63u) == 63u) {
        unsigned long long t1;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
        if (t1 - t0 > 2000000000ull) {     // 2 s: some block of the grid never arrived
          atomicMax(&status[0], MOE_B200_DEV_TIMEOUT);
          status[1] = 41;
          status[2] = b;
          break;
        }
      }
    }
    left = atomicAdd(counter, 1);      // looked at in the end
  }
  __syncthreads();
  // totals, and the rows that earlier blocks put in front of this block's: a warp each (16 bits: 2048 tokens)
  for (int je = warp; je < k * E; je += kMidWarps) {
    unsigned both = 0;
    for (int bb = lane; bb < nb; bb += 32) {
      const unsigned c = (unsigned)__ldcg(&xch[je * nb + bb]);
      both += c | (bb < b ? c << 16 : 0u);
    }
    both = __reduce_add_sync(0xffffffffu, both);
    if (lane == 0) {
      s_tot[je] = (int)(both & 0xffffu);
      if (both >> 16) atomicAdd(&s_base[je % E], (int)(both >> 16));
    }
  }
  float* s_sum = &s_part[0][0][0];
  if (b == 0)
    for (int i = tid; i < nb * E; i += 32 * kMidWarps) s_sum[i] = __ldcg(&xps[i]);
  __syncthreads();

  // ---- offsets (every warp), stable ranks in (token, slot) order: a warp per expert, 32 pairs at a time ----
  int tot = 0;
  if (lane < E)
    for (int j = 0; j < k; ++j) tot += s_tot[j * E + lane];
  int incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  const int mine0 = incl - tot + (lane < E ? s_base[lane] : 0);      // first row of this block's tokens
  const int npair = N * k;
  for (int e = warp; e < E; e += kMidWarps) {
    int next = __shfl_sync(0xffffffffu, mine0, e);
    for (int p0 = 0; p0 < npair; p0 += 32) {
      const int p = p0 + lane;
      const bool mine = p < npair && s_idx[p] == e;
      const unsigned hit = __ballot_sync(0xffffffffu, mine);
      if (mine) {
        const int r = next + __popc(hit & ((1u << lane) - 1u));
        s_row[p] = r;
        row_of[p] = r;
      }
      next += __popc(hit);
    }
  }
  __syncthreads();

  // ---- row copies: a warp per token ----
  if (warp < N)
    for (int j = 0; j < k; ++j) {
      const int r = s_row[warp * k + j];
      if ((unsigned)r >= (unsigned)(Ntotal * k)) continue;      // (counts of a block that never arrived)
      uint4* to = reinterpret_cast<uint4*>(perm + (size_t)r * d);
#pragma unroll
      for (int u = 0; u < kInFlight; ++u)
        if (lane + 32 * u < pieces) to[lane + 32 * u] = pre[u];
      for (int p = lane + 32 * kInFlight; p < pieces; p += 32) to[p] = __ldcg(row + p);
    }
  if (b == 0) {
    if (warp == kMidWarps - 1) {
      if (lane < E) {
        for (int j = 0; j < k; ++j) cnt_slot[j * E + lane] = s_tot[j * E + lane];
        offsets[lane] = incl - tot;
      }
      if (lane == 31) offsets[E] = incl;
    }
    if (warp == kMidWarps - 2) {      // the loss (model.py:213-216)
      float term = 0.f;
      if (lane < E) {
        float ps = 0.f;
#pragma unroll 8
        for (int bb = 0; bb < nb; ++bb) ps += s_sum[bb * E + lane];      // in block order
        psum[lane] = ps;
        term = (ps / (float)Ntotal) * ((float)s_tot[lane] / (float)Ntotal);
      }
      float a = 0.f;
      for (int e = 0; e < E; ++e) a += __shfl_sync(0xffffffffu, term, e);
      if (lane == 0) aux[0] = a / (float)E * (float)(E * E);
    }
  }
  // the last block to leave puts the meeting counter back to zero for the next call
  if (tid == 0 && left == 2 * nb - 1) *counter = 0;
}

template <int NT, typename T>
int launch(const void* x, const void* Wg, const void* bg, int N, int d, int E, int k,
           float* out_logits, int32_t* out_idx, float* out_w, int32_t* cnt_slot, int32_t* offsets,
           int32_t* row_of, void* perm, void* planes, float* psum, float* aux, int* xch, int* counter,
           int32_t* status, cudaStream_t s) {
  // beyond 128 tokens repeating the routing in every block costs more than one exchange
  constexpr bool F32 = sizeof(T) == 4;
  if constexpr (!F32) {
    if (xch != nullptr && counter != nullptr && status != nullptr && N > 128) {
      MOE_CUDA_CHECK(launch_pdl(front_mid_kernel<NT>, dim3((N + kMidTok - 1) / kMidTok), dim3(32 * kMidWarps), 0, s,
                                static_cast<const T*>(x), static_cast<const T*>(Wg), static_cast<const T*>(bg), N, d, E, k,
                                out_logits, out_idx, out_w, cnt_slot, offsets, row_of, static_cast<T*>(perm), psum, aux, xch,
                                counter, status));
      return 0;
    }
  }
  const int per = F32 ? f32_tokens_per_block(N) : 16;
  const size_t smem = front_small_smem_bytes(NT, F32 ? per : N, E, k) + (F32 ? front_f32_chunk_bytes(NT) : 0);
  static PerDeviceOnce once;
  auto fn = front_small_kernel<NT, T>;
  int rc = ensure_dynamic_smem(once, fn, 160 * 1024);
  if (rc) return rc;
  const int blocks = (N + per - 1) / per;
  MOE_CUDA_CHECK(launch_pdl_as(fn, dim3(blocks), dim3(kThreads), 0, F32 && blocks > 1, smem, s, static_cast<const T*>(x),
                               static_cast<const T*>(Wg), static_cast<const T*>(bg), N, d, E, k, out_logits, out_idx,
                               out_w, cnt_slot, offsets, row_of, static_cast<T*>(perm),
                               static_cast<__nv_bfloat16*>(planes), psum, aux, xch, status, per));
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
