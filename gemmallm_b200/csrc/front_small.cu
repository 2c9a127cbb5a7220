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
// 16, which stores 160 KB at d 512: 512 tokens 81.8 -> 76.0 us, 51 tokens 58.5 -> 55.1, 1024 134 -> 130). Up to 16 are one
// block's, which need not meet any other.
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

// bf16 calls of more than 128 tokens: blocks of up to 16 tokens that share the work, of 16 warps. What a warp does counts four
// times and not eight, its loads (both its chunks of the tokens and of the weights, its token's row for the copy) are in flight
// together without spills, a token's softmax and top-k are a warp's and not a few lanes', and no step divides. Blocks meet
// at a grid barrier (up to 128 of them, one an SM, launched cooperatively).
// (front_small_body did it with 32 warps: 9.4 us from the wait to the end at 300 tokens, where this kernel takes 7.2. The
// cooperative launch takes 2 us of that again: front_small_body's blocks met under an ordinary launch, as if the GPU were
// theirs. Whole calls, d 1024, f 4096, 8 experts, that one -> this one: 130 tokens 52.3 -> 51.5 us, 300 58.3 -> 58.7, 400 61.3 ->
// 61.6, 600 64.4 -> 65.2, 1173 89.5 -> 90.3.)
constexpr int kMidWarps = 16, kMidTok = 16, kMidMaxE = 64;

// Tokens of a block, a power of two: fewer of them shorten the row copies, which the block's warps then share, and more blocks
// lengthen the meeting and read the router's weights more often. 2, 4, 8 and 16 of them, us a call: 64 experts, d 2048, f 1408,
// four slots, 60 tokens 189, 189, 190, 194; 100 200, 198, 198, 200; 300 203, 207, 205, 206; 1000 228, 226, 231, 230; 8 experts,
// d 1024, f 4096, 130 tokens 51.7, 51.3, 51.6, 53.0; 300 59.3, 59.4, 58.6, 59.7; 600 65.7, 65.5, 65.4, 65.5.
// Up to 8 tokens stay one block's, which need not meet any other.
int mid_tokens_per_block(int64_t N) {
  if (N <= 64) return N > 4 && N <= 8 ? 8 : 4;
  return N <= 512 ? 8 : kMidTok;
}

// More than 32 experts, two a lane, logits that are not finite as in front_many.cu: calls of up to 2048 tokens and 4096 rows,
// from one token on (d 2048, 64 experts of f 1408, four slots, whole calls against the general router and dispatch: 1 token
// 58.6 -> 37.3 us, 8 112 -> 90, 100 212 -> 199, 1000 245 -> 229).
template <int NT>      // 8 NT >= E
__global__ void __launch_bounds__(32 * kMidWarps, 1)
front_mid_kernel(const __nv_bfloat16* x, const __nv_bfloat16* Wg, const __nv_bfloat16* bg, int Ntotal, int d, int E, int k,
                 float* __restrict__ out_logits, int32_t* __restrict__ out_idx, float* __restrict__ out_w,
                 int32_t* __restrict__ cnt_slot, int32_t* __restrict__ offsets, int32_t* __restrict__ row_of,
                 __nv_bfloat16* __restrict__ perm, float* __restrict__ psum, float* __restrict__ aux, int* __restrict__ xch,
                 int per, int share) {
  constexpr int ET = 8 * NT, EL = ET > 32 ? 2 : 1, GL = ET / EL, P = 32 / GL;      // experts a lane, lanes of a token
  constexpr int kInFlight = 4, kChunks = NT > 4 ? 1 : 2;       // of a row to copy; of K
  extern __shared__ __align__(16) float s_dyn[];
  float (*s_part)[kMidTok][ET] = reinterpret_cast<float (*)[kMidTok][ET]>(s_dyn);   // [kMidWarps]; then block 0's probability
                                                                                    // sums of all blocks
  __shared__ float s_prob[kMidTok][ET];
  __shared__ int s_idx[kMidTok * kMaxTopK], s_row[kMidTok * kMaxTopK], s_tot[kMaxTopK * ET], s_base[ET];
  static_assert(kMidWarps * kMidTok >= 128, "the sums of 128 blocks");
  static_assert(kMaxTopK * ET <= 32 * kMidWarps, "a thread per count");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int b = (int)blockIdx.x, nb = (int)gridDim.x;
  const int N = min(per, Ntotal - b * per);
  const int pieces = d >> 3, nchunk = (d + 31) >> 5;
  x += (size_t)b * per * d;
  out_idx += (size_t)b * per * k;
  out_w += (size_t)b * per * k;
  row_of += (size_t)b * per * k;
  if (tid < ET) s_base[tid] = 0;
  if (tid < kMaxTopK * ET) s_tot[tid] = 0;
  pdl_wait();                 // x may come from the kernel before this one
  pdl_launch_dependents();

  // ---- logits: a warp's chunks of 32 of K, as in the body above ----
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const int own = warp / share, step = 32 * share, first_p = lane + 32 * (warp - own * share);     // the row this warp copies, from which
  const uint4* row = reinterpret_cast<const uint4*>(x) + (size_t)min(own, N - 1) * pieces;         // piece on
  uint4 pre[kInFlight];
#pragma unroll
  for (int u = 0; u < kInFlight; ++u) pre[u] = first_p + step * u < pieces ? __ldcg(row + first_p + step * u) : zero;
  const uint4* xa = reinterpret_cast<const uint4*>(x) + (size_t)min(g, N - 1) * pieces + t;
  const uint4* xb = reinterpret_cast<const uint4*>(x) + (size_t)min(g + 8, N - 1) * pieces + t;
  const uint4* wg = reinterpret_cast<const uint4*>(Wg) + t;
  float bias[EL];
#pragma unroll
  for (int i = 0; i < EL; ++i) bias[i] = lane % GL + 32 * i < E ? to_f32(bg[lane % GL + 32 * i]) : 0.f;
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
  for (int c0 = warp; c0 < nchunk; c0 += kChunks * kMidWarps) {
    uint4 A[kChunks], B[kChunks], W[kChunks][NT];
#pragma unroll
    for (int u = 0; u < kChunks; ++u) {
      const int p = 4 * (c0 + u * kMidWarps);
      const bool ok = p + t < pieces;
      A[u] = ok ? __ldcg(xa + p) : zero;
      B[u] = ok ? __ldcg(xb + p) : zero;
#pragma unroll
      for (int j = 0; j < NT; ++j) W[u][j] = ok ? wg[(size_t)min(8 * j + g, E - 1) * pieces + p] : zero;
    }
#pragma unroll
    for (int u = 0; u < kChunks; ++u)
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
    const int e0 = lane % GL;
    float v[EL], p[EL], sum = 0.f;
    unsigned key[EL], kmax = 0u;
#pragma unroll
    for (int i = 0; i < EL; ++i) {
      const int e = e0 + 32 * i;
      v[i] = 0.f;
#pragma unroll
      for (int q = 0; q < kMidWarps / P; ++q) v[i] += s_part[q * P + lane / GL][warp][e];
#pragma unroll
      for (int o = GL; o < 32; o <<= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
      v[i] += bias[i];
      if (out_logits != nullptr && lane < GL && e < E) out_logits[((size_t)b * per + warp) * E + e] = v[i];
      const bool live = e < E;
      v[i] = live ? v[i] + 0.f : -INFINITY;      // + 0: no negative zero
      const unsigned u = __float_as_uint(v[i]);
      key[i] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);      // order-preserving
      if (EL > 1 && !(live && v[i] == v[i])) key[i] = live ? 1u : 0u;      // below every number's: chosen last; never
      kmax = max(kmax, key[i]);
    }
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    const float m = __uint_as_float((kmax & 0x80000000u) ? (kmax & 0x7fffffffu) : ~kmax);
#pragma unroll
    for (int i = 0; i < EL; ++i) {
      p[i] = e0 + 32 * i < E ? expf(v[i] - m) : 0.f;
      sum += p[i];
    }
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv_sum = __frcp_rn(sum);
#pragma unroll
    for (int i = 0; i < EL; ++i)
      if (lane < GL) s_prob[warp][lane + 32 * i] = p[i] * inv_sum;
    int my_sel = 0;
    float my_val = 0.f, total = 0.f;
#pragma unroll 1
    for (int j = 0; j < k; ++j) {
      unsigned km = key[0];
      if (EL > 1) km = max(km, key[EL - 1]);
      km = __reduce_max_sync(0xffffffffu, km);
      const unsigned low = __ballot_sync(0xffffffffu, key[0] == km);      // (the first group's lanes come first)
      const unsigned high = EL > 1 ? __ballot_sync(0xffffffffu, key[EL - 1] == km) : 0u;
      const int winner = low != 0u ? __ffs(low) - 1 : 31 + __ffs(high);
      const float bv = __uint_as_float((km & 0x80000000u) ? (km & 0x7fffffffu) : ~km);
      const float val = EL > 1 ? expf(bv - m) : expf(bv - m) * inv_sum;      // (as router_tc_kernel: their sum cancels the denominator)
      total += val;
      if (lane == j) { my_sel = winner; my_val = val; }
#pragma unroll
      for (int i = 0; i < EL; ++i)
        if (e0 + 32 * i == winner) key[i] = 0u;     // below every real key
    }
    if (lane < k) {
      s_idx[warp * k + lane] = my_sel;
      out_idx[warp * k + lane] = my_sel;
      out_w[warp * k + lane] = EL > 1 ? my_val / total : my_val * __frcp_rn(total);
    }
  } else {      // (no token: below, nothing has to ask)
    if (lane < k) s_idx[warp * k + lane] = -1;
    for (int e = lane; e < ET; e += 32) s_prob[warp][e] = 0.f;
  }
  __syncthreads();

  // ---- this block's counts per (slot, expert), a count's blocks side by side (where there are many counts, a block's), and its
  // probability sums ----
  float* s_sum = s_dyn;
  const int ke = k * E;
  const bool wide = ke > 2 * kMidWarps;
  float* xps = reinterpret_cast<float*>(xch + nb * ke);    // [nb][E]
  for (int i = tid; i < ke; i += 32 * kMidWarps) {
    int c = 0;
    const int j = i / E, e = i - j * E;
#pragma unroll
    for (int tok = 0; tok < kMidTok; ++tok) c += s_idx[tok * k + j] == e ? 1 : 0;
    if (nb == 1) s_tot[i] = c;
    else xch[wide ? b * ke + i : i * nb + b] = c;
  }
  if (tid >= 32 * kMidWarps - E) {
    const int e = tid - (32 * kMidWarps - E);
    float ps = 0.f;
#pragma unroll
    for (int tok = 0; tok < kMidTok; ++tok) ps += s_prob[tok][e];
    if (nb == 1) s_sum[e] = ps;
    else xps[b * E + e] = ps;
  }
  if (nb == 1) {
    __syncthreads();
  } else {
    cooperative_groups::this_grid().sync();
    // totals, and the rows that earlier blocks put in front of this block's (16 bits: 2048 tokens)
    if (!wide) {      // a warp per count
      for (int je = warp; je < ke; je += kMidWarps) {
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
    } else {          // a thread per count, or several (a warp per count: 16 rounds of loads one after the other)
      const int per = 32 * kMidWarps / ke, q = tid / ke, je = tid - q * ke;
      if (q < per) {
        unsigned both = 0;
#pragma unroll 16
        for (int bb = q; bb < nb; bb += per) {
          const unsigned c = (unsigned)__ldcg(&xch[bb * ke + je]);
          both += c | (bb < b ? c << 16 : 0u);
        }
        if (both & 0xffffu) atomicAdd(&s_tot[je], (int)(both & 0xffffu));
        if (both >> 16) atomicAdd(&s_base[je % E], (int)(both >> 16));
      }
    }
    if (b == 0)
      for (int i = tid; i < nb * E; i += 32 * kMidWarps) s_sum[i] = __ldcg(&xps[i]);
    __syncthreads();
  }

  // ---- offsets (every warp), stable ranks in (token, slot) order: a warp per expert, 32 pairs at a time ----
  int first[EL], mine0[EL], before = 0;      // of experts lane, 32 + lane: first row; first row of this block's tokens
#pragma unroll
  for (int i = 0; i < EL; ++i) {
    const int e = lane + 32 * i;
    int tot = 0;
    if (e < E)
      for (int j = 0; j < k; ++j) tot += s_tot[j * E + e];
    int incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    first[i] = before + incl - tot;
    mine0[i] = first[i] + (e < E ? s_base[e] : 0);
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
  const int npair = N * k;
  for (int e = warp; e < E; e += kMidWarps) {
    int next = __shfl_sync(0xffffffffu, EL > 1 && e >= 32 ? mine0[EL - 1] : mine0[0], e & 31);
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

  // ---- row copies: `share` warps per token ----
  if (own < N)
    for (int j = 0; j < k; ++j) {
      const int r = s_row[own * k + j];
      uint4* to = reinterpret_cast<uint4*>(perm + (size_t)r * d);
#pragma unroll
      for (int u = 0; u < kInFlight; ++u)
        if (first_p + step * u < pieces) to[first_p + step * u] = pre[u];
      for (int p = first_p + step * kInFlight; p < pieces; p += step) to[p] = __ldcg(row + p);
    }
  if (b == 0) {
    if (warp == kMidWarps - 1) {
#pragma unroll
      for (int i = 0; i < EL; ++i) {
        const int e = lane + 32 * i;
        if (e < E) {
          for (int j = 0; j < k; ++j) cnt_slot[j * E + e] = s_tot[j * E + e];
          offsets[e] = first[i];
        }
      }
      if (lane == 31) offsets[E] = before;
    }
    if (warp == kMidWarps - 2) {      // the loss (model.py:213-216)
      float a = 0.f;
#pragma unroll
      for (int i = 0; i < EL; ++i) {
        const int e = lane + 32 * i;
        float term = 0.f;
        if (e < E) {
          float ps = 0.f;
#pragma unroll 8
          for (int bb = 0; bb < nb; ++bb) ps += s_sum[bb * E + e];      // in block order
          psum[e] = ps;
          term = (ps / (float)Ntotal) * ((float)s_tot[e] / (float)Ntotal);
        }
        for (int q = 0; q < 32 && q + 32 * i < E; ++q) a += __shfl_sync(0xffffffffu, term, q);
      }
      if (lane == 0) aux[0] = a / (float)E * (float)(E * E);
    }
  }
}

template <int NT>
int launch_mid(const void* x, const void* Wg, const void* bg, int N, int d, int E, int k, float* out_logits, int32_t* out_idx,
               float* out_w, int32_t* cnt_slot, int32_t* offsets, int32_t* row_of, void* perm, float* psum, float* aux, int* xch,
               int per, cudaStream_t s) {
  const size_t smem = sizeof(float) * kMidWarps * kMidTok * 8 * NT;
  static PerDeviceOnce once;
  int rc = ensure_dynamic_smem(once, front_mid_kernel<NT>, smem);
  if (rc) return rc;
  // cooperative, since its blocks wait for one another: beside those of other streams they start when all of them fit
  const int blocks = (N + per - 1) / per;
  MOE_CUDA_CHECK(launch_pdl_as(front_mid_kernel<NT>, dim3(blocks), dim3(32 * kMidWarps), 0, blocks > 1, smem, s,
                            static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(Wg),
                            static_cast<const __nv_bfloat16*>(bg), N, d, E, k, out_logits, out_idx, out_w, cnt_slot, offsets,
                            row_of, static_cast<__nv_bfloat16*>(perm), psum, aux, xch, per, kMidWarps / per));
  return 0;
}

template <int NT, typename T>
int launch(const void* x, const void* Wg, const void* bg, int N, int d, int E, int k,
           float* out_logits, int32_t* out_idx, float* out_w, int32_t* cnt_slot, int32_t* offsets,
           int32_t* row_of, void* perm, void* planes, float* psum, float* aux, int* xch, int32_t* status, cudaStream_t s) {
  constexpr bool F32 = sizeof(T) == 4;
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

// With the exchange buffer (blocks share the work): as many tokens as give a grid
// whose blocks are all resident at once with room to spare.
// (More than 32 experts where the general router is the tcgen05 kernel, whose choice among logits that are not finite is also
// always an expert.)
bool front_split_supported(int64_t N, int d, int E, int k, int dtype) {
  return dtype == MOE_B200_BF16 && N >= 1 && N <= 16 * 128 && E <= kMidMaxE && (E <= kMaxE || d >= 64) && k <= kMaxTopK;
}

// xch: int32 scratch of at least front_small_exchange_ints(N, E, k) words (only used beyond 128 tokens or 32 experts; without
// it every block repeats the whole routing at every size). per: tokens of a block that shares the work, 0 for the best number; with 16 the public
// entry's smaller exchange buffer does.
int64_t front_small_exchange_ints(int64_t N, int E, int k) {
  const int64_t nb = N < 512 ? (N + 3) / 4 : 128;      // the most that either type has
  return nb * k * E + nb * E;
}

// fp32 calls: the general kernels took 36 us at 512 tokens (d 512, 8 experts: router 22, dispatch 14, with a memset in front).
// One block an SM, 128 of them at most: up to 2048 tokens on a whole GPU, fewer where a part of one is at hand.
bool front_f32_supported(int64_t N, int E, int k) {
  return N >= 1 && N <= 16 * 128 && E <= kMaxE && k <= kMaxTopK && N * k <= kRowsPathMaxRows;
}

int front_resident(int64_t N, int dtype, bool* yes) {
  int sms = 0;
  int rc = N > 8 ? sm_count(&sms) : 0;
  const int per = dtype == MOE_B200_F32 ? f32_tokens_per_block(N) : mid_tokens_per_block(N);
  *yes = rc == 0 && (N + per - 1) / per <= (N > 8 ? sms : 1);
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
                       cudaStream_t s, int* xch, int32_t* status, int dtype, void* planes, int per) {
  if (dtype == MOE_B200_F32)
    return launch_by_experts<float>(E, x, Wg, bg, (int)N, d, E, k, out_logits, out_idx, out_w, cnt_slot, offsets, row_of,
                                    perm, planes, psum, aux, xch, status, s);
  // beyond 128 tokens repeating the routing in every block costs more than one exchange
  if (xch != nullptr && (N > 128 || E > kMaxE)) {
    auto mid = E <= 8 ? launch_mid<1> : E <= 16 ? launch_mid<2> : E <= 32 ? launch_mid<4> : launch_mid<8>;
    return mid(x, Wg, bg, (int)N, d, E, k, out_logits, out_idx, out_w, cnt_slot, offsets, row_of, perm, psum, aux, xch,
               per > 0 ? per : mid_tokens_per_block(N), s);
  }
  return launch_by_experts<__nv_bfloat16>(E, x, Wg, bg, (int)N, d, E, k, out_logits, out_idx, out_w, cnt_slot, offsets,
                                          row_of, perm, nullptr, psum, aux, xch, status, s);
}

}  // namespace moe
