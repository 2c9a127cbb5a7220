// Router and dispatch of a few thousand tokens in ONE launch (bf16): logits, softmax, top-k, counts, offsets, ranks, the sorted
// copies of the rows and the load-balancing loss (reference model.py:206-253), and for a training step the pair of every row.
//
// A block routes a range of tokens, 16 at a time, exchanges its counts with the other blocks at a grid barrier and
// copies its tokens' rows. What bounds it is latency, not bandwidth: a group of 16 tokens is one round trip for its rows, one
// meeting of the block's warps and one chain of softmax and top-k, so the next group's rows are under way during that chain
// (its partial sums go to the other half of a double buffer, one block barrier a group), and the first rows to copy during
// the exchange. The blocks are at most one an SM and are launched cooperatively, since they wait for one another.
//
// Logits that are not finite are treated as by the general kernels that take the larger calls: up to 16 experts neither NaN nor
// minus infinity is ever chosen, a slot without an expert has the index 0x7fffffff and no row, and the status says so; beyond,
// every slot gets an expert, NaN after all others, and the weights are formed of the chosen logits alone: one expert whose
// logits are NaN does not make those of the others NaN.
#include "front_small.cuh"

namespace moe {

namespace {

constexpr int kWarps = 16, kGroup = 16, kMaxPer = 128;      // tokens of a block, at most

// NORM: Wg is the folded weight of norm.cu and norm_c its constants, stats the (mean, rstd) of every row; logits as the general
// router forms them then, copies of the normalised rows `xn`.
template <int NT, bool NORM>      // 8 NT >= E
__global__ void __launch_bounds__(32 * kWarps, 1)
front_many_kernel(const __nv_bfloat16* x, const __nv_bfloat16* xn, const float* stats, const float* norm_c,
                  const __nv_bfloat16* Wg, const __nv_bfloat16* bg, int Ntotal, int d, int E, int k,
                  float* __restrict__ out_logits, int32_t* __restrict__ out_idx, float* __restrict__ out_w,
                  int32_t* __restrict__ cnt_slot, int32_t* __restrict__ offsets, int32_t* __restrict__ row_of,
                  __nv_bfloat16* __restrict__ perm, int32_t* __restrict__ pair_of, float* __restrict__ psum,
                  float* __restrict__ aux, int* __restrict__ xch, int32_t* __restrict__ status, int per, int share,
                  bool clear) {
  constexpr int ET = 8 * NT, EL = ET > 32 ? 2 : 1, GL = ET / EL, P = 32 / GL;      // experts a lane, lanes of a token
  constexpr bool STRICT = NT <= 2;
  static_assert(!NORM || STRICT, "with a folded LayerNorm the general router is the strict one at any number of experts");
  constexpr int kInFlight = 4, kChunks = NT > 4 ? 1 : 2;       // of a row to copy; of K
  extern __shared__ __align__(16) float s_dyn[];
  float (*s_part)[kWarps][kGroup][ET] = reinterpret_cast<float (*)[kWarps][kGroup][ET]>(s_dyn);      // [2]; then block 0's
  int* s_idx = reinterpret_cast<int*>(s_dyn + 2 * kWarps * kGroup * ET);                             // probability sums of all
  int* s_row = s_idx + per * k;                                                                      // blocks
  static_assert(2 * kWarps * kGroup >= kNumSMs, "the sums of all blocks");
  __shared__ float s_prob[kWarps][ET];
  __shared__ int s_cnt[kMaxTopK * ET], s_tot[kMaxTopK * ET], s_base[ET];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int b = (int)blockIdx.x, nb = (int)gridDim.x, ke = k * E;
  const bool wide = ke > 2 * kWarps;      // many counts
  const int N = min(per, Ntotal - b * per);
  const int pieces = d >> 3, nchunk = (d + 31) >> 5;
  x += (size_t)b * per * d;
  xn += (size_t)b * per * d;
  if (NORM) stats += (size_t)b * per * 2;
  out_idx += (size_t)b * per * k;
  out_w += (size_t)b * per * k;
  row_of += (size_t)b * per * k;
  for (int i = tid; i < kMaxTopK * ET; i += 32 * kWarps) s_cnt[i] = s_tot[i] = 0;
  if (tid < ET) s_base[tid] = 0;
  pdl_wait();                 // x may come from the kernel before this one
  pdl_launch_dependents();
  // (in front of the exchange: nothing is reported or counted before it)
  if (clear && b == 0)
    for (int i = tid; i < MOE_B200_READY_OFFSET + MOE_B200_READY_INTS; i += 32 * kWarps) status[i] = 0;
  __syncthreads();

  // ---- routing, 16 tokens at a time: a warp's chunks of 32 of K for all of them, then a token for every warp ----
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const uint4* xp = reinterpret_cast<const uint4*>(x);
  const uint4* wg = reinterpret_cast<const uint4*>(Wg) + t;
  float bias[EL], c1[EL], psum_acc[EL];
#pragma unroll
  for (int i = 0; i < EL; ++i) {
    const int e = lane % GL + 32 * i;
    bias[i] = e < E ? (NORM ? __ldcg(&norm_c[E + e]) : to_f32(bg[e])) : 0.f;
    c1[i] = NORM && e < E ? __ldcg(&norm_c[e]) : 0.f;
    psum_acc[i] = 0.f;
  }
  uint4 A[kChunks], B[kChunks], W[kChunks][NT];
  auto load = [&](int t0, int c0) {
    const uint4* xa = xp + (size_t)min(t0 + g, N - 1) * pieces + t;
    const uint4* xb = xp + (size_t)min(t0 + g + 8, N - 1) * pieces + t;
#pragma unroll
    for (int u = 0; u < kChunks; ++u) {
      const int p = 4 * (c0 + u * kWarps);
      const bool ok = p + t < pieces;
      A[u] = ok ? __ldcg(xa + p) : zero;
      B[u] = ok ? __ldcg(xb + p) : zero;
#pragma unroll
      for (int j = 0; j < NT; ++j) W[u][j] = ok ? wg[(size_t)min(8 * j + g, E - 1) * pieces + p] : zero;
    }
  };
  load(0, warp);
  int half = 0;
  for (int t0 = 0; t0 < N; t0 += kGroup, half ^= 1) {
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
    for (int c0 = warp; c0 < nchunk; c0 += kChunks * kWarps) {
      if (c0 != warp) load(t0, c0);
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
      *reinterpret_cast<float2*>(&s_part[half][warp][g][8 * j + 2 * t]) = make_float2(acc[j][0], acc[j][1]);
      *reinterpret_cast<float2*>(&s_part[half][warp][g + 8][8 * j + 2 * t]) = make_float2(acc[j][2], acc[j][3]);
    }
    if (t0 + kGroup < N) load(t0 + kGroup, warp);
    __syncthreads();      // (the one before it: all warps are done with the other half)

    const int tok = t0 + warp;
    if (tok < N) {
      const int e0 = lane % GL;
      const float mean = NORM ? __ldcg(&stats[2 * tok]) : 0.f, rstd = NORM ? __ldcg(&stats[2 * tok + 1]) : 1.f;
      float v[EL], p[EL], sum = 0.f;
      unsigned key[EL], kmax = 0u;
#pragma unroll
      for (int i = 0; i < EL; ++i) {
        const int e = e0 + 32 * i;
        v[i] = 0.f;
#pragma unroll
        for (int q = 0; q < kWarps / P; ++q) v[i] += s_part[half][q * P + lane / GL][warp][e];
#pragma unroll
        for (int o = GL; o < 32; o <<= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        v[i] = NORM ? rstd * (v[i] - mean * c1[i]) + bias[i] : v[i] + bias[i];
        const bool live = e < E;
        if (lane < GL && live) out_logits[((size_t)b * per + tok) * E + e] = v[i];
        v[i] = live ? v[i] + 0.f : -INFINITY;      // + 0: no negative zero
        const unsigned u = __float_as_uint(v[i]);
        key[i] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);      // order-preserving
        if (STRICT && !(v[i] > -INFINITY)) key[i] = 0u;           // never chosen
        if (!STRICT && !(live && v[i] == v[i])) key[i] = live ? 1u : 0u;      // below every number's: chosen last; never
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
#pragma unroll
      for (int i = 0; i < EL; ++i) psum_acc[i] += p[i] / sum;
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
        const bool none = STRICT && km == 0u;
        // (beyond 16 experts as router_tc_kernel: the denominator, which the sum of the chosen cancels, is left out)
        const float val = STRICT ? (none ? 0.f : expf(bv - m)) / sum : expf(bv - m);
        total += val;                    // left-to-right sum, as model.py:221
        if (lane == j) { my_sel = none ? 0x7fffffff : winner; my_val = val; }
#pragma unroll
        for (int i = 0; i < EL; ++i)
          if (e0 + 32 * i == winner) key[i] = 0u;     // below every real key
      }
      if (lane < k) {
        s_idx[tok * k + lane] = my_sel;
        out_idx[tok * k + lane] = my_sel;
        out_w[tok * k + lane] = my_val / total;
        if (!STRICT || my_sel < E) atomicAdd(&s_cnt[lane * E + my_sel], 1);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < EL; ++i)
    if (lane < GL) s_prob[warp][lane + 32 * i] = psum_acc[i];
  // `share` warps copy a row together: from piece first_p of token `own` on, and of every (16 / share)-th after it
  const int own = warp / share, step = 32 * share, first_p = lane + 32 * (warp - own * share), stride = kWarps / share;
  uint4 cur[kInFlight], nxt[kInFlight];
  auto fetch = [&](uint4 (&v)[kInFlight], int tok) {
    const uint4* row = reinterpret_cast<const uint4*>(xn) + (size_t)min(tok, N - 1) * pieces;
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) v[u] = first_p + step * u < pieces ? __ldcg(row + first_p + step * u) : zero;
  };
  fetch(cur, own);
  __syncthreads();

  // ---- the exchange: this block's counts per (slot, expert) and its probability sums ----
  float* s_sum = s_dyn;
  float* xps = reinterpret_cast<float*>(xch + nb * ke);    // [nb][E]
  for (int i = tid; i < ke; i += 32 * kWarps) {
    if (nb == 1) s_tot[i] = s_cnt[i];
    else xch[wide ? b * ke + i : i * nb + b] = s_cnt[i];
  }
  if (tid >= 32 * kWarps - E) {
    const int e = tid - (32 * kWarps - E);
    float ps = 0.f;
#pragma unroll
    for (int q = 0; q < kWarps; ++q) ps += s_prob[q][e];
    if (nb == 1) s_sum[e] = ps;
    else xps[b * E + e] = ps;
  }
  if (nb == 1) {
    __syncthreads();
  } else {
    cooperative_groups::this_grid().sync();
    // totals, and the rows that earlier blocks put in front of this block's (16 bits: fewer than 65536 tokens)
    if (!wide) {      // a warp per count
      for (int je = warp; je < ke; je += kWarps) {
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
    } else {          // a thread per count, or several
      const int shares = 32 * kWarps / ke, q = tid / ke, je = tid - q * ke;
      if (q < shares) {
        unsigned both = 0;
#pragma unroll 16
        for (int bb = q; bb < nb; bb += shares) {
          const unsigned c = (unsigned)__ldcg(&xch[bb * ke + je]);
          both += c | (bb < b ? c << 16 : 0u);
        }
        if (both & 0xffffu) atomicAdd(&s_tot[je], (int)(both & 0xffffu));
        if (both >> 16) atomicAdd(&s_base[je % E], (int)(both >> 16));
      }
    }
    if (b == 0)
      for (int i = tid; i < nb * E; i += 32 * kWarps) s_sum[i] = __ldcg(&xps[i]);
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
  for (int e = warp; e < E; e += kWarps) {
    int next = __shfl_sync(0xffffffffu, EL > 1 && e >= 32 ? mine0[EL - 1] : mine0[0], e & 31);
    for (int p0 = 0; p0 < npair; p0 += 32) {
      const int p = p0 + lane;
      const bool mine = p < npair && s_idx[p] == e;
      const unsigned hit = __ballot_sync(0xffffffffu, mine);
      if (mine) {
        const int r = next + __popc(hit & ((1u << lane) - 1u));
        s_row[p] = r;
        row_of[p] = r;
        if (pair_of != nullptr) pair_of[r] = b * per * k + p;
      }
      next += __popc(hit);
    }
  }
  if (STRICT)
    for (int p = tid; p < npair; p += 32 * kWarps)
      if (s_idx[p] >= E) {
        s_row[p] = row_of[p] = -1;
        atomicMax(&status[0], MOE_B200_DEV_BAD_INDEX);
      }
  __syncthreads();

  // ---- row copies ----
  for (int tok = own; tok < N; tok += stride) {
    if (tok + stride < N) fetch(nxt, tok + stride);
    const uint4* row = reinterpret_cast<const uint4*>(xn) + (size_t)tok * pieces;
    for (int j = 0; j < k; ++j) {
      const int r = s_row[tok * k + j];
      if (r < 0) continue;
      uint4* to = reinterpret_cast<uint4*>(perm + (size_t)r * d);
#pragma unroll
      for (int u = 0; u < kInFlight; ++u)
        if (first_p + step * u < pieces) to[first_p + step * u] = cur[u];
    }
    for (int p0 = first_p + step * kInFlight; p0 < pieces; p0 += step * kInFlight) {
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) cur[u] = p0 + step * u < pieces ? __ldcg(row + p0 + step * u) : zero;
      for (int j = 0; j < k; ++j) {
        const int r = s_row[tok * k + j];
        if (r < 0) continue;
        uint4* to = reinterpret_cast<uint4*>(perm + (size_t)r * d);
#pragma unroll
        for (int u = 0; u < kInFlight; ++u)
          if (p0 + step * u < pieces) to[p0 + step * u] = cur[u];
      }
    }
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) cur[u] = nxt[u];
  }
  if (b == 0) {
    if (warp == kWarps - 1) {
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
    if (warp == kWarps - 2) {      // the loss (model.py:213-216)
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

template <int NT, bool NORM>
int launch(const void* x, const void* xn, const float* stats, const float* norm_c, const void* Wg, const void* bg, int N, int d,
           int E, int k, float* logits, int32_t* idx, float* w, int32_t* cnt_slot, int32_t* offsets, int32_t* row_of, void* perm,
           int32_t* pair_of, float* psum, float* aux, int32_t* xch, int32_t* status, int per, bool clear,
           cudaStream_t s) {
  constexpr size_t part = sizeof(float) * 2 * kWarps * kGroup * 8 * NT;
  static PerDeviceOnce once;
  int rc = ensure_dynamic_smem(once, front_many_kernel<NT, NORM>, part + 2 * sizeof(int) * kMaxPer * kMaxTopK);
  if (rc) return rc;
  const int blocks = (N + per - 1) / per;
  MOE_CUDA_CHECK(launch_pdl_as(front_many_kernel<NT, NORM>, dim3(blocks), dim3(32 * kWarps), 0, blocks > 1,
                               part + 2 * sizeof(int) * per * k, s, static_cast<const __nv_bfloat16*>(x),
                               static_cast<const __nv_bfloat16*>(xn), stats, norm_c,
                               static_cast<const __nv_bfloat16*>(Wg), static_cast<const __nv_bfloat16*>(bg), N, d, E, k, logits,
                               idx, w, cnt_slot, offsets, row_of, static_cast<__nv_bfloat16*>(perm), pair_of, psum, aux, xch,
                               status, per, per < kWarps ? kWarps / per : 1, clear));
  return 0;
}

}  // namespace

// Tokens of a block for a call that this kernel takes, 0 for any other: as many as give every SM one block, a few (a power of
// two) where that shortens the copies. A block reads the router's weights once per 16 tokens and has its groups one after the
// other, which the general kernels do not: the more experts, the fewer tokens. Whole calls, general kernels -> this
// one (medians of three, a memset in front of both, which this one has no more): 8 experts, d 1024, f 4096: 2100 tokens 143 -> 128 us, 4000 191 -> 178, 12000 551 -> 540,
// 18000 780 -> 776; d 512, f 2048: 4000 85.5 -> 70.0, 12000 173 -> 165, 18000 243 -> 235; 16 experts, d 1024, f 2048: 2200 108 ->
// 88, 8000 225 -> 207, 15360 380 -> 367; 32 experts, d 2048, f 1408: 2200 156 -> 139, 5000 240 -> 230, 9400 362 -> 365; 64 experts,
// four slots: 1100 244 -> 228, 2000 277 -> 267, 3500 324 -> 324, but 4096 378 -> 407. Training steps, 8 experts, d 512 with 2560
// tokens 325 -> 285; of a few hundred tokens they are as long on the host. With a folded LayerNorm, whose rows a launch of their own
// normalises: 2100 tokens 146 -> 133, 4000 201 -> 193, 9400 451 -> 448; in front of the products 12800 44 -> 43, 16384 45 -> 49.
int front_many_tokens(int64_t N, int d, int E, int k, int dtype, bool norm, int* per) {
  *per = 0;
  if (norm && E > 16) return 0;
  if (dtype != MOE_B200_BF16 || N < 1 || N > (int64_t)kMaxPer * kNumSMs || E > 64 || (E > 16 && d < 64) || k > kMaxTopK) return 0;
  int sms = 0;
  int rc = sm_count(&sms);
  if (rc) return rc;
  sms = sms < kNumSMs ? sms : kNumSMs;
  int64_t p = N <= 64 ? 4 : N <= 512 ? 8 : 16;
  if (p * sms < N) p = (N + sms - 1) / sms;
  if (p < kGroup && p != 4 && p != 8) p = kGroup;
  if (p <= (norm ? kMaxPer / 2 : E <= 16 ? kMaxPer : E <= 32 ? kMaxPer / 2 : 24)) *per = (int)p;
  return 0;
}

// norm_c, or nullptr: a folded LayerNorm, with `stats` and the normalised rows `xn` of layernorm_rows.
// xch: int32 scratch, (k + 1) * E words for each of kNumSMs blocks. clear: the status words and the counters behind them, none of
// which this kernel uses itself, are zeroed here first, whatever they held (a memset in front of the launch takes 2.0 to 2.6 us:
// 3000 tokens, d 256, f 64, 8 experts 32.3 us with it and 29.8 without).
int launch_front_many(const void* x, const void* xn, const float* stats, const float* norm_c, const void* Wg, const void* bg,
                      int64_t N, int d, int E, int k, float* logits, int32_t* idx, float* w, int32_t* cnt_slot,
                      int32_t* offsets, int32_t* row_of, void* perm, int32_t* pair_of, float* psum, float* aux, int32_t* xch,
                      int32_t* status, int per, bool clear, cudaStream_t s) {
  auto fn = norm_c != nullptr ? (E <= 8 ? launch<1, true> : launch<2, true>)
            : E <= 8 ? launch<1, false> : E <= 16 ? launch<2, false> : E <= 32 ? launch<4, false> : launch<8, false>;
  return fn(x, norm_c != nullptr ? xn : x, stats, norm_c, Wg, bg, (int)N, d, E, k, logits, idx, w, cnt_slot, offsets, row_of,
            perm, pair_of, psum, aux, xch, status, per, clear, s);
}

}  // namespace moe
