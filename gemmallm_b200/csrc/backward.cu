// Backward pass of the block (the reference trains through MOE.forward with torch.autograd:
// loss.backward() in train.py:140-141 reaches model.py:200-276 and 173-190). The two input
// gradients and the two weight gradients of the expert Linears are grouped products on the
// tcgen05 kernel of experts_tc2.cu, whose epilogue also takes dh back through dropout, product and
// GELU; this file holds what surrounds them, all HBM-bound:
//
//   combine_bwd      dy[r] = w[pair] * dOut[token], dw[pair] = dOut[token] . y[r]   (model.py:271)
//   router_bwd       dw -> d(renormalised scores) -> d(softmax) -> dlogits, plus the gradient
//                    of the load-balancing loss through the mean probabilities
//                    (model.py:207-223; the counts of model.py:213 carry no gradient), and in the
//                    same pass dWg = dlogits^T x, dbg = sum dlogits                 (model.py:206)
//   combine_dx       dx[t] = the sum of its rows' gradients + dlogits[t] Wg    (model.py:248-253, 206)
//   colsum           bias gradients per expert
// They start under programmatic dependent launch (each launch cost 1.5 to 2.9 us behind the kernel before it) and read
// what that kernel may have written through L2, behind pdl_wait.
#include "common.cuh"

namespace moe {

namespace {

__global__ void pair_of_kernel(const int32_t* row_of, int64_t M, int32_t* __restrict__ pair_of) {
  pdl_wait();
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < M) {
    const int r = __ldcg(&row_of[p]);
    if (r >= 0) pair_of[r] = (int32_t)p;
  }
}

// One warp per sorted row. Rows behind the last expert's (pairs whose router index was out of range, such as those of
// a token with NaN logits, have none) belong to no pair, and pair_of says nothing about them.
__global__ void __launch_bounds__(256)
combine_bwd_kernel(const __nv_bfloat16* dout, const __nv_bfloat16* y, const int32_t* pair_of, const int32_t* offsets,
                   int E, const float* w, int64_t M, int d, int k, __nv_bfloat16* __restrict__ dy,
                   float* __restrict__ dw) {
  const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  pdl_wait();
  if (r >= M || r >= __ldcg(&offsets[E])) return;
  const int p = __ldcg(&pair_of[r]);
  const int64_t t = p / k;
  const float wp = __ldcg(&w[p]);
  float dot = 0.f;
  for (int c = lane * 8; c < d; c += 256) {
    float g[8], yv[8], o[8];
    load8(dout + t * d + c, g);
    load8(y + r * d + c, yv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      dot = fmaf(g[i], yv[i], dot);
      o[i] = wp * g[i];
    }
    store8(dy + r * d + c, o);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if (lane == 0) dw[p] = dot;
}

// Gradient of a token's logits by G lanes; lane l of them holds experts l, l + G, ... (PER of them).
//   w_j = v_j / total, v_j = p[idx_j]:  dv_j = (dw_j - sum_i dw_i w_i) / total
//   aux = E * sum_e mean_n p[n,e] * cnt0_e / N:  dp[e] += grad_aux * E * cnt0_e / N^2
//   dl[e] = p[e] * (dp[e] - sum_e' p[e'] dp[e'])
template <int PER, int G>
__device__ __forceinline__ void token_dlogits(const float* __restrict__ logits, const int32_t* __restrict__ idx,
                                              const float* __restrict__ w, const float* dw,
                                              const int32_t* __restrict__ cnt0, float aux_c, int64_t t, int E, int k,
                                              int lane, float (&dl)[PER]) {
  static_assert(G == 32 || PER == 1, "experts of a token over part of a warp");
  float p[PER], dp[PER];
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + G * i;
    p[i] = e < E ? logits[t * E + e] : -INFINITY;
    m = fmaxf(m, p[i]);
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + G * i;
    p[i] = e < E ? expf(p[i] - m) : 0.f;
    sum += p[i];
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  // total of the chosen probabilities and sum_i dw_i w_i (every lane computes them: k <= 8)
  float total = 0.f, dww = 0.f;
  for (int j = 0; j < k; ++j) dww = fmaf(__ldcg(&dw[t * k + j]), w[t * k + j], dww);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + G * i;
    p[i] = p[i] / sum;
    dp[i] = e < E ? aux_c * (float)cnt0[e] : 0.f;
  }
  for (int j = 0; j < k; ++j) {
    // p[e] lives in lane e mod G, slice e / G
    const int e = idx[t * k + j];
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (i == e / G) v = p[i];
    total += __shfl_sync(0xffffffffu, v, e % G, G);
  }
  for (int j = 0; j < k; ++j) {
    const int e = idx[t * k + j];
    const float dv = (__ldcg(&dw[t * k + j]) - dww) / total;
    if (e % G == lane) {
#pragma unroll
      for (int i = 0; i < PER; ++i)
        if (i == e / G) dp[i] += dv;
    }
  }
  float pdp = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) pdp = fmaf(p[i], dp[i], pdp);
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) pdp += __shfl_xor_sync(0xffffffffu, pdp, o);
#pragma unroll
  for (int i = 0; i < PER; ++i) dl[i] = p[i] * (dp[i] - pdp);
}

constexpr int kDlTokens = 32;    // tokens of a step
constexpr int kDlExperts = 8;    // experts of a block's accumulators
constexpr int kDlCols = 1024;    // columns of a block, four per thread

// grid: (column blocks, token ranges, expert groups). Every block forms the logits' gradients of its tokens (the
// first column block and expert group store them) and the products of its eight experts with its columns of
// x; the partial sums of a token range go to part [range][E][d] and part_b [range][E] (no atomics: the same
// result every time). What bounds it is latency: a step's loads of x are under way while its logits' gradients are formed,
// and up to 16 experts a warp takes four or two tokens side by side (16384 tokens, d 1024, 8 experts: 40 -> 20 us,
// 1024 tokens 17 -> 8).
template <int PER, int G>
__global__ void __launch_bounds__(256)
router_bwd_kernel(const float* __restrict__ logits, const int32_t* __restrict__ idx,
                  const float* __restrict__ w, const float* dw,
                  const int32_t* __restrict__ cnt0, float grad_aux_host, const float* __restrict__ grad_aux_dev,
                  const __nv_bfloat16* __restrict__ x, int64_t N, int d, int E, int k, int tokens_per_block,
                  float* __restrict__ dl_out, float* __restrict__ part, float* __restrict__ part_b) {
  __shared__ float s_dl[kDlTokens][kDlExperts];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int e0 = blockIdx.z * kDlExperts;
  const int c = blockIdx.x * kDlCols + tid * 4;
  const int64_t t_begin = (int64_t)blockIdx.y * tokens_per_block;
  const int64_t t_end = min(t_begin + tokens_per_block, N);
  pdl_wait();
  const float grad_aux = grad_aux_dev != nullptr ? __ldg(grad_aux_dev) : grad_aux_host;
  const float aux_c = grad_aux * (float)E / ((float)N * (float)N);
  const bool store_dl = blockIdx.x == 0 && blockIdx.z == 0;
  float acc[kDlExperts][4];
#pragma unroll
  for (int i = 0; i < kDlExperts; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[i][q] = 0.f;
  float bsum = 0.f;
  for (int64_t t0 = t_begin; t0 < t_end; t0 += kDlTokens) {
    const int nt = (int)min((int64_t)kDlTokens, t_end - t0);
    const uint2* xp = reinterpret_cast<const uint2*>(x + t0 * d + c);
    const size_t pitch = (size_t)d >> 2;
    uint2 v[8];
    auto request = [&](int tb) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        v[u] = c < d && tb + u < nt ? __ldg(xp + (size_t)(tb + u) * pitch) : make_uint2(0, 0);
    };
    request(0);
    __syncthreads();
    for (int tb = warp * (32 / G); tb < nt; tb += 8 * (32 / G)) {      // (whole warps stay together)
      const int tl = tb + lane / G, l = lane % G;
      float dl[PER];
      token_dlogits<PER, G>(logits, idx, w, dw, cnt0, aux_c, t0 + min(tl, nt - 1), E, k, l, dl);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int e = l + G * i;
        if (tl < nt && e < E && store_dl) dl_out[(t0 + tl) * E + e] = dl[i];
        if (tl < nt && e >= e0 && e < e0 + kDlExperts) s_dl[tl][e - e0] = e < E ? dl[i] : 0.f;
      }
    }
    __syncthreads();
    if (blockIdx.x == 0 && tid < kDlExperts)
      for (int tl = 0; tl < nt; ++tl) bsum += s_dl[tl][tid];
    if (c < d) {
      for (int tb = 0; tb < nt; tb += 8) {
        uint2 now[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) now[u] = v[u];
        if (tb + 8 < nt) request(tb + 8);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (tb + u < nt) {
            const float xv[4] = {bf16_lo(now[u].x), bf16_hi(now[u].x), bf16_lo(now[u].y), bf16_hi(now[u].y)};
            const float4 ga = *reinterpret_cast<const float4*>(&s_dl[tb + u][0]);
            const float4 gb = *reinterpret_cast<const float4*>(&s_dl[tb + u][4]);
            const float g[kDlExperts] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
            for (int i = 0; i < kDlExperts; ++i)
#pragma unroll
              for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(g[i], xv[q], acc[i][q]);
          }
      }
    }
  }
  if (c < d) {
#pragma unroll
    for (int i = 0; i < kDlExperts; ++i)
      if (e0 + i < E)
        *reinterpret_cast<float4*>(part + ((size_t)blockIdx.y * E + e0 + i) * d + c) =
            make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  }
  if (blockIdx.x == 0 && tid < kDlExperts && e0 + tid < E) part_b[(size_t)blockIdx.y * E + e0 + tid] = bsum;
}

// out[i] = sum over `ranges` of part[r][i], in order; eight groups of 32 threads take every eighth.
__global__ void __launch_bounds__(256)
router_bwd_finish_kernel(const float* part, const float* part_b, int ranges, int64_t n,
                         int E, __nv_bfloat16* __restrict__ dWg, __nv_bfloat16* __restrict__ dbg) {
  __shared__ float s_sum[8][33];
  const int grp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool bias = blockIdx.x == gridDim.x - 1;
  pdl_wait();
  for (int64_t i0 = bias ? 0 : (int64_t)blockIdx.x * 32; i0 < (bias ? (int64_t)E : n); i0 += bias ? 32 : n) {
    const float* p = bias ? part_b : part;
    const int64_t len = bias ? (int64_t)E : n, i = i0 + lane;
    float sum = 0.f;
    if (i < len) {
#pragma unroll 4
      for (int r = grp; r < ranges; r += 8) sum += __ldcg(&p[(size_t)r * len + i]);
    }
    s_sum[grp][lane] = sum;
    __syncthreads();
    if (threadIdx.x < 32 && i < len) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q) t += s_sum[q][lane];
      __nv_bfloat16* out = bias ? dbg : dWg;
      if (out != nullptr) out[i] = __float2bfloat16_rn(t);
    }
    __syncthreads();
  }
}

// dx[t] = sum_j dxs[row_of[t, j]] + sum_e dl[t, e] Wg[e]; a thread takes eight columns of four tokens, so that a
// piece of Wg is used four times. Latency bounds it: with two slots (TWO) the rows of all four tokens are looked up,
// then all eight pieces requested, before anything is added (16384 tokens, d 1024: 15 us of the step less than with
// each row looked up and fetched in turn).
template <bool TWO>
__global__ void __launch_bounds__(256)
combine_dx_kernel(const __nv_bfloat16* __restrict__ dxs, const int32_t* __restrict__ row_of,
                  const float* __restrict__ dl, const __nv_bfloat16* __restrict__ Wg, int64_t N, int d, int E, int k,
                  __nv_bfloat16* __restrict__ dx) {
  constexpr int kTok = 4;
  const int pieces = d >> 3;
  const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t t0 = item / pieces * kTok;
  const int c = (int)(item % pieces) << 3;
  pdl_wait();
  if (t0 >= N) return;
  float acc[kTok][8];
  if constexpr (TWO) {
    int2 rows[kTok];
#pragma unroll
    for (int u = 0; u < kTok; ++u)
      rows[u] = t0 + u < N ? *reinterpret_cast<const int2*>(row_of + (t0 + u) * 2) : make_int2(-1, -1);
    uint4 v[kTok][2];
#pragma unroll
    for (int u = 0; u < kTok; ++u) {
      v[u][0] = rows[u].x >= 0 ? *reinterpret_cast<const uint4*>(dxs + (int64_t)rows[u].x * d + c) : make_uint4(0, 0, 0, 0);
      v[u][1] = rows[u].y >= 0 ? *reinterpret_cast<const uint4*>(dxs + (int64_t)rows[u].y * d + c) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < kTok; ++u) {
      const uint32_t a[4] = {v[u][0].x, v[u][0].y, v[u][0].z, v[u][0].w};
      const uint32_t b[4] = {v[u][1].x, v[u][1].y, v[u][1].z, v[u][1].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[u][2 * q] = bf16_lo(a[q]) + bf16_lo(b[q]);
        acc[u][2 * q + 1] = bf16_hi(a[q]) + bf16_hi(b[q]);
      }
    }
  } else {
#pragma unroll
    for (int u = 0; u < kTok; ++u) {
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[u][i] = 0.f;
      if (t0 + u < N)
        for (int j = 0; j < k; ++j) {
          const int row = row_of[(t0 + u) * k + j];
          if (row < 0) continue;
          float v[8];
          load8(dxs + (int64_t)row * d + c, v);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[u][i] += v[i];
        }
    }
  }
#pragma unroll 4
  for (int e = 0; e < E; ++e) {
    float wv[8];
    load8_ldg(Wg + (size_t)e * d + c, wv);
#pragma unroll
    for (int u = 0; u < kTok; ++u)
      if (t0 + u < N) {
        const float g = __ldg(&dl[(t0 + u) * E + e]);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[u][i] = fmaf(g, wv[i], acc[u][i]);
      }
  }
#pragma unroll
  for (int u = 0; u < kTok; ++u)
    if (t0 + u < N) store8(dx + (t0 + u) * d + c, acc[u]);
}

// Partial column sums: one block per 256-row tile of an expert (blockIdx.x, which alone counts beyond 65535: tiles over
// the experts in order, as the grouped products count them) and 64 columns (blockIdx.y); eight threads cover a row's 128 bytes,
// 32 such groups take every 32nd row, eight loads in flight each.
__global__ void __launch_bounds__(256)
colsum_kernel(const __nv_bfloat16* src, const int32_t* offsets, int E, int C,
              float* __restrict__ part) {
  __shared__ float s_part[32][65];
  __shared__ int s_row0, s_row1;
  pdl_wait();
  if (threadIdx.x == 0) {
    int tile = blockIdx.x, r0 = 0, r1 = 0;
    for (int e = 0; e < E; ++e) {
      const int beg = offsets[e], end = offsets[e + 1], tiles = (end - beg + 255) / 256;
      if (tile < tiles) {
        r0 = beg + tile * 256;
        r1 = min(end, r0 + 256);
        break;
      }
      tile -= tiles;
    }
    s_row0 = r0;
    s_row1 = r1;
  }
  __syncthreads();
  const int r0 = s_row0, r1 = s_row1;
  if (r0 == r1) return;      // behind the last tile
  const int pc = threadIdx.x & 7, lane_r = threadIdx.x >> 3;
  const int c = blockIdx.y * 64 + pc * 8;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if (c < C) {
    uint4 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = r0 + lane_r + 32 * q;
      v[q] = r < r1 ? __ldcg(reinterpret_cast<const uint4*>(src + (size_t)r * C + c)) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t w[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[2 * i] += bf16_lo(w[i]);
        acc[2 * i + 1] += bf16_hi(w[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) s_part[lane_r][pc * 8 + i] = acc[i];
  __syncthreads();
  if (threadIdx.x < 64) {
    const int col = blockIdx.y * 64 + threadIdx.x;
    if (col < C) {
      float sum = 0.f;
#pragma unroll
      for (int q = 0; q < 32; ++q) sum += s_part[q][threadIdx.x];
      part[(size_t)blockIdx.x * C + col] = sum;
    }
  }
}

// db[e][c] = sum of the expert's slots of part (`slots` per 256-row tile), in order: eight groups of
// 32 threads take every eighth slot.
__global__ void __launch_bounds__(256)
colsum_finish_kernel(const float* part, int slots, const int32_t* offsets, int C,
                     __nv_bfloat16* __restrict__ db) {
  __shared__ float s_sum[8][33];
  __shared__ int s_first, s_count;
  const int e = blockIdx.y;
  pdl_wait();
  if (threadIdx.x == 0) {
    int first = 0;
    for (int i = 0; i < e; ++i) first += (offsets[i + 1] - offsets[i] + 255) / 256;
    s_first = first * slots;
    s_count = (offsets[e + 1] - offsets[e] + 255) / 256 * slots;
  }
  __syncthreads();
  const int col = blockIdx.x * 32 + (threadIdx.x & 31), grp = threadIdx.x >> 5;
  float sum = 0.f;
  if (col < C) {
    const float* p = part + (size_t)s_first * C + col;
#pragma unroll 4
    for (int i = grp; i < s_count; i += 8) sum += __ldcg(&p[(size_t)i * C]);
  }
  s_sum[grp][threadIdx.x & 31] = sum;
  __syncthreads();
  if (threadIdx.x < 32 && col < C) {
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += s_sum[q][threadIdx.x];
    db[(size_t)e * C + col] = __float2bfloat16_rn(t);
  }
}

unsigned blocks_for(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }

}  // namespace

int launch_pair_of(const int32_t* row_of, int64_t M, int32_t* pair_of, cudaStream_t s) {
  if (M == 0) return 0;
  MOE_CUDA_CHECK(launch_pdl(pair_of_kernel, dim3(blocks_for(M, 256)), dim3(256), 0, s, row_of, M, pair_of));
  return 0;
}

int launch_combine_bwd(const void* dout, const void* y, const int32_t* pair_of, const int32_t* offsets, int E,
                       const float* w, int64_t M, int d, int k, void* dy, float* dw, cudaStream_t s) {
  if (M == 0) return 0;
  MOE_CUDA_CHECK(launch_pdl(combine_bwd_kernel, dim3(blocks_for(M, 8)), dim3(256), 0, s,
                            static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(y), pair_of,
                            offsets, E, w, M, d, k, static_cast<__nv_bfloat16*>(dy), dw));
  return 0;
}

// Token ranges of router_bwd_kernel: about two blocks per SM, their partial sums at most 16 MB.
static int64_t router_bwd_tokens(int64_t N, int d, int E) {
  const int64_t groups = (int64_t)((d + kDlCols - 1) / kDlCols) * ((E + kDlExperts - 1) / kDlExperts);
  int64_t ranges = (2 * kNumSMs + groups - 1) / groups;
  const int64_t most = ((int64_t)16 << 20) / ((int64_t)E * d * 4);
  if (ranges > most) ranges = most;
  if (ranges < 1) ranges = 1;
  const int64_t per = (N + ranges - 1) / ranges;
  return (per + kDlTokens - 1) / kDlTokens * kDlTokens;
}

int64_t router_bwd_scratch_floats(int64_t N, int d, int E) {
  const int64_t per = router_bwd_tokens(N > 0 ? N : 1, d, E);
  return (N + per - 1) / per * ((int64_t)E * d + E);
}

int launch_router_bwd(const float* logits, const int32_t* idx, const float* w, const float* dw,
                      const int32_t* cnt0, float grad_aux, const float* grad_aux_dev, const void* x,
                      int64_t N, int d, int E, int k, float* dl, float* scratch, void* dWg, void* dbg, cudaStream_t s) {
  if (N == 0) return 0;
  const int64_t per = router_bwd_tokens(N, d, E);
  const int64_t ranges = (N + per - 1) / per;
  float* part_b = scratch + (size_t)ranges * E * d;
  auto fn = E <= 8 ? router_bwd_kernel<1, 8>
                   : (E <= 16 ? router_bwd_kernel<1, 16>
                              : (E <= 32 ? router_bwd_kernel<1, 32>
                                         : (E <= 64 ? router_bwd_kernel<2, 32> : router_bwd_kernel<kMaxExperts / 32, 32>)));
  const dim3 grid((d + kDlCols - 1) / kDlCols, (unsigned)ranges, (E + kDlExperts - 1) / kDlExperts);
  MOE_CUDA_CHECK(launch_pdl(fn, grid, dim3(256), 0, s, logits, idx, w, dw, cnt0, grad_aux, grad_aux_dev,
                            static_cast<const __nv_bfloat16*>(x), N, d, E, k, (int)per, dl, scratch, part_b));
  if (dWg == nullptr && dbg == nullptr) return 0;
  const int64_t n = (int64_t)E * d;
  MOE_CUDA_CHECK(launch_pdl(router_bwd_finish_kernel, dim3(blocks_for(n, 32) + 1), dim3(256), 0, s, scratch, part_b,
                            (int)ranges, n, E, static_cast<__nv_bfloat16*>(dWg), static_cast<__nv_bfloat16*>(dbg)));
  return 0;
}

int launch_combine_dx(const void* dxs, const int32_t* row_of, const float* dl, const void* Wg, int64_t N, int d, int E,
                      int k, void* dx, cudaStream_t s) {
  if (N == 0) return 0;
  const int64_t items = (N + 3) / 4 * (d >> 3);
  MOE_CUDA_CHECK(launch_pdl(k == 2 ? combine_dx_kernel<true> : combine_dx_kernel<false>, dim3(blocks_for(items, 256)), dim3(256), 0, s,
                            static_cast<const __nv_bfloat16*>(dxs), row_of, dl, static_cast<const __nv_bfloat16*>(Wg),
                            N, d, E, k, static_cast<__nv_bfloat16*>(dx)));
  return 0;
}

int launch_colsum_finish(const float* part, int slots, const int32_t* offsets, int E, int C, void* db,
                         cudaStream_t s) {
  MOE_CUDA_CHECK(launch_pdl(colsum_finish_kernel, dim3((C + 31) / 32, E), dim3(256), 0, s, part, slots, offsets, C,
                            static_cast<__nv_bfloat16*>(db)));
  return 0;
}

int launch_colsum(const void* src, const int32_t* offsets, int64_t M, int E, int C, float* part, void* db,
                  cudaStream_t s) {
  const unsigned tiles = blocks_for(M, 256) + (unsigned)E;    // at least as many as there are
  MOE_CUDA_CHECK(launch_pdl(colsum_kernel, dim3(tiles, (C + 63) / 64), dim3(256), 0, s,
                            static_cast<const __nv_bfloat16*>(src), offsets, E, C, part));
  return launch_colsum_finish(part, 1, offsets, E, C, db, s);
}

}  // namespace moe
