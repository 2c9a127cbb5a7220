// Backward pass of the block (the reference trains through MOE.forward with torch.autograd:
// loss.backward() in train.py:140-141 reaches model.py:200-276 and 173-190). The two input
// gradients and the two weight gradients of the expert Linears are grouped products on the
// tcgen05 kernel of experts_tc2.cu, whose epilogue also takes dh back through dropout, product and
// GELU; this file holds what surrounds them, all HBM-bound:
//
//   combine_bwd      dy[r] = w[pair] * dOut[token], dw[pair] = dOut[token] . y[r]   (model.py:271)
//   router_bwd       dw -> d(renormalised scores) -> d(softmax) -> dlogits, plus the gradient
//                    of the load-balancing loss through the mean probabilities
//                    (model.py:207-223; the counts of model.py:213 carry no gradient)
//   router_bwd_wx    dWg = dlogits^T x, dbg = sum dlogits, dx += dlogits Wg       (model.py:206)
//   colsum           bias gradients per expert
#include "common.cuh"

namespace moe {

namespace {

__global__ void pair_of_kernel(const int32_t* __restrict__ row_of, int64_t M, int32_t* __restrict__ pair_of) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < M) {
    const int r = row_of[p];
    if (r >= 0) pair_of[r] = (int32_t)p;
  }
}

// One warp per sorted row.
__global__ void __launch_bounds__(256)
combine_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ y,
                   const int32_t* __restrict__ pair_of, const float* __restrict__ w, int64_t M, int d,
                   int k, __nv_bfloat16* __restrict__ dy, float* __restrict__ dw) {
  const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= M) return;
  const int p = pair_of[r];
  const int64_t t = p / k;
  const float wp = w[p];
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

// One warp per token; lane e handles experts e, e+32, ...
//   w_j = v_j / total, v_j = p[idx_j]:  dv_j = (dw_j - sum_i dw_i w_i) / total
//   aux = E * sum_e mean_n p[n,e] * cnt0_e / N:  dp[e] += grad_aux * E * cnt0_e / N^2
//   dl[e] = p[e] * (dp[e] - sum_e' p[e'] dp[e'])
__global__ void __launch_bounds__(256)
router_bwd_kernel(const float* __restrict__ logits, const int32_t* __restrict__ idx,
                  const float* __restrict__ w, const float* __restrict__ dw,
                  const int32_t* __restrict__ cnt0, float grad_aux_host, const float* __restrict__ grad_aux_dev,
                  int64_t N, int E, int k, float* __restrict__ dl) {
  const int64_t t = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= N) return;
  constexpr int kPer = kMaxExperts / 32;
  float l[kPer], p[kPer], dp[kPer];
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = lane + 32 * i;
    l[i] = e < E ? logits[t * E + e] : -INFINITY;
    m = fmaxf(m, l[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = lane + 32 * i;
    p[i] = e < E ? expf(l[i] - m) : 0.f;
    sum += p[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  // total of the chosen probabilities and sum_i dw_i w_i (every lane computes them: k <= 8)
  float total = 0.f, dww = 0.f;
  for (int j = 0; j < k; ++j) dww = fmaf(dw[t * k + j], w[t * k + j], dww);
  const float grad_aux = grad_aux_dev != nullptr ? __ldg(grad_aux_dev) : grad_aux_host;
  const float aux_c = grad_aux * (float)E / ((float)N * (float)N);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = lane + 32 * i;
    p[i] = p[i] / sum;
    dp[i] = e < E ? aux_c * (float)cnt0[e] : 0.f;
  }
  for (int j = 0; j < k; ++j) {
    // p[e] lives in lane e & 31, slice e >> 5
    const int e = idx[t * k + j];
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (i == (e >> 5)) v = p[i];
    total += __shfl_sync(0xffffffffu, v, e & 31);
  }
  for (int j = 0; j < k; ++j) {
    const int e = idx[t * k + j];
    const float dv = (dw[t * k + j] - dww) / total;
    if ((e & 31) == lane) {
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        if (i == (e >> 5)) dp[i] += dv;
    }
  }
  float pdp = 0.f;
#pragma unroll
  for (int i = 0; i < kPer; ++i) pdp = fmaf(p[i], dp[i], pdp);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) pdp += __shfl_xor_sync(0xffffffffu, pdp, o);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = lane + 32 * i;
    if (e < E) dl[t * E + e] = p[i] * (dp[i] - pdp);
  }
}

// dWg[e][c] += sum_t dl[t][e] x[t][c] (fp32 atomics into a zeroed buffer), dbg[e] += sum_t dl[t][e],
// dxr[t][c] = sum_e dl[t][e] Wg[e][c]. A block owns 256 columns and a range of tokens; experts in
// groups of 32 (E > 32 re-reads the token range from L2).
__global__ void __launch_bounds__(256)
router_bwd_wx_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ Wg,
                     const float* __restrict__ dl, int64_t N, int d, int E, int tokens_per_block,
                     float* __restrict__ dWg, float* __restrict__ dbg,
                     __nv_bfloat16* __restrict__ dxr) {
  __shared__ float s_dl[64][33];
  const int c = blockIdx.x * 256 + threadIdx.x;
  const int64_t t_begin = (int64_t)blockIdx.y * tokens_per_block;
  const int64_t t_end = t_begin + tokens_per_block < N ? t_begin + tokens_per_block : N;
  const bool col_ok = c < d;
  for (int e0 = 0; e0 < E; e0 += 32) {
    const int ne = E - e0 < 32 ? E - e0 : 32;
    float acc[32], wg[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      acc[i] = 0.f;
      wg[i] = (col_ok && i < ne) ? __bfloat162float(Wg[(size_t)(e0 + i) * d + c]) : 0.f;
    }
    float bsum = 0.f;   // thread i < ne of column block 0 sums dl[:, e0 + i]
    for (int64_t t0 = t_begin; t0 < t_end; t0 += 64) {
      const int nt = (int)(t_end - t0 < 64 ? t_end - t0 : 64);
      __syncthreads();
      for (int i = threadIdx.x; i < 64 * 32; i += 256) {
        const int tl = i >> 5, el = i & 31;
        s_dl[tl][el] = (tl < nt && el < ne) ? dl[(t0 + tl) * E + e0 + el] : 0.f;
      }
      __syncthreads();
      if (blockIdx.x == 0 && (int)threadIdx.x < ne)
        for (int tl = 0; tl < nt; ++tl) bsum += s_dl[tl][threadIdx.x];
      if (col_ok) {
        for (int tl = 0; tl < nt; ++tl) {
          const float xv = __bfloat162float(x[(t0 + tl) * d + c]);
          float dx = 0.f;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float g = s_dl[tl][i];
            acc[i] = fmaf(g, xv, acc[i]);
            dx = fmaf(g, wg[i], dx);
          }
          // more than 32 experts: the sum over expert groups passes through the bf16 buffer
          // (one extra rounding per group of 32 experts)
          float prev = e0 == 0 ? 0.f : __bfloat162float(dxr[(t0 + tl) * d + c]);
          dxr[(t0 + tl) * d + c] = __float2bfloat16_rn(prev + dx);
        }
      }
    }
    if (col_ok)
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i < ne) atomicAdd(&dWg[(size_t)(e0 + i) * d + c], acc[i]);
    if (blockIdx.x == 0 && (int)threadIdx.x < ne) atomicAdd(&dbg[e0 + threadIdx.x], bsum);
  }
}

__global__ void iota_kernel(int32_t* __restrict__ p, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = (int32_t)i;
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ src, int64_t n, __nv_bfloat16* __restrict__ dst) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = __float2bfloat16_rn(src[i]);
}

__global__ void fill_f32_kernel(float* __restrict__ p, int64_t n, float v) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

// Partial column sums: one block per 256-row tile of an expert (tiles counted over the experts in
// order, as the grouped products count them) and 64 columns; eight threads cover a row's 128 bytes,
// 32 such groups take every 32nd row, eight loads in flight each.
__global__ void __launch_bounds__(256)
colsum_kernel(const __nv_bfloat16* __restrict__ src, const int32_t* __restrict__ offsets, int E, int C,
              float* __restrict__ part) {
  __shared__ float s_part[32][65];
  __shared__ int s_row0, s_row1;
  if (threadIdx.x == 0) {
    int tile = blockIdx.y, r0 = 0, r1 = 0;
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
  const int c = blockIdx.x * 64 + pc * 8;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if (c < C) {
    uint4 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = r0 + lane_r + 32 * q;
      v[q] = r < r1 ? __ldg(reinterpret_cast<const uint4*>(src + (size_t)r * C + c)) : make_uint4(0, 0, 0, 0);
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
    const int col = blockIdx.x * 64 + threadIdx.x;
    if (col < C) {
      float sum = 0.f;
#pragma unroll
      for (int q = 0; q < 32; ++q) sum += s_part[q][threadIdx.x];
      part[(size_t)blockIdx.y * C + col] = sum;
    }
  }
}

// db[e][c] = sum of the expert's slots of part (`slots` per 256-row tile), in order: eight groups of
// 32 threads take every eighth slot.
__global__ void __launch_bounds__(256)
colsum_finish_kernel(const float* __restrict__ part, int slots, const int32_t* __restrict__ offsets, int C,
                     __nv_bfloat16* __restrict__ db) {
  __shared__ float s_sum[8][33];
  __shared__ int s_first, s_count;
  const int e = blockIdx.y;
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
    for (int i = grp; i < s_count; i += 8) sum += p[(size_t)i * C];
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
  pair_of_kernel<<<blocks_for(M, 256), 256, 0, s>>>(row_of, M, pair_of);
  MOE_CUDA_CHECK(cudaGetLastError());
  return 0;
}

int launch_combine_bwd(const void* dout, const void* y, const int32_t* pair_of, const float* w,
                       int64_t M, int d, int k, void* dy, float* dw, cudaStream_t s) {
  if (M == 0) return 0;
  combine_bwd_kernel<<<blocks_for(M, 8), 256, 0, s>>>(
      static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(y), pair_of, w, M, d,
      k, static_cast<__nv_bfloat16*>(dy), dw);
  MOE_CUDA_CHECK(cudaGetLastError());
  return 0;
}

int launch_router_bwd(const float* logits, const int32_t* idx, const float* w, const float* dw,
                      const int32_t* cnt0, float grad_aux, const float* grad_aux_dev, const void* x, const void* Wg,
                      int64_t N, int d, int E, int k, float* dl, float* dWg_f32, float* dbg_f32, void* dWg,
                      void* dbg, void* dxr, cudaStream_t s) {
  if (N == 0) return 0;
  router_bwd_kernel<<<blocks_for(N, 8), 256, 0, s>>>(logits, idx, w, dw, cnt0, grad_aux, grad_aux_dev, N, E, k, dl);
  MOE_CUDA_CHECK(cudaGetLastError());
  MOE_CUDA_CHECK(cudaMemsetAsync(dWg_f32, 0, sizeof(float) * (size_t)E * d, s));
  MOE_CUDA_CHECK(cudaMemsetAsync(dbg_f32, 0, sizeof(float) * (size_t)E, s));
  // about two token ranges per SM column block
  int sms = 0;
  int rc = sm_count(&sms);
  if (rc) return rc;
  const int col_blocks = (d + 255) / 256;
  int64_t ranges = (2 * (int64_t)sms + col_blocks - 1) / col_blocks;
  int64_t per = (N + ranges - 1) / ranges;
  per = (per + 63) / 64 * 64;
  ranges = (N + per - 1) / per;
  router_bwd_wx_kernel<<<dim3(col_blocks, (unsigned)ranges), 256, 0, s>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(Wg), dl, N, d, E,
      (int)per, dWg_f32, dbg_f32, static_cast<__nv_bfloat16*>(dxr));
  MOE_CUDA_CHECK(cudaGetLastError());
  if (dWg != nullptr)
    f32_to_bf16_kernel<<<blocks_for((int64_t)E * d, 256), 256, 0, s>>>(dWg_f32, (int64_t)E * d,
                                                                       static_cast<__nv_bfloat16*>(dWg));
  if (dbg != nullptr)
    f32_to_bf16_kernel<<<blocks_for(E, 256), 256, 0, s>>>(dbg_f32, E, static_cast<__nv_bfloat16*>(dbg));
  MOE_CUDA_CHECK(cudaGetLastError());
  return 0;
}

int launch_iota(int32_t* p, int64_t n, cudaStream_t s) {
  if (n == 0) return 0;
  iota_kernel<<<blocks_for(n, 256), 256, 0, s>>>(p, n);
  MOE_CUDA_CHECK(cudaGetLastError());
  return 0;
}

int launch_fill_f32(float* p, int64_t n, float v, cudaStream_t s) {
  if (n == 0) return 0;
  fill_f32_kernel<<<blocks_for(n, 256), 256, 0, s>>>(p, n, v);
  MOE_CUDA_CHECK(cudaGetLastError());
  return 0;
}

int launch_colsum_finish(const float* part, int slots, const int32_t* offsets, int E, int C, void* db,
                         cudaStream_t s) {
  colsum_finish_kernel<<<dim3((C + 31) / 32, E), 256, 0, s>>>(part, slots, offsets, C,
                                                             static_cast<__nv_bfloat16*>(db));
  MOE_CUDA_CHECK(cudaGetLastError());
  return 0;
}

int launch_colsum(const void* src, const int32_t* offsets, int64_t M, int E, int C, float* part, void* db,
                  cudaStream_t s) {
  const unsigned tiles = blocks_for(M, 256) + (unsigned)E;    // at least as many as there are
  colsum_kernel<<<dim3((C + 63) / 64, tiles), 256, 0, s>>>(static_cast<const __nv_bfloat16*>(src), offsets, E, C,
                                                            part);
  MOE_CUDA_CHECK(cudaGetLastError());
  return launch_colsum_finish(part, 1, offsets, E, C, db, s);
}

}  // namespace moe
