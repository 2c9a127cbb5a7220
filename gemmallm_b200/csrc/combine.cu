// Combine kernel: weighted un-permute of the expert outputs back to token
// order, fused with the caller's residual add.
//   out[t] = sum_j w[t,j] * y[row_of[t,j]]  (+ residual[t])
// in fp32, slots in order, rounded once. Replaces the two zero-filled fp32
// scatter buffers, the index_copy_ calls and the weighted sum of reference
// model.py:264-271, and the `tensor += skip_connection` of model.py:319.
//
// HBM-bound gather (no atomics, deterministic): each thread produces eight
// consecutive output elements from k 16-byte (bf16) or 32-byte (fp32) loads, which for one, two and four slots are all under
// way together with the skip connection's (one slot after the other, behind a division of 64 bits: 65536 tokens, d 2048, four
// slots, nothing in L2, 291 us, now 244 = 6.6 TB/s; 16384, d 1024, two 34.8 and 29.7).
#include "common.cuh"
#include "ep_sync.cuh"

namespace moe {

namespace {

// Eight elements as they lie in memory.
template <typename T>
struct Eight {
  uint4 raw[sizeof(T) / 2];
  __device__ __forceinline__ void load(const T* p) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(T) / 2; ++i) raw[i] = __ldcg(reinterpret_cast<const uint4*>(p) + i);
  }
  __device__ __forceinline__ void get(float (&v)[8]) const {
    if constexpr (sizeof(T) == 2) {
      v[0] = bf16_lo(raw[0].x); v[1] = bf16_hi(raw[0].x);
      v[2] = bf16_lo(raw[0].y); v[3] = bf16_hi(raw[0].y);
      v[4] = bf16_lo(raw[0].z); v[5] = bf16_hi(raw[0].z);
      v[6] = bf16_lo(raw[0].w); v[7] = bf16_hi(raw[0].w);
    } else {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        v[4 * i] = __uint_as_float(raw[i].x); v[4 * i + 1] = __uint_as_float(raw[i].y);
        v[4 * i + 2] = __uint_as_float(raw[i].z); v[4 * i + 3] = __uint_as_float(raw[i].w);
      }
    }
  }
};

// K: the number of slots, 0 for any other (the workloads have one, two or four; unrolled, three slots of 32768 tokens, d 1024,
// would take 47 us and not 54, six of 16384, d 2048, 85 and not 92, eight 113 as they do). FEW: N * pieces < 2^31.
// (y comes from the kernel in front, which may still run where this one starts, row_of and w perhaps as well: no loads of
// constant data, so no __restrict__)
template <typename T, int K, bool FEW>
__global__ void __launch_bounds__(256)
combine_kernel(const T* y, const int32_t* row_of, const float* w, const T* residual, int64_t N, int d,
               int k, T* __restrict__ out, const EpSync sy, int32_t* __restrict__ status) {
  const int pieces = d >> 3;
  const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t t = FEW ? (int64_t)((unsigned)item / (unsigned)pieces) : item / pieces;
  const int c = (int)(item - t * pieces) << 3;
  pdl_wait();
  // expert-parallel: y is the return buffer the expert owners store into; wait for all of them
  if (!epsync::block_wait(sy, status, 25)) return;
  if (item >= N * pieces) return;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  Eight<T> res;
  if (residual != nullptr) res.load(residual + t * d + c);
  // row_of == nullptr: y is already in (token, slot) order (expert-parallel return buffer)
  // mul then add, not fma: the reference forms w0*a + w1*b from rounded products
  if constexpr (K > 0) {
    int row[K];
    float wj[K];
    Eight<T> yj[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      row[j] = row_of != nullptr ? row_of[t * K + j] : (int)(t * K + j);
      wj[j] = w[t * K + j];
    }
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (row[j] >= 0) yj[j].load(y + (int64_t)row[j] * d + c);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (row[j] < 0) continue;
      float v[8];
      yj[j].get(v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = __fadd_rn(acc[i], __fmul_rn(wj[j], v[i]));
    }
  } else {
    for (int j = 0; j < k; ++j) {
      const int row = row_of != nullptr ? row_of[t * k + j] : (int)(t * k + j);
      if (row < 0) continue;
      const float wj = w[t * k + j];
      Eight<T> yj;
      yj.load(y + (int64_t)row * d + c);
      float v[8];
      yj.get(v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = __fadd_rn(acc[i], __fmul_rn(wj, v[i]));
    }
  }
  if (residual != nullptr) {
    float r[8];
    res.get(r);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = __fadd_rn(acc[i], r[i]);
  }
  store8(out + t * d + c, acc);
}

template <typename T>
auto combine_kernel_of(int k, bool few) {
  if (!few) return combine_kernel<T, 0, false>;
  return k == 1 ? combine_kernel<T, 1, true> : k == 2 ? combine_kernel<T, 2, true>
         : k == 4 ? combine_kernel<T, 4, true> : combine_kernel<T, 0, true>;
}

// Small-N variant: the down product arrives as `ksplit` fp32 partial buffers
// part[s][M][d] without bias; sum them in order s = 0..ksplit-1, add the
// expert's down.bias, then weight and add as above.
// TWO: the call has two slots per token (the reference's k): the routing of both and all the
// partial sums of both are requested before anything is added, so that the kernel is two
// round trips to L2 long instead of one per slot and kind of load.
template <bool TWO>
__global__ void __launch_bounds__(64)
combine_decode_kernel(const float* __restrict__ part, int ksplit, int64_t part_stride,
                      const int32_t* __restrict__ row_of, const int32_t* __restrict__ idx,
                      const float* __restrict__ w, const void* const* __restrict__ b2,
                      const __nv_bfloat16* __restrict__ residual, int64_t N, int d, int k,
                      __nv_bfloat16* __restrict__ out) {
  const int pieces = d >> 3;
  const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();   // the next kernel may become resident; it waits before it reads
  pdl_wait();
  if (item >= N * pieces) return;
  const int64_t t = item / pieces;
  const int c = (int)(item - t * pieces) << 3;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if constexpr (TWO) {
    // (routing through L2 after the wait, as below)
    int row[2], e[2];
    float wj[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      row[j] = __ldcg(&row_of[t * 2 + j]);
      e[j] = __ldcg(&idx[t * 2 + j]);
      wj[j] = __ldcg(&w[t * 2 + j]);
    }
    float r[8];
    if (residual != nullptr) load8(residual + t * d + c, r);
    float v[2][8], pv[2][8][8];
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (row[j] >= 0) {
        load8_ldg(static_cast<const __nv_bfloat16*>(b2[e[j]]) + c, v[j]);
#pragma unroll
        for (int sp = 0; sp < 8; ++sp)
          if (sp < ksplit) load8(part + (int64_t)sp * part_stride + (int64_t)row[j] * d + c, pv[j][sp]);
      }
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (row[j] >= 0) {
        float s2[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) s2[i] = 0.f;
#pragma unroll
        for (int sp = 0; sp < 8; ++sp)
          if (sp < ksplit) {
#pragma unroll
            for (int i = 0; i < 8; ++i) s2[i] += pv[j][sp][i];
          }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float yv = __bfloat162float(__float2bfloat16_rn(s2[i] + v[j][i]));
          acc[i] = __fadd_rn(acc[i], __fmul_rn(wj[j], yv));
        }
      }
    if (residual != nullptr) {
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = __fadd_rn(acc[i], r[i]);
    }
    store8(out + t * d + c, acc);
    return;
  }
  for (int j = 0; j < k; ++j) {
    // row_of, idx and w come from the routing kernel, which may still be running when this
    // kernel becomes resident: read them through L2 after the wait, never through the read-only
    // path (whose loads the compiler may move above the wait)
    const int row = __ldcg(&row_of[t * k + j]);
    if (row < 0) continue;
    const int e = __ldcg(&idx[t * k + j]);
    const float wj = __ldcg(&w[t * k + j]);
    float v[8];
    load8_ldg(static_cast<const __nv_bfloat16*>(b2[e]) + c, v);
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = 0.f;
    // all partial loads in flight at once; summed in order sp = 0, 1, ...
    float pv[8][8];
#pragma unroll
    for (int sp = 0; sp < 8; ++sp)
      if (sp < ksplit) load8(part + (int64_t)sp * part_stride + (int64_t)row * d + c, pv[sp]);
#pragma unroll
    for (int sp = 0; sp < 8; ++sp)
      if (sp < ksplit) {
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += pv[sp][i];
      }
    // the expert's output is rounded to bf16 before weighting, as on the large-N path
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float yv = __bfloat162float(__float2bfloat16_rn(s[i] + v[i]));
      acc[i] = __fadd_rn(acc[i], __fmul_rn(wj, yv));
    }
  }
  if (residual != nullptr) {
    float r[8];
    load8(residual + t * d + c, r);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = __fadd_rn(acc[i], r[i]);
  }
  store8(out + t * d + c, acc);
}

// fp32: the down product as `splits` partial sums part[s][M][d] without bias, added in order, with the expert's down.bias,
// then weighted as above. A thread: four elements of a token. 512 tokens, d 512, four parts, two slots: 8 MB that lie in L2.
__global__ void __launch_bounds__(128)
combine_parts_f32_kernel(const float* __restrict__ part, int splits, int64_t part_stride, const int32_t* __restrict__ row_of,
                         const int32_t* __restrict__ idx, const float* __restrict__ w, const void* const* __restrict__ b2,
                         const float* __restrict__ residual, int64_t N, int d, int k, float* __restrict__ out) {
  const int pieces = d >> 2;
  const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  pdl_wait();
  if (item >= N * pieces) return;
  const int64_t t = item / pieces;
  const int c = (int)(item - t * pieces) << 2;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int j = 0; j < k; ++j) {
    const int row = __ldcg(&row_of[t * k + j]);
    if (row < 0) continue;
    const float wj = __ldcg(&w[t * k + j]);
    const float* b = static_cast<const float*>(b2[__ldcg(&idx[t * k + j])]) + c;    // (of any alignment)
    const float bias[4] = {__ldg(b), __ldg(b + 1), __ldg(b + 2), __ldg(b + 3)};
    const float* p = part + (int64_t)row * d + c;
    float4 u[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (q < splits) u[q] = __ldcg(reinterpret_cast<const float4*>(p + q * part_stride));
    float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (q < splits) { y[0] += u[q].x; y[1] += u[q].y; y[2] += u[q].z; y[3] += u[q].w; }
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = __fadd_rn(acc[i], __fmul_rn(wj, y[i] + bias[i]));
  }
  if (residual != nullptr) {
    const float4 r = *reinterpret_cast<const float4*>(residual + t * d + c);
    acc[0] = __fadd_rn(acc[0], r.x); acc[1] = __fadd_rn(acc[1], r.y);
    acc[2] = __fadd_rn(acc[2], r.z); acc[3] = __fadd_rn(acc[3], r.w);
  }
  *reinterpret_cast<float4*>(out + t * d + c) = make_float4(acc[0], acc[1], acc[2], acc[3]);
}

}  // namespace

int launch_combine_parts_f32(const float* part, int splits, int64_t M, const int32_t* row_of, const int32_t* idx,
                             const float* w, const void* plan, int E, const void* residual, int64_t N, int d, int k,
                             void* out, cudaStream_t s) {
  if (N == 0) return 0;
  const int64_t blocks = (N * (d >> 2) + 127) / 128;
  MOE_CUDA_CHECK(launch_pdl(combine_parts_f32_kernel, dim3((unsigned)blocks), dim3(128), 0, s, part, splits, M * (int64_t)d,
                            row_of, idx, w, plan_view(plan, E).b2, static_cast<const float*>(residual), N, d, k,
                            static_cast<float*>(out)));
  return 0;
}

int launch_combine_decode(const float* part, int ksplit, int64_t M, const int32_t* row_of,
                          const int32_t* idx, const float* w, const void* plan, int E,
                          const void* residual, int64_t N, int d, int k, void* out, cudaStream_t s) {
  if (N == 0) return 0;
  PlanView pv = plan_view(plan, E);
  const int64_t items = N * (d >> 3);
  const int64_t blocks = (items + 63) / 64;   // small blocks: spread few items over many SMs
  if (k == 2)
    MOE_CUDA_CHECK(launch_pdl(combine_decode_kernel<true>, dim3((unsigned)blocks), dim3(64), 0, s, part, ksplit,
                              M * (int64_t)d, row_of, idx, w, pv.b2,
                              static_cast<const __nv_bfloat16*>(residual), N, d, k,
                              static_cast<__nv_bfloat16*>(out)));
  else
    MOE_CUDA_CHECK(launch_pdl(combine_decode_kernel<false>, dim3((unsigned)blocks), dim3(64), 0, s, part, ksplit,
                              M * (int64_t)d, row_of, idx, w, pv.b2,
                              static_cast<const __nv_bfloat16*>(residual), N, d, k,
                              static_cast<__nv_bfloat16*>(out)));
  return 0;
}

int launch_combine(const void* y, const int32_t* row_of, const float* w, const void* residual,
                   int64_t N, int d, int k, int dtype, void* out, cudaStream_t s,
                   const EpSync* ep_wait, int32_t* status) {
  if (N == 0) return 0;
  const EpSync nosync = {};
  const EpSync& sy = ep_wait != nullptr ? *ep_wait : nosync;
  const int64_t items = N * (d >> 3);
  const int64_t blocks = (items + 255) / 256;
  const bool few = blocks * 256 < (int64_t)1 << 31;
  if (dtype == MOE_B200_BF16) {
    MOE_CUDA_CHECK(launch_pdl(combine_kernel_of<__nv_bfloat16>(k, few), dim3((unsigned)blocks), dim3(256), 0, s,
                              static_cast<const __nv_bfloat16*>(y), row_of, w,
                              static_cast<const __nv_bfloat16*>(residual), N, d, k,
                              static_cast<__nv_bfloat16*>(out), sy, status));
  } else {
    MOE_CUDA_CHECK(launch_pdl(combine_kernel_of<float>(k, few), dim3((unsigned)blocks), dim3(256), 0, s,
                              static_cast<const float*>(y), row_of, w,
                              static_cast<const float*>(residual), N, d, k, static_cast<float*>(out),
                              sy, status));
  }
  return 0;
}

}  // namespace moe

