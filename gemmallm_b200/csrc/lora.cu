// LoRA branch of an expert's Linear folded into its weight (reference
// model.py:175-179 and 185-189, fine_tuning=True):
//   x W^T + b + s * (B (A x + a) + b_lora)  =  x (W + s B A)^T + (b + s (B a + b_lora))
// so the grouped GEMM kernels run unchanged on W' = W + s B A and b' = b + s (B a + b_lora).
// W [out,in], A [r,in], B [out,r]; fp32 arithmetic, one rounding to the parameter dtype.
// W is read once and W' written once; A and B reach the arithmetic through shared memory. What bounds it is the
// arithmetic as much as the memory (rank 16: 16 FMA an element): a thread owns 8 rows x 8 columns, so that an element
// of A is read from shared memory and unpacked once for eight outputs, and fma.rn.f32x2 takes two columns at a time,
// the same sums in the same order as with plain FMA. [8192,1024] and [1024,4096], rank 16, nothing in L2: 20 + 12 us
// (4 rows a thread, plain FMA) -> 16 + 9 us.
#include "common.cuh"

namespace moe {

namespace {

constexpr int kMaxRank = 64;

constexpr int kTileRows = 64, kTileCols = 256;
constexpr int kBPitch = kTileRows + 4;      // floats: rows of 272 bytes, so that ranks fall into different banks

// Eight consecutive elements as they lie in memory. Through L2: the parameters may come from the kernel before this one
// (an optimizer step), which read-only loads must not be used for behind pdl_wait.
__device__ __forceinline__ void raw8(const __nv_bfloat16* p, uint4 (&v)[1]) {
  v[0] = __ldcg(reinterpret_cast<const uint4*>(p));
}
__device__ __forceinline__ void raw8(const float* p, uint4 (&v)[2]) {
  v[0] = __ldcg(reinterpret_cast<const uint4*>(p));
  v[1] = __ldcg(reinterpret_cast<const uint4*>(p) + 1);
}
__device__ __forceinline__ uint64_t pair_of_floats(float lo, float hi) {
  return (uint64_t)__float_as_uint(hi) << 32 | __float_as_uint(lo);
}
__device__ __forceinline__ void unpack8(const uint4 (&v)[1], uint64_t (&o)[4]) {
  const uint32_t w[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = pair_of_floats(bf16_lo(w[i]), bf16_hi(w[i]));
}
__device__ __forceinline__ void unpack8(const uint4 (&v)[2], uint64_t (&o)[4]) {
  o[0] = (uint64_t)v[0].y << 32 | v[0].x;
  o[1] = (uint64_t)v[0].w << 32 | v[0].z;
  o[2] = (uint64_t)v[1].y << 32 | v[1].x;
  o[3] = (uint64_t)v[1].w << 32 | v[1].z;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float lo_float(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_float(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

// One block per 64 x 256 tile of W: the tile's slice of A [rank][256] and the scaled rows of
// B [rank][64] wait in shared memory, every thread owns 8 rows x 8 columns, and W streams through once.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? 2 : 1)
lora_merge_kernel(const T* W, const T* b, const T* A, const T* a_bias, const T* B, const T* b_lora,
                  float scale, int out_f, int in_f, int rank, T* out_W, T* out_b) {
  constexpr int kRaw = sizeof(T) / 2;      // 16-byte pieces of eight elements
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* s_a = reinterpret_cast<T*>(smem_raw);                                                  // [rank][256]
  float* s_b = reinterpret_cast<float*>(smem_raw + (size_t)rank * kTileCols * sizeof(T));   // [rank][kBPitch]
  const int c0 = blockIdx.x * kTileCols, r0 = blockIdx.y * kTileRows;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = c0 + tx * 8;
  pdl_wait();
  // W first: its loads are in flight while the tables are filled
  uint4 raw[8][kRaw];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = r0 + ty * 8 + i;
    if (row < out_f && c < in_f) {
      raw8(W + (size_t)row * in_f + c, raw[i]);
    } else {
#pragma unroll
      for (int q = 0; q < kRaw; ++q) raw[i][q] = make_uint4(0, 0, 0, 0);
    }
  }
  const int rows = min(kTileRows, out_f - r0);
#pragma unroll 4
  for (int i = threadIdx.x; i < kTileRows * rank; i += 256) {      // neighbours in memory are ranks of a row
    const int rr = i / rank, r = i - rr * rank;
    s_b[r * kBPitch + rr] = rr < rows ? scale * to_f32(B[(size_t)r0 * rank + i]) : 0.f;
  }
  for (int i = threadIdx.x; i < rank * (kTileCols / 8); i += 256) {
    const int r = i / (kTileCols / 8), pc = i - r * (kTileCols / 8);
    uint4 v[kRaw];
    if (c0 + pc * 8 < in_f) {
      raw8(A + (size_t)r * in_f + c0 + pc * 8, v);
    } else {
#pragma unroll
      for (int q = 0; q < kRaw; ++q) v[q] = make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int q = 0; q < kRaw; ++q) reinterpret_cast<uint4*>(s_a + (size_t)r * kTileCols + pc * 8)[q] = v[q];
  }
  __syncthreads();
  uint64_t acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) unpack8(raw[i], acc[i]);
  for (int r = 0; r < rank; ++r) {
    uint4 v[kRaw];
#pragma unroll
    for (int q = 0; q < kRaw; ++q) v[q] = reinterpret_cast<const uint4*>(s_a + (size_t)r * kTileCols + tx * 8)[q];
    uint64_t a[4];
    unpack8(v, a);
    float br[8];
    load8(s_b + r * kBPitch + ty * 8, br);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint64_t bb = pair_of_floats(br[i], br[i]);
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][q] = fma2(bb, a[q], acc[i][q]);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = r0 + ty * 8 + i;
    if (row < out_f && c < in_f) {
      float o[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        o[2 * q] = lo_float(acc[i][q]);
        o[2 * q + 1] = hi_float(acc[i][q]);
      }
      store8(out_W + (size_t)row * in_f + c, o);
    }
  }
  if (blockIdx.x == 0 && (int)threadIdx.x < rows) {
    const int row = r0 + threadIdx.x;
    float sum = 0.f;
    for (int r = 0; r < rank; ++r) sum = fmaf(s_b[r * kBPitch + threadIdx.x], to_f32(a_bias[r]), sum);
    T v;
    from_f32(v, to_f32(b[row]) + sum + scale * to_f32(b_lora[row]));
    out_b[row] = v;
  }
}

template <typename T>
int launch_merge(const void* W, const void* b, const void* A, const void* a_bias, const void* B,
                 const void* b_lora, float scale, int out_f, int in_f, int rank, void* out_W,
                 void* out_b, cudaStream_t s) {
  const size_t smem = (size_t)rank * (kTileCols * sizeof(T) + kBPitch * sizeof(float));
  static PerDeviceOnce once;
  if (smem > 48 * 1024) {
    int rc = ensure_dynamic_smem(once, lora_merge_kernel<T>, 96 * 1024);
    if (rc) return rc;
  }
  MOE_CUDA_CHECK(launch_pdl(lora_merge_kernel<T>, dim3((in_f + kTileCols - 1) / kTileCols, (out_f + kTileRows - 1) / kTileRows),
                            dim3(256), smem, s, static_cast<const T*>(W), static_cast<const T*>(b),
                            static_cast<const T*>(A), static_cast<const T*>(a_bias), static_cast<const T*>(B),
                            static_cast<const T*>(b_lora), scale, out_f, in_f, rank, static_cast<T*>(out_W),
                            static_cast<T*>(out_b)));
  return 0;
}

}  // namespace
}  // namespace moe

using namespace moe;

extern "C" int moe_b200_lora_merge(const void* W, const void* b, const void* A, const void* a_bias,
                                   const void* B, const void* b_lora, float scale, int out_features,
                                   int in_features, int rank, int dtype, void* out_W, void* out_b,
                                   void* stream) {
  if (dtype != MOE_B200_F32 && dtype != MOE_B200_BF16)
    return set_error(MOE_B200_ERR_DTYPE, "dtype must be MOE_B200_F32 or MOE_B200_BF16");
  if (out_features < 1 || in_features < 8 || (in_features & 7) || rank < 1 || rank > kMaxRank)
    return set_error(MOE_B200_ERR_SHAPE, "in_features must be a multiple of 8 and rank in [1,64]");
  if (!W || !b || !A || !a_bias || !B || !b_lora || !out_W || !out_b)
    return set_error(MOE_B200_ERR_NULL, "NULL argument");
  if (!aligned16(W) || !aligned16(A) || !aligned16(out_W))
    return set_error(MOE_B200_ERR_ALIGN, "W, A and out_W must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == MOE_B200_BF16)
    return launch_merge<__nv_bfloat16>(W, b, A, a_bias, B, b_lora, scale, out_features, in_features, rank,
                                       out_W, out_b, s);
  return launch_merge<float>(W, b, A, a_bias, B, b_lora, scale, out_features, in_features, rank, out_W,
                             out_b, s);
}
