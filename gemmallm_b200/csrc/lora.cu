// LoRA branch of an expert's Linear folded into its weight (reference
// model.py:175-179 and 185-189, fine_tuning=True):
//   x W^T + b + s * (B (A x + a) + b_lora)  =  x (W + s B A)^T + (b + s (B a + b_lora))
// so the grouped GEMM kernels run unchanged on W' = W + s B A and b' = b + s (B a + b_lora).
// W [out,in], A [r,in], B [out,r]; sums in fp32, one rounding to the parameter dtype.
// W is read once and W' written once. bf16: B A by mma.sync, the rest is the stream of W and W' (4 KiB units a warp, the
// next one asked for before this one is stored): [8192,1024] and [1024,4096], rank 16, nothing in L2: 16 + 9 us with the
// sums on the CUDA cores (packed FMA, which bound it), now 10.7 + 6.9; a LoRA step of the dense feed-forward, 1632 rows, 223
// -> 215 us. The tensor core cuts its fp32 sums off where FMA rounds them, but adds 16 products at once and takes B
// unscaled: fewer W' are not the nearest bf16 to their 64-bit value than with FMA ([8192,1024], rank 16, N(0, 0.02^2): 11 of
// 8388608 against 42; rank 64 37 against 147; rank 33, A and B five times as large, [2816,2048]: 101 of 5767168 against 513).
// fp32: the sums on the CUDA cores, a thread owning 8 rows x 8 columns, A and B in shared memory.
#include "common.cuh"
#include "internal.h"

namespace moe {

namespace {

constexpr int kMaxRank = 64;

constexpr int kTileRows = 64, kTileCols = 256;
constexpr int kBPitch = kTileRows + 4;      // floats: rows of 272 bytes, so that ranks fall into different banks

// Eight consecutive elements as they lie in memory. Through L2: the parameters may come from the kernel before this one
// (an optimizer step), which read-only loads must not be used for behind pdl_wait.
__device__ __forceinline__ void raw8(const float* p, uint4 (&v)[2]) {
  v[0] = __ldcg(reinterpret_cast<const uint4*>(p));
  v[1] = __ldcg(reinterpret_cast<const uint4*>(p) + 1);
}
__device__ __forceinline__ uint64_t pair_of_floats(float lo, float hi) {
  return (uint64_t)__float_as_uint(hi) << 32 | __float_as_uint(lo);
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

// fp32. One block per 64 x 256 tile of W: the tile's slice of A [rank][256] and the scaled rows of
// B [rank][64] wait in shared memory, every thread owns 8 rows x 8 columns, and W streams through once.
__global__ void __launch_bounds__(256, 1)
lora_merge_f32_kernel(const float* W, const float* b, const float* A, const float* a_bias, const float* B, const float* b_lora,
                      float scale, int out_f, int in_f, int rank, float* out_W, float* out_b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* s_a = reinterpret_cast<float*>(smem_raw);       // [rank][256]
  float* s_b = s_a + (size_t)rank * kTileCols;           // [rank][kBPitch]
  const int c0 = blockIdx.x * kTileCols, r0 = blockIdx.y * kTileRows;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = c0 + tx * 8;
  pdl_wait();
  // W first: its loads are in flight while the tables are filled
  uint4 raw[8][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = r0 + ty * 8 + i;
    if (row < out_f && c < in_f) {
      raw8(W + (size_t)row * in_f + c, raw[i]);
    } else {
      raw[i][0] = raw[i][1] = make_uint4(0, 0, 0, 0);
    }
  }
  const int rows = min(kTileRows, out_f - r0);
#pragma unroll 4
  for (int i = threadIdx.x; i < kTileRows * rank; i += 256) {      // neighbours in memory are ranks of a row
    const int rr = i / rank, r = i - rr * rank;
    s_b[r * kBPitch + rr] = rr < rows ? scale * B[(size_t)r0 * rank + i] : 0.f;
  }
  for (int i = threadIdx.x; i < rank * (kTileCols / 8); i += 256) {
    const int r = i / (kTileCols / 8), pc = i - r * (kTileCols / 8);
    uint4 v[2];
    if (c0 + pc * 8 < in_f) {
      raw8(A + (size_t)r * in_f + c0 + pc * 8, v);
    } else {
      v[0] = v[1] = make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) reinterpret_cast<uint4*>(s_a + (size_t)r * kTileCols + pc * 8)[q] = v[q];
  }
  __syncthreads();
  uint64_t acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) unpack8(raw[i], acc[i]);
  for (int r = 0; r < rank; ++r) {
    uint4 v[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) v[q] = reinterpret_cast<const uint4*>(s_a + (size_t)r * kTileCols + tx * 8)[q];
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
    for (int r = 0; r < rank; ++r) sum = fmaf(s_b[r * kBPitch + threadIdx.x], a_bias[r], sum);
    out_b[row] = b[row] + sum + scale * b_lora[row];
  }
}

// bf16: B A on the tensor cores (products of bf16 are exact in fp32, the sums fp32, cut off), so that one pass over W is left.
// A warp takes units of 16 rows x 128 columns of its block's 128 columns; the slice of A [rank][128] waits in shared
// memory with its columns in the order that gives a thread eight neighbouring ones: tile j, place n of a group of 32 columns
// is column 8 (n / 2) + 2 j + n % 2. The next unit of W is requested when this one's products have been added, before the
// result is stored. A launch takes several Linears, one after the other in its blocks (both of a feed-forward of d 1024, f 4096:
// 17 us of a fine-tuning step with a launch each, which the second one's blocks could not begin before the first's end).
constexpr int kMergeCols = 128;
constexpr int kMergePitch = kMergeCols + 8;      // elements: rows 16 bytes apart modulo the banks
constexpr int kMergeWarps = 8;
constexpr int kMergeJobs = 32;      // of a launch: 3 KB of arguments

struct MergeJob {
  const __nv_bfloat16 *W, *b, *A, *a_bias, *B, *b_lora;
  __nv_bfloat16 *out_W, *out_b;
  float scale;
  int out_f, in_f, rank;
  int end, strips, sharing;      // blocks of the launch up to this Linear's last; strips of columns; blocks that share one
};
struct MergeJobs {
  MergeJob job[kMergeJobs];
};

__global__ void __launch_bounds__(32 * kMergeWarps, 2) lora_merge_tc_kernel(const __grid_constant__ MergeJobs jobs) {
  int which = 0, before = 0;
  for (; (int)blockIdx.x >= jobs.job[which].end; ++which) before = jobs.job[which].end;
  const MergeJob& job = jobs.job[which];
  const __nv_bfloat16 *W = job.W, *b = job.b, *A = job.A, *a_bias = job.a_bias, *B = job.B, *b_lora = job.b_lora;
  __nv_bfloat16 *out_W = job.out_W, *out_b = job.out_b;
  const float scale = job.scale;
  const int out_f = job.out_f, in_f = job.in_f, rank = job.rank;
  const int share = ((int)blockIdx.x - before) / job.strips, strip = (int)blockIdx.x - before - share * job.strips;
  __shared__ __align__(16) __nv_bfloat16 s_a[kMaxRank][kMergePitch];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int c0 = strip * kMergeCols;
  const int ksteps = (rank + 15) >> 4;
  const int units = (out_f + 15) >> 4, stride = job.sharing * kMergeWarps;
  pdl_wait();
  uint4 w[2][4];      // rows g and g + 8; columns 32 q + 8 t
  auto request = [&](int u) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = u * 16 + g + 8 * h;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = c0 + q * 32 + t * 8;
        w[h][q] = row < out_f && c < in_f ? __ldcg(reinterpret_cast<const uint4*>(W + (size_t)row * in_f + c))
                                          : make_uint4(0, 0, 0, 0);
      }
    }
  };
  int u = share * kMergeWarps + warp;
  if (u < units) request(u);
  for (int i = tid; i < ksteps * 16 * (kMergeCols / 8); i += 32 * kMergeWarps) {
    const int r = i / (kMergeCols / 8), p = i - r * (kMergeCols / 8);      // eight columns of a rank
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < rank && c0 + p * 8 < in_f) v = __ldcg(reinterpret_cast<const uint4*>(A + (size_t)r * in_f + c0 + p * 8));
    const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
    __nv_bfloat16* to = &s_a[r][(p >> 2) * 32 + (p & 3) * 2];
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<uint32_t*>(to + j * 8) = vw[j];
  }
  __syncthreads();
  for (; u < units; u += stride) {
    const int row0 = u * 16;
    float acc[4][4][4];      // group of 32 columns, tile, fragment
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[q][j][i] = 0.f;
    for (int ks = 0; ks < ksteps; ++ks) {
      // rows g and g + 8 of B, ranks 16 ks + 2 t + {0, 1} and + 8 (element by element: rank may be odd)
      uint32_t a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = row0 + g + 8 * (i & 1), r = ks * 16 + 2 * t + 8 * (i >> 1);
        const unsigned short* p = reinterpret_cast<const unsigned short*>(B) + (size_t)row * rank + r;
        const uint32_t lo = row < out_f && r < rank ? __ldcg(p) : 0, hi = row < out_f && r + 1 < rank ? __ldcg(p + 1) : 0;
        a[i] = hi << 16 | lo;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          uint32_t f[4];       // tiles j and j + 1: ranks 0-7 and 8-15 of the step each
          const uint32_t at = (uint32_t)__cvta_generic_to_shared(
              &s_a[ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8][q * 32 + (j + (lane >> 4)) * 8]);
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                       : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(at) : "memory");
#pragma unroll
          for (int h = 0; h < 2; ++h)
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                : "+f"(acc[q][j + h][0]), "+f"(acc[q][j + h][1]), "+f"(acc[q][j + h][2]), "+f"(acc[q][j + h][3])
                : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(f[2 * h]), "r"(f[2 * h + 1]));
        }
    }
    // rows g and g + 8, columns 8 t + 2 j + {0, 1} of every group
    uint4 o[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t vw[4] = {w[h][q].x, w[h][q].y, w[h][q].z, w[h][q].w};
        uint32_t r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          r[j] = pack_bf16x2(fmaf(scale, acc[q][j][2 * h], bf16_lo(vw[j])), fmaf(scale, acc[q][j][2 * h + 1], bf16_hi(vw[j])));
        o[h][q] = make_uint4(r[0], r[1], r[2], r[3]);
      }
    if (u + stride < units) request(u + stride);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = row0 + g + 8 * h;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = c0 + q * 32 + t * 8;
        if (row < out_f && c < in_f) *reinterpret_cast<uint4*>(out_W + (size_t)row * in_f + c) = o[h][q];
      }
    }
    if (strip == 0 && lane < 16 && row0 + lane < out_f) {
      const int row = row0 + lane;
      float sum = 0.f;
      for (int r = 0; r < rank; ++r) sum = fmaf(scale * to_f32(B[(size_t)row * rank + r]), to_f32(a_bias[r]), sum);
      out_b[row] = __float2bfloat16_rn(to_f32(b[row]) + sum + scale * to_f32(b_lora[row]));
    }
  }
}

int launch_merges_bf16(const LoraMerge* merges, int n, cudaStream_t s) {
  typedef const __nv_bfloat16* In;
  typedef __nv_bfloat16* Out;
  MergeJobs jobs;
  unsigned grid = 0;
  for (int i = 0; i < n; ++i) {
    const LoraMerge& m = merges[i];
    const unsigned strips = (unsigned)((m.in_f + kMergeCols - 1) / kMergeCols);
    const unsigned blocks = (unsigned)(((m.out_f + 15) / 16 + kMergeWarps - 1) / kMergeWarps);
    const unsigned most = (2 * kNumSMs + strips - 1) / strips, sharing = blocks < most ? blocks : most;
    grid += strips * sharing;
    jobs.job[i] = {static_cast<In>(m.W), static_cast<In>(m.b), static_cast<In>(m.A), static_cast<In>(m.a_bias),
                   static_cast<In>(m.B), static_cast<In>(m.b_lora), static_cast<Out>(m.out_W), static_cast<Out>(m.out_b),
                   m.scale, m.out_f, m.in_f, m.rank, (int)grid, (int)strips, (int)sharing};
  }
  MOE_CUDA_CHECK(launch_pdl(lora_merge_tc_kernel, dim3(grid), dim3(32 * kMergeWarps), 0, s, jobs));
  return 0;
}

int launch_merge_f32(const void* W, const void* b, const void* A, const void* a_bias, const void* B, const void* b_lora,
                     float scale, int out_f, int in_f, int rank, void* out_W, void* out_b, cudaStream_t s) {
  typedef const float* In;
  const size_t smem = (size_t)rank * (kTileCols + kBPitch) * sizeof(float);
  static PerDeviceOnce once;
  if (smem > 48 * 1024) {
    int rc = ensure_dynamic_smem(once, lora_merge_f32_kernel, 96 * 1024);
    if (rc) return rc;
  }
  MOE_CUDA_CHECK(launch_pdl(lora_merge_f32_kernel, dim3((in_f + kTileCols - 1) / kTileCols, (out_f + kTileRows - 1) / kTileRows),
                            dim3(256), smem, s, static_cast<In>(W), static_cast<In>(b), static_cast<In>(A),
                            static_cast<In>(a_bias), static_cast<In>(B), static_cast<In>(b_lora), scale, out_f, in_f, rank,
                            static_cast<float*>(out_W), static_cast<float*>(out_b)));
  return 0;
}

}  // namespace
}  // namespace moe

namespace moe {

int lora_merges(const LoraMerge* merges, int n, int dtype, void* stream) {
  if (dtype != MOE_B200_F32 && dtype != MOE_B200_BF16)
    return set_error(MOE_B200_ERR_DTYPE, "dtype must be MOE_B200_F32 or MOE_B200_BF16");
  for (int i = 0; i < n; ++i) {
    const LoraMerge& m = merges[i];
    if (m.out_f < 1 || m.in_f < 8 || (m.in_f & 7) || m.rank < 1 || m.rank > kMaxRank)
      return set_error(MOE_B200_ERR_SHAPE, "in_features must be a multiple of 8 and rank in [1,64]");
    if (!m.W || !m.b || !m.A || !m.a_bias || !m.B || !m.b_lora || !m.out_W || !m.out_b)
      return set_error(MOE_B200_ERR_NULL, "NULL argument");
    if (!aligned16(m.W) || !aligned16(m.A) || !aligned16(m.out_W))
      return set_error(MOE_B200_ERR_ALIGN, "W, A and out_W must be 16-byte aligned");
  }
  cudaStream_t s = (cudaStream_t)stream;
  int rc = 0;
  if (dtype == MOE_B200_BF16) {
    for (int i = 0; i < n && rc == 0; i += kMergeJobs)
      rc = launch_merges_bf16(merges + i, n - i < kMergeJobs ? n - i : kMergeJobs, s);
  } else {
    for (int i = 0; i < n && rc == 0; ++i) {
      const LoraMerge& m = merges[i];
      rc = launch_merge_f32(m.W, m.b, m.A, m.a_bias, m.B, m.b_lora, m.scale, m.out_f, m.in_f, m.rank, m.out_W, m.out_b, s);
    }
  }
  return rc;
}

}  // namespace moe

using namespace moe;

extern "C" int moe_b200_lora_merge(const void* W, const void* b, const void* A, const void* a_bias,
                                   const void* B, const void* b_lora, float scale, int out_features,
                                   int in_features, int rank, int dtype, void* out_W, void* out_b,
                                   void* stream) {
  const LoraMerge m = {W, b, A, a_bias, B, b_lora, out_W, out_b, scale, out_features, in_features, rank};
  return lora_merges(&m, 1, dtype, stream);
}
