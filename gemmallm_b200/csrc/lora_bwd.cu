// Gradients of the LoRA tensors of grouped Linears (reference model.py:175-179,185-189 under autograd). The
// kernels of a training step run on merged weights W' = W + s B A, b' = b + s (B a + b_lora); with In and Out' the
// Linear's input and output gradient on an expert's rows and G = Out'^T In, g = colsum(Out'):
//   dB = s (G A^T + g a^T) = s Out'^T Q,  Q = In A^T + a      [rows, r]
//   dA = s B^T G           = s P^T In,    P = Out' B          [rows, r]
//   da = s B^T g           = s colsum(P),  db_lora = s g
// so G itself, a full weight gradient, is not needed, and where the base weights are frozen it is not formed: all
// that is left are products with one side of the rank's width (16), bound by reading In and Out' twice. Three
// launches for both Linears of all experts:
//   lora_rows_kernel    P and Q, K cut into ranges (partial sums): rows are the 16-row operand of mma.sync,
//                       straight from global memory; A and B wait in shared memory
//   lora_cols_kernel    X^T S over segments of rows: X^T fragments by transposing ldmatrix; P and Q enter as
//                       bf16 head and remainder, two products each, so that their rounding is that of fp32
//   lora_finish_kernel  sums over an expert's segments in order, scale, rounding
#include "common.cuh"

namespace moe {

namespace {

constexpr int kRank = 16;          // ranks in steps of 16, padded with zeros
constexpr int kRowTile = 64;
constexpr int kRange = 512;        // contraction range of a block of lora_rows_kernel
constexpr int kColTile = 128;
constexpr int kWPitch = kRange + 8;
constexpr int kXPitch = kColTile + 8;
constexpr int kSPitch = 2 * kRank + 8;

// What the four products of either kind read; index 2 * linear + (0: Q / dB, 1: P / dA).
struct Jobs {
  const __nv_bfloat16* x[4];       // rows kernel: In, Out';  cols kernel: Out', In
  int C[4];                        // their widths
  int ranges[4];                   // rows kernel: K ranges of the product
  float* part[4];                  // [ranges][M][R] of the rows kernel
  float* out[4];                   // [segments][C][R] of the cols kernel
  float* colsum[2];                // [segments][R] of P, per Linear
  const void* const* tab;          // [2][E][3]: A, a, B of every expert
};

// Row tile `tile` of `rows_per` rows, counted over the experts in order.
__device__ __forceinline__ bool find_tile(const int32_t* offsets, int E, int tile, int rows_per, int& e, int& row0,
                                          int& rows) {
  for (e = 0; e < E; ++e) {
    const int beg = offsets[e], n = offsets[e + 1] - beg, tiles = (n + rows_per - 1) / rows_per;
    if (tile < tiles) {
      row0 = beg + tile * rows_per;
      rows = min(rows_per, n - tile * rows_per);
      return true;
    }
    tile -= tiles;
  }
  return false;
}

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}

// grid: (row tiles, sum of the jobs' ranges, rank steps); part[job][range][row][r] = x[row, range] . W[range, r]
__global__ void __launch_bounds__(256)
lora_rows_kernel(const Jobs jobs, const int32_t* __restrict__ offsets, int E, int64_t M, int rank, int R) {
  __shared__ __align__(16) __nv_bfloat16 s_w[kRank * kWPitch];
  __shared__ float s_red[4][32][8];
  int job = 0, range = blockIdx.y;
  while (range >= jobs.ranges[job]) range -= jobs.ranges[job++];
  int e, row0, rows;
  if (!find_tile(offsets, E, blockIdx.x, kRowTile, e, row0, rows)) return;
  const int C = jobs.C[job], k0 = range * kRange, n0 = blockIdx.z * kRank;
  const int klen = min(kRange, C - k0);             // a multiple of 8
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the range's weights, [rank][k]: A [rank][C] as it lies, B [C][rank] transposed
  const bool is_b = (job & 1) != 0;
  const __nv_bfloat16* W =
      static_cast<const __nv_bfloat16*>(jobs.tab[((size_t)(job >> 1) * E + e) * 3 + (is_b ? 2 : 0)]);
  if (!is_b) {
    for (int i = tid; i < kRank * kRange / 8; i += 256) {
      const int r = i / (kRange / 8), k = (i - r * (kRange / 8)) * 8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (n0 + r < rank && k < klen) v = __ldg(reinterpret_cast<const uint4*>(W + (size_t)(n0 + r) * C + k0 + k));
      *reinterpret_cast<uint4*>(s_w + r * kWPitch + k) = v;
    }
  } else {
    // a thread takes whole rows of B, 16 ranks of one k (32 contiguous bytes where rows allow 16-byte loads), and
    // a warp's stores of one rank are 64 contiguous bytes (with k along the lanes of the loads, a sector for
    // every two bytes, this kernel took 38 instead of 15 us at 1632 rows, d 1024, f 4096)
    const bool wide = rank % 8 == 0 && (reinterpret_cast<uintptr_t>(W) & 15) == 0;
#pragma unroll
    for (int u = 0; u < kRange / 256; ++u) {
      const int k = tid + u * 256;
      uint4 v[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
      if (k < klen) {
        const __nv_bfloat16* row = W + (size_t)(k0 + k) * rank + n0;
        if (wide) {
          v[0] = __ldg(reinterpret_cast<const uint4*>(row));
          if (n0 + 8 < rank) v[1] = __ldg(reinterpret_cast<const uint4*>(row) + 1);
        } else {
          unsigned short* h = reinterpret_cast<unsigned short*>(v);
#pragma unroll
          for (int r = 0; r < kRank; ++r)
            if (n0 + r < rank) h[r] = __ldg(reinterpret_cast<const unsigned short*>(row) + r);
        }
      }
      const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(v);
#pragma unroll
      for (int r = 0; r < kRank; ++r) s_w[r * kWPitch + k] = h[r];
    }
  }
  __syncthreads();
  // warp = 16 rows x half of the range; the contraction index inside 32 elements is permuted alike for both sides
  const int g = lane >> 2, t = lane & 3, rg = warp & 3, half = warp >> 2;
  const int ra = rg * 16 + g, rb = ra + 8;
  const uint4* xa = reinterpret_cast<const uint4*>(jobs.x[job] + (size_t)(row0 + min(ra, rows - 1)) * C + k0);
  const uint4* xb = reinterpret_cast<const uint4*>(jobs.x[job] + (size_t)(row0 + min(rb, rows - 1)) * C + k0);
  const int pieces = klen >> 3;
  float acc[2][4] = {};
  const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll 1
  for (int c0 = half * 8; c0 < half * 8 + 8; c0 += 4) {     // 16 chunks of 32 elements in a range
    uint4 a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = 4 * (c0 + u) + t;
      a[u] = p < pieces ? __ldg(xa + p) : zero;
      b[u] = p < pieces ? __ldg(xb + p) : zero;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = 4 * (c0 + u) + t;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint4 w = *reinterpret_cast<const uint4*>(s_w + (8 * j + g) * kWPitch + p * 8);
        mma16816(acc[j], a[u].x, b[u].x, a[u].y, b[u].y, w.x, w.y);
        mma16816(acc[j], a[u].z, b[u].z, a[u].w, b[u].w, w.z, w.w);
      }
    }
  }
  if (half == 1) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) s_red[rg][lane][j * 4 + i] = acc[j][i];
  }
  __syncthreads();
  if (half == 0) {
    float* out = jobs.part[job] + ((size_t)range * M + row0) * R + n0;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][i] += s_red[rg][lane][j * 4 + i];
      const int c = 8 * j + 2 * t;
      if (ra < rows) *reinterpret_cast<float2*>(out + (size_t)ra * R + c) = make_float2(acc[j][0], acc[j][1]);
      if (rb < rows) *reinterpret_cast<float2*>(out + (size_t)rb * R + c) = make_float2(acc[j][2], acc[j][3]);
    }
  }
}

// grid: (segments of `seg_rows` rows, sum of the jobs' column tiles, rank steps);
// out[job][segment][c][r] = sum over the segment's rows of x[row, c] * S[row, r]
__global__ void __launch_bounds__(256)
lora_cols_kernel(const Jobs jobs, const int32_t* __restrict__ offsets, int E, int64_t M, int rank, int R,
                 int seg_rows) {
  __shared__ __align__(16) __nv_bfloat16 s_x[kRowTile * kXPitch];
  __shared__ __align__(16) __nv_bfloat16 s_s[kRowTile * kSPitch];
  int job = 0, ct = blockIdx.y;
  for (;; ++job) {
    const int tiles = (jobs.C[job] + kColTile - 1) / kColTile;
    if (ct < tiles) break;
    ct -= tiles;
  }
  int e, row0, rows;
  if (!find_tile(offsets, E, blockIdx.x, seg_rows, e, row0, rows)) return;
  const int C = jobs.C[job], c0 = ct * kColTile, n0 = blockIdx.z * kRank;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sj = job;                               // dB takes Q (even), dA takes P (odd)
  const bool with_bias = (job & 1) == 0;
  const __nv_bfloat16* a_bias =
      with_bias ? static_cast<const __nv_bfloat16*>(jobs.tab[((size_t)(job >> 1) * E + e) * 3 + 1]) : nullptr;
  const int ranges = jobs.ranges[sj];
  const bool sums = !with_bias && ct == 0;          // this block also forms colsum(P)
  float acc[2][4] = {};
  float psum = 0.f;
  for (int r0 = 0; r0 < rows; r0 += kRowTile) {
    __syncthreads();
    // S: four threads per row, four columns each; the K ranges in order
    {
      const int rr = tid >> 2, q = (tid & 3) * 4;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (r0 + rr < rows) {
        for (int k = 0; k < ranges; ++k) {
          const float4 p = *reinterpret_cast<const float4*>(jobs.part[sj] + ((size_t)k * M + row0 + r0 + rr) * R + n0 + q);
          v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
        }
        if (with_bias) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (n0 + q + i < rank) v[i] += __bfloat162float(a_bias[n0 + q + i]);
        }
      }
      float lo[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) lo[i] = v[i] - __bfloat162float(__float2bfloat16_rn(v[i]));
      __nv_bfloat16* s = s_s + rr * kSPitch + q;
      *reinterpret_cast<uint2*>(s) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      *reinterpret_cast<uint2*>(s + kRank) = make_uint2(pack_bf16x2(lo[0], lo[1]), pack_bf16x2(lo[2], lo[3]));
    }
    // X: 64 rows x 128 columns
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = tid + u * 256, rr = i >> 4, c = (i & 15) * 8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (r0 + rr < rows && c0 + c < C)
        v = __ldg(reinterpret_cast<const uint4*>(jobs.x[job ^ 1] + (size_t)(row0 + r0 + rr) * C + c0 + c));
      *reinterpret_cast<uint4*>(s_x + rr * kXPitch + c) = v;
    }
    __syncthreads();
    if (sums && tid < kRank)
      for (int rr = 0; rr < kRowTile; ++rr)
        psum += __bfloat162float(s_s[rr * kSPitch + tid]) + __bfloat162float(s_s[rr * kSPitch + kRank + tid]);
#pragma unroll
    for (int kk = 0; kk < kRowTile / 16; ++kk) {
      uint32_t a[4], hi[4], lo[4];
      // matrices (rows kk*16 + {0,8}) x (columns +{0,8}): transposed they are the fragments a0..a3 of X^T
      const int mr = kk * 16 + (lane & 7) + ((lane >> 4) << 3), mc = warp * 16 + (((lane >> 3) & 1) << 3);
      ldmatrix_x4_trans(a, s_x + mr * kXPitch + mc);
      const int sr = kk * 16 + (lane & 7) + (((lane >> 3) & 1) << 3), sc = (lane >> 4) << 3;
      ldmatrix_x4_trans(hi, s_s + sr * kSPitch + sc);
      ldmatrix_x4_trans(lo, s_s + sr * kSPitch + kRank + sc);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        mma16816(acc[j], a[0], a[1], a[2], a[3], hi[2 * j], hi[2 * j + 1]);
        mma16816(acc[j], a[0], a[1], a[2], a[3], lo[2 * j], lo[2 * j + 1]);
      }
    }
  }
  const int g = lane >> 2, t = lane & 3;
  float* out = jobs.out[job] + ((size_t)blockIdx.x * C + c0 + warp * 16) * R + n0;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (c0 + warp * 16 + g < C)
      *reinterpret_cast<float2*>(out + (size_t)g * R + 8 * j + 2 * t) = make_float2(acc[j][0], acc[j][1]);
    if (c0 + warp * 16 + g + 8 < C)
      *reinterpret_cast<float2*>(out + (size_t)(g + 8) * R + 8 * j + 2 * t) = make_float2(acc[j][2], acc[j][3]);
  }
  if (sums && tid < kRank) jobs.colsum[job >> 1][(size_t)blockIdx.x * R + n0 + tid] = psum;
}

struct Results {
  __nv_bfloat16 *dA[2], *da[2], *dB[2], *db[2];   // [E][rank][in], [E][rank], [E][out][rank], [E][out]
  const __nv_bfloat16* g[2];                      // [E][out] gradients of the merged biases
};

// grid: (blocks over C * R of the widest job, 4 jobs, E)
__global__ void __launch_bounds__(256)
lora_finish_kernel(const Jobs jobs, const Results res, const int32_t* __restrict__ offsets, int rank, int R,
                   int seg_rows, float scale) {
  const int job = blockIdx.y, l = job >> 1, e = blockIdx.z;
  const int C = jobs.C[job];
  __shared__ int s_first, s_count;
  if (threadIdx.x == 0) {
    int first = 0;
    for (int i = 0; i < e; ++i) first += (offsets[i + 1] - offsets[i] + seg_rows - 1) / seg_rows;
    s_first = first;
    s_count = (offsets[e + 1] - offsets[e] + seg_rows - 1) / seg_rows;
  }
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (int64_t)C * rank) return;
  // dB [C][rank]; dA [rank][C]
  const bool is_a = (job & 1) != 0;
  const int c = (int)(is_a ? i % C : i / rank), r = (int)(is_a ? i / C : i % rank);
  float sum = 0.f;
  for (int q = 0; q < s_count; ++q) sum += jobs.out[job][((size_t)(s_first + q) * C + c) * R + r];
  const __nv_bfloat16 v = __float2bfloat16_rn(sum * scale);
  if (!is_a) {
    res.dB[l][(size_t)e * C * rank + i] = v;
    if (r == 0)
      res.db[l][(size_t)e * C + c] = __float2bfloat16_rn(scale * __bfloat162float(res.g[l][(size_t)e * C + c]));
  } else {
    res.dA[l][(size_t)e * C * rank + i] = v;
    if (c == 0) {
      float ps = 0.f;
      for (int q = 0; q < s_count; ++q) ps += jobs.colsum[l][(size_t)(s_first + q) * R + r];
      res.da[l][(size_t)e * rank + r] = __float2bfloat16_rn(ps * scale);
    }
  }
}

struct Plan {
  int R, seg_rows;
  int64_t row_tiles, segs;
  int ranges[4];
  size_t part[4], out[4], colsum[2], total;     // in floats
};

Plan make_plan(int64_t M, int d, int f, int E, int rank) {
  Plan p;
  p.R = (rank + kRank - 1) / kRank * kRank;
  // segments long enough that their partial results stay small next to the activations
  p.seg_rows = M > 8192 ? 1024 : 256;
  p.row_tiles = (M + kRowTile - 1) / kRowTile + E;
  p.segs = (M + p.seg_rows - 1) / p.seg_rows + E;
  const int width[4] = {d, 2 * f, f, d};       // In, Out' of gate_and_up, then of down
  size_t at = 0;
  for (int j = 0; j < 4; ++j) {
    p.ranges[j] = (width[j] + kRange - 1) / kRange;
    p.part[j] = at;
    at += (size_t)p.ranges[j] * M * p.R;
  }
  for (int j = 0; j < 4; ++j) {
    p.out[j] = at;
    at += (size_t)p.segs * width[j ^ 1] * p.R;
  }
  for (int l = 0; l < 2; ++l) {
    p.colsum[l] = at;
    at += (size_t)p.segs * p.R;
  }
  p.total = at;
  return p;
}

}  // namespace

size_t lora_grads_scratch_floats(int64_t M, int d, int f, int E, int rank) { return make_plan(M, d, f, E, rank).total; }

int launch_lora_grads(const void* const* tab, const void* x, const void* dgu, const void* h, const void* dy,
                      const int32_t* offsets, int64_t M, int d, int f, int E, int rank, float scale, float* scratch,
                      const void* const (&g)[2], void* const (&dA)[2], void* const (&da)[2], void* const (&dB)[2],
                      void* const (&db)[2], cudaStream_t s) {
  if (M == 0) return 0;
  const Plan p = make_plan(M, d, f, E, rank);
  Jobs rows = {}, cols = {};
  const void* act[4] = {x, dgu, h, dy};
  const int width[4] = {d, 2 * f, f, d};
  unsigned ranges = 0, tiles = 0;
  for (int j = 0; j < 4; ++j) {
    rows.x[j] = cols.x[j] = static_cast<const __nv_bfloat16*>(act[j]);   // the cols kernel takes x[job ^ 1]
    rows.C[j] = width[j];
    cols.C[j] = width[j ^ 1];
    rows.ranges[j] = cols.ranges[j] = p.ranges[j];
    rows.part[j] = cols.part[j] = scratch + p.part[j];
    cols.out[j] = scratch + p.out[j];
    ranges += (unsigned)p.ranges[j];
    tiles += (unsigned)((width[j] + kColTile - 1) / kColTile);
  }
  rows.tab = cols.tab = tab;
  Results res;
  for (int l = 0; l < 2; ++l) {
    cols.colsum[l] = scratch + p.colsum[l];
    res.dA[l] = static_cast<__nv_bfloat16*>(dA[l]);
    res.da[l] = static_cast<__nv_bfloat16*>(da[l]);
    res.dB[l] = static_cast<__nv_bfloat16*>(dB[l]);
    res.db[l] = static_cast<__nv_bfloat16*>(db[l]);
    res.g[l] = static_cast<const __nv_bfloat16*>(g[l]);
  }
  const unsigned steps = (unsigned)(p.R / kRank);
  lora_rows_kernel<<<dim3((unsigned)p.row_tiles, ranges, steps), 256, 0, s>>>(rows, offsets, E, M, rank, p.R);
  MOE_CUDA_CHECK(cudaGetLastError());
  lora_cols_kernel<<<dim3((unsigned)p.segs, tiles, steps), 256, 0, s>>>(cols, offsets, E, M, rank, p.R, p.seg_rows);
  MOE_CUDA_CHECK(cudaGetLastError());
  const int64_t widest = (int64_t)(2 * f > d ? 2 * f : d) * rank;
  lora_finish_kernel<<<dim3((unsigned)((widest + 255) / 256), 4, (unsigned)E), 256, 0, s>>>(cols, res, offsets, rank, p.R,
                                                                                         p.seg_rows, scale);
  MOE_CUDA_CHECK(cudaGetLastError());
  return 0;
}

}  // namespace moe
