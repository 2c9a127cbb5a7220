// Gradients of the LoRA tensors of grouped Linears (reference model.py:175-179,185-189 under autograd). The
// kernels of a training step run on merged weights W' = W + s B A, b' = b + s (B a + b_lora); with G = dL/dW' [out, in]
// and g = dL/db' [out] as the weight-gradient product and the column sums give them, rounded to bf16:
//   dB = s (G A^T + g a^T),  db_lora = s g,  dA = s B^T G,  da = s B^T g
// G carries the rounding of a base weight's gradient into the LoRA tensors, and it has to: forming the products from
// the activations instead (two products with one side of the rank's width, no G where the base weights are frozen)
// is as exact, but a step then rounds elsewhere, and after one SGD step the two ways are 1.0e-2 of the outputs
// apart (2-norm, 14912 rows, d 1024, f 4096, rank 16), where a step repeated the same way differs by nothing.
// Two launches for both Linears of a run of experts, bound by reading G twice:
//   lora_products_kernel  blocks of two kinds, side by side:
//     rows  Q = G A^T, `in` cut into ranges (partial sums): rows of G are the 16-row operand of
//           mma.sync, straight from global memory; A waits in shared memory
//     cols  P = G^T B over segments of G's rows: G^T fragments by transposing ldmatrix, the next tile of G
//           requested before the products of this one
//   lora_finish_kernel  sums over ranges and segments in order, the bias terms, scale, rounding
// (Two kernels one after the other, without the request ahead and with one thread a rank for B^T g, took 9 + 24 us
// for both Linears at d 1024, f 4096, rank 16, with launches 11 + 26 + 10; now 15 + 7.)
// (A step of the dense feed-forward at 1632 rows, d 1024, f 4096: 239 us.)
// Products of bf16 are exact in fp32 and all sums are fp32, so the only rounding behind G is that of the results.
#include "common.cuh"
#include "internal.h"

namespace moe {

namespace {

constexpr int kRank = 16;          // ranks in steps of 16, padded with zeros
constexpr int kRowTile = 64;
constexpr int kRange = 512;        // contraction range of a block of rows
constexpr int kSegRows = 256;      // rows of G of a block of columns
constexpr int kColTile = 128;
constexpr int kWPitch = kRange + 8;
constexpr int kXPitch = kColTile + 8;
constexpr int kSPitch = kRank + 8;

// One of the two Linears; E experts from the first one of the launch.
struct Linear {
  const __nv_bfloat16* G;          // [E][out][in]
  const __nv_bfloat16* g;          // [E][out]
  const void* const* tab;          // [E][3]: A, a, B of every expert
  int out, in, rank, R;            // R: rank rounded up to kRank
  int row_tiles, ranges, segs, col_tiles;
  float* q;                        // [ranges][E][out][R]
  float* p;                        // [segs][E][in][R]
  float* pb;                       // [segs][E][R]: B^T g
  __nv_bfloat16 *dA, *da, *dB, *db;   // [E][rank][in], [E][rank], [E][out][rank], [E][out]
};
struct Jobs {
  Linear lin[2];
  int E;
  unsigned db[2], da[2];            // the same for the finishing kernel: dB and db of both, then dA and da
  unsigned cols[2], rows[2];       // where each Linear's blocks end: first all `cols` blocks (the longer ones), then `rows`
};

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

constexpr int kRowsSmem = kRank * kWPitch * 2 + 4 * 32 * 8 * 4;
constexpr int kColsSmem = kRowTile * kXPitch * 2 + kRowTile * kSPitch * 2;
constexpr int kProductsSmem = kRowsSmem > kColsSmem ? kRowsSmem : kColsSmem;

// block b of a Linear's (expert, row tile, range) x rank steps; q[range][e][row][r] = G[row, range] . A[r, range]
__device__ __forceinline__ void rows_block(const Linear& L, int E, unsigned b, unsigned char* smem) {
  __nv_bfloat16* s_w = reinterpret_cast<__nv_bfloat16*>(smem);                             // [kRank][kWPitch]
  float (*s_red)[32][8] = reinterpret_cast<float (*)[32][8]>(smem + kRank * kWPitch * 2);    // [4]
  const int n0 = blockIdx.y * kRank;
  if (n0 >= L.R) return;               // the other Linear's rank is larger
  const int range = (int)(b % L.ranges), tile = (int)(b / L.ranges % L.row_tiles), e = (int)(b / L.ranges / L.row_tiles);
  const int C = L.in, k0 = range * kRange, row0 = tile * kRowTile, rows = min(kRowTile, L.out - row0);
  const int klen = min(kRange, C - k0);             // a multiple of 8
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const __nv_bfloat16* A = static_cast<const __nv_bfloat16*>(L.tab[(size_t)e * 3]);
  for (int i = tid; i < kRank * kRange / 8; i += 256) {
    const int r = i / (kRange / 8), k = (i - r * (kRange / 8)) * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (n0 + r < L.rank && k < klen) v = __ldg(reinterpret_cast<const uint4*>(A + (size_t)(n0 + r) * C + k0 + k));
    *reinterpret_cast<uint4*>(s_w + r * kWPitch + k) = v;
  }
  __syncthreads();
  // warp = 16 rows x half of the range; the contraction index inside 32 elements is permuted alike for both sides
  const int g = lane >> 2, t = lane & 3, rg = warp & 3, half = warp >> 2;
  const int ra = rg * 16 + g, rb = ra + 8;
  const __nv_bfloat16* G = L.G + ((size_t)e * L.out + row0) * C + k0;
  const uint4* xa = reinterpret_cast<const uint4*>(G + (size_t)min(ra, rows - 1) * C);
  const uint4* xb = reinterpret_cast<const uint4*>(G + (size_t)min(rb, rows - 1) * C);
  const int pieces = klen >> 3;
  float acc[2][4] = {};
  const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll 1
  for (int c0 = half * 8; c0 < half * 8 + 8; c0 += 4) {     // 16 chunks of 32 elements in a range
    uint4 a[4], b4[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = 4 * (c0 + u) + t;
      a[u] = p < pieces ? __ldcg(xa + p) : zero;
      b4[u] = p < pieces ? __ldcg(xb + p) : zero;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = 4 * (c0 + u) + t;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint4 w = *reinterpret_cast<const uint4*>(s_w + (8 * j + g) * kWPitch + p * 8);
        mma16816(acc[j], a[u].x, b4[u].x, a[u].y, b4[u].y, w.x, w.y);
        mma16816(acc[j], a[u].z, b4[u].z, a[u].w, b4[u].w, w.z, w.w);
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
    float* out = L.q + (((size_t)range * E + e) * L.out + row0) * L.R + n0;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][i] += s_red[rg][lane][j * 4 + i];
      const int c = 8 * j + 2 * t;
      if (ra < rows) *reinterpret_cast<float2*>(out + (size_t)ra * L.R + c) = make_float2(acc[j][0], acc[j][1]);
      if (rb < rows) *reinterpret_cast<float2*>(out + (size_t)rb * L.R + c) = make_float2(acc[j][2], acc[j][3]);
    }
  }
}

// block b of a Linear's (expert, segment, column tile) x rank steps;
// p[segment][e][c][r] = sum over the segment's rows of G[row, c] * B[row, r]
__device__ __forceinline__ void cols_block(const Linear& L, int E, unsigned b, unsigned char* smem) {
  __nv_bfloat16* s_x = reinterpret_cast<__nv_bfloat16*>(smem);       // [kRowTile][kXPitch]
  __nv_bfloat16* s_s = s_x + kRowTile * kXPitch;                      // [kRowTile][kSPitch]
  const int n0 = blockIdx.y * kRank;
  if (n0 >= L.R) return;               // the other Linear's rank is larger
  const int ct = (int)(b % L.col_tiles), seg = (int)(b / L.col_tiles % L.segs), e = (int)(b / L.col_tiles / L.segs);
  const int C = L.in, c0 = ct * kColTile, row0 = seg * kSegRows, rows = min(kSegRows, L.out - row0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const __nv_bfloat16* B = static_cast<const __nv_bfloat16*>(L.tab[(size_t)e * 3 + 2]) + (size_t)row0 * L.rank + n0;
  const __nv_bfloat16* G = L.G + ((size_t)e * L.out + row0) * C + c0;
  const __nv_bfloat16* gb = L.g + (size_t)e * L.out + row0;
  float acc[2][4] = {};
  float psum = 0.f;
  // G: 64 rows x 128 columns at a time, 16 bytes of four rows a thread
  uint4 v[4];
  auto request = [&](int r0) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = tid + u * 256, rr = i >> 4, c = (i & 15) * 8;
      v[u] = r0 + rr < rows && c0 + c < C ? __ldcg(reinterpret_cast<const uint4*>(G + (size_t)(r0 + rr) * C + c))
                                          : make_uint4(0, 0, 0, 0);
    }
  };
  request(0);
  for (int r0 = 0; r0 < rows; r0 += kRowTile) {
    __syncthreads();
    // B: four threads per row, four ranks each (rows of B are as wide as the rank: no wider loads)
    {
      const int rr = tid >> 2, q = (tid & 3) * 4;
      __nv_bfloat16 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        w[i] = r0 + rr < rows && n0 + q + i < L.rank ? B[(size_t)(r0 + rr) * L.rank + q + i] : __float2bfloat16_rn(0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) s_s[rr * kSPitch + q + i] = w[i];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = tid + u * 256;
      *reinterpret_cast<uint4*>(s_x + (i >> 4) * kXPitch + (i & 15) * 8) = v[u];
    }
    if (r0 + kRowTile < rows) request(r0 + kRowTile);
    __syncthreads();
    if (ct == 0) {       // this block also forms B^T g: sixteen threads a rank, four rows each
      const int r = tid & 15, q = (tid >> 4) * 4;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (r0 + q + i < rows)
          psum = fmaf(__bfloat162float(s_s[(q + i) * kSPitch + r]),
                      __bfloat162float(__ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(gb + r0 + q + i)))), psum);
    }
#pragma unroll
    for (int kk = 0; kk < kRowTile / 16; ++kk) {
      uint32_t a[4], w[4];
      // matrices (rows kk*16 + {0,8}) x (columns +{0,8}): transposed they are the fragments a0..a3 of G^T
      const int mr = kk * 16 + (lane & 7) + ((lane >> 4) << 3), mc = warp * 16 + (((lane >> 3) & 1) << 3);
      ldmatrix_x4_trans(a, s_x + mr * kXPitch + mc);
      const int sr = kk * 16 + (lane & 7) + (((lane >> 3) & 1) << 3), sc = (lane >> 4) << 3;
      ldmatrix_x4_trans(w, s_s + sr * kSPitch + sc);
#pragma unroll
      for (int j = 0; j < 2; ++j) mma16816(acc[j], a[0], a[1], a[2], a[3], w[2 * j], w[2 * j + 1]);
    }
  }
  const int g = lane >> 2, t = lane & 3;
  float* out = L.p + (((size_t)seg * E + e) * C + c0 + warp * 16) * L.R + n0;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (c0 + warp * 16 + g < C)
      *reinterpret_cast<float2*>(out + (size_t)g * L.R + 8 * j + 2 * t) = make_float2(acc[j][0], acc[j][1]);
    if (c0 + warp * 16 + g + 8 < C)
      *reinterpret_cast<float2*>(out + (size_t)(g + 8) * L.R + 8 * j + 2 * t) = make_float2(acc[j][2], acc[j][3]);
  }
  if (ct == 0) {
    __syncthreads();
    float* s_psum = reinterpret_cast<float*>(smem);
    s_psum[tid] = psum;
    __syncthreads();
    if (tid < kRank) {
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) sum += s_psum[i * 16 + tid];
      L.pb[((size_t)seg * E + e) * L.R + n0 + tid] = sum;
    }
  }
}

__global__ void __launch_bounds__(256)
lora_products_kernel(const __grid_constant__ Jobs jobs) {
  __shared__ __align__(16) unsigned char smem[kProductsSmem];
  pdl_wait();
  const unsigned b = blockIdx.x;
  if (b < jobs.cols[0]) cols_block(jobs.lin[0], jobs.E, b, smem);
  else if (b < jobs.cols[1]) cols_block(jobs.lin[1], jobs.E, b - jobs.cols[0], smem);
  else if (b < jobs.rows[0]) rows_block(jobs.lin[0], jobs.E, b - jobs.cols[1], smem);
  else rows_block(jobs.lin[1], jobs.E, b - jobs.rows[0], smem);
}

constexpr int kFinishCols = 16;

// `n` values `step` apart, added in order, eight requested at a time.
__device__ __forceinline__ float sum_of(const float* p, int n, size_t step) {
  float sum = 0.f;
  for (int k = 0; k < n; k += 8) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __ldcg(p + (size_t)min(k + i, n - 1) * step);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (k + i < n) sum += v[i];
  }
  return sum;
}

// blocks: 256 elements of dB, or 16 columns x 16 ranks of dA (its partial sums lie by column, dA by rank: through shared
// memory), of one expert
__global__ void __launch_bounds__(256)
lora_finish_kernel(const __grid_constant__ Jobs jobs, float scale) {
  __shared__ float s_t[kRank][kFinishCols + 1];
  const unsigned bx = blockIdx.x;
  const bool is_a = bx >= jobs.db[1];
  const int l = is_a ? (bx >= jobs.da[0] ? 1 : 0) : (bx >= jobs.db[0] ? 1 : 0);
  const Linear& L = jobs.lin[l];
  const unsigned at = bx - (is_a ? (l ? jobs.da[0] : jobs.db[1]) : (l ? jobs.db[0] : 0u));
  const int tid = threadIdx.x;
  pdl_wait();
  if (!is_a) {                         // dB [out][rank], db [out]
    const unsigned per = ((unsigned)(L.out * L.rank) + 255) / 256;
    const int e = (int)(at / per);
    const int64_t i = (int64_t)(at % per) * 256 + tid;
    if (i >= (int64_t)L.out * L.rank) return;
    const int c = (int)(i / L.rank), r = (int)(i % L.rank);
    const size_t step = (size_t)jobs.E * L.out * L.R;
    const float sum = sum_of(L.q + ((size_t)e * L.out + c) * L.R + r, L.ranges, step);
    const float gc = __bfloat162float(L.g[(size_t)e * L.out + c]);
    const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(L.tab[(size_t)e * 3 + 1]);
    L.dB[(size_t)e * L.out * L.rank + i] = __float2bfloat16_rn(scale * fmaf(gc, __bfloat162float(a[r]), sum));
    if (r == 0) L.db[(size_t)e * L.out + c] = __float2bfloat16_rn(scale * gc);
  } else {                             // dA [rank][in], da [rank]
    const int tiles = (L.in + kFinishCols - 1) / kFinishCols, steps = L.R / kRank;
    const int c0 = (int)(at % tiles) * kFinishCols, n0 = (int)(at / tiles % steps) * kRank, e = (int)(at / tiles / steps);
    const size_t step = (size_t)jobs.E * L.in * L.R;
    const int r = tid & 15, cc = tid >> 4;
    s_t[r][cc] = sum_of(L.p + ((size_t)e * L.in + min(c0 + cc, L.in - 1)) * L.R + n0 + r, L.segs, step);
    __syncthreads();
    const int rr = tid / kFinishCols, c = tid % kFinishCols;
    if (n0 + rr < L.rank && c0 + c < L.in)
      L.dA[((size_t)e * L.rank + n0 + rr) * L.in + c0 + c] = __float2bfloat16_rn(scale * s_t[rr][c]);
    if (c0 == 0 && tid < kRank && n0 + tid < L.rank) {
      const float ps = sum_of(L.pb + (size_t)e * L.R + n0 + tid, L.segs, (size_t)jobs.E * L.R);
      L.da[(size_t)e * L.rank + n0 + tid] = __float2bfloat16_rn(scale * ps);
    }
  }
}

// Sizes of both Linears and their places in the scratch buffer; returns its floats.
size_t lay_out(Jobs* jobs, int d, int f, const LoraRun& run, float* scratch) {
  size_t at = 0;
  const int E = jobs->E = run.count;
  for (int l = 0; l < 2; ++l) {
    Linear& L = jobs->lin[l];
    L.out = l == 0 ? 2 * f : d;
    L.in = l == 0 ? d : f;
    L.rank = run.rank[l];
    L.R = (L.rank + kRank - 1) / kRank * kRank;
    L.row_tiles = (L.out + kRowTile - 1) / kRowTile;
    L.ranges = (L.in + kRange - 1) / kRange;
    L.segs = (L.out + kSegRows - 1) / kSegRows;
    L.col_tiles = (L.in + kColTile - 1) / kColTile;
    L.q = scratch + at;
    at += (size_t)L.ranges * E * L.out * L.R;
    L.p = scratch + at;
    at += (size_t)L.segs * E * L.in * L.R;
    L.pb = scratch + at;
    at += (size_t)L.segs * E * L.R;
  }
  return at;
}

}  // namespace

size_t lora_grads_scratch_floats(int d, int f, const LoraRun& run) {
  Jobs jobs = {};
  return lay_out(&jobs, d, f, run, nullptr);
}

int launch_lora_grads(const void* const* tab, int d, int f, int all, const LoraRun& run, float* scratch,
                      const void* const (&G)[2], const void* const (&g)[2], cudaStream_t s) {
  Jobs jobs = {};
  lay_out(&jobs, d, f, run, scratch);
  const int E = run.count;
  for (int l = 0; l < 2; ++l) {
    Linear& L = jobs.lin[l];
    L.tab = tab + ((size_t)l * all + run.first) * 3;
    L.G = static_cast<const __nv_bfloat16*>(G[l]) + (size_t)run.first * L.out * L.in;
    L.g = static_cast<const __nv_bfloat16*>(g[l]) + (size_t)run.first * L.out;
    L.dA = static_cast<__nv_bfloat16*>(run.dA[l]);
    L.da = static_cast<__nv_bfloat16*>(run.da[l]);
    L.dB = static_cast<__nv_bfloat16*>(run.dB[l]);
    L.db = static_cast<__nv_bfloat16*>(run.db[l]);
  }
  const Linear &a = jobs.lin[0], &b = jobs.lin[1];
  const unsigned steps = (unsigned)((a.R > b.R ? a.R : b.R) / kRank);
  jobs.cols[0] = (unsigned)(a.segs * a.col_tiles * E);
  jobs.cols[1] = jobs.cols[0] + (unsigned)(b.segs * b.col_tiles * E);
  jobs.rows[0] = jobs.cols[1] + (unsigned)(a.row_tiles * a.ranges * E);
  jobs.rows[1] = jobs.rows[0] + (unsigned)(b.row_tiles * b.ranges * E);
  MOE_CUDA_CHECK(launch_pdl(lora_products_kernel, dim3(jobs.rows[1], steps), dim3(256), 0, s, jobs));
  unsigned at = 0;
  for (int l = 0; l < 2; ++l) jobs.db[l] = at += (unsigned)((jobs.lin[l].out * jobs.lin[l].rank + 255) / 256 * E);
  for (int l = 0; l < 2; ++l)
    jobs.da[l] = at += (unsigned)((jobs.lin[l].in + kFinishCols - 1) / kFinishCols * (jobs.lin[l].R / kRank) * E);
  MOE_CUDA_CHECK(launch_pdl(lora_finish_kernel, dim3(at), dim3(256), 0, s, jobs, run.scale));
  return 0;
}

}  // namespace moe
